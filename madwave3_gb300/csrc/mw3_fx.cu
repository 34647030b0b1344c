// The radial DST-I products and the angular terms on the tensor cores (tcgen05.mma,
// kind::f16) from exact base-256 digits (mw3_fx.cuh): the FP64 path, and the mixed path's
// shapes outside its fused chain and its 64-angle kernel.
//
// A DST along R or along r1 is y_k = sum_i S[k][i] x_i.  With S[k][n-1-i] = (-1)^k S[k][i]
// the even outputs come from u_i = x_i + x_{n-1-i} and the odd ones from v_i = x_i -
// x_{n-1-i}, i < ceil(n/2) (formed as integers, so exactly): half the products.  Along r1
// a length up to 128 fills one 128-row operand without that, so it stays whole.
// The k-space rectangle keeps the even outputs first and the odd ones behind them where n
// is even: the lanes of the accumulators (outputs) then store contiguously, and the next
// transform's pairs (k, n-1-k) are again positions (q, n-1-q), with the columns S[.][2q].
#include "mw3_internal.h"
#include "mw3_fx.cuh"

#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>

namespace mw3 {
namespace fx {

// one CTA tile: up to NV vectors of one segment against one 128-row block of one matrix
struct alignas(16) Item {
    int seg;
    int v0;          // first vector: r1 row (transforms along R) or column (along r1)
    int mode;        // 0 whole, 1 even outputs (sums), 2 odd outputs (differences); bits 2..: 128-row block
    int nn;          // the segment's r1 length, or the r1 row of an angular tile
    int nks;         // K steps
    int a[2];        // its matrix in the first and in the second transform, in 256-byte units
    int nv_m8;       // vectors | rows of its matrix planes (a multiple of 8) << 8
};

template <typename T>
struct Args {
    const Item *items;
    int nitems;
    int n1, n2, na;
    const T *src;
    T *dst;
    const unsigned char *planes;
    int pass;                    // 0, 1: the first or the second transform along this axis
    int nst;                     // stages of the ring of A
    int perm;                    // outputs stored even part first
    const T *etab;               // along r1, first product: k-space factor [n2][nn], by etoff
    const int64_t *etoff;        // [W][na]
    int drop;                    // bits the first digit gives up (long sums along R)
    const int *blk_wave;
    // gather epilogue
    double *H;
    const int *mapT;
    const int64_t *foff;
    const double *psi;           // the vector itself, for the points that the transforms do not reach
    const int *qptr, *qlist;     // per (wave, angle): stored points with r1 beyond the length
    // angular terms
    const int *map;
    const T *yj;                 // [G][na][n1] yyy(j, r1) by ladder slot
    const T *l2;                 // [G][3][na][n2] xl2mat_j(Om, Om + q; R), slot q + 1, by ladder slot
    const int *cpl;              // [G][3][2]: the block Omega + q of the same wave and state, -1 where there is none
    // [G][na] each angle's scale: its entries of the angular matrices stand x 2^sa, the vector's
    // over it.  Next to the poles every entry of a high Omega is tiny (60 angles, Omega = 10:
    // 2e-13), and one scale for the whole matrix kept it to 3e-5 of itself.  Costs the angular
    // kernels 0.1 to 1 % in FP64, 1.6 % in FP32 (384 x 192 x 80, three states: 637 -> 647 us)
    const int *sa;
    int *err;
};

// eight consecutive numbers, zero from n on; vec: they start on 32 bytes (one 256-bit load
// takes a whole sector a lane: half the cache lines a load instruction touches)
__device__ __forceinline__ void load8(const double *x, int n, bool vec, double (&v)[8])
{
    if (vec && n >= 8) {
#pragma unroll
        for (int c = 0; c < 8; c += 4)
            asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                         : "=d"(v[c]), "=d"(v[c + 1]), "=d"(v[c + 2]), "=d"(v[c + 3])
                         : "l"(x + c));
    } else {
#pragma unroll
        for (int c = 0; c < 8; c++) v[c] = c < n ? x[c] : 0.0;
    }
}

__device__ __forceinline__ void load8(const float *x, int n, bool vec, float (&v)[8])
{
    if (vec && n >= 8) {
        asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                     : "l"(x));
    } else {
#pragma unroll
        for (int c = 0; c < 8; c++) v[c] = c < n ? x[c] : 0.f;
    }
}

__device__ __forceinline__ void store4(double *q, int n, bool vec, const double (&y)[4])
{
    if (vec && n >= 4) {
        asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};"
                     :
                     : "l"(q), "d"(y[0]), "d"(y[1]), "d"(y[2]), "d"(y[3])
                     : "memory");
    } else {
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (c < n) q[c] = y[c];
    }
}

__device__ __forceinline__ void store4(float *q, int n, bool vec, const float (&y)[4])
{
    if (vec && n >= 4) {
        *reinterpret_cast<float4 *>(q) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (c < n) q[c] = y[c];
    }
}

// the bits of a fixed-point number kept where a vector's entry was
__device__ __forceinline__ long long as_int(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ int as_int(float x) { return __float_as_int(x); }
__device__ __forceinline__ void as_num(long long v, double &x) { x = __longlong_as_double(v); }
__device__ __forceinline__ void as_num(int v, float &x) { x = __int_as_float(v); }

// a barrier of the filling warps; true for all of them where any of them passes true
__device__ __forceinline__ bool barrier_or(bool x)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)x), "n"(FILL)
        : "memory");
    return r != 0;
}

enum Epi { EPI_ROWS = 0, EPI_GATHER = 1, EPI_COLS_E = 2, EPI_COLS = 3, EPI_ANG_J = 4, EPI_ANG_G = 5 };

// eight j-basis values of block g at ladder slot j, r1 row r1 and columns R0..: the j^2 and
// l^2 terms with the Omega +- 1 blocks, H_b,j = (yyy + l2_0) B_b + l2_- B_{b-1} + l2_+ B_{b+1}
template <typename T>
__device__ __forceinline__ void ang_values(const Args<T> &p, int g, int j, int r1, int R0, int nv, bool vec,
                                           T (&v)[8])
{
    const size_t at = ((size_t)j * p.n1 + r1) * p.n2 + R0, blk = (size_t)p.na * p.n1 * p.n2;
    const T *l = p.l2 + ((size_t)g * 3 * p.na + j) * p.n2 + R0;
    const size_t slot = (size_t)p.na * p.n2;
    const T y = p.yj[((size_t)g * p.na + j) * p.n1 + r1];
    T b[8];
    load8(p.src + g * blk + at, nv, vec, b);
    load8(l + slot, nv, vec, v);
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = (y + v[c]) * b[c];
#pragma unroll
    for (int q = 0; q < 3; q += 2) {
        const int s = p.cpl[(g * 3 + q) * 2];
        if (s < 0) continue;
        T f[8];
        load8(p.src + s * blk + at, nv, vec, b);
        load8(l + q * slot, nv, vec, f);
#pragma unroll
        for (int c = 0; c < 8; c++) v[c] = fma(f[c], b[c], v[c]);
    }
}

// One persistent CTA per SM takes its tiles in turn, four roles at work on different tiles:
// warps 0-7 load vectors, find each one's largest entry and write digits (two B blocks in
// shared memory), warp 17 copies the matrix steps through a ring, warp 16 issues the MMAs (two
// sets of accumulators in tensor memory), warps 8-15 put the sums together and store them.
// With every warp of a CTA going through these phases in turn, two CTAs an SM, a tile of 32
// FP64 vectors took 40 k cycles a CTA: 5 k for the loads, 7 k for the digits, 11 k for the
// MMAs, 7-20 k for the way back.  The MMAs of a K step take 500 cycles; with the copies and
// their waits on the issuing thread it was 1400.  Cycles a tile now (FP64, 384 x 192 x 80):
// along R 14 k, the MMAs; along r1 13-16 k, fill and way back 10 k each beside them; to the j
// basis 10 k, back 12 k, of which the loads of the coupled blocks 9 k.
template <typename T, int EPI, bool FOLD>
__global__ void __launch_bounds__(THREADS, 1) k_fx_dst(Args<T> p)
{
    typedef typename Num<T>::Int Int;
    constexpr int ND = Num<T>::ND, NV = Num<T>::NV;
    constexpr uint32_t BSTEP = Size<T>::BSTEP, BBYTES = Size<T>::BBYTES, ABYTES = Size<T>::ABYTES;
    // eight vectors a filling warp; the WPG warps of a group of eight share its K
    constexpr int NG = NV / 8, WPG = FILL / 32 / NG, KT = 32 * WPG, U = KB / KT;
    constexpr bool ROWS = EPI == EPI_ROWS || EPI == EPI_GATHER, ANG = EPI == EPI_ANG_J || EPI == EPI_ANG_G;
    static_assert(!ROWS || FOLD, "transforms along R are folded");
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char *As = sm, *Bs = sm + ABYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + ABYTES + 2 * BBYTES);
    uint64_t *empty = full + MAXST;           // the ring of A
    uint64_t *bfull = empty + MAXST, *bempty = bfull + 2;      // the B blocks
    uint64_t *tfull = bempty + 2, *tempty = tfull + 2;         // the accumulators
    uint32_t *slot = reinterpret_cast<uint32_t *>(tempty + 2);
    volatile int *fail = reinterpret_cast<volatile int *>(slot + 1);
    unsigned *s_max = reinterpret_cast<unsigned *>(slot + 2);      // [NEF][WPG][NV]: largest |x| of a tile's vectors
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nst = p.nst;
    const uint32_t astage = (ABYTES / nst) & ~127u;
    if (warp == 0) tc::tmem_alloc(slot, 512);
    if (threadIdx.x == 0) {
        for (int i = 0; i < nst; i++) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&bfull[i], FILL / 32);
            tc::mbar_init(&bempty[i], 1);
            tc::mbar_init(&tfull[i], 1);
            tc::mbar_init(&tempty[i], WAYBACK / 32);
        }
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tb = *slot;
    tc::dependents_launch();
    const int n2 = p.n2, n1 = p.n1;
    const bool vec = n2 % (32 / (int)sizeof(T)) == 0;     // rows start on 32 bytes
    auto length = [&](const Item &it) { return ANG ? p.na : ROWS ? n2 : it.nn; };
    // this CTA's tiles.  Along R a run of the list, where the tiles of the same vectors stand
    // together: first the even outputs' 128-row blocks, then the odd ones'.  A second block
    // takes the digits of the first (K is above 128 then and fills both B blocks), an odd
    // tile what its even one has loaded.  With a fill for every tile that was 22 k cycles at
    // K = 192, against 10-14 k for the MMAs (mixed 384 x 192 x 80, first transform: 623 us,
    // sharing 419).  Along r1 (K up to 128, one row block) runs of tiles gained nothing in
    // FP32 (740 -> 738 us) and lost in FP64 (1248 -> 1354): strided there
    const int step_i = ROWS ? 1 : (int)gridDim.x;
    const int begin = ROWS ? (int)((int64_t)p.nitems * blockIdx.x / gridDim.x) : (int)blockIdx.x;
    const int end = ROWS ? (int)((int64_t)p.nitems * (blockIdx.x + 1) / gridDim.x) : p.nitems;
    auto same_vectors = [](const Item &x, const Item &y) { return ROWS && x.seg == y.seg && x.v0 == y.v0; };
    auto same_digits = [&](const Item &x, const Item &y) { return same_vectors(x, y) && ((x.mode ^ y.mode) & 3) == 0; };
    // the largest entries' exponent field of vector n of the j-th tile
    auto field = [&](int j, int n) {
        const unsigned *sx = s_max + (j % NEF) * WPG * NV;
        return (int)((WPG == 2 ? max(sx[n], sx[NV + n]) : sx[n]) >> Num<T>::EBITS);
    };

    constexpr int MMA_WARP = (FILL + WAYBACK) / 32;
    if (warp >= MMA_WARP) {
        regs_down<REG_AUX>();
        if (warp == MMA_WARP + 1 && lane == 0) {
            // ---- the matrix steps of every tile in turn, nst in flight ----
            int ct = 0, cs = 0, cph = 0;                   // copies issued; the next one's stage and phase
            bool ok = true;
            for (int i = begin; i < end && ok; i += step_i) {
                const int n = p.items[i].nks;
                const uint32_t cb = (uint32_t)(p.items[i].nv_m8 >> 8) * (ND * 32);
                const unsigned char *ca = p.planes + (int64_t)p.items[i].a[p.pass] * 256;
                for (int ks = 0; ks < n; ks++) {
                    if (ct == nst) tc::dependents_wait();      // the waits have a limit, the kernel ahead has none
                    if (ct >= nst && !(ok = wait(&empty[cs], cph ^ 1, fail))) break;
                    tc::mbar_expect_tx(&full[cs], cb);
                    tc::bulk_g2s(As + cs * astage, ca + (int64_t)ks * cb, cb, &full[cs]);
                    ct++;
                    if (++cs == nst) {
                        cs = 0;
                        cph ^= 1;
                    }
                }
            }
            // no copy stays in flight
            for (int c = max(0, ct - nst); c < ct; c++) tc::mbar_wait(&full[c % nst], (c / nst) & 1);
        } else if (warp == MMA_WARP && lane == 0) {
            // ---- the MMAs ----
            const uint64_t a0 = tc::sdesc(tc::smem_u32(As), LBO, SBO), b0 = tc::sdesc(tc::smem_u32(Bs), LBO, SBO);
            int t = 0, ts = 0, tph = 0;                    // steps issued; the next one's stage and phase
            int nb = 0, ni = 0;
            tc::dependents_wait();                         // as the copies
            bool ok = begin < end && wait(&full[0], 0, fail);
            Item it = {}, nxt = {};
            if (ok) it = p.items[begin];
            for (int i = begin; i < end && ok; i += step_i, ni++) {
                const bool more = i + step_i < end;
                if (more) nxt = p.items[i + step_i];
                const int nks = it.nks, m8 = it.nv_m8 >> 8;
                const bool keep = more && same_digits(it, nxt);     // the next tile takes these B blocks again
                const int nb0 = nb;
                if (ni >= 2) ok = wait(&tempty[ni & 1], ((ni >> 1) - 1) & 1, fail);
                const uint32_t d = tb + 256u * (ni & 1);
                for (int ks = 0; ks < nks && ok; ks++) {
                    if (ks % (KB / KS) == 0 && !(ok = wait(&bfull[nb & 1], (nb >> 1) & 1, fail))) break;
                    const bool lastk = ks + 1 == nks;
                    const int s = ts;
                    t++;
                    if (++ts == nst) {
                        ts = 0;
                        tph ^= 1;
                    }
                    tc::fence_after_sync();
                    step<T>(d, a0 + (uint64_t)(s * (astage >> 4)), m8,
                            b0 + (uint64_t)(((nb & 1) * BBYTES + (ks % (KB / KS)) * BSTEP) >> 4), ROWS ? 0 : 1, ks == 0,
                            [&] {      // the next step's matrix
                                if (!lastk || more) ok = wait(&full[ts], tph, fail);
                            });
                    tc::mma_commit(&empty[s]);
                    if (lastk || (ks + 1) % (KB / KS) == 0) {
                        if (!keep) tc::mma_commit(&bempty[nb & 1]);
                        nb++;
                    }
                    if (lastk) tc::mma_commit(&tfull[ni & 1]);
                }
                if (keep) nb = nb0;
                it = nxt;
            }
            // no MMA stays in flight
            for (int c = max(0, t - nst); c < t; c++) tc::mbar_wait(&empty[c % nst], (c / nst) & 1);
        }
        __syncwarp();
    } else if (warp >= FILL / 32) {
        // ---- the way back: lane = output, half the tile's vectors a thread ----
        regs_down<REG_WAY>();
        const int q4 = warp & 3, half = (warp >> 2) & 1, m = q4 * 32 + lane;
        const uint32_t lrow = tb + ((uint32_t)(q4 * 32) << 16);
        int ni = 0, nf = 0;                       // tiles done; the fill that this one's digits are from
        Item nxt = {};
        if (begin < end) nxt = p.items[begin];
        tc::dependents_wait();
        for (int i = begin; i < end; i += step_i, ni++) {
            const Item it = nxt;
            bool keep = false;
            if (i + step_i < end) {
                nxt = p.items[i + step_i];
                keep = same_digits(it, nxt);
            }
            const int a = ANG ? 0 : it.seg % p.na;
            const int md = it.mode & 3, mt = it.mode >> 2;
            const int L = length(it), nv = it.nv_m8 & 255;
            const int L2 = (L + 1) >> 1;                                // even outputs
            const int out = 128 * mt + m;                               // index within its parity
            const bool on = md == 0 ? out < L : out < (md == 1 ? L2 : L - L2);
            const int sh = Num<T>::SH - (md ? 1 : 0) - p.drop;
            const auto ls = lane_scale(EPI == EPI_ANG_G && on ? p.sa[(size_t)it.seg * p.na + out] : 0, (T)0);
            const int k = md == 0 ? out : 2 * out + md - 1;             // the output itself
            const int pos = md == 0 ? out : p.perm && !(L & 1) ? out + (md == 1 ? 0 : L2) : k;
            const bool any = __any_sync(0xffffffffu, on);
            if (EPI == EPI_GATHER && it.v0 == 0 && it.mode == 1) {
                // once a segment: the stored points beyond the r1 length keep psi
                const int wa = p.blk_wave[it.seg / p.na] * p.na + a, q1 = p.qptr[wa + 1];
                const int64_t o = p.foff[it.seg];
                for (int q = p.qptr[wa] + (int)threadIdx.x - FILL; q < q1; q += WAYBACK) {
                    const int ir = p.qlist[q];
                    p.H[o + ir] = p.psi[o + ir];
                }
                __syncwarp();
            }
            const bool ok = wait(&tfull[ni & 1], (ni >> 1) & 1, fail);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc::fence_after_sync();
            const uint32_t trow = lrow + 256u * (ni & 1);
            const int64_t fo = EPI == EPI_GATHER ? p.foff[it.seg]
                               : EPI == EPI_ANG_G && on ? p.foff[(size_t)it.seg * p.na + out] : 0;
            const T *et = EPI == EPI_COLS_E && on
                              ? p.etab + p.etoff[p.blk_wave[it.seg / p.na] * p.na + a] + (size_t)it.v0 * it.nn + k : nullptr;
            const int cend = min(nv, (half + 1) * (NV / 2));
#pragma unroll 1
            for (int c0 = half * (NV / 2); c0 < cend && any; c0 += 4) {
                // what the stores need is on its way while the sums are put together
                int idx[4];
                T e[4];
                if (EPI == EPI_GATHER || EPI == EPI_ANG_G) {
                    const int *mp = EPI == EPI_GATHER ? p.mapT + ((size_t)a * n2 + k) * n1 + it.v0 + c0
                                                      : p.map + ((size_t)out * n1 + it.nn) * n2 + it.v0 + c0;
#pragma unroll
                    for (int c = 0; c < 4; c++) idx[c] = on && c0 + c < nv ? mp[c] : -1;
                }
                if (EPI == EPI_COLS_E)
#pragma unroll
                    for (int c = 0; c < 4; c++) e[c] = on && c0 + c < nv ? et[(size_t)(c0 + c) * it.nn] : (T)0;
                uint32_t v[ND][4];
                load_groups(trow + c0, NV, v);
                T y[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    uint32_t g[ND];
#pragma unroll
                    for (int q = 0; q < ND; q++) g[q] = v[q][c];
                    y[c] = combine(g, field(nf, c0 + c), sh, ls);
                }
                if (on) {
                    if (EPI == EPI_ROWS) {
                        T *q = p.dst + ((size_t)it.seg * n1 + it.v0 + c0) * n2 + pos;
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (c0 + c < nv) q[(size_t)c * n2] = y[c];
                    } else if (EPI == EPI_GATHER) {
                        double *h0 = p.H + fo;
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (idx[c] >= 0) h0[idx[c]] = (double)y[c];
                    } else if (EPI == EPI_ANG_G) {
                        // one writer per point: adds at L2, no load in the way
                        double *h0 = p.H + fo;
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (idx[c] >= 0) atomicAdd(h0 + idx[c], (double)y[c]);
                    } else {
                        T *q = EPI == EPI_ANG_J
                                   ? p.dst + (((size_t)it.seg * p.na + out) * n1 + it.nn) * n2 + it.v0 + c0
                                   : p.dst + ((size_t)it.seg * n1 + pos) * n2 + it.v0 + c0;
                        if (EPI == EPI_COLS_E)
#pragma unroll
                            for (int c = 0; c < 4; c++) y[c] *= e[c];
                        store4(q, nv - c0, vec, y);
                    }
                }
                __syncwarp();
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive(&tempty[ni & 1]);
            if (!keep) nf++;
        }
    } else {
        // ---- vectors into digits ----
        regs_up<REG_FILL>();
        const int grp = warp % NG, hf = warp / NG;
        const int rn = (lane & 7) + 8 * grp, rp = (lane >> 3) + 4 * hf;      // along R: this thread's row and k group
        T kv[U][8], kw[FOLD ? U : 1][8];                      // entries of the first B block, and their mirrors
        unsigned kmax[ROWS ? 1 : 8];                          // the largest |x| past the first block
        int ka[EPI == EPI_ANG_J ? U : 1];                     // the scales of kv's angles
        // entry k of this thread's eight vectors (transforms along r1, angles)
        auto column = [&](const Item &it, int k, T (&v)[8]) {
            const int n = (it.nv_m8 & 255) - 8 * grp;
            if (EPI == EPI_ANG_G)
                ang_values(p, it.seg, k, it.nn, it.v0 + 8 * grp, n, vec, v);
            else if (EPI == EPI_ANG_J)
                load8(p.src + (((size_t)it.seg * p.na + k) * n1 + it.nn) * n2 + it.v0 + 8 * grp, n, vec, v);
            else
                load8(p.src + ((size_t)it.seg * n1 + k) * n2 + it.v0 + 8 * grp, n, vec, v);
        };
        auto scale = [&](const Item &it, int k) { return EPI == EPI_ANG_J ? p.sa[(size_t)it.seg * p.na + k] : 0; };
        auto scaled = [&](T x, int u) {
            return EPI == EPI_ANG_J ? mag_down<T>(mag(x), ka[EPI == EPI_ANG_J ? u : 0]) : mag(x);
        };
        // along R: entries k..k+7 of this thread's row, and their mirrors L-1-k downwards
        auto row = [&](const Item &it, int L, int k, T (&v)[8], T (&w)[8]) {
            const T *x = p.src + ((size_t)it.seg * n1 + it.v0 + rn) * n2;
            load8(x + k, ((L + 1) >> 1) - k, vec, v);
            const int e = L - 8 - k;
            if (e >= 0) {
                load8(x + e, 8, vec && e % (32 / (int)sizeof(T)) == 0, w);
            } else {
#pragma unroll
                for (int c = 0; c < 8; c++) w[c] = e + c >= 0 ? x[e + c] : (T)0;
            }
        };
        // a tile's first B block into registers, and the largest entries past it
        auto fetch = [&](const Item &it, bool known) {
            const int L = length(it), md = it.mode & 3, K = md ? (L + 1) >> 1 : L;
            if (ROWS) {
                const bool on = rn < (it.nv_m8 & 255);
                if (known && K <= KB) return;
                kmax[0] = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int k = 8 * (rp + 4 * WPG * u);
#pragma unroll
                    for (int c = 0; c < 8; c++) kv[u][c] = kw[FOLD ? u : 0][c] = (T)0;
                    if (on && k < K) row(it, L, k, kv[u], kw[FOLD ? u : 0]);
                }
                if (on && !known)
#pragma unroll 1
                    for (int k = KB + 8 * rp; k < K; k += 32 * WPG) {
                        T v[8], w[8];
                        row(it, L, k, v, w);
#pragma unroll
                        for (int c = 0; c < 8; c++) kmax[0] = max(kmax[0], max(mag(v[c]), mag(w[c])));
                    }
            } else {
#pragma unroll
                for (int c = 0; c < 8; c++) kmax[ROWS ? 0 : c] = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int k = lane + 32 * hf + KT * u;
#pragma unroll
                    for (int c = 0; c < 8; c++) kv[u][c] = (T)0;
                    if (EPI == EPI_ANG_J) ka[EPI == EPI_ANG_J ? u : 0] = k < K ? scale(it, k) : 0;
                    if (k < K) column(it, k, kv[u]);
                    if (FOLD) {
#pragma unroll
                        for (int c = 0; c < 8; c++) kw[u][c] = (T)0;
                        if (md && k < K) column(it, L - 1 - k, kw[u]);
                    }
                }
#pragma unroll 1
                for (int k = lane + 32 * hf + KB; k < K; k += KT) {
                    T v[8];
                    column(it, k, v);
                    const int s = scale(it, k);
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        kmax[ROWS ? 0 : c] = max(kmax[ROWS ? 0 : c], EPI == EPI_ANG_J ? mag_down<T>(mag(v[c]), s) : mag(v[c]));
                }
            }
        };
        int nb = 0, ni = 0;                       // B blocks written, tiles filled
        bool bad = false, known = false;          // known: the tile before had the same vectors
        unsigned mrow = 0;                        // along R: the row's largest |x|
        Item nxt = {};
        if (begin < end) nxt = p.items[begin];
        tc::dependents_wait();
        if (begin < end) fetch(nxt, false);
        for (int i = begin, in; i < end; i = in, ni++) {
            const Item it = nxt;
            const int md = it.mode & 3, L = length(it), K = md ? (L + 1) >> 1 : L;
            const int nv = it.nv_m8 & 255;
            const int sh = Num<T>::SH - (md ? 1 : 0) - p.drop;
            // ---- the largest |x| of each vector.  One of subnormal numbers has the scale of the
            // smallest normal ones, which is theirs ----
            unsigned *sx = s_max + (ni % NEF) * WPG * NV;
            if (ROWS) {
                if (!known) {
                    mrow = kmax[0];
#pragma unroll
                    for (int u = 0; u < U; u++)
#pragma unroll
                        for (int c = 0; c < 8; c++) mrow = max(mrow, max(mag(kv[u][c]), mag(kw[FOLD ? u : 0][c])));
                    mrow = max(mrow, __shfl_xor_sync(0xffffffffu, mrow, 8));
                    mrow = max(mrow, __shfl_xor_sync(0xffffffffu, mrow, 16));
                }
                if (lane < 8) sx[hf * NV + rn] = max(mrow, 1u << Num<T>::EBITS);
            } else {
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    unsigned mx = kmax[ROWS ? 0 : c];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        mx = max(mx, scaled(kv[u][c], u));
                        if (FOLD) mx = max(mx, mag(kw[FOLD ? u : 0][c]));
                    }
                    mx = __reduce_max_sync(0xffffffffu, mx);
                    if (lane == c) sx[hf * NV + 8 * grp + c] = max(mx, 1u << Num<T>::EBITS);
                }
            }
            if (barrier_or(bad)) break;           // every filling thread, or none
            const bool formed = known && K <= KB;      // the differences are in the registers
            in = i + step_i;
            known = false;
            for (; in < end; in += step_i) {
                nxt = p.items[in];
                if (!same_digits(it, nxt)) {
                    known = same_vectors(it, nxt);
                    break;
                }
            }
            // ---- digits, one block of K at a time.  Every entry is converted and masked: a
            // branch round each kept the eight chains of a thread from overlapping ----
            for (int kb = 0; kb < K; kb += KB, nb++) {
                const int kr = (min(K - kb, KB) + KS - 1) & ~(KS - 1);
                unsigned char *Bb = Bs + (nb & 1) * BBYTES;
                if (nb >= 2 && !bad) bad = !wait(&bempty[nb & 1], ((nb >> 1) - 1) & 1, fail);
                tc::fence_after_sync();
                if (kb > 0) {                     // a later block's entries, all on their way together
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int k = ROWS ? kb + 8 * (rp + 4 * WPG * u) : kb + lane + 32 * hf + KT * u;
                        if (k >= K) continue;
                        if (EPI == EPI_ANG_J) ka[EPI == EPI_ANG_J ? u : 0] = scale(it, k);
                        if (!ROWS) column(it, k, kv[u]);
                        else if (rn < nv) row(it, L, k, kv[u], kw[FOLD ? u : 0]);
                    }
                }
                if (ROWS) {
                    const int ef = field(ni, rn);
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int kg = rp + 4 * WPG * u, k = kb + 8 * kg;
                        if (8 * kg >= kr) continue;
                        Int X[8];
                        if (formed) {
#pragma unroll
                            for (int c = 0; c < 8; c++) X[c] = as_int(kv[u][c]);
                        } else {
#pragma unroll
                            for (int c = 0; c < 8; c++) {
                                const Int x = to_fixed(kv[u][c], ef, sh), y = to_fixed(kw[FOLD ? u : 0][7 - c], ef, sh);
                                // the middle of an odd length pairs with itself
                                const Int on = -(Int)(rn < nv && k + c < K), two = -(Int)(L - 1 - (k + c) != k + c);
                                const Int z = (x - y) & on & two;
                                X[c] = md == 1 ? (x + (y & two)) & on : z;
                                if (K <= KB) as_num(z, kv[u][c]);
                            }
                        }
                        put_digits(X, Bb + (kg >> 1) * BSTEP + (rn >> 3) * SBO + (kg & 1) * LBO + (rn & 7) * 16,
                                   NV / 8 * SBO);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int kl = lane + 32 * hf + KT * u, k = kb + kl;
                        if (kl - lane >= kr) continue;
                        Int X[8];
#pragma unroll
                        for (int c = 0; c < 8; c++) {
                            const int ef = field(ni, 8 * grp + c) + (EPI == EPI_ANG_J ? ka[EPI == EPI_ANG_J ? u : 0] : 0);
                            const Int on = -(Int)(k < K);
                            X[c] = to_fixed(kv[u][c], ef, sh) & on;
                            if (FOLD) {
                                // a length kept whole pairs with nothing, an odd one's middle with itself
                                const Int y = to_fixed(kw[FOLD ? u : 0][c], ef, sh) & on;
                                const Int two = -(Int)(L - 1 - k != k);
                                X[c] = md == 2 ? (X[c] - y) & two : X[c] + (y & two & -(Int)(md == 1));
                            }
                        }
                        put_digits(X, Bb + (kl >> 4) * BSTEP + grp * SBO + ((kl >> 3) & 1) * LBO + (kl & 7) * 16,
                                   NV / 8 * SBO);
                    }
                }
                tc::fence_async_smem();
                __syncwarp();
                if (lane == 0 && !bad) arrive(&bfull[nb & 1]);
            }
            bad = __any_sync(0xffffffffu, bad);
            if (in < end) fetch(nxt, known);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && *fail) atomicExch(p.err, 1);
    if (warp == 0) tc::tmem_dealloc(tb, 512);
}

}  // namespace fx

namespace {

// rows of the planes of a matrix of M rows (of each of its 128-row blocks)
inline int plane_rows(int M) { return std::min(128, (M + 7) & ~7); }

// bytes of one K step of them, in the 256-byte units of a tile's matrix index
template <typename T>
int step_units(int m8) { return fx::Num<T>::ND * m8 / 8; }

// stages of the ring of A for planes of up to m8 rows
template <typename T>
int ring_stages(int m8)
{
    int n = fx::MAXST;
    while (((fx::Size<T>::ABYTES / n) & ~127u) < (uint32_t)step_units<T>(m8) * 256) n--;
    return n;
}

// digits of the rows of one constant matrix as K steps of planes of m8 rows (canonical
// K-major), one 128-row block after the other, appended to `out`.  Returns the bits a vector's first digit (up to
// 512, or 64 of FP32) has to give up so that no group g <= 4 of a row can sum past 2^24.
// value(m, k): the entry x 2^SBITS, an integer of at most 2^(SBITS+1)
template <typename T, typename F>
int append_planes(std::vector<__half> &out, int M, int m8, int K, F &&value)
{
    constexpr int ND = fx::Num<T>::ND;
    static const std::vector<__half> half_of = [] {
        std::vector<__half> h(513);
        for (int d = 0; d <= 512; d++) h[d] = __float2half((float)(d - 256));
        return h;
    }();
    const double first = sizeof(T) == 8 ? 512.0 : 64.0;       // a vector's first digit
    const int nks = (K + fx::KS - 1) / fx::KS;
    const int nmt = (M + 127) / 128;
    const size_t base = out.size(), plane = (size_t)m8 * fx::KS, ast = ND * plane;
    out.resize(base + (size_t)nmt * nks * ast, half_of[256]);
    int drop = 0;
    for (int m = 0; m < M; m++) {
        long long sum[ND] = {};                 // of |digit| over k
        for (int k = 0; k < K; k++) {
            long long v = value(m, k);
            __half *st = out.data() + base + ((size_t)(m / 128) * nks + k / fx::KS) * ast +
                         fx::a_off(m % 128, k % fx::KS) / 2;
            for (int d = ND - 1; d >= 0; d--) {
                const int g = d > 0 ? (int)((v + 128) & 255) - 128 : (int)v;
                v = (v - g) >> 8;
                st[d * plane] = half_of[g + 256];
                sum[d] += g < 0 ? -g : g;
            }
        }
        double low = 0.0;                       // digits of x past the first: up to 128
        for (int g = 0; g < std::min(5, ND); g++) {
            while (drop < 3 && ldexp(first, -drop) * (double)sum[g] + 128.0 * low > 16777216.0) drop++;
            low += (double)sum[g];
        }
    }
    return drop;
}

// S[i][k] = 2 sin(pi (i+1)(k+1)/(n+1)) x 2^SBITS, rounded from long double
template <typename T>
struct Sine {
    int n;
    std::vector<long long> s;
    explicit Sine(int n_) : n(n_), s((size_t)2 * (n_ + 1))
    {
        const long double pi = 3.141592653589793238462643383279502884L;
        for (int m = 0; m <= n + 1; m++) {
            const int q = std::min(m, n + 1 - m);          // the first quadrant
            s[m] = llrintl(ldexpl(2.0L * sinl(pi * (long double)q / (long double)(n + 1)), fx::Num<T>::SBITS));
            if (m > 0 && m <= n) s[2 * (n + 1) - m] = -s[m];
        }
    }
    long long operator()(int i, int k) const { return s[(long long)(i + 1) * (k + 1) % (2 * (n + 1))]; }
};

// resident CTAs of the persistent kernel: one per SM
int fx_ctas()
{
    int dev = 0, nsm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

template <typename V>
int fx_upload(Ctx &c, V **dst, const std::vector<V> &v)
{
    void *q = nullptr;
    const size_t bytes = sizeof(V) * std::max<size_t>(v.size(), 1);
    if (cudaMalloc(&q, bytes) != cudaSuccess) {
        cudaGetLastError();
        c.err = "cudaMalloc: radial digit tables";
        return MW3_ERR_NOMEM;
    }
    c.allocs.push_back(q);
    *dst = reinterpret_cast<V *>(q);
    if (!v.empty()) MW3_CUDA_TRY(cudaMemcpy(q, v.data(), sizeof(V) * v.size(), cudaMemcpyHostToDevice));
    return MW3_OK;
}

// the kernel's shared memory granted, and compiled with the registers that its warps share out
template <typename T, int EPI, bool FOLD>
bool ready()
{
    cudaFuncAttributes a;
    const bool ok = cudaFuncSetAttribute(fx::k_fx_dst<T, EPI, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)fx::Size<T>::SMEM) == cudaSuccess &&
                    cudaFuncGetAttributes(&a, fx::k_fx_dst<T, EPI, FOLD>) == cudaSuccess &&
                    a.numRegs * fx::THREADS >= fx::REGS;
    if (!ok) cudaGetLastError();
    return ok;
}

template <typename T, int EPI, bool FOLD>
void launch(Ctx &c, const fx::Args<T> &p)
{
    launch_early(fx::k_fx_dst<T, EPI, FOLD>, dim3(std::min(p.nitems, c.fx_grid)), fx::THREADS, fx::Size<T>::SMEM, c.stream, p);
    c.launches++;
}

template <typename T>
int build_fx_t(Ctx &c)
{
    constexpr int NV = fx::Num<T>::NV;
    c.use_fx = false;
    c.d_fxZ = nullptr;
    // K of one product is at most 256: npun2 <= 512 folded, npun1 <= 256 (which mw3_create asks for)
    if (c.n2 > 512 || c.n1 > 256) return MW3_OK;
    if (!(ready<T, fx::EPI_ROWS, true>() && ready<T, fx::EPI_GATHER, true>() && ready<T, fx::EPI_COLS_E, false>() &&
          ready<T, fx::EPI_COLS, false>() && ready<T, fx::EPI_COLS_E, true>() && ready<T, fx::EPI_COLS, true>()))
        return MW3_OK;
    const int n1 = c.n1, n2 = c.n2, na = c.na, W = (int)c.waves.size();
    int dropR = 0, drop1 = 0;
    // along R: [pass][parity][128-row block][K step]
    {
        const Sine<T> S(n2);
        const int he = (n2 + 1) / 2, ho = n2 / 2, K = he, m8 = plane_rows(he);
        const bool perm = n2 % 2 == 0;
        for (int pass = 0; pass < 2; pass++) {
            std::vector<__half> pl;
            auto col = [&](int q) { return pass && perm ? 2 * q : q; };
            for (int par = 0; par < 2; par++) {
                const size_t b = pl.size();
                dropR = std::max(dropR, append_planes<T>(pl, par ? ho : he, m8, K,
                                                      [&](int m, int k) { return S(2 * m + par, col(k)); }));
                // both parities take the even one's block count
                const size_t want = (size_t)((he + 127) / 128) * ((K + fx::KS - 1) / fx::KS) * step_units<T>(m8) * 128;
                pl.resize(b + want, __float2half(0.f));
            }
            __half *d = nullptr;
            const int rc = fx_upload(c, &d, pl);
            if (rc) return rc;
            c.d_fxR[pass] = d;
        }
    }
    std::vector<int> off1((size_t)W * na), off2((size_t)W * na);      // K steps before the length's matrices
    // along r1: every length once; a length above 128 folded (even, odd) and, for the second
    // product, with the columns of the stored order
    {
        std::map<int, std::pair<std::pair<int64_t, int64_t>, int64_t>> at;
        std::vector<__half> pl;
        std::vector<T> et;
        std::vector<int64_t> eoff((size_t)W * na);
        const int he = (n2 + 1) / 2;
        bool fold = false;
        for (int w = 0; w < W; w++)
            for (int a = 0; a < na; a++) {
                const WaveTables &t = c.waves[w];
                const int nn = t.nopr1[a];
                auto f = at.find(nn);
                if (f == at.end()) {
                    const Sine<T> S(nn);
                    std::pair<int64_t, int64_t> o;
                    o.first = o.second = (int64_t)pl.size() * 2;
                    if (nn <= 128) {
                        drop1 = std::max(drop1, append_planes<T>(pl, nn, plane_rows(nn), nn, [&](int m, int k) { return S(m, k); }));
                    } else {
                        fold = true;
                        const int K = (nn + 1) / 2;
                        for (int pass = 0; pass < (nn % 2 ? 1 : 2); pass++) {
                            if (pass) o.second = (int64_t)pl.size() * 2;
                            for (int par = 0; par < 2; par++)
                                drop1 = std::max(drop1, append_planes<T>(pl, par ? nn / 2 : K, plane_rows(K), K, [&](int m, int k) {
                                                     return S(2 * m + par, pass ? 2 * k : k);
                                                 }));
                        }
                    }
                    // min(p1 + p2, radcut) / (4 (nn+1) (n2+1)) by stored column; the momenta depend on the length only
                    const int64_t eo = (int64_t)et.size();
                    const double divi = 1.0 / (4.0 * (double)(nn + 1) * (double)(n2 + 1));
                    for (int q = 0; q < n2; q++) {
                        const int R = n2 % 2 ? q : (q < he ? 2 * q : 2 * (q - he) + 1);
                        for (int m = 0; m < nn; m++) {
                            double ek = t.p2r1[(size_t)a * n1 + m] + t.p2r2[(size_t)a * n2 + R];
                            if (ek > c.grid.radcutmax) ek = c.grid.radcutmax;
                            et.push_back((T)(ek * divi));
                        }
                    }
                    f = at.emplace(nn, std::make_pair(o, eo)).first;
                }
                off1[(size_t)w * na + a] = (int)(f->second.first.first / 256);
                off2[(size_t)w * na + a] = (int)(f->second.first.second / 256);
                eoff[(size_t)w * na + a] = f->second.second;
            }
        if (dropR > 1 || drop1 > 0) return MW3_OK;
        c.fx_drop = dropR;
        int rc;
        __half *d = nullptr;
        if ((rc = fx_upload(c, &d, pl))) return rc;
        c.d_fxr = d;
        T *de = nullptr;
        if ((rc = fx_upload(c, &de, et))) return rc;
        c.d_fxe = de;
        if ((rc = fx_upload(c, &c.d_fxe_off, eoff))) return rc;
        // a folded product reads rows that another tile of it writes: its own output rectangle
        if (fold) {
            void *z = nullptr;
            const size_t bytes = sizeof(T) * (size_t)c.G * na * n1 * n2;
            if (cudaMalloc(&z, bytes) != cudaSuccess) {
                cudaGetLastError();
                c.err = "cudaMalloc: second rectangle of the digit transforms";
                return MW3_ERR_NOMEM;
            }
            c.allocs.push_back(z);
            MW3_CUDA_TRY(cudaMemset(z, 0, bytes));
            c.d_fxZ = z;
        }
    }
    // the tiles, in segment order; hphi of a part of the blocks takes a range of them
    std::vector<fx::Item> rows, cols;
    c.h_fx_row0.assign(1, 0);
    c.h_fx_col0.assign(1, 0);
    const int he = (n2 + 1) / 2, nmt = (he + 127) / 128, nmto = (n2 / 2 + 127) / 128, ksR = (he + fx::KS - 1) / fx::KS;
    const int mR = plane_rows(he), uR = ksR * step_units<T>(mR);
    int m1max = 8;
    for (int w = 0; w < W; w++)
        for (int b = 0; b < c.waves[w].ncan; b++)
            for (int a = 0; a < na; a++) {
                const int seg = (c.waves[w].g0 + b) * na + a, nn = c.waves[w].nopr1[a];
                const int o1 = off1[(size_t)w * na + a], o2 = off2[(size_t)w * na + a];
                for (int v = 0; v < nn; v += NV)
                    for (int par = 0; par < 2; par++)
                        for (int mt = 0; mt < (par ? nmto : nmt); mt++) {
                            const int at = (par * nmt + mt) * uR;
                            rows.push_back(fx::Item{seg, v, (par + 1) | (mt << 2), nn, ksR, {at, at},
                                                    std::min(NV, nn - v) | (mR << 8)});
                        }
                const int K1 = nn <= 128 ? nn : (nn + 1) / 2, ks1 = (K1 + fx::KS - 1) / fx::KS, m1 = plane_rows(K1);
                const int u1 = ks1 * step_units<T>(m1);
                m1max = std::max(m1max, m1);
                for (int v = 0; v < n2; v += NV)
                    for (int par = 0; par < (nn <= 128 ? 1 : 2); par++)
                        cols.push_back(fx::Item{seg, v, nn <= 128 ? 0 : par + 1, nn, ks1, {o1 + par * u1, o2 + par * u1},
                                                std::min(NV, n2 - v) | (m1 << 8)});
                c.h_fx_row0.push_back((int)rows.size());
                c.h_fx_col0.push_back((int)cols.size());
            }
    c.fx_nst[0] = ring_stages<T>(mR);
    c.fx_nst[1] = ring_stages<T>(m1max);
    fx::Item *d;
    int rc;
    if ((rc = fx_upload(c, &d, rows))) return rc;
    c.d_fx_rows = d;
    if ((rc = fx_upload(c, &d, cols))) return rc;
    c.d_fx_cols = d;
    c.fx_grid = fx_ctas();
    c.use_fx = true;
    return MW3_OK;
}

// the angular terms through the j basis, B = D X, the j-diagonal scaling with the
// Omega +- 1 coupling, H += D^T Hb, both products from exact digits.  Leaves c.use_fx_ang
// false where the explicit matrices are needed (over 256 angles, a block whose j list leaves
// the ladder j0 + k inc, or matrices the digits do not cover)
template <typename T>
int build_fx_ang_t(Ctx &c)
{
    constexpr int NV = fx::Num<T>::NV;
    const int na = c.na, n1 = c.n1, n2 = c.n2, G = c.G, ne = c.ne;
    const int nks = (na + fx::KS - 1) / fx::KS, nmt = (na + 127) / 128, m8 = plane_rows(na);
    const int units = nks * step_units<T>(m8);
    if (!(ready<T, fx::EPI_ANG_J, false>() && ready<T, fx::EPI_ANG_G, false>())) return MW3_OK;
    for (auto &t : c.waves)
        for (double d : t.djmmp)
            if (!(fabs(d) <= 2.0)) return MW3_OK;
    std::vector<__half> pl;
    std::vector<int> sa((size_t)G * na), sd(na);
    std::vector<const double *> seen;                 // the (Omega, state) columns already cut
    std::vector<int> seen_at, seen_lad;
    std::vector<T> yj((size_t)G * na * n1, (T)0), l2((size_t)G * 3 * na * n2, (T)0);
    std::vector<int> at((size_t)G * 2);
    int drop = 0;
    for (auto &t : c.waves) {
        int njl = 0;                                  // ladder j = j0 + k inc <= (na-1) inc and <= nangu2
        while (njl < t.nj2 && t.j0 + njl * t.inc <= (na - 1) * t.inc && t.j0 + njl * t.inc <= t.nangu2) njl++;
        if (njl > na) return MW3_OK;
        for (int b = 0; b < t.ncan; b++)
            for (int s = 0; s < b; s++)
                if (t.iombas[s] == t.iombas[b] && t.nelebas[s] == t.nelebas[b]) return MW3_OK;
        for (int b = 0; b < t.ncan; b++) {
            const int g = t.g0 + b, om = t.iombas[b], e = t.nelebas[b];
            const double *D = t.djmmp.data() + ((size_t)om * ne + (e - 1)) * (t.nangu2 + 1) * na;
            const int lad = (t.j0 * 4 + t.inc) * 4096 + njl;
            // an angle's largest entry of the ladder just below 2
            for (int a = 0; a < na; a++) {
                double dmax = 0.0;
                for (int js = 0; js < njl; js++) dmax = std::max(dmax, fabs(D[(size_t)(t.j0 + js * t.inc) * na + a]));
                int ex = 1;
                if (dmax > 0.0) frexp(dmax, &ex);         // dmax < 2^ex
                sd[a] = std::min((int)fx::Num<T>::SAMAX, std::max(0, 1 - ex));
            }
            std::copy(sd.begin(), sd.end(), sa.begin() + (size_t)g * na);
            int f = -1;
            for (size_t i = 0; i < seen.size() && f < 0; i++)
                if (seen_lad[i] == lad && !memcmp(seen[i], D, sizeof(double) * (t.nangu2 + 1) * na)) f = (int)i;
            if (f < 0) {
                f = (int)seen.size();
                seen.push_back(D);
                seen_lad.push_back(lad);
                seen_at.push_back((int)(pl.size() / 128));
                auto d = [&](int js, int a) {
                    return js < njl ? llrint(ldexp(D[(size_t)(t.j0 + js * t.inc) * na + a], sd[a] + fx::Num<T>::SBITS))
                                    : 0LL;
                };
                drop = std::max(drop, append_planes<T>(pl, na, m8, na, [&](int m, int k) { return d(m, k); }));
                drop = std::max(drop, append_planes<T>(pl, na, m8, na, [&](int m, int k) { return d(k, m); }));
            }
            at[2 * g] = seen_at[f];
            at[2 * g + 1] = seen_at[f] + nmt * units;
            // yyy of the block's own j list, by ladder slot
            for (int k = 0; k < t.nojbas[b]; k++) {
                const int jb = t.jbas[(size_t)b * na + k];
                bool any = false;
                for (int ir1 = 0; ir1 < n1; ir1++) any |= t.yj2[((size_t)b * n1 + ir1) * na + k] != 0.0;
                if (!any) continue;
                if ((jb - t.j0) % t.inc != 0 || (jb - t.j0) / t.inc < 0 || (jb - t.j0) / t.inc >= njl) return MW3_OK;
                const int js = (jb - t.j0) / t.inc;
                for (int ir1 = 0; ir1 < n1; ir1++)
                    yj[((size_t)g * na + js) * n1 + ir1] += (T)t.yj2[((size_t)b * n1 + ir1) * na + k];
            }
            // xl2mat_j(Om, Om + q; R) for the sources Om + q
            for (int q = -1; q <= 1; q++) {
                const int oms = om + q;
                if (oms < t.iommin || oms > t.iommax) continue;
                for (int js = 0; js < std::min(njl, t.nj2); js++) {
                    const size_t u = (((size_t)(e - 1) * t.nj2 + js) * t.nom + (om - t.iommin)) * t.nom + (oms - t.iommin);
                    if (!t.l2used[u]) continue;
                    for (int ir2 = 0; ir2 < n2; ir2++)
                        l2[(((size_t)g * 3 + (q + 1)) * na + js) * n2 + ir2] =
                            (T)t.l2tab[((((size_t)(e - 1) * t.nj2 + js) * n2 + ir2) * t.nom + (om - t.iommin)) * t.nom +
                                       (oms - t.iommin)];
                }
            }
        }
    }
    if (drop > 1) return MW3_OK;
    // tiles of one r1 row x NV R that hold stored points
    const int t2n = (n2 + NV - 1) / NV;
    std::vector<char> on((size_t)n1 * t2n, 0);
    for (int a = 0; a < na; a++)
        for (int ir = 0; ir < c.npunreal[a]; ir++)
            on[(size_t)(c.indr1[(size_t)a * c.npt + ir] - 1) * t2n + (c.indr2[(size_t)a * c.npt + ir] - 1) / NV] = 1;
    std::vector<fx::Item> items;
    c.h_fx_ang0.assign(1, 0);
    for (int g = 0; g < G; g++) {
        for (int i = 0; i < n1; i++)
            for (int j = 0; j < t2n; j++)
                if (on[(size_t)i * t2n + j])
                    for (int mt = 0; mt < nmt; mt++)
                        items.push_back(fx::Item{g, j * NV, mt << 2, i, nks, {at[2 * g] + mt * units, at[2 * g + 1] + mt * units},
                                                 std::min(NV, n2 - j * NV) | (m8 << 8)});
        c.h_fx_ang0.push_back((int)items.size());
    }
    int rc;
    __half *d = nullptr;
    fx::Item *di = nullptr;
    if ((rc = fx_upload(c, &d, pl))) return rc;
    if ((rc = fx_upload(c, &di, items))) return rc;
    if ((rc = fx_upload(c, &c.d_fx_sa, sa))) return rc;
    T *dy = nullptr, *dl = nullptr;
    if ((rc = fx_upload(c, &dy, yj))) return rc;
    if ((rc = fx_upload(c, &dl, l2))) return rc;
    c.d_fx_yj = dy;
    c.d_fx_l2 = dl;
    c.d_fx_ang = di;
    c.d_fxD = d;
    c.fx_nst[2] = ring_stages<T>(m8);
    c.fx_drop_ang = drop;
    c.fx_grid = fx_ctas();
    c.use_fx_ang = true;
    return MW3_OK;
}

}  // namespace

// tables of the digit DSTs; leaves c.use_fx false where another path is asked for or the shape
// is outside them.  Mixed: the fused chain is faster (256 x 128 x 60, J = 10: 141 us against 449),
// and the three-kernel 3xTF32 form keeps its shapes (every r1 length up
// to 128): results there would otherwise move by its own error, 2e-5 of psi after 32 iterations
// at npun2 = 436; what is left ran on FP32 CUDA cores (512 x 256 x 120: 1.56 ms against 0.47)
int build_fx(Ctx &c)
{
    c.use_fx = false;
    c.d_fxZ = nullptr;
    c.fx_allocs.clear();
    if (c.k_dst >= 0 || (!c.fp64 && (c.use_tc_dst2d || tc_dst_supported(c)))) return MW3_OK;
    const size_t n0 = c.allocs.size();
    const int rc = c.fp64 ? build_fx_t<double>(c) : build_fx_t<float>(c);
    c.fx_allocs.assign(c.allocs.begin() + (long)n0, c.allocs.end());
    if (!c.use_fx) drop_fx(c);
    return rc == MW3_ERR_NOMEM ? MW3_OK : rc;        // no room: the dense transforms need none of this
}

void drop_fx(Ctx &c)
{
    for (void *p : c.fx_allocs) {
        cudaFree(p);
        c.allocs.erase(std::find(c.allocs.begin(), c.allocs.end(), p));
    }
    c.fx_allocs.clear();
    c.d_fxR[0] = c.d_fxR[1] = c.d_fxr = c.d_fxe = c.d_fxZ = c.d_fx_rows = c.d_fx_cols = nullptr;
    c.d_fxe_off = nullptr;
    c.use_fx = false;
}

int build_fx_ang(Ctx &c)
{
    c.use_fx_ang = false;
    if (c.k_ang == 0 || c.na < 2 || c.na > 256 || c.use_tc_ang) return MW3_OK;
    const size_t n0 = c.allocs.size();
    const int rc = c.fp64 ? build_fx_ang_t<double>(c) : build_fx_ang_t<float>(c);
    if (!c.use_fx_ang)
        while (c.allocs.size() > n0) {
            cudaFree(c.allocs.back());
            c.allocs.pop_back();
        }
    return rc == MW3_ERR_NOMEM ? MW3_OK : rc;
}

// j^2, l^2 and the Omega coupling of blocks [g_begin, g_end) (whole waves): X -> B in Y, then H +=
template <typename T>
void launch_fx_ang(Ctx &c, const T *X, T *Y, double *H, int g_begin, int g_end)
{
    fx::Args<T> p = {};
    p.n1 = c.n1; p.n2 = c.n2; p.na = c.na;
    p.blk_wave = c.d_blk_wave;
    p.H = H; p.map = c.d_map; p.foff = c.d_foff;
    p.err = c.d_tc_err;
    p.planes = (const unsigned char *)c.d_fxD;
    p.yj = (const T *)c.d_fx_yj; p.l2 = (const T *)c.d_fx_l2; p.cpl = c.d_cpl;
    p.drop = c.fx_drop_ang; p.sa = c.d_fx_sa; p.nst = c.fx_nst[2];
    p.items = (const fx::Item *)c.d_fx_ang + c.h_fx_ang0[g_begin];
    p.nitems = c.h_fx_ang0[g_end] - c.h_fx_ang0[g_begin];
    p.src = X; p.dst = Y; p.pass = 0;
    launch<T, fx::EPI_ANG_J, false>(c, p);
    p.src = Y; p.dst = nullptr; p.pass = 1;
    launch<T, fx::EPI_ANG_G, false>(c, p);
}

// the four products of the radial kinetic term of blocks [g_begin, g_end): X -> Y, Y in place
// (or through Z), Y -> H at the stored points
template <typename T>
void launch_fx_dst(Ctx &c, const T *X, T *Y, double *H, const double *psi, int g_begin, int g_end, bool mark)
{
    const int s0 = g_begin * c.na, s1 = g_end * c.na;
    fx::Args<T> p = {};
    p.n1 = c.n1; p.n2 = c.n2; p.na = c.na;
    p.blk_wave = c.d_blk_wave;
    p.H = H; p.mapT = c.d_mapT; p.foff = c.d_foff;
    p.psi = psi; p.qptr = c.d_quirk_ptr; p.qlist = c.d_quirk;
    p.err = c.d_tc_err;
    p.etab = (const T *)c.d_fxe; p.etoff = c.d_fxe_off;
    const fx::Item *rows = (const fx::Item *)c.d_fx_rows + c.h_fx_row0[s0];
    const fx::Item *cols = (const fx::Item *)c.d_fx_cols + c.h_fx_col0[s0];
    const int nr = c.h_fx_row0[s1] - c.h_fx_row0[s0], nc = c.h_fx_col0[s1] - c.h_fx_col0[s0];
    if (mark) stage_mark(c, 0);
    p.items = rows; p.nitems = nr;
    p.src = X; p.dst = Y; p.planes = (const unsigned char *)c.d_fxR[0]; p.perm = 1; p.pass = 0; p.drop = c.fx_drop;
    p.nst = c.fx_nst[0];
    launch<T, fx::EPI_ROWS, true>(c, p);
    if (mark) stage_mark(c, 1);
    T *Z = c.d_fxZ ? (T *)c.d_fxZ : Y;
    p.items = cols; p.nitems = nc;
    p.src = Y; p.dst = Z; p.planes = (const unsigned char *)c.d_fxr; p.drop = 0;
    p.nst = c.fx_nst[1];
    if (c.d_fxZ) launch<T, fx::EPI_COLS_E, true>(c, p);
    else launch<T, fx::EPI_COLS_E, false>(c, p);
    p.src = Z; p.dst = Y; p.perm = 0; p.pass = 1;
    if (c.d_fxZ) launch<T, fx::EPI_COLS, true>(c, p);
    else launch<T, fx::EPI_COLS, false>(c, p);
    if (mark) stage_mark(c, 2);
    p.items = rows; p.nitems = nr;
    p.src = Y; p.dst = nullptr; p.planes = (const unsigned char *)c.d_fxR[1]; p.drop = c.fx_drop;
    p.nst = c.fx_nst[0];
    launch<T, fx::EPI_GATHER, true>(c, p);
}

template void launch_fx_dst<double>(Ctx &, const double *, double *, double *, const double *, int, int, bool);
template void launch_fx_dst<float>(Ctx &, const float *, float *, double *, const double *, int, int, bool);
template void launch_fx_ang<double>(Ctx &, const double *, double *, double *, int, int);
template void launch_fx_ang<float>(Ctx &, const float *, float *, double *, int, int);

}  // namespace mw3
