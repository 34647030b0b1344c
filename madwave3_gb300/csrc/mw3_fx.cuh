// Exact products on the tensor cores from base-256 digits: a vector x with |x| < 2^E
// is the integer round(x 2^(57-E)), cut into signed base-256 digits d_0..d_6 (the first up
// to 512) that FP16 holds exactly, and so is a constant matrix S (|S| <= 2, x 2^54) from
// long double.  The products s_i d_j of one weight i + j = g sum to integers up to 2^24
// for g <= 4 and K <= 256, which the FP32 accumulators of tcgen05.mma hold exactly; the
// groups g = 0..6 are kept in seven accumulators and put together as one integer.  The
// groups past 6 that are left out are 2^-54 of a typical row sum, below one FP64 rounding.  (Error-free splitting
// of matrix products after Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012.)
//
// All digits of one K step of B stand one below the other (row = NV digit + vector), so
// digit i of A takes the first ND - i digits of B in one MMA of N = NV (ND - i) whose
// columns start at NV i: group g = i + j lands in columns NV g .. NV g + NV - 1 by itself.
#pragma once
#include "mw3_tc.cuh"

#include <cuda_fp16.h>

namespace mw3 {
namespace fx {

constexpr int KS = 16;                             // K of one MMA
constexpr int KB = 128;                            // K of one B block in shared memory
constexpr uint32_t APL = 128 * KS * 2;             // one digit of one K step of A: 4 KB
constexpr uint32_t SBO = 256, LBO = 128;
constexpr int FILL = 256;                          // threads that cut vectors into digits: warps 0-7
constexpr int WAYBACK = 256;                       // and that put the sums together: warps 8-15
constexpr int THREADS = FILL + WAYBACK + 128;      // and one warp for the MMAs, one for the copies
// registers a thread: 96 at launch (640 threads), then shared out by warpgroup: 256 x 128 +
// 256 x 80 + 128 x 64 = 61440, all that the CTA was launched with
constexpr int REG_FILL = 128, REG_WAY = 80, REG_AUX = 64;
// (with fewer at launch the filling warps would wait for theirs without end: the host asks
// the compiled kernel before it takes it)
constexpr int REGS = FILL * REG_FILL + WAYBACK * REG_WAY + 128 * REG_AUX;
static_assert(REGS <= THREADS * 96, "more registers than at launch");
constexpr int NEF = 8;                             // tiles whose exponents are kept (up to five are under way)

// What depends on the type of the vectors.  FP32 vectors take four digits of 30 bits
// (|X| <= 2^30, the constant matrix x 2^29), FP64 vectors seven; the accumulators of all
// groups of one tile take up to 256 tensor-memory columns, half of them.
template <typename T> struct Num;
template <> struct Num<double> {
    enum { ND = 7, NV = 32, SH = 4, EBITS = 20, EMAX = 0x7FF, SBITS = 54, SAMAX = 1000 };
    typedef long long Int;
};
template <> struct Num<float> {
    enum { ND = 4, NV = 64, SH = 6, EBITS = 23, EMAX = 0xFF, SBITS = 29, SAMAX = 80 };
    typedef int Int;
};
template <typename T> struct Size {
    static constexpr uint32_t ABYTES = sizeof(T) == 8 ? 114688 : 98304;            // the ring of K steps of A
    static constexpr uint32_t BSTEP = Num<T>::ND * Num<T>::NV * KS * 2;            // 7 or 8 KB
    static constexpr uint32_t BBYTES = (KB / KS) * BSTEP;                          // 56 or 64 KB, twice
    static constexpr uint32_t SMEM = ABYTES + 2 * BBYTES + 3072;                   // 227 KB: one CTA an SM
};
constexpr int MAXST = 8;                           // stages of the ring

// element (row, k) of one digit of a K step of A
__host__ __device__ constexpr uint32_t a_off(int r, int k)
{
    return (uint32_t)((r & 7) * 16 + (r >> 3) * SBO + (k & 7) * 2 + (k >> 3) * LBO);
}

// the bits of |x| that order vectors' entries: the high word, or all of an FP32 number
__device__ __forceinline__ unsigned mag(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ unsigned mag(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// mag of x / 2^s (as far as its exponent field); infinities and NaN stay
template <typename T>
__device__ __forceinline__ unsigned mag_down(unsigned m, int s)
{
    return m >> Num<T>::EBITS >= (unsigned)Num<T>::EMAX ? m : (unsigned)max((int)m - (s << Num<T>::EBITS), 0);
}

// round(x 2^(57 - E)) for |x| < 2^E, E = ef - 1022 with ef the exponent field of the
// largest |x| of the vector; sh = 4, or 3 to leave a bit for a sum of two; x / 2^s with s added to ef
__device__ __forceinline__ long long to_fixed(double x, int ef, int sh)
{
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    const int ex = (int)((h >> 20) & 0x7FFu);
    const unsigned mh = (h & 0xFFFFFu) | (ex ? 0x100000u : 0u);
    const unsigned r = min((unsigned)(ef - max(ex, 1)), 63u);
    unsigned long long v = (((unsigned long long)mh << 32) | l) << sh;
    v = (v + ((1ull << r) >> 1)) >> r;
    const long long s = (long long)((int)h >> 31);
    return ((long long)v ^ s) - s;
}

// the same in 32 bits: round(x 2^(30 - E)), E = ef - 126, for sh = 6
__device__ __forceinline__ int to_fixed(float x, int ef, int sh)
{
    const unsigned b = __float_as_uint(x);
    const int ex = (int)((b >> 23) & 0xFFu);
    const unsigned r = min((unsigned)(ef - max(ex, 1)), 31u);
    unsigned v = ((b & 0x7FFFFFu) | (ex ? 0x800000u : 0u)) << sh;
    v = (v + ((1u << r) >> 1)) >> r;
    const int s = (int)b >> 31;
    return ((int)v ^ s) - s;
}

__device__ __forceinline__ uint32_t h2sub(uint32_t u, __half2 off)
{
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&u), off);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// the seven digits of eight integers (|X| <= 2^57) as FP16, 16 bytes a digit
__device__ __forceinline__ void put_digits(const long long *X, unsigned char *dst, uint32_t digit_stride)
{
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const unsigned long long b = (unsigned long long)X[i] + 0x0200808080808080ull;
        hi[i] = (uint32_t)(b >> 32);
        lo[i] = (uint32_t)b;
    }
    // 1024 of the bit pattern and the bias, 512 or 128
    const __half2 off0 = __floats2half2_rn(1536.f, 1536.f), off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
    for (int d = 0; d < 7; d++) {
        uint32_t w[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            uint32_t u;
            if (d == 0) u = __byte_perm(hi[2 * p], hi[2 * p + 1], 0x7632) + 0x64006400u;
            else if (d == 1) u = (__byte_perm(hi[2 * p], hi[2 * p + 1], 0x0501) & 0x00FF00FFu) | 0x64006400u;
            else if (d == 2) u = (__byte_perm(hi[2 * p], hi[2 * p + 1], 0x0400) & 0x00FF00FFu) | 0x64006400u;
            else {
                const int by = 6 - d;
                u = (__byte_perm(lo[2 * p], lo[2 * p + 1], (unsigned)(by | ((4 + by) << 8))) & 0x00FF00FFu) |
                    0x64006400u;
            }
            w[p] = h2sub(u, d ? off : off0);
        }
        *reinterpret_cast<uint4 *>(dst + d * digit_stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// the four digits of eight integers (|X| <= 2^30)
__device__ __forceinline__ void put_digits(const int *X, unsigned char *dst, uint32_t digit_stride)
{
    uint32_t b[8];
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = (uint32_t)X[i] + 0x80808080u;
    const __half2 off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const int by = 3 - d;
        uint32_t w[4];
#pragma unroll
        for (int p = 0; p < 4; p++)
            w[p] = h2sub((__byte_perm(b[2 * p], b[2 * p + 1], (unsigned)(by | ((4 + by) << 8))) & 0x00FF00FFu) |
                             0x64006400u,
                         off);
        *reinterpret_cast<uint4 *>(dst + d * digit_stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// what combine takes a row's power of two s back with: the exponent, or the factor 2^-s (s up to
// 80, and f below is 2^-24 at least or 0, so nothing is lost)
__device__ __forceinline__ int lane_scale(int s, double) { return s; }
__device__ __forceinline__ float lane_scale(int s, float) { return __uint_as_float((unsigned)(127 - s) << 23); }

// one output: its seven groups -> the sum over k of S x.  ef: exponent field of the vector's
// largest |x|, sh as in to_fixed, ls: the power of two that this output's row of S stands
// multiplied with (lane_scale).  (Conversions by FP32 additions and integer instructions
// instead of the quarter-rate and FP64 units were no faster.)
__device__ __forceinline__ double combine(const uint32_t (&v)[7], int ef, int sh, int ls)
{
    int a[7];
#pragma unroll
    for (int g = 0; g < 7; g++) a[g] = __float2int_rn(__uint_as_float(v[g]));
    const long long H = ((long long)a[0] << 24) + ((long long)a[1] << 16) + ((long long)a[2] << 8) + a[3];
    const long long L = ((long long)a[4] << 16) + ((long long)a[5] << 8) + a[6];
    // the leading 62 bits of H 2^24 + L, in units 2^(72-z) of 2^54 2^(57-E)
    const int z = min(24, __clzll(H < 0 ? ~H : H) - 2);
    const long long V = (H << z) + (L >> (24 - z));
    if (ef >= 0x7FF) return __longlong_as_double(0x7FF8000000000000ll);   // an infinity or NaN in the vector
    if (V == 0) return 0.0;
    const double y = (double)V;
    const int sc = ef - 1061 + (4 - sh) - z - ls;    // E - 39 - z, one more for a folded vector
    const int e = (int)(((unsigned)__double2hiint(y) >> 20) & 0x7FFu) + sc;
    if (e > 0 && e < 0x7FF)
        return __hiloint2double(__double2hiint(y) + (sc << 20), __double2loint(y));
    return scalbn(y, sc);
}

// the groups are exact; their FP32 sum rounds once at the size of the first
__device__ __forceinline__ float combine(const uint32_t (&v)[4], int ef, int sh, float ls)
{
    const float r = 1.f / 256.f;
    const float f = ls * fmaf(fmaf(fmaf(__uint_as_float(v[3]), r, __uint_as_float(v[2])), r, __uint_as_float(v[1])), r,
                              __uint_as_float(v[0]));
    if (ef >= 0xFF) return __uint_as_float(0x7FC00000u);
    const int sc = ef - 137 + (6 - sh);              // E - 11 (48 - 29 - 30), one more for a folded vector
    const int s0 = max(sc, -100);
    float y = f * __uint_as_float((unsigned)(s0 + 127) << 23);
    if (sc < -100) y *= __uint_as_float((unsigned)(sc + 227) << 23);
    return y;
}

__device__ __forceinline__ bool wait(uint64_t *mbar, uint32_t parity, volatile int *fail)
{
    const uint32_t a = tc::smem_u32(mbar);
    long long t0 = 0;
    for (int i = 0;; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 31) == 31) {
            if (*fail) return false;
            const long long t = clock64();
            if (t0 == 0) t0 = t;
            else if (t - t0 > tc::kWaitCycles) {
                *fail = 1;
                return false;
            }
        }
    }
}

__device__ __forceinline__ void arrive(uint64_t *mbar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" : : "r"(tc::smem_u32(mbar)) : "memory");
}

__device__ __forceinline__ void mma_f16(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t idesc, int accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(dtmem), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
}

// kind::f16, FP16 operands, FP32 accumulate; bmn: B stored with its rows (N) contiguous
__host__ __device__ constexpr uint32_t idesc(int M, int N, int bmn)
{
    return (1u << 4) | ((uint32_t)bmn << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// the MMAs of one K step: A at a (ND planes of m8 rows, m8 a multiple of 8: the rows past them
// that the MMA reads are the next plane's and give lanes that nothing reads), B at b.  The
// issuing thread stays one or two MMAs ahead of the tensor cores, so what it has to wait for
// besides (mid) goes before the last and largest MMA
template <typename T, typename F>
__device__ __forceinline__ void step(uint32_t d, uint64_t a, int m8, uint64_t b, int bmn, bool first, F &&mid)
{
    constexpr int ND = Num<T>::ND, NV = Num<T>::NV;
    if (first) {                       // digit 0 spans every group: it clears them
        mma_f16(d, a, b, idesc(128, NV * ND, bmn), 0);
#pragma unroll
        for (int i = ND - 1; i > 0; i--) {
            if (i == 1) mid();
            mma_f16(d + NV * i, a + (uint64_t)(i * m8 * 2), b, idesc(128, NV * (ND - i), bmn), 1);
        }
    } else {
#pragma unroll
        for (int i = ND - 1; i >= 0; i--) {
            if (i == 0) mid();
            mma_f16(d + NV * i, a + (uint64_t)(i * m8 * 2), b, idesc(128, NV * (ND - i), bmn), 1);
        }
    }
}

template <int N> __device__ __forceinline__ void regs_up()
{
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void regs_down()
{
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// four columns of this thread's lane, without the wait
__device__ __forceinline__ void ld4_nw(uint32_t taddr, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}

// the accumulators of four columns of this thread's lane, groups nv columns apart
template <int ND>
__device__ __forceinline__ void load_groups(uint32_t taddr, int nv, uint32_t (&v)[ND][4])
{
#pragma unroll
    for (int g = 0; g < ND; g++) ld4_nw(taddr + nv * g, v[g]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int g = 0; g < ND; g++)
        asm volatile("" : "+r"(v[g][0]), "+r"(v[g][1]), "+r"(v[g][2]), "+r"(v[g][3]));
}

}  // namespace fx
}  // namespace mw3
