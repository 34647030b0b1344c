// Exact products on the tensor cores from base-256 digits: a vector x with |x| < 2^E
// is the integer round(x 2^(57-E)), cut into signed base-256 digits d_0..d_6 (the first up
// to 512) that FP16 holds exactly, and so is a constant matrix S (|S| <= 2, x 2^54) from
// long double.  The products s_i d_j of one weight i + j = g sum to integers up to 2^24
// for g <= 4 and K <= 256, which the FP32 accumulators of tcgen05.mma hold exactly; the
// groups g = 0..6 are kept in seven accumulators and put together as one integer.  The
// groups past 6 that are left out are 2^-54 of a typical row sum, below one FP64 rounding.  (Error-free splitting
// of matrix products after Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012.)
//
// All digits of one K step of B stand one below the other (row = 32 digit + vector), so
// digit i of A takes the first 7 - i digits of B in one MMA of N = 32 (7 - i) whose
// columns start at 32 i: group g = i + j lands in columns 32 g .. 32 g + 31 by itself.
#pragma once
#include "mw3_tc.cuh"

#include <cuda_fp16.h>

namespace mw3 {
namespace fx {

constexpr int ND = 7;                              // digits
constexpr int NV = 32;                             // vectors of one tile
constexpr int KS = 16;                             // K of one MMA
constexpr int KB = 128;                            // K of one B block in shared memory
constexpr uint32_t APL = 128 * KS * 2;             // one digit of one K step of A: 4 KB
constexpr uint32_t ASTEP = ND * APL;               // 28 KB
constexpr uint32_t BSTEP = ND * NV * KS * 2;       // 7 KB
constexpr uint32_t BBYTES = (KB / KS) * BSTEP;     // 56 KB
constexpr uint32_t SBO = 256, LBO = 128;
constexpr int WORKERS = 256;
constexpr uint32_t SMALL = 1024;
constexpr uint32_t SMEM = BBYTES + 2 * ASTEP + SMALL;   // 113 KB: two CTAs per SM

// element (row, k) of one digit of a K step of A
__host__ __device__ constexpr uint32_t a_off(int r, int k)
{
    return (uint32_t)((r & 7) * 16 + (r >> 3) * SBO + (k & 7) * 2 + (k >> 3) * LBO);
}

__device__ __forceinline__ unsigned hi_abs(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }

// round(x 2^(57 - E)) for |x| < 2^E, E = ef - 1022 with ef the exponent field of the
// largest |x| of the vector; sh = 4, or 3 to leave a bit for a sum of two
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
    for (int d = 0; d < ND; d++) {
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
            const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&u), d ? off : off0);
            w[p] = *reinterpret_cast<const uint32_t *>(&v);
        }
        *reinterpret_cast<uint4 *>(dst + d * digit_stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// one accumulator row of eight vectors: v[g][c], g the group; the sum over k S x in FP64.
// ef: exponent field of the vector's largest |x|, sh as in to_fixed
__device__ __forceinline__ double combine(const uint32_t (&v)[ND][8], int c, int ef, int sh)
{
    int a[ND];
#pragma unroll
    for (int g = 0; g < ND; g++) a[g] = __float2int_rn(__uint_as_float(v[g][c]));
    const long long H = ((long long)a[0] << 24) + ((long long)a[1] << 16) + ((long long)a[2] << 8) + a[3];
    const long long L = ((long long)a[4] << 16) + ((long long)a[5] << 8) + a[6];
    // the leading 62 bits of H 2^24 + L, in units 2^(72-z) of 2^54 2^(57-E)
    const int z = min(24, __clzll(H < 0 ? ~H : H) - 2);
    const long long V = (H << z) + (L >> (24 - z));
    if (ef >= 0x7FF) return __longlong_as_double(0x7FF8000000000000ll);   // an infinity or NaN in the vector
    if (V == 0) return 0.0;
    const double y = (double)V;
    const int sc = ef - 1061 + (4 - sh) - z;         // E - 39 - z, one more for a folded vector
    const int e = (int)(((unsigned)__double2hiint(y) >> 20) & 0x7FFu) + sc;
    if (e > 0 && e < 0x7FF)
        return __hiloint2double(__double2hiint(y) + (sc << 20), __double2loint(y));
    return scalbn(y, sc);
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

// the MMAs of one K step: A at a (ND planes), B at b
__device__ __forceinline__ void step(uint32_t d, uint64_t a, uint64_t b, int bmn, int accumulate)
{
#pragma unroll
    for (int i = 0; i < ND; i++)
        mma_f16(d + NV * i, a + (uint64_t)(i * (APL >> 4)), b, idesc(128, NV * (ND - i), bmn), i ? 1 : accumulate);
}

// eight columns of this thread's lane, without the wait
__device__ __forceinline__ void ld8_nw(uint32_t taddr, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void regs8(uint32_t *r)
{
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]));
}

// the ND accumulators of eight columns of this thread's lane
__device__ __forceinline__ void load_groups(uint32_t taddr, uint32_t (&v)[ND][8])
{
#pragma unroll
    for (int g = 0; g < ND; g++) ld8_nw(taddr + NV * g, v[g]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int g = 0; g < ND; g++) regs8(v[g]);
}

}  // namespace fx
}  // namespace mw3
