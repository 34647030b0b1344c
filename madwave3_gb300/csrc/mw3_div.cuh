#pragma once

namespace mw3 {

// a / b, correctly rounded, for a divisor that every point shares: z = 1 / b rounded
// once on the host, then one multiply and two FMAs (Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is known
// in advance", 2004).  That needs every intermediate clear of under- and overflow:
// zdiv_ok says so for b, the exponent test for a; a zero keeps its sign, and the rest
// (tiny, huge, infinite, NaN) is divided.  The tests are integer instructions, off
// the FP64 pipe.
// The FP64 update is bound by that pipe (two operations a clock an SM): a division of
// each point took k_update 204 us an iteration at 256 x 128 x 60, J = 10 (11 blocks),
// this 158 us, with the same bits.
__host__ __device__ inline bool zdiv_ok(double b) { return b >= 0x1p-100 && b < 0x1p100; }

__device__ __forceinline__ double div_shared(double a, double b, double z, bool ok)
{
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7FFFFFFFu;
    const double q = a * z;
    if (ok && hi - (200u << 20) < (1600u << 20)) return fma(fma(-q, b, a), z, q);   // 2^-823 <= |a| < 2^777
    if (ok && (hi | (unsigned)__double2loint(a)) == 0u) return q;
    return a / b;
}

}  // namespace mw3
