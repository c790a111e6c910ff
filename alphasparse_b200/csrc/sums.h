// Sums of fp64 products with what their roundings leave out: two-sum (Knuth, The Art of Computer Programming 2, 4.2.2), with the products' own
// errors by fma as in the dot product of Ogita, Rump and Oishi (Accurate sum and dot product, 2005).
#ifndef ASP_SUMS_H
#define ASP_SUMS_H

namespace asp
{
struct TwoSum
{
    double hi = 0, lo = 0;
    // (__dmul_rn: a product that the compiler contracts into the sums that follow would not be the one whose error is taken)
    __device__ __forceinline__ void add(double v, double x)
    {
        const double p = __dmul_rn(v, x), t = hi + p, b = t - hi;
        lo += (hi - (t - b)) + (p - b) + fma(v, x, -p);
        hi = t;
    }
    __device__ __forceinline__ void add(const TwoSum &o)
    {
        const double t = hi + o.hi, b = t - hi;
        lo += (hi - (t - b)) + (o.hi - b) + o.lo;
        hi = t;
    }
    __device__ __forceinline__ double value() const { return isfinite(hi) ? hi + lo : hi; } // (the errors of an infinite sum are no numbers)
};
} // namespace asp
#endif
