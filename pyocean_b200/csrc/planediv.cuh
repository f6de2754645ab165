// Index divisions of the advection launches as multiplies: plane index -> layer of the k-major (layer, tracer) planes, and
// CTA -> tile of a batched launch (compiled for the host too by tests/hostcore).
#pragma once

#ifdef __CUDACC__
#define PO_PD __host__ __device__ __forceinline__
#else
#define PO_PD inline
#endif

namespace po {

// Division of a plane index p by the tracer count nt as a multiply-high (Granlund & Montgomery 1994, "Division by
// invariant integers using multiplication"): with m = ceil(2^32 / nt) and e = m nt - 2^32 < nt,
// floor(p m / 2^32) = floor(p / nt) whenever p e < 2^32, which holds for 0 <= p < 2^16 and 1 <= nt < 2^16 (the
// entry points bound nt * nz by 65535).  nt = 1 is encoded as m = 0 and divides by identity.
PO_PD unsigned plane_magic(int nt)
{
    return nt <= 1 ? 0u : (unsigned)((0x100000000ull + (unsigned long long)nt - 1) / (unsigned long long)nt);
}

PO_PD int plane_div(int p, unsigned m)
{
    return m == 0u ? p : (int)(((unsigned long long)(unsigned)p * m) >> 32);
}

// x / d for 0 <= x < d count as a multiply: with m = ceil(2^47 / d), e = m d - 2^47 < d, floor(x m / 2^47) = x / d
// whenever x e < 2^47 (the same method), which d d count < 2^47 ensures.  x m < 2^47 (count + 1) must fit 64 bits, and m
// itself is 2^47 for d = 1: counts up to 65535 take the multiply, larger ones (a domain of that many rows of tiles, one
// tile wide) and products beyond the bound m = 0, the division itself.
inline unsigned long long tile_magic(long long d, long long count)
{
    constexpr unsigned long long one = 1ull << 47;
    if (count > 65535 || (double)d * (double)d * (double)count >= 1.4e14) return 0ull;
    return (one + (unsigned long long)d - 1) / (unsigned long long)d;
}

PO_PD int tile_div(int x, unsigned long long m, int d)
{
    return m ? (int)(((unsigned long long)(unsigned)x * m) >> 47) : x / d;
}

}  // namespace po
