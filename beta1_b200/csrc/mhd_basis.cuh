// The basis vector an operator product of the persistent GMRES solve starts
// from, element by element, from vectors that are complete at the last grid
// barrier.  Shared by the kernel and host builds of the same code.
#pragma once

#include <cstdint>

#ifndef __CUDACC__
#define MHD_BASIS_HD
#else
#define MHD_BASIS_HD __host__ __device__ __forceinline__
#endif

namespace mhd
{

// V_j = (v - sum_{c < nc} d[c] V_c) / div.  For j > 0 v is w', what the first
// Gram-Schmidt pass left, and d the second pass's products: no thread stores
// the corrected vector over v, so an element reads the same whether its owner
// has gone on already or not (a product's aliases and copies take elements of
// other CTAs, and no barrier lies between the correction and the product).
struct BasisVec
{
    const double *v;
    double div;
    const double *V; // V_c at V + c n
    const double *d;
    int nc;
    int64_t n;

    MHD_BASIS_HD double at(int64_t t) const
    {
        double s = v[t];
        for (int c = 0; c < nc; ++c)
            s -= d[c] * V[int64_t(c) * n + t];
        return s / div;
    }
};

} // namespace mhd
