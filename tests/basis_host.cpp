// Host build of the persistent solve's basis vectors (mhd_basis.cuh) for
// tests/test_cpu_basis_order.py.
#include "../beta1_b200/csrc/mhd_basis.cuh"

using namespace mhd;

extern "C" {

// Elements idx[0..m) of V_j as a product reads them, from the state that the
// second reduction of step j - 1 leaves (w: w', d: its products), with the
// owners of the elements named in gone[0..g) a step further: they have stored
// their elements of V_j.
void basis_read(int64_t n, int j, const double *w, double div, double *V, const double *d, const int64_t *gone, int64_t g,
                const int64_t *idx, int64_t m, double *out)
{
    const BasisVec x{w, div, V, d, j, n};
    for (int64_t q = 0; q < g; ++q)
        V[int64_t(j) * n + gone[q]] = x.at(gone[q]);
    for (int64_t q = 0; q < m; ++q)
        out[q] = x.at(idx[q]);
}
}
