// Host build of the hot kernels' point arithmetic (mhd_hot.cuh) for
// tests/test_cpu_hot_args.py, and of the weights' order (mhd_layout.cuh).
#include "../beta1_b200/csrc/mhd_hot.cuh"

using namespace mhd;

extern "C" {

// quotients of numerators t[0..n) by d, as the kernels form them
void hot_quot(uint32_t d, const uint32_t *t, uint32_t *q, int n)
{
    const FastDiv f = fast_div(d);
    for (int i = 0; i < n; ++i)
        q[i] = fast_quot(t[i], f);
}

int hot_plane_of(int f) { return plane_of(f); }

// the weights' order on a block: cell[p] and back[cell[p]] of every padded point p
void weight_order(int ni, int nj, int nk, int G, int64_t *cell, int64_t *back)
{
    BlockView b{};
    b.ni = ni, b.nj = nj, b.nk = nk, b.G = G;
    b.NJ = nj + 1 + 2 * G, b.NK = nk + 1 + 2 * G;
    b.vol = (int64_t(ni + 1 + 2 * G) * b.NJ * b.NK + 31) & ~int64_t(31);
    int64_t p = 0;
    for (int i = -G; i <= ni + G; ++i)
        for (int j = -G; j <= nj + G; ++j)
            for (int k = -G; k <= nk + G; ++k, ++p)
            {
                cell[p] = weight_cell(b, i, j, k);
                back[p] = weight_point(b, cell[p]);
            }
}

int64_t weight_value(int64_t d, int ncomp, int m) { return weight_tile(d, ncomp) + int64_t(m) * kWTile; }
}
