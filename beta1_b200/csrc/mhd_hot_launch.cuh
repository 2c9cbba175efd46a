// Host side of the hot kernels' launches (mhd_hot.cuh).
#pragma once

#include "mhd_hot.cuh"

#include <type_traits>
#include <utility>

namespace mhd
{

constexpr unsigned kHotCta = 256;

template <class... P, class... Q>
inline void hot_launch(void (*kernel)(P...), dim3 grid, cudaStream_t st, Q &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kHotCta);
    cfg.stream = st;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Q>(args)...);
}

// f(arguments, grid) for every chunk of blocks over a kind's points, or, with
// nreg > 0, over region boxes of at most nreg points; returns the launches
template <class F> inline int hot_for(const HotGrid &h, int kind, F f, int64_t nreg = 0)
{
    for (const HotChunk &c : h.chunks)
    {
        const unsigned x = nreg > 0 ? unsigned((nreg + kHotCta - 1) / kHotCta) : c.ctas[kind];
        const dim3 g(x, c.args.flat ? 1u : unsigned(c.args.n));
        if (c.args.n <= kHotFew)
            f(c.few, g);
        else
            f(c.args, g);
    }
    return int(h.chunks.size());
}

// the same over every point of the blocks with their ghost layers, one grid row per block
template <class F> inline int hot_for_padded(const HotGrid &h, F f)
{
    for (const HotChunk &c : h.chunks)
    {
        const dim3 g(unsigned((c.padded + kHotCta - 1) / kHotCta), unsigned(c.args.n));
        if (c.args.n <= kHotFew)
            f(c.few, g);
        else
            f(c.args, g);
    }
    return int(h.chunks.size());
}

} // namespace mhd
