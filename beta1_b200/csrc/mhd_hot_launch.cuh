// Host side of the hot kernels' launches (mhd_hot.cuh).
#pragma once

#include "mhd_hot.cuh"

#include <type_traits>
#include <utility>

namespace mhd
{

constexpr unsigned kHotCta = 256;

// A launch that may start while the kernel before it on the stream drains
// (the kernel waits before it reads what others write, pdl_wait): about 1 us
// less from kernel to kernel inside the step's graph.
template <class... P, class... Q>
inline void pdl_launch(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                       Q &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Q>(args)...);
}

template <class... P, class... Q>
inline void hot_launch(void (*kernel)(P...), dim3 grid, cudaStream_t st, Q &&...args)
{
    pdl_launch(kernel, grid, kHotCta, 0, st, std::forward<Q>(args)...);
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
