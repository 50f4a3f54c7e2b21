// Chained launches: a kernel of a sequence whose blocks may become resident while the one before it finishes.
//
// The solves of the linear system are sequences of short kernels (3 to 20 us each at 250,000 cells), in which the drain of
// one and the start of the next took up to a tenth of the time: GMRES(30) on 249,600 tets in FP64 3.91 -> 3.49 ms,
// GMRES(10) with the block ILU(0) 4.50 -> 4.27 ms, GMRES(30) on 1,996,800 tets in FP32 12.99 -> 12.44 ms.  The kernels of
// a residual on a small mesh are shorter still: 30.7 -> 23.4 us on 8,192 triangles, an ESDIRK4 step there 10.3 -> 7.8 ms.
//
// A kernel launched by launch_chained may start early; it must call chain_wait before it reads what an earlier kernel of
// the sequence wrote, or writes what one may still read (the wait ends when all earlier kernels have completed and their
// writes are visible), and chain_release after it, which lets the next one start in turn.  Ahead of its wait a kernel may
// read what was written before the sequence began, and what a kernel of the sequence wrote if another one stands between
// the two: that one releases its successor only after its own wait, so the writer has completed by then.  The solve's
// sweeps read the operator that way; its builder is part of the sequence, and the gather of the right-hand side stands
// between them.  A reader that follows its writer directly has to wait first, or be launched unchained.  Arrays that a
// sequence writes are not __restrict__ parameters, so that the compiler moves no load of them ahead of the wait.
#pragma once
#include "platform.cuh"
#include <utility>

namespace dndsb
{
DNDSB_D void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
DNDSB_D void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
DNDSB_D void chain_step()
{
    chain_wait();
    chain_release();
}

template <typename... P, typename... A>
void launch_chained_shared(void (*kernel)(P...), unsigned grid, unsigned block, size_t shared, cudaStream_t st, A &&...args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid), cfg.blockDim = dim3(block), cfg.dynamicSmemBytes = shared, cfg.stream = st, cfg.attrs = &at, cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <typename... P, typename... A>
void launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t st, A &&...args)
{
    launch_chained_shared(kernel, grid, block, 0, st, std::forward<A>(args)...);
}
// DNDSB_LAUNCH, chained
#define DNDSB_CHAIN(kernel, n, block, stream, ...)                                                           \
    do                                                                                                       \
    {                                                                                                        \
        if ((n) > 0)                                                                                         \
            ::dndsb::launch_chained(kernel, ::dndsb::grid_for((n), (block)), (block), (stream), __VA_ARGS__); \
    } while (0)
} // namespace dndsb
