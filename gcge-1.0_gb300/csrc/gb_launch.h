// gb_launch.h -- kernel launches of a context's stream.
//
// A solve of a few thousand unknowns is some thousand launches of kernels of a few
// microseconds, one after the other, and between two of them the chip drains, flushes and
// starts again: 2 to 3 us each time. Launches therefore carry the programmatic
// stream-serialisation attribute: a kernel's blocks are placed while its predecessor's last
// ones retire, and every kernel begins with GB_PDL(), which waits until the predecessor is
// complete and its writes are visible, before it touches memory. The order of the stream's
// work is what it was. (Where the operation before is no kernel, or the kernel was launched
// without the attribute, the instruction does nothing.) No kernel lets its successor in
// before its own end (griddepcontrol.launch_dependents): the blocks that then sit waiting
// take shared memory from the L1 of the kernel that still runs, and the block Gram product
// over 262144 rows rose from 484 to 512 us, a whole orthonormalisation from 5.51 to 5.70 ms.
// Measured, without the attribute -> with it: 30 x 30 grid (6 pairs) 21.6 -> 19.6 ms,
// 100 x 100 grid 56.2 -> 52.2 ms, 48^3 cells in mixed precision 454 -> 400 ms, 64^3 brick
// orthonormalisation 5.57 -> 5.51 ms.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "gb_internal.h"

#define GB_PDL() asm volatile("griddepcontrol.wait;" ::: "memory")

template <typename... P, typename... A>
static inline cudaError_t gb_launch(cudaStream_t stream, dim3 grid, dim3 block, size_t smem, void (*kern)(P...), A &&...args)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

#define GB_LAUNCH(ctx, kern, grid, block, smem, ...)                                   \
    do {                                                                               \
        gb_launch((ctx)->stream, (grid), (block), (smem), kern, __VA_ARGS__);          \
        (ctx)->launches++;                                                             \
        if ((ctx)->prof) gb_prof_end(ctx);                                             \
        int _st = gb_check_launch(ctx);                                                \
        if (_st) return _st;                                                           \
    } while (0)
