// gb_noalloc.cu -- the Gram product V^T W for callers that cannot allocate
// device memory.
//
// Some embedding applications own the whole GPU memory through their own pool
// or arena and may not call cudaMalloc / cudaFree (those calls can synchronise
// the device and would take memory the pool has already claimed). This entry
// point computes the same Gram block as GCGE_GPU_MultiVecInnerProd into memory
// the caller passes, with its partial sums in a fixed file-scope device array
// instead of the library's context scratch, and allocates nothing. It runs on the
// tensor cores (gb_ozaki.cu: gb_gram_fixed) where that is the shorter way and the
// operands prove that the digits which column scales leave them keep every entry within
// the bound of a plain FP64 sum, and on the FP64 pipe (k_gram_partial, plain FP64 fused multiply-adds
// with a fixed-order second stage) otherwise: at 262,144 x (178, 64) 5.45 ms on the
// FP64 pipe, 0.42 ms on the tensor cores; at 600,000 x (256, 128) 33.0 and 1.82 ms.
//
// The array is GB_NOALLOC_DOUBLES doubles (8 MiB) and a control block of 64 KiB beside
// it (column scales); every GPU that loads the library holds them until the process
// exits. All calls share it and it keeps the
// last call's contents: every call writes each partial it later reads, so
// nothing needs to start at zero. Calls that overlap on the GPU (different
// streams, or different host threads on one device) race on the array.
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "gb_internal.h"

#define GB_NOALLOC_DOUBLES (1u << 20)
#define GB_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) double g_noalloc_partials[GB_NOALLOC_DOUBLES];
static __device__ __align__(256) char g_noalloc_ctl[GB_GRAM_FIXED_CTL];

// Per-device address of the array and SM count, set up on the first call on a
// device with that device current (host code must not pass the array's name:
// on the host it is only a stand-in symbol, not a device address). The set-up
// runs under a lock; the address is published with a release store after the SM
// count, and read with an acquire load, so a thread that sees the address also
// sees the count, whichever host thread made the first call.
static std::atomic<double *> s_part_addr[GB_NOALLOC_MAX_DEVICES];
static std::atomic<void *> s_ctl_addr[GB_NOALLOC_MAX_DEVICES];
static std::atomic<int> s_num_sms[GB_NOALLOC_MAX_DEVICES];
static std::mutex s_setup_lock;

static int setup_device(int dev, double **part, void **ctl, int *num_sms)
{
    double *p = s_part_addr[dev].load(std::memory_order_acquire);
    if (!p) {
        std::lock_guard<std::mutex> guard(s_setup_lock);
        p = s_part_addr[dev].load(std::memory_order_acquire);
        if (!p) {
            void *addr = nullptr, *caddr = nullptr;
            if (cudaGetSymbolAddress(&addr, g_noalloc_partials) != cudaSuccess || !addr) return GCGE_GPU_ERR_CUDA;
            if (cudaGetSymbolAddress(&caddr, g_noalloc_ctl) != cudaSuccess || !caddr) return GCGE_GPU_ERR_CUDA;
            if (gb_gram_fixed_ctl_bytes() > GB_GRAM_FIXED_CTL) return GCGE_GPU_ERR_CUDA;
            int sms = 0;
            if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
                return GCGE_GPU_ERR_CUDA;
            s_num_sms[dev].store(sms, std::memory_order_relaxed);
            s_ctl_addr[dev].store(caddr, std::memory_order_relaxed);
            p = (double *)addr;
            s_part_addr[dev].store(p, std::memory_order_release);
        }
    }
    *part = p;
    *ctl = s_ctl_addr[dev].load(std::memory_order_relaxed);
    *num_sms = s_num_sms[dev].load(std::memory_order_relaxed);
    return GCGE_GPU_OK;
}

extern "C" int GCGE_GPU_InnerProdNoAlloc(int n, int k1, int k2, const double *V, long ldv, const double *W, long ldw,
                                         double *a, int lda, int sym, void *stream)
{
    if (n <= 0 || k1 <= 0 || k2 <= 0 || !V || !W || !a || lda < k1 || ldv < k1 || ldw < k2 || (sym && k1 != k2))
        return GCGE_GPU_ERR_ARG;
    if ((size_t)k1 * k2 > GB_NOALLOC_DOUBLES / 4) return GCGE_GPU_ERR_ARG;   // at most 262,144 entries
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= GB_NOALLOC_MAX_DEVICES) return GCGE_GPU_ERR_CUDA;
    double *part = nullptr;
    int num_sms = 0;
    void *ctl = nullptr;
    int st = setup_device(dev, &part, &ctl, &num_sms);
    if (st) return st;
    return gb_gram_fixed((cudaStream_t)stream, num_sms, n, k1, k2, V, ldv, W, ldw, a, lda, sym, part,
                         GB_NOALLOC_DOUBLES, ctl);
}
