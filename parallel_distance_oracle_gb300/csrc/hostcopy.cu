// hostcopy.cu -- host <-> device copies that the SMs carry out.
//
// Page-locked host memory (cudaHostAlloc / cudaHostRegister) has a device
// alias that kernels can read and write directly.  Copies to and from such
// memory are done here by a plain copy kernel rather than by the copy engines
// (cudaMemcpyAsync): on hosts where the copy engines are slowed by other work,
// half of the 1.5 GB exports of an R-MAT s20 index took 120 ms through them and
// 8-27 ms through the SMs.  Any other host memory goes through cudaMemcpyAsync.

#include "pado_internal.cuh"

namespace pado {
namespace {

// Up to five copies of one launch; grid row y takes copy y.
constexpr int MAX_COPIES = 5;
struct CopyList {
    const unsigned char *src[MAX_COPIES];
    unsigned char *dst[MAX_COPIES];
    uint64_t bytes[MAX_COPIES];
};

// dst[0, bytes) = src[0, bytes): 16 bytes of the destination, aligned, per
// thread step, the few before and after them bytewise.  Bound by the link to
// host memory (193 GB/s written, 211 read by this kernel at any grid of 152
// blocks and more, the same as the copy engines).  A source that is not
// aligned alike is read in 4-byte words and shifted into place; every word read
// holds a byte that is copied.  (Bytewise, a program that keeps many indexes' labels
// in one array, so that most start anywhere, waited 5.1 ms for the exports of 64
// graphs.)
__global__ void __launch_bounds__(256) sm_copy_kernel(const __grid_constant__ CopyList list)
{
    const unsigned char *src = list.src[blockIdx.y];
    unsigned char *dst = list.dst[blockIdx.y];
    const uint64_t bytes = list.bytes[blockIdx.y];
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t mis = (16 - ((uintptr_t)dst & 15)) & 15;
    const uint64_t head = mis < bytes ? mis : bytes;
    const uint64_t body = (bytes - head) / 16;
    if (tid < head) dst[tid] = src[tid];
    const uint64_t tail = head + body * 16 + tid;
    if (tail < bytes) dst[tail] = src[tail];
    src += head;
    uint4 *d4 = reinterpret_cast<uint4 *>(dst + head);
    if (((uintptr_t)src & 15) == 0) {
        const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
        for (uint64_t i = tid; i < body; i += nth) d4[i] = s4[i];
        return;
    }
    const uint32_t off = (uint32_t)((uintptr_t)src & 3), sh = 8 * off;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(src - off);
    for (uint64_t i = tid; i < body; i += nth) {
        const uint32_t w0 = w[4 * i], w1 = w[4 * i + 1], w2 = w[4 * i + 2], w3 = w[4 * i + 3];
        const uint32_t w4 = sh ? w[4 * i + 4] : 0u;
        d4[i] = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh),
                           __funnelshift_r(w3, w4, sh));
    }
}

void sm_copies(const CopyList &list, int n, cudaStream_t s, const char *name)
{
    uint64_t most = 0;
    for (int i = 0; i < n; ++i) most = std::max(most, list.bytes[i]);
    if (!n) return;
    // the first block's 256 threads alone cover a head and a tail (15 bytes each)
    const dim3 grid(grid_for(most / 16 + 1, 256, 152u * 16u), (unsigned)n);
    PADO_LAUNCH(name, s, sm_copy_kernel<<<grid, 256, 0, s>>>(list));
}

}  // namespace

void *mapped_host(const void *p)
{
    if (!p) return nullptr;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();  // an unknown pointer is not an error here
        return nullptr;
    }
    return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

void download_all(std::initializer_list<HostCopy> copies, cudaStream_t s)
{
    CopyList list;
    int n = 0;
    for (const HostCopy &c : copies) {
        if (!c.bytes) continue;
        if (void *dh = mapped_host(c.h)) {
            list.src[n] = static_cast<const unsigned char *>(c.d);
            list.dst[n] = static_cast<unsigned char *>(dh);
            list.bytes[n] = c.bytes;
            if (++n == MAX_COPIES) {
                sm_copies(list, n, s, "host_write_kernel");
                n = 0;
            }
        } else {
            PADO_CUDA(cudaMemcpyAsync(c.h, c.d, c.bytes, cudaMemcpyDeviceToHost, s));
        }
    }
    sm_copies(list, n, s, "host_write_kernel");
}

void upload_bytes(void *d, const void *h, uint64_t bytes, cudaStream_t s)
{
    if (!bytes) return;
    if (const void *dh = mapped_host(h)) {
        CopyList list;
        list.src[0] = static_cast<const unsigned char *>(dh);
        list.dst[0] = static_cast<unsigned char *>(d);
        list.bytes[0] = bytes;
        sm_copies(list, 1, s, "host_read_kernel");
    } else {
        PADO_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s));
    }
}

}  // namespace pado
