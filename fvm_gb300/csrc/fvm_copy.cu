// fvm_copy.cu -- the state copies of upload_state / download_state.
//
// A call moves 7 (2-D) or 9 (3-D) arrays.  One cudaMemcpyAsync per array cost 2.3 to 3.5 us
// of GPU time and 3 to 4 us of host time each on small grids, and one copy at a time
// reached 183 to 205 GB/s on large ones.  Where the caller's buffers are page-locked the
// arrays go in one kernel that reads or writes the host memory directly; any other
// buffer takes cudaMemcpyAsync as before.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "fvm_internal.cuh"

namespace fvm {
namespace {

constexpr int MOST = 9;

struct Copies {
    double *dst[MOST];
    const double *src[MOST];
    int vec[MOST];   // both addresses 16-byte aligned
};

__global__ void __launch_bounds__(256) k_copy(const __grid_constant__ Copies c, long long n)
{
    double *dst = c.dst[blockIdx.y];
    const double *src = c.src[blockIdx.y];
    const long long i0 = blockIdx.x * 256LL + threadIdx.x, step = 256LL * gridDim.x;
    if (c.vec[blockIdx.y]) {
        const long long h = n / 2;
        double2 *d2 = reinterpret_cast<double2 *>(dst);
        const double2 *s2 = reinterpret_cast<const double2 *>(src);
        for (long long i = i0; i < h; i += 4 * step) {   // four loads in flight per thread
            double2 v[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (i + q * step < h) v[q] = s2[i + q * step];
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (i + q * step < h) d2[i + q * step] = v[q];
        }
        if (i0 == 0 && (n & 1)) dst[n - 1] = src[n - 1];
    } else {
        for (long long i = i0; i < n; i += step) dst[i] = src[i];
    }
}

// Whether [p, p + bytes) lies in one page-locked host allocation or registration that the
// device reaches at the same address.
bool pinned(const void *p, size_t bytes)
{
    using Fn = CUresult (*)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
    static Fn get = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 7000, cudaEnableDefault, &r) == cudaSuccess &&
            r == cudaDriverEntryPointSuccess)
            get = reinterpret_cast<Fn>(f);
        else cudaGetLastError();
    });
    if (!get) return false;
    unsigned type = 0, managed = 1;
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute at[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void *out[] = {&type, &managed, &dev, &start, &size};
    const CUdeviceptr a = reinterpret_cast<CUdeviceptr>(p);
    if (get(5, at, out, a) != CUDA_SUCCESS) return false;
    return type == CU_MEMORYTYPE_HOST && !managed && dev == a && start != 0 && start <= a && a + bytes <= start + size;
}

}  // namespace

// Copies of n doubles each on the stream, dst[k] <- src[k], entries with a null address
// left out (kind: host to device or device to host; at most 9).
cudaError_t copy_arrays(double *const *dst, const double *const *src, int count, size_t n, cudaMemcpyKind kind,
                        cudaStream_t st)
{
    const size_t bytes = n * sizeof(double);
    Copies c{};
    int m = 0;
    for (int k = 0; k < count; k++) {
        if (!dst[k] || !src[k]) continue;
        const void *host = kind == cudaMemcpyHostToDevice ? (const void *)src[k] : (const void *)dst[k];
        bool direct = (reinterpret_cast<uintptr_t>(host) & 7u) == 0 && pinned(host, bytes);
        // overlapping targets keep the order of separate copies
        for (int q = 0; q < count; q++)
            if (q != k && dst[q] && dst[q] < dst[k] + n && dst[k] < dst[q] + n) direct = false;
        if (!direct) {
            const cudaError_t e = cudaMemcpyAsync(dst[k], src[k], bytes, kind, st);
            if (e != cudaSuccess) return e;
            continue;
        }
        c.dst[m] = dst[k];
        c.src[m] = src[k];
        c.vec[m] = ((reinterpret_cast<uintptr_t>(dst[k]) | reinterpret_cast<uintptr_t>(src[k])) & 15u) == 0;
        m++;
    }
    if (m == 0) return cudaSuccess;
    const long long blocks = std::min<long long>((long long)((n + 2047) / 2048), 152LL * 8 / m);
    k_copy<<<dim3((unsigned)std::max<long long>(blocks, 1), m), 256, 0, st>>>(c, (long long)n);
    return cudaGetLastError();
}

}  // namespace fvm
