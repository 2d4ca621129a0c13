// The Transform trait of the reference (montmul/src/transform.rs:22-46), as its Gpu backend
// implements it (gpu/mod.rs:286-319): buffers of `count` vectors of L/2 elements in GF(M31^2) x
// GF(M61^2), batched forward (weight by zeta^j, DIF), inverse (DIT, unweight by zeta^-j / n)
// and pointwise products with per-vector scales. Lengths up to L = 16,384 transform one vector
// per block in shared memory; longer ones in global mode (passes over device memory plus
// bulk-copied shared-memory tiles).
//
// On the device a vector of a shared-memory length is in the reference's element order, so a
// download is one copy per field. A global-mode vector keeps the kernels' order (element j at
// swz(j), a permutation within aligned 16-element blocks); upload and download apply and remove it
// on the device. Coefficients cross the bus as the caller's 32-bit limbs and become field elements on
// the device: 64 vectors of L = 8,192 through load_forward twice, pointwise, inverse and
// download_raw take 3.8 ms where the host expanding and permuting them took 13.9 (medians of 200 passes
// of one process; on a shared host single passes and whole processes vary by more than that). The rest is
// the 6.3 MB result into fresh pages and the allocations.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <string>
#include <vector>

#include "../../include/montmul_b200.h"
#include "mm_global.cuh"
#include "mm_host.hpp"

using namespace mm;

// Defined in mm_backend.cu.
extern "C++" int mm_set_error(int code, const std::string& msg);
extern "C++" int mm_device_tables(mm_b200_device* dev, int m, bool global, const F2K** t2, const F1** t1,
                                  KernelSet* ks, GlobalKernels* gk);
extern "C++" int mm_device_ordinal(const mm_b200_device* dev);

struct mm_b200_tbuf {
    mm_b200_device* dev = nullptr;
    size_t len = 0, count = 0, n = 0;
    F2* d2 = nullptr;
    F1* d1 = nullptr;
};

namespace {

#define TK(call)                                                                                      \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) return mm_set_error(MM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int log2_len(size_t len) {
    int l = 0;
    while (((size_t)1 << l) < len) ++l;
    return ((size_t)1 << l) == len ? l : -1;
}

// out = scale a b per element (cpu.rs:395-407): canonical GF(p^2) products; the scale of vector
// v is scales[v] (reduced mod M31 for the M31 part), or 1.
__global__ void pointwise_kernel(F2* o2, F1* o1, const F2* a2, const F1* a1, const F2* b2, const F1* b1,
                                 const uint32_t* scales, int logn, size_t total) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        F2 x = cmul(a2[e], b2[e]);
        F1 y = cmul(a1[e], b1[e]);
        const uint32_t c = scales ? scales[e >> logn] : 1u;
        if (c != 1) {
            x = cmul_r((uint64_t)c, x);
            y = cmul_r(c % P1, y);
        }
        o2[e] = x;
        o1[e] = y;
    }
}

// Field elements of a buffer from rows of k 32-bit coefficients, zero from k on (cpu.rs:349-358):
// coefficient j in the real part of element j, j + n in the imaginary part, as it is for M61 and mod
// M31. SWZ: the buffer is in the kernels' element order. The rows are in the memory that the M31 elements
// will take (8 bytes an element, the 4 bytes of two coefficients), so the M31 elements are made from
// the M61 ones by a second kernel.
template <bool SWZ>
__global__ void expand_kernel(const uint32_t* __restrict__ c, uint32_t k, int logn, size_t total, F2* o2) {
    const uint32_t n = 1u << logn;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t v = e >> logn;
        const uint32_t j = (uint32_t)e & (n - 1);
        const uint32_t* row = c + v * k;
        o2[SWZ ? (v << logn) + (size_t)swz((int)j) : e] = f2(j < k ? row[j] : 0u, j + n < k ? row[j + n] : 0u);
    }
}
__global__ void expand_m31_kernel(const F2* __restrict__ in, size_t total, F1* o1) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const uint32_t re = (uint32_t)in[e].re, im = (uint32_t)in[e].im;
        o1[e] = f1(csubp1((re & P1) + (re >> 31)), csubp1((im & P1) + (im >> 31)));
    }
}

// Elements first .. first + part - 1 of a buffer in the kernels' order, to natural order.
template <class T>
__global__ void natural_kernel(const T* __restrict__ in, int logn, size_t first, size_t part, T* out) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < part; i += (size_t)gridDim.x * blockDim.x) {
        const size_t e = first + i;
        out[i] = in[(e >> logn << logn) + (size_t)swz((int)(e & (((size_t)1 << logn) - 1)))];
    }
}

unsigned grid_for(size_t total) { return (unsigned)std::min<size_t>((total + 255) / 256, 148 * 16); }

// A device allocation released at the end of its scope.
struct DevMem {
    void* p = nullptr;
    ~DevMem() { cudaFree(p); }
};

// Bound of the device staging of a global-mode download, in elements.
constexpr size_t kStageElements = (size_t)1 << 20;

bool swizzled(size_t n) { return log2_len(n) > kMaxSharedLogN; }

// A new buffer of `count` vectors of length len from rows of k coefficients each.
int upload_rows(mm_b200_device* dev, const uint32_t* rows, size_t k, size_t len, size_t count, const char* what,
                mm_b200_tbuf** out) {
    const int l = log2_len(len);
    if (l < 3 || l > kMaxGlobalLogN + 1)
        return mm_set_error(MM_ERR_ARG, std::string(what) + ": length must be a power of two in 8 .. 2^24");
    const size_t n = len / 2, total = count * n;
    TK(cudaSetDevice(mm_device_ordinal(dev)));
    std::unique_ptr<mm_b200_tbuf, void (*)(mm_b200_tbuf*)> b(new mm_b200_tbuf(), mm_b200_t_free);
    b->dev = dev;
    b->len = len;
    b->count = count;
    b->n = n;
    TK(cudaMalloc(&b->d2, std::max<size_t>(1, total) * sizeof(F2)));
    TK(cudaMalloc(&b->d1, std::max<size_t>(1, total) * sizeof(F1)));
    if (total) {
        uint32_t* c = reinterpret_cast<uint32_t*>(b->d1);
        if (k) TK(cudaMemcpyAsync(c, rows, count * k * 4, cudaMemcpyHostToDevice, cudaStreamLegacy));
        if (swizzled(n)) expand_kernel<true><<<grid_for(total), 256, 0, cudaStreamLegacy>>>(c, (uint32_t)k, l - 1, total, b->d2);
        else expand_kernel<false><<<grid_for(total), 256, 0, cudaStreamLegacy>>>(c, (uint32_t)k, l - 1, total, b->d2);
        TK(cudaGetLastError());
        expand_m31_kernel<<<grid_for(total), 256, 0, cudaStreamLegacy>>>(b->d2, total, b->d1);
        TK(cudaGetLastError());
        TK(cudaStreamSynchronize(cudaStreamLegacy));   // the caller's rows are free again
    }
    *out = b.release();
    return MM_OK;
}

// A buffer's `total` elements in natural order to the host.
template <class T>
int download(const T* d, size_t n, size_t total, void* host) {
    if (!swizzled(n)) {
        TK(cudaMemcpy(host, d, total * sizeof(T), cudaMemcpyDeviceToHost));
        return MM_OK;
    }
    const size_t step = std::min(total, kStageElements);
    DevMem stage;
    if (cudaMalloc(&stage.p, step * sizeof(T)) != cudaSuccess) {
        // No room for the staging: the order is undone in place on the host (swz permutes within 16 elements).
        cudaGetLastError();
        stage.p = nullptr;
        TK(cudaMemcpy(host, d, total * sizeof(T), cudaMemcpyDeviceToHost));
        T* h = static_cast<T*>(host);
        for (size_t e = 0; e < total; e += 16) {
            T in[16];
            std::copy(h + e, h + e + 16, in);
            const int j0 = (int)(e & (n - 1));
            for (int j = 0; j < 16; ++j) h[e + j] = in[swz_c(j0 + j) & 15];
        }
        return MM_OK;
    }
    for (size_t e = 0; e < total; e += step) {
        const size_t part = std::min(step, total - e);
        natural_kernel<<<grid_for(part), 256, 0, cudaStreamLegacy>>>(d, log2_len(n), e, part, static_cast<T*>(stage.p));
        TK(cudaGetLastError());
        TK(cudaMemcpy(static_cast<T*>(host) + e, stage.p, part * sizeof(T), cudaMemcpyDeviceToHost));
    }
    return MM_OK;
}

int check_buf(const mm_b200_tbuf* b, size_t len, size_t count, const char* what) {
    if (!b) return mm_set_error(MM_ERR_ARG, std::string(what) + ": null buffer");
    if (b->len != len || b->count < count)
        return mm_set_error(MM_ERR_ARG, std::string(what) + ": buffer holds " + std::to_string(b->count) +
                                            " vectors of length " + std::to_string(b->len));
    return MM_OK;
}

int transform(mm_b200_tbuf* b, size_t len, size_t count, bool inverse) {
    const char* what = inverse ? "t_inverse" : "t_forward";
    int rc = check_buf(b, len, count, what);
    if (rc || count == 0) return rc;
    const int m = log2_len(len) - 1;
    TK(cudaSetDevice(mm_device_ordinal(b->dev)));
    const bool global = m > kMaxSharedLogN;
    const F2K* t2 = nullptr;
    const F1* t1 = nullptr;
    KernelSet ks{};
    GlobalKernels gk{};
    rc = mm_device_tables(b->dev, m, global, &t2, &t1, &ks, &gk);
    if (rc) return rc;
    uint32_t* d_err = nullptr;
    if (global) {
        TK(cudaFuncSetAttribute((const void*)gtransform_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGlobalSmem));
        TK(cudaMalloc(&d_err, 4));
        TK(cudaMemset(d_err, 0, 4));
    }
    for (size_t v0 = 0; v0 < count; v0 += 65535) {
        const unsigned grid = (unsigned)std::min<size_t>(65535, count - v0);
        if (global)
            gtransform_kernel<256><<<grid, 256, kGlobalSmem>>>(b->d2, b->d1, t2, t1, m, (uint32_t)v0, inverse ? 1 : 0, d_err);
        else
            ks.transform<<<grid, ks.threads, ks.smem>>>(b->d2, b->d1, t2, t1, (uint32_t)v0, inverse ? 1 : 0);
        TK(cudaGetLastError());
    }
    TK(cudaDeviceSynchronize());
    if (global) {
        uint32_t err = 0;
        TK(cudaMemcpy(&err, d_err, 4, cudaMemcpyDeviceToHost));
        TK(cudaFree(d_err));
        if (err) return mm_set_error(MM_ERR_CUDA, std::string(what) + ": a bulk copy did not complete within its time limit");
    }
    return MM_OK;
}

}  // namespace

extern "C" {

int mm_b200_t_upload(mm_b200_device* dev, const uint32_t* coeffs, size_t len, size_t count, mm_b200_tbuf** out) {
    if (!dev || !out || (!coeffs && count)) return mm_set_error(MM_ERR_ARG, "t_upload: null argument");
    return upload_rows(dev, coeffs, len, len, count, "t_upload", out);
}

int mm_b200_t_download_raw(const mm_b200_tbuf* b, uint32_t* f1, uint64_t* f2) {
    if (!b || (!f1 && !f2)) return mm_set_error(MM_ERR_ARG, "t_download_raw: null argument");
    TK(cudaSetDevice(mm_device_ordinal(b->dev)));
    const size_t total = b->count * b->n;
    if (!total) return MM_OK;
    // F2 and F1 are (re, im) pairs, the layout of f2 and f1.
    if (f2) {
        const int rc = download(b->d2, b->n, total, f2);
        if (rc) return rc;
    }
    return f1 ? download(b->d1, b->n, total, f1) : (int)MM_OK;
}

int mm_b200_t_forward(mm_b200_tbuf* b, size_t len, size_t count) { return transform(b, len, count, false); }
int mm_b200_t_inverse(mm_b200_tbuf* b, size_t len, size_t count) { return transform(b, len, count, true); }

int mm_b200_t_pointwise(mm_b200_tbuf* out, const mm_b200_tbuf* a, const mm_b200_tbuf* bb, const uint32_t* scales,
                        size_t len, size_t count) {
    int rc = check_buf(out, len, count, "t_pointwise");
    if (!rc) rc = check_buf(a, len, count, "t_pointwise");
    if (!rc) rc = check_buf(bb, len, count, "t_pointwise");
    if (rc || count == 0) return rc;
    TK(cudaSetDevice(mm_device_ordinal(out->dev)));
    uint32_t* d_sc = nullptr;
    if (scales) {
        TK(cudaMalloc(&d_sc, count * 4));
        TK(cudaMemcpy(d_sc, scales, count * 4, cudaMemcpyHostToDevice));
    }
    const size_t total = count * out->n;
    const int logn = log2_len(out->n);
    const unsigned grid = (unsigned)std::min<size_t>((total + 255) / 256, 148 * 16);
    pointwise_kernel<<<grid, 256>>>(out->d2, out->d1, a->d2, a->d1, bb->d2, bb->d1, d_sc, logn, total);
    TK(cudaGetLastError());
    TK(cudaDeviceSynchronize());
    if (d_sc) TK(cudaFree(d_sc));
    return MM_OK;
}

int mm_b200_t_load_forward(mm_b200_device* dev, const uint32_t* limbs, size_t k, size_t len, size_t count,
                           mm_b200_tbuf** out) {
    if (!dev || !out || (!limbs && count && k)) return mm_set_error(MM_ERR_ARG, "t_load_forward: null argument");
    if (k > len) return mm_set_error(MM_ERR_ARG, "t_load_forward: more limbs than coefficients");
    int rc = upload_rows(dev, limbs, k, len, count, "t_upload", out);
    if (rc) return rc;
    rc = mm_b200_t_forward(*out, len, count);
    if (rc) {
        mm_b200_t_free(*out);
        *out = nullptr;
    }
    return rc;
}

size_t mm_b200_t_count(const mm_b200_tbuf* b) { return b ? b->count : 0; }
size_t mm_b200_t_len(const mm_b200_tbuf* b) { return b ? b->len : 0; }

void mm_b200_t_free(mm_b200_tbuf* b) {
    if (!b) return;
    cudaSetDevice(mm_device_ordinal(b->dev));
    cudaFree(b->d2);
    cudaFree(b->d1);
    delete b;
}

}  // extern "C"
