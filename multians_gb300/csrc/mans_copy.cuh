// Many small copies in one launch: between device memory and pinned host
// memory the GPU can address.
//
// A copy-engine copy of a few KB takes the engine 3.6 us and the host 1.7 us
// to issue, the link 0.1 us; the kernel moves bytes at the same rate as the
// engine (48 MB in: 206 against 207 GB/s, out 191 and 191, with 64 CTAs), so
// only large copies are left to the engine.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mans {

struct CopyItem {
    const uint8_t* src;
    uint8_t* dst;
    uint64_t bytes;
};

constexpr uint32_t kCopyItems = 128;           // a launch takes: 3 KB of parameters
constexpr uint32_t kCopyThreads = 128;         // few enough to fit beside a decode's CTAs
constexpr uint32_t kCopyCtas = 8;              // per item
constexpr uint64_t kCopyBytesMax = 256 << 10;  // of an item: 16 KB per CTA and pass

struct CopyList {
    CopyItem item[kCopyItems];
    uint32_t n = 0;
};

// 16-byte stores to the destination; loads as wide as the source's offset to
// them allows (4-byte words shifted together for odd ones: a word that holds
// a byte of the source, but no other, is read).
__global__ void __launch_bounds__(kCopyThreads) k_copy_list(const __grid_constant__ CopyList l) {
    const CopyItem c = l.item[blockIdx.y];
    const uint64_t t = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
    const uint64_t to_line = (16 - ((uintptr_t) c.dst & 15)) & 15;
    const uint64_t head = to_line < c.bytes ? to_line : c.bytes;
    for (uint64_t i = t; i < head; i += stride) c.dst[i] = c.src[i];
    const uint8_t* s = c.src + head;
    uint4* d = reinterpret_cast<uint4*>(c.dst + head);
    const uint64_t nv = (c.bytes - head) >> 4;
    const uint32_t off = (uint32_t) (uintptr_t) s & 15u;
    if (off == 0) {
        const uint4* v = reinterpret_cast<const uint4*>(s);
        uint64_t i = t;
        for (; i + 3 * stride < nv; i += 4 * stride) {
            const uint4 a = v[i], b = v[i + stride], e = v[i + 2 * stride], f = v[i + 3 * stride];
            d[i] = a;
            d[i + stride] = b;
            d[i + 2 * stride] = e;
            d[i + 3 * stride] = f;
        }
        for (; i < nv; i += stride) d[i] = v[i];
    } else {
        const uint32_t sh = 8 * (off & 3u);
        const uint32_t* w = reinterpret_cast<const uint32_t*>(s - (off & 3u));
        for (uint64_t i = t; i < nv; i += stride) {
            const uint32_t* q = w + 4 * i;
            const uint32_t w0 = q[0], w1 = q[1], w2 = q[2], w3 = q[3], w4 = sh ? q[4] : 0u;
            d[i] = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                              __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
        }
    }
    const uint64_t done = head + 16 * nv;
    for (uint64_t i = done + t; i < c.bytes; i += stride) c.dst[i] = c.src[i];
}

inline cudaError_t copy_list(const CopyList& l, cudaStream_t st) {
    if (l.n == 0) return cudaSuccess;
    k_copy_list<<<dim3(kCopyCtas, l.n), kCopyThreads, 0, st>>>(l);
    return cudaGetLastError();
}

}  // namespace mans
