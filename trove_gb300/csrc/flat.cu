// Width-agnostic kernels: the flat vector copy (TRV_PATH_VECTOR), the TMA
// bulk copy (TRV_PATH_BULK), byte-wise gather/scatter of what neither the struct
// kernels nor packed.cu take, and the seeded input generator.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fetch.cuh"
#include "flat.h"

namespace trv {

// ---- seeded input stream (stream_word, flat.h) --------------------------
__global__ void fill_u32_kernel(unsigned* __restrict__ dst, long long nwords, unsigned long long seed) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nwords; k += stride)
        dst[k] = stream_word(seed, (unsigned long long)k);
}

void launch_fill_u32(unsigned* dst, long long nwords, unsigned long long seed, int grid, cudaStream_t st) {
    fill_u32_kernel<<<grid, 256, 0, st>>>(dst, nwords, seed);
}

// idx[i] = stream_bounded(seed, i, bound): n indices uniform in [0, bound).
__global__ void uniform_indices_kernel(int* __restrict__ idx, long long n, unsigned bound, unsigned long long seed) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride)
        idx[k] = (int)stream_bounded(seed, (unsigned long long)k, bound);
}

void launch_uniform_indices(int* idx, long long n, unsigned bound, unsigned long long seed, int grid,
                            cudaStream_t st) {
    uniform_indices_kernel<<<grid, 256, 0, st>>>(idx, n, bound, seed);
}

// Run pattern over n >= 32 indices: output chunk c (32 aligned outputs) is,
// when bit 0 of word 2c is set, a run start + 0..31 with start drawn from
// word 2c + 1 over [0, n - 32]; otherwise 32 independent draws over [0, n)
// from the stream seed ^ 0x5bd1e995 at the output's own position.  Every
// output depends only on its chunk, so one thread per output.
__global__ void run_indices_kernel(int* __restrict__ idx, long long n, unsigned long long seed) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const unsigned long long c = (unsigned long long)k >> 5;
        if (stream_word(seed, 2 * c) & 1u)
            idx[k] = (int)(stream_bounded(seed, 2 * c + 1, (unsigned)(n - 31)) + (unsigned)(k & 31));
        else
            idx[k] = (int)stream_bounded(seed ^ 0x5bd1e995ull, (unsigned long long)k, (unsigned)n);
    }
}

void launch_run_indices(int* idx, long long n, unsigned long long seed, int grid, cudaStream_t st) {
    run_indices_kernel<<<grid, 256, 0, st>>>(idx, n, seed);
}

// ---- flat vector copy ----------------------------------------------------
// Copies nbytes from s to d.  The first `head` bytes bring both pointers to
// V alignment; the aligned middle moves as V vectors, U per thread per pass
// (all U loads issued before the stores); block 0 also copies the head and
// the sub-vector tail byte by byte.
template <typename V, int U>
__global__ void __launch_bounds__(256)
flat_copy_kernel(const unsigned char* __restrict__ s, unsigned char* __restrict__ d, long long nbytes,
                 int head) {
    const long long body = (nbytes - head) / (long long)sizeof(V);
    const V* __restrict__ sv = reinterpret_cast<const V*>(s + head);
    V* __restrict__ dv = reinterpret_cast<V*>(d + head);
    const long long step = (long long)gridDim.x * blockDim.x * U;
    for (long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x; base < body; base += step) {
        V r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = base + (long long)u * blockDim.x;
            if (k < body) r[u] = __ldg(sv + k);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = base + (long long)u * blockDim.x;
            if (k < body) __stcs(dv + k, r[u]);
        }
    }
    if (blockIdx.x == 0) {
        const long long tail_begin = head + body * (long long)sizeof(V);
        if ((long long)threadIdx.x < head) d[threadIdx.x] = s[threadIdx.x];
        const long long t = tail_begin + threadIdx.x;
        if (t < nbytes) d[t] = s[t];
    }
}

template <typename V, int U>
static void launch_flat_v(const unsigned char* s, unsigned char* d, long long nbytes, int head, int grid,
                          cudaStream_t st) {
    flat_copy_kernel<V, U><<<grid, 256, 0, st>>>(s, d, nbytes, head);
}

const void* flat_copy_func(int vec_bytes, int unroll) {
#define TRV_FLAT_FUNC(V, U) \
    if (sizeof(V) == (size_t)vec_bytes && U == unroll) return (const void*)&flat_copy_kernel<V, U>;
    TRV_FLAT_FUNC(uint4, 1) TRV_FLAT_FUNC(uint4, 2) TRV_FLAT_FUNC(uint4, 4) TRV_FLAT_FUNC(uint4, 8)
    TRV_FLAT_FUNC(uint2, 1) TRV_FLAT_FUNC(uint2, 2) TRV_FLAT_FUNC(uint2, 4) TRV_FLAT_FUNC(uint2, 8)
    TRV_FLAT_FUNC(unsigned, 1) TRV_FLAT_FUNC(unsigned, 2) TRV_FLAT_FUNC(unsigned, 4) TRV_FLAT_FUNC(unsigned, 8)
    TRV_FLAT_FUNC(unsigned char, 1) TRV_FLAT_FUNC(unsigned char, 2) TRV_FLAT_FUNC(unsigned char, 4)
    TRV_FLAT_FUNC(unsigned char, 8)
#undef TRV_FLAT_FUNC
    return nullptr;
}

void launch_flat_copy(const void* src, void* dst, long long nbytes, int vec_bytes, int head, int unroll, int grid,
                      cudaStream_t st) {
    const unsigned char* s = static_cast<const unsigned char*>(src);
    unsigned char* d = static_cast<unsigned char*>(dst);
#define TRV_FLAT_CASE(V)                                                  \
    switch (unroll) {                                                     \
        case 1: launch_flat_v<V, 1>(s, d, nbytes, head, grid, st); break; \
        case 2: launch_flat_v<V, 2>(s, d, nbytes, head, grid, st); break; \
        case 4: launch_flat_v<V, 4>(s, d, nbytes, head, grid, st); break; \
        default: launch_flat_v<V, 8>(s, d, nbytes, head, grid, st); break; \
    }
    switch (vec_bytes) {
        case 16: TRV_FLAT_CASE(uint4) break;
        case 8: TRV_FLAT_CASE(uint2) break;
        case 4: TRV_FLAT_CASE(unsigned) break;
        default: TRV_FLAT_CASE(unsigned char) break;
    }
#undef TRV_FLAT_CASE
}

// ---- copy between different alignments -------------------------------------
// Source and destination differ modulo 16: the destination is written as
// aligned 16-byte vectors, each joined from the two aligned source vectors that
// hold its bytes (the second one is the next thread's first: a hit in L1).  WS
// = whole words between the two alignments, `bits` what is left of a word.
// Without it the copy moved by the largest power of two that both sides share,
// down to single bytes: 1 GiB took 444 us by words and 1282 by bytes, against
// 301 us joined, which is what a copy between equal alignments takes.
// The vectors of the body have all of their source inside the array: up to 31
// bytes at either end move by bytes.
template <int WS, int U>
__global__ void __launch_bounds__(256)
shift_copy_kernel(const unsigned char* __restrict__ s, unsigned char* __restrict__ d, long long nbytes, int head,
                  long long body, unsigned bits) {
    const uint4* __restrict__ sv = reinterpret_cast<const uint4*>(s + head - (WS * 4 + bits / 8));
    uint4* __restrict__ dv = reinterpret_cast<uint4*>(d + head);
    const long long step = (long long)gridDim.x * blockDim.x * U;
    for (long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x; base < body; base += step) {
        uint4 a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = base + (long long)u * blockDim.x;
            if (k < body) {
                a[u] = __ldg(sv + k);
                b[u] = __ldg(sv + k + 1);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = base + (long long)u * blockDim.x;
            if (k < body) {
                const unsigned w[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
                __stcs(dv + k, make_uint4(__funnelshift_r(w[WS], w[WS + 1], bits),
                                          __funnelshift_r(w[WS + 1], w[WS + 2], bits),
                                          __funnelshift_r(w[WS + 2], w[WS + 3], bits),
                                          __funnelshift_r(w[WS + 3], w[WS + 4], bits)));
            }
        }
    }
    if (blockIdx.x == 0) {
        const long long t = head + 16 * body + threadIdx.x;
        if ((long long)threadIdx.x < head) d[threadIdx.x] = s[threadIdx.x];
        if (t < nbytes) d[t] = s[t];
    }
}

template <int WS>
static void launch_shift(const unsigned char* s, unsigned char* d, long long nbytes, int head, long long body,
                         unsigned bits, int unroll, int grid, cudaStream_t st) {
    switch (unroll) {
        case 1: shift_copy_kernel<WS, 1><<<grid, 256, 0, st>>>(s, d, nbytes, head, body, bits); break;
        case 2: shift_copy_kernel<WS, 2><<<grid, 256, 0, st>>>(s, d, nbytes, head, body, bits); break;
        default: shift_copy_kernel<WS, 4><<<grid, 256, 0, st>>>(s, d, nbytes, head, body, bits); break;
    }
}

ShiftPlan plan_shift_copy(const void* src, const void* dst, long long nbytes) {
    const long long a = (long long)(reinterpret_cast<uintptr_t>(src) & 15u);
    const long long b = (long long)(reinterpret_cast<uintptr_t>(dst) & 15u);
    ShiftPlan p;
    p.shift = int((a - b) & 15);
    p.head = int((16 - b) & 15);
    if (p.head < p.shift) p.head += 16;  // the first vector's source starts at head - shift
    p.body = (nbytes - p.head + p.shift) / 16 - 1;
    return p;
}

const void* shift_copy_func() { return (const void*)&shift_copy_kernel<1, 4>; }

void launch_shift_copy(const void* src, void* dst, long long nbytes, const ShiftPlan& p, int unroll, int grid,
                       cudaStream_t st) {
    const unsigned char* s = static_cast<const unsigned char*>(src);
    unsigned char* d = static_cast<unsigned char*>(dst);
    const unsigned bits = unsigned(p.shift % 4) * 8;
    switch (p.shift / 4) {
        case 0: return launch_shift<0>(s, d, nbytes, p.head, p.body, bits, unroll, grid, st);
        case 1: return launch_shift<1>(s, d, nbytes, p.head, p.body, bits, unroll, grid, st);
        case 2: return launch_shift<2>(s, d, nbytes, p.head, p.body, bits, unroll, grid, st);
        default: return launch_shift<3>(s, d, nbytes, p.head, p.body, bits, unroll, grid, st);
    }
}

// ---- byte-wise gather / scatter: rows too narrow or few for packed.cu -------
__global__ void gather_bytes_kernel(const unsigned char* __restrict__ s, long long src_n,
                                    const int* __restrict__ idx, unsigned char* __restrict__ d, long long n,
                                    unsigned width) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int j = idx[i];
        if (j < 0 || (long long)j >= src_n) continue;
        const unsigned char* p = s + (long long)j * width;
        unsigned char* q = d + i * (long long)width;
        for (unsigned b = 0; b < width; ++b) q[b] = p[b];
    }
}

__global__ void scatter_bytes_kernel(const unsigned char* __restrict__ s, const int* __restrict__ idx,
                                     unsigned char* __restrict__ d, long long dst_n, long long n,
                                     unsigned width, bool sampled) {
    if (sampled && !IndexSample(idx, n, int(threadIdx.x & 31u)).rows_adjoin(int(width))) return;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int j = idx[i];
        if (j < 0 || (long long)j >= dst_n) continue;
        const unsigned char* p = s + i * (long long)width;
        unsigned char* q = d + (long long)j * width;
        for (unsigned b = 0; b < width; ++b) q[b] = p[b];
    }
}

void launch_gather_bytes(const void* src, long long src_n, const int* idx, void* dst, long long n,
                         unsigned width, int grid, cudaStream_t st) {
    gather_bytes_kernel<<<grid, 256, 0, st>>>(static_cast<const unsigned char*>(src), src_n, idx,
                                              static_cast<unsigned char*>(dst), n, width);
}

void launch_scatter_bytes(const void* src, const int* idx, void* dst, long long dst_n, long long n,
                          unsigned width, int grid, bool sampled, cudaStream_t st) {
    scatter_bytes_kernel<<<grid, 256, 0, st>>>(static_cast<const unsigned char*>(src), idx,
                                               static_cast<unsigned char*>(dst), dst_n, n, width, sampled);
}

}  // namespace trv
