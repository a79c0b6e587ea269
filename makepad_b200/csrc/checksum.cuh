// FNV-1a 64 of a buffer in device memory, the same value as the byte-by-byte loop on the host.
//
//   h = (h ^ byte) * p   (mod 2^64, p = 2^40 + 0x1B3)
//
// The loop is one chain of multiplications per byte: about 1 ns a byte on a host core, 31 ms for the 28 MB of a
// 12288 x 4096 Q4 weight, whose copy to the GPU takes 0.6 ms.  Two facts cut the chain:
//   * the lowest byte of h depends on the lowest byte alone: l' = (l ^ byte) * 0xB3 mod 256.  A chunk of bytes is a map
//     of l; as 0xB3 is odd, starts that differ in bit 7 alone stay apart by bit 7 alone, so 128 starts give the map;
//   * with l known the rest is linear: h ^ byte = h + ((l ^ byte) - l), so over a chunk of n bytes
//     h_end = (h - l) * p^n + F, with F the plain loop started from l.
// fnv_map_kernel forms the maps (one warp per chunk, four starts per lane), fnv_group_kernel composes them by groups,
// fnv_walk_kernel follows the one true l through the groups, fnv_sum_kernel runs the plain loop of each chunk from its
// true start and folds a group; the host folds the groups.  Bound by the integer pipe of the map kernel (about six
// instructions per byte and warp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include "launch.h"

namespace mpq {

constexpr int FNV_CHUNK = 4096;               // bytes per warp of the map kernel: 7000 warps for 28 MB, three quarters of what the SMs hold
constexpr int FNV_GROUP = 64;                 // chunks per group: its maps are 8 KB of shared memory
constexpr uint64_t FNV_PRIME = 0x100000001B3ull;

// map[c][s] = low byte after chunk c from start s, s < 128 (start s + 128 gives map ^ 0x80).  Chunks past the end: identity.
__global__ void __launch_bounds__(256) fnv_map_kernel(const uint8_t* __restrict__ buf, int64_t bytes, int64_t chunks, uint32_t* __restrict__ map)
{
    const int64_t c = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (c >= chunks) return;
    const int64_t at = c * FNV_CHUNK;
    const int n = (int)max((int64_t)0, min((int64_t)FNV_CHUNK, bytes - at));
    // starts 4 lane .. 4 lane + 3: the even ones in the halves of e, the odd ones in the halves of o
    uint32_t e = (uint32_t)(4 * lane) | (uint32_t)(4 * lane + 2) << 16, o = e + 0x00010001u;
    int i = 0;
    for (; i + 16 <= n; i += 16) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(buf + at + i));          // the whole warp reads the same 16 bytes
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const uint32_t b = __byte_perm(w[k >> 2], 0u, 0x4040u | (uint32_t)((k & 3) * 0x0101));      // the byte in both halves
            e = ((e & 0x00FF00FFu) ^ b) * 0xB3u;
            o = ((o & 0x00FF00FFu) ^ b) * 0xB3u;
        }
    }
    for (; i < n; ++i) {
        const uint32_t b = (uint32_t)buf[at + i] * 0x00010001u;
        e = ((e & 0x00FF00FFu) ^ b) * 0xB3u;
        o = ((o & 0x00FF00FFu) ^ b) * 0xB3u;
    }
    map[c * 32 + lane] = (e & 0x00FF00FFu) | (o & 0x00FF00FFu) << 8;
}

__device__ __forceinline__ uint32_t fnv_step(const uint8_t* map, uint32_t l) { return map[l & 127u] ^ (l & 128u); }

// gmap[g] = the composed map of the group's chunks.  128 threads, one per start.
__global__ void __launch_bounds__(128) fnv_group_kernel(const uint32_t* __restrict__ map, int64_t chunks, uint8_t* __restrict__ gmap)
{
    __shared__ uint32_t s_map[FNV_GROUP * 32];
    const int64_t c0 = (int64_t)blockIdx.x * FNV_GROUP;
    const int n = (int)min((int64_t)FNV_GROUP, chunks - c0);
    for (int i = threadIdx.x; i < n * 32; i += 128) s_map[i] = map[c0 * 32 + i];
    __syncthreads();
    uint32_t l = threadIdx.x;
    for (int k = 0; k < n; ++k) l = fnv_step(reinterpret_cast<const uint8_t*>(s_map + k * 32), l);
    gmap[(int64_t)blockIdx.x * 128 + threadIdx.x] = (uint8_t)l;
}

// start[g] = the low byte in front of group g.  One block; 64 groups' maps at a time in shared memory.
__global__ void __launch_bounds__(256) fnv_walk_kernel(const uint32_t* __restrict__ gmap, int64_t groups, uint32_t l, uint8_t* __restrict__ start)
{
    __shared__ uint32_t s_map[64 * 32];
    for (int64_t g0 = 0; g0 < groups; g0 += 64) {
        const int n = (int)min((int64_t)64, groups - g0);
        for (int i = threadIdx.x; i < n * 32; i += 256) s_map[i] = gmap[g0 * 32 + i];
        __syncthreads();
        if (threadIdx.x == 0)
            for (int k = 0; k < n; ++k) {
                start[g0 + k] = (uint8_t)l;
                l = fnv_step(reinterpret_cast<const uint8_t*>(s_map + k * 32), l);
            }
        __syncthreads();
    }
}

// sum[g] = what the plain loop makes of the group's bytes when started from h = start[g]
__global__ void __launch_bounds__(FNV_GROUP) fnv_sum_kernel(const uint8_t* __restrict__ buf, int64_t bytes, const uint32_t* __restrict__ map, int64_t chunks,
                                                            const uint8_t* __restrict__ start, uint64_t* __restrict__ sum)
{
    __shared__ uint32_t s_map[FNV_GROUP * 32];
    __shared__ uint64_t s_f[FNV_GROUP];
    __shared__ uint8_t s_l[FNV_GROUP];
    const int64_t c0 = (int64_t)blockIdx.x * FNV_GROUP;
    const int n = (int)min((int64_t)FNV_GROUP, chunks - c0), t = threadIdx.x;
    for (int i = t; i < n * 32; i += FNV_GROUP) s_map[i] = map[c0 * 32 + i];
    __syncthreads();
    if (t == 0) {
        uint32_t l = start[blockIdx.x];
        for (int k = 0; k < n; ++k) {
            s_l[k] = (uint8_t)l;
            l = fnv_step(reinterpret_cast<const uint8_t*>(s_map + k * 32), l);
        }
    }
    __syncthreads();
    uint64_t pn = 1;                                       // p^(bytes of this thread's chunk)
    if (t < n) {
        const int64_t at = (c0 + t) * FNV_CHUNK;
        const int len = (int)min((int64_t)FNV_CHUNK, bytes - at);
        uint64_t h = s_l[t];
        int i = 0;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (len >= 16) v = __ldg(reinterpret_cast<const uint4*>(buf + at));
        for (; i + 16 <= len; i += 16) {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            if (i + 32 <= len) v = __ldg(reinterpret_cast<const uint4*>(buf + at + i + 16));      // ahead of the chain
#pragma unroll
            for (int k = 0; k < 16; ++k) h = (h ^ ((w[k >> 2] >> (8 * (k & 3))) & 0xFFu)) * FNV_PRIME;
        }
        for (; i < len; ++i) h = (h ^ buf[at + i]) * FNV_PRIME;
        s_f[t] = h;
        uint64_t sq = FNV_PRIME;
        for (int b = len; b; b >>= 1, sq *= sq)
            if (b & 1) pn *= sq;
    }
    __shared__ uint64_t s_p[FNV_GROUP];
    s_p[t] = pn;
    __syncthreads();
    if (t == 0) {
        uint64_t h = s_l[0];
        for (int k = 0; k < n; ++k) h = (h - s_l[k]) * s_p[k] + s_f[k];
        sum[blockIdx.x] = h;
    }
}

// device memory fnv1a64_device wants: 1/32 of the buffer
inline size_t fnv1a64_scratch_bytes(int64_t bytes)
{
    if (bytes <= 0) return 0;
    const int64_t chunks = (bytes + FNV_CHUNK - 1) / FNV_CHUNK, groups = (chunks + FNV_GROUP - 1) / FNV_GROUP;
    return ((size_t)groups * 8 + 127) / 128 * 128 + (size_t)groups * 129 + (size_t)chunks * 128;
}

// *h = FNV-1a 64 of buf[0, bytes) continued from *h.  buf: 16-byte aligned device memory; scratch: fnv1a64_scratch_bytes of
// device memory.  Waits for the stream; *h is unchanged on an error.
inline cudaError_t fnv1a64_device(const void* buf, int64_t bytes, uint64_t* h, uint8_t* scratch, cudaStream_t s)
{
    if (bytes <= 0) return cudaSuccess;
    const int64_t chunks = (bytes + FNV_CHUNK - 1) / FNV_CHUNK, groups = (chunks + FNV_GROUP - 1) / FNV_GROUP;
    // sums (8 B per group) | group maps (128 B) | chunk maps (128 B) | group starts (1 B)
    const size_t off_gmap = ((size_t)groups * 8 + 127) / 128 * 128, off_map = off_gmap + (size_t)groups * 128, off_start = off_map + (size_t)chunks * 128;
    const uint8_t* b = static_cast<const uint8_t*>(buf);
    uint64_t* sum = reinterpret_cast<uint64_t*>(scratch);
    uint32_t* map = reinterpret_cast<uint32_t*>(scratch + off_map);
    cudaError_t e = launch(fnv_map_kernel, (unsigned)((chunks + 7) / 8), 256, s, b, bytes, chunks, map);
    if (e == cudaSuccess) e = launch(fnv_group_kernel, (unsigned)groups, 128, s, map, chunks, scratch + off_gmap);
    if (e == cudaSuccess) e = launch(fnv_walk_kernel, 1, 256, s, reinterpret_cast<const uint32_t*>(scratch + off_gmap), groups, (uint32_t)(*h & 0xFFu), scratch + off_start);
    if (e == cudaSuccess) e = launch(fnv_sum_kernel, (unsigned)groups, FNV_GROUP, s, b, bytes, map, chunks, scratch + off_start, sum);
    uint64_t* host = static_cast<uint64_t*>(malloc((size_t)groups * 9));
    uint8_t* host_l = host ? reinterpret_cast<uint8_t*>(host + groups) : nullptr;
    if (!host && e == cudaSuccess) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, sum, (size_t)groups * 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(host_l, scratch + off_start, (size_t)groups, cudaMemcpyDeviceToHost, s);
    const cudaError_t done = cudaStreamSynchronize(s);                  // (on an error too: nobody still uses the scratch)
    if (e == cudaSuccess) e = done;
    for (int64_t g = 0; e == cudaSuccess && g < groups; ++g) {
        uint64_t pn = 1, sq = FNV_PRIME;
        for (int64_t n = bytes - g * FNV_CHUNK * FNV_GROUP < FNV_CHUNK * FNV_GROUP ? bytes - g * FNV_CHUNK * FNV_GROUP : FNV_CHUNK * FNV_GROUP; n; n >>= 1, sq *= sq)
            if (n & 1) pn *= sq;
        *h = (*h - host_l[g]) * pn + host[g];
    }
    free(host);
    return e;
}

}  // namespace mpq
