// sm_103a decode kernels for OpenZL's numeric codec graph.
//
// All work here is integer and HBM/latency bound: no tensor cores. Each
// kernel takes a task array plus, for data-parallel kinds, a tile list; the
// host planner (dec_plan.cpp) builds both. Kernels never trap: malformed
// input sets the batch status word (first error wins) and the kernel moves
// on. Every spin-wait is bounded.
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include <cuda_runtime.h>

#include "dec_tasks.h"
#include "dec_exec.h"
#include "fse_shape.h"
#include "huf_split.h"
#include "stream_ring.cuh"

namespace ozl {

// ---------------------------------------------------------------------------
// helpers

__device__ __forceinline__ void reportError(uint32_t* status, uint32_t code)
{
    atomicCAS(status, 0u, code);
}

// 8 bytes from any address inside a buffer that this library allocated with
// at least 16 bytes of slack on both sides of every stream it reads this way.
__device__ __forceinline__ uint64_t ld64Any(const uint8_t* p)
{
    uintptr_t const a = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(7);
    unsigned const s = unsigned(reinterpret_cast<uintptr_t>(p) - a) * 8u;
    uint64_t const lo = *reinterpret_cast<const uint64_t*>(a);
    if (s == 0) return lo;
    uint64_t const hi = *reinterpret_cast<const uint64_t*>(a + 8);
    return (lo >> s) | (hi << (64u - s));
}

__device__ __forceinline__ uint64_t ldElem(const uint8_t* p, uint32_t w)
{
    switch (w) {
        case 1: return *p;
        case 2: return (reinterpret_cast<uintptr_t>(p) & 1) ? (uint64_t(p[0]) | (uint64_t(p[1]) << 8))
                                                           : *reinterpret_cast<const uint16_t*>(p);
        case 4:
            if (!(reinterpret_cast<uintptr_t>(p) & 3)) return *reinterpret_cast<const uint32_t*>(p);
            return uint64_t(p[0]) | (uint64_t(p[1]) << 8) | (uint64_t(p[2]) << 16) | (uint64_t(p[3]) << 24);
        default:
            if (!(reinterpret_cast<uintptr_t>(p) & 7)) return *reinterpret_cast<const uint64_t*>(p);
            {
                uint64_t v = 0;
                for (int b = 0; b < 8; b++) v |= uint64_t(p[b]) << (8 * b);
                return v;
            }
    }
}

__device__ __forceinline__ void stElem(uint8_t* p, uint64_t v, uint32_t w)
{
    switch (w) {
        case 1: *p = uint8_t(v); break;
        case 2:
            if (!(reinterpret_cast<uintptr_t>(p) & 1)) *reinterpret_cast<uint16_t*>(p) = uint16_t(v);
            else { p[0] = uint8_t(v); p[1] = uint8_t(v >> 8); }
            break;
        case 4:
            if (!(reinterpret_cast<uintptr_t>(p) & 3)) *reinterpret_cast<uint32_t*>(p) = uint32_t(v);
            else for (int b = 0; b < 4; b++) p[b] = uint8_t(v >> (8 * b));
            break;
        default:
            if (!(reinterpret_cast<uintptr_t>(p) & 7)) *reinterpret_cast<uint64_t*>(p) = v;
            else for (int b = 0; b < 8; b++) p[b] = uint8_t(v >> (8 * b));
    }
}

__device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

__device__ __forceinline__ uint64_t widthMask(uint32_t w)
{
    return w >= 8 ? ~0ull : ((1ull << (8 * w)) - 1);
}

// ---------------------------------------------------------------------------
// copy / constant: tiles of kTileBytes output bytes

// Copies one tile: bytes up to the destination's 16-byte boundary, then
// 16-byte stores, each from the two aligned 16-byte source blocks that hold
// its bytes (both blocks hold bytes of the source, so nothing outside the
// source's blocks is read), then the tail bytes.
__global__ void __launch_bounds__(256) kCopy(const CopyTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    CopyTask const t = tasks[tr.task];
    uint64_t const b0 = uint64_t(tr.tile) * kTileBytes;
    uint64_t const b1 = min(t.bytes, b0 + kTileBytes);
    uint64_t const head = min(b1 - b0, uint64_t((16 - (reinterpret_cast<uintptr_t>(t.dst + b0) & 15)) & 15));
    for (uint64_t i = b0 + threadIdx.x; i < b0 + head; i += blockDim.x) t.dst[i] = t.src[i];
    uint64_t const a0 = b0 + head;
    uint64_t const nv = (b1 - a0) / 16;
    uint4* const d = reinterpret_cast<uint4*>(t.dst + a0);
    uintptr_t const sa = reinterpret_cast<uintptr_t>(t.src + a0);
    uint32_t const off = uint32_t(sa & 15);
    const uint4* const s = reinterpret_cast<const uint4*>(sa - off);
    if (off == 0) {
#pragma unroll 4
        for (uint64_t i = threadIdx.x; i < nv; i += blockDim.x) d[i] = __ldg(s + i);
    } else {
        uint32_t const q = off >> 2, r = (off & 3) * 8;
#pragma unroll 4
        for (uint64_t i = threadIdx.x; i < nv; i += blockDim.x) d[i] = shiftCombine(__ldg(s + i), __ldg(s + i + 1), q, r);
    }
    for (uint64_t i = a0 + nv * 16 + threadIdx.x; i < b1; i += blockDim.x) t.dst[i] = t.src[i];
}

__global__ void kConst(const ConstTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    ConstTask const t = tasks[tr.task];
    uint64_t const total = t.n * t.w;
    uint64_t const b0 = uint64_t(tr.tile) * kTileBytes;
    uint64_t const b1 = min(total, b0 + kTileBytes);
    if (t.w == 1) {
        uint8_t const v = t.value[0];
        uint32_t const v4 = v * 0x01010101u;
        // head bytes up to 16-byte alignment, then 16-byte stores
        uint64_t a = b0;
        uintptr_t const base = reinterpret_cast<uintptr_t>(t.out);
        uint64_t const alignStart = min(b1, (((base + b0 + 15) & ~uintptr_t(15)) - base));
        for (uint64_t i = a + threadIdx.x; i < alignStart; i += blockDim.x) t.out[i] = v;
        a = alignStart;
        uint64_t const nv = (b1 - a) / 16;
        uint4 const q = make_uint4(v4, v4, v4, v4);
        uint4* d = reinterpret_cast<uint4*>(t.out + a);
        for (uint64_t i = threadIdx.x; i < nv; i += blockDim.x) d[i] = q;
        for (uint64_t i = a + nv * 16 + threadIdx.x; i < b1; i += blockDim.x) t.out[i] = v;
    } else {
        for (uint64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) t.out[i] = t.value[i % t.w];
    }
}

// XXH3's published secret and primes (the checksum kernels below and the
// content-checksum block sums fused into the numeric pipeline).
struct XxhSecret {
    uint8_t b[192];
};
constexpr XxhSecret kXxhSecretBytes = { {
    0xb8, 0xfe, 0x6c, 0x39, 0x23, 0xa4, 0x4b, 0xbe, 0x7c, 0x01, 0x81, 0x2c, 0xf7, 0x21, 0xad, 0x1c,
    0xde, 0xd4, 0x6d, 0xe9, 0x83, 0x90, 0x97, 0xdb, 0x72, 0x40, 0xa4, 0xa4, 0xb7, 0xb3, 0x67, 0x1f,
    0xcb, 0x79, 0xe6, 0x4e, 0xcc, 0xc0, 0xe5, 0x78, 0x82, 0x5a, 0xd0, 0x7d, 0xcc, 0xff, 0x72, 0x21,
    0xb8, 0x08, 0x46, 0x74, 0xf7, 0x43, 0x24, 0x8e, 0xe0, 0x35, 0x90, 0xe6, 0x81, 0x3a, 0x26, 0x4c,
    0x3c, 0x28, 0x52, 0xbb, 0x91, 0xc3, 0x00, 0xcb, 0x88, 0xd0, 0x65, 0x8b, 0x1b, 0x53, 0x2e, 0xa3,
    0x71, 0x64, 0x48, 0x97, 0xa2, 0x0d, 0xf9, 0x4e, 0x38, 0x19, 0xef, 0x46, 0xa9, 0xde, 0xac, 0xd8,
    0xa8, 0xfa, 0x76, 0x3f, 0xe3, 0x9c, 0x34, 0x3f, 0xf9, 0xdc, 0xbb, 0xc7, 0xc7, 0x0b, 0x4f, 0x1d,
    0x8a, 0x51, 0xe0, 0x4b, 0xcd, 0xb4, 0x59, 0x31, 0xc8, 0x9f, 0x7e, 0xc9, 0xd9, 0x78, 0x73, 0x64,
    0xea, 0xc5, 0xac, 0x83, 0x34, 0xd3, 0xeb, 0xc3, 0xc5, 0x81, 0xa0, 0xff, 0xfa, 0x13, 0x63, 0xeb,
    0x17, 0x0d, 0xdd, 0x51, 0xb7, 0xf0, 0xda, 0x49, 0xd3, 0x16, 0x55, 0x26, 0x29, 0xd4, 0x68, 0x9e,
    0x2b, 0x16, 0xbe, 0x58, 0x7d, 0x47, 0xa1, 0xfc, 0x8f, 0xf8, 0xb8, 0xd1, 0x7a, 0xd0, 0x31, 0xce,
    0x45, 0xcb, 0x3a, 0x8f, 0x95, 0x16, 0x04, 0x28, 0xaf, 0xd7, 0xfb, 0xca, 0xbb, 0x4b, 0x40, 0x7e,
} };
__constant__ XxhSecret kXxhSecret = kXxhSecretBytes;

#define XP32_1 0x9E3779B1u
#define XP32_2 0x85EBCA77u
#define XP32_3 0xC2B2AE3Du
#define XP64_1 0x9E3779B185EBCA87ull
#define XP64_2 0xC2B2AE3D27D4EB4Full
#define XP64_3 0x165667B19E3779F9ull
#define XP64_4 0x85EBCA77C2B2AE63ull
#define XP64_5 0x27D4EB2F165667C5ull
#define XPMX1 0x165667919E3779F9ull
#define XPMX2 0x9FB21C651E98DF25ull

// The secret as the 64-bit words that the checksum kernels index per lane:
// at byte offsets 0, 8, ..., 184; at 121 + 8 i (the final stripe); at
// 11 + 8 k (the merge).
struct XxhWords {
    uint64_t w8[24], last[8], merge[8];
};
constexpr XxhWords xxhWords()
{
    XxhWords x{};
    for (int k = 0; k < 24; k++)
        for (int b = 0; b < 8; b++) x.w8[k] |= uint64_t(kXxhSecretBytes.b[8 * k + b]) << (8 * b);
    for (int k = 0; k < 8; k++)
        for (int b = 0; b < 8; b++) {
            x.last[k] |= uint64_t(kXxhSecretBytes.b[121 + 8 * k + b]) << (8 * b);
            x.merge[k] |= uint64_t(kXxhSecretBytes.b[11 + 8 * k + b]) << (8 * b);
        }
    return x;
}
__constant__ XxhWords kXxhWords = xxhWords();

__device__ __forceinline__ uint64_t secret64(int off)
{
    uint64_t v = 0;
    for (int b = 0; b < 8; b++) v |= uint64_t(kXxhSecret.b[off + b]) << (8 * b);
    return v;
}
__device__ __forceinline__ uint32_t secret32(int off)
{
    return uint32_t(kXxhSecret.b[off]) | (uint32_t(kXxhSecret.b[off + 1]) << 8) | (uint32_t(kXxhSecret.b[off + 2]) << 16)
            | (uint32_t(kXxhSecret.b[off + 3]) << 24);
}
// ---------------------------------------------------------------------------
// Fused numeric pipeline: source (plain elements, byte planes or LSB-first
// bit-packed fields) -> optional zigzag -> optional delta -> output elements.
//
// Delta decoding is an exclusive prefix sum: out[i] = first + sum(src[0..i))
// modulo 2^(8w), src holding n-1 elements (decode_delta_kernel.c:232). A tile
// is kNumTileBytes of output (kNumTileBytes / w elements); thread t owns the
// 64 output bytes 64t..64t+63 of its tile and holds them as 16 words of
// little-endian elements, so every width keeps 64 bytes of loads in flight
// per thread. Byte and 16-bit elements are zigzagged and scanned four or two
// to a word with SIMD byte/halfword adds. Plain sources and planes are read
// with 16- or 8-byte loads (shifted into place when misaligned); bit-packed
// sources are staged through shared memory with coalesced loads, one pad
// word after every 32 so that the threads' field reads spread over the
// banks. Delta tasks take three launches, none of which waits on another
// CTA: the sum of every tile's sources, an exclusive scan of those sums per
// task (one CTA per task), then the final pass that scans inside the tile
// and adds the tile's prefix. (One CTA running a whole task, tile after tile,
// reads the sources once, but a tile then takes 2.5 us of a serial task: 4.8
// ms for 4096 mixed frames against 1.8 in three passes.)
constexpr int kNPThreads = 256;
constexpr int kNW = 16;                                   // words per thread
constexpr uint32_t kNPBytes = 4 * kNW;                    // 64 output bytes per thread
static_assert(kNPBytes * kNPThreads == kNumTileBytes, "tile = threads x bytes per thread");
constexpr uint32_t kNPStageWords = kNumTileBytes / 4 + 8; // the fields of a tile plus partial blocks at both ends
constexpr uint32_t kNPStagePadded = kNPStageWords + kNPStageWords / 32 + 1;

__device__ __forceinline__ uint32_t npPad(uint32_t q) { return q + (q >> 5); }

// NQ 16-byte blocks from p (any alignment; every block read holds bytes of
// the range) into w[0 .. 4 NQ)
template <int NQ>
__device__ __forceinline__ void npLdq(const uint8_t* p, uint32_t* w)
{
    uintptr_t const a = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15);
    uint32_t const off = uint32_t(reinterpret_cast<uintptr_t>(p) - a);
    const uint4* const s = reinterpret_cast<const uint4*>(a);
    if (off == 0) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            uint4 const u = __ldg(s + q);
            w[4 * q] = u.x; w[4 * q + 1] = u.y; w[4 * q + 2] = u.z; w[4 * q + 3] = u.w;
        }
    } else {
        uint32_t const qq = off >> 2, r = (off & 3) * 8;
        uint4 prev = __ldg(s);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            uint4 const nxt = __ldg(s + q + 1);
            uint4 const u = shiftCombine(prev, nxt, qq, r);
            w[4 * q] = u.x; w[4 * q + 1] = u.y; w[4 * q + 2] = u.z; w[4 * q + 3] = u.w;
            prev = nxt;
        }
    }
}

// 8 bytes from p (any alignment) into w[0], w[1], from the aligned 8-byte
// words that hold them
__device__ __forceinline__ void npLd8(const uint8_t* p, uint32_t* w)
{
    uintptr_t const a = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(7);
    uint32_t const off = uint32_t(reinterpret_cast<uintptr_t>(p) - a);
    const uint2* const s = reinterpret_cast<const uint2*>(a);
    uint2 const u0 = __ldg(s);
    if (off == 0) {
        w[0] = u0.x;
        w[1] = u0.y;
    } else {
        uint2 const u1 = __ldg(s + 1);
        uint32_t const r = (off & 3) * 8;
        uint32_t const x0 = off < 4 ? u0.x : u0.y, x1 = off < 4 ? u0.y : u1.x, x2 = off < 4 ? u1.x : u1.y;
        w[0] = __funnelshift_r(x0, x1, r);
        w[1] = __funnelshift_r(x1, x2, r);
    }
}

// Loads the thread's source elements j0 .. j0 + 64/W (those below nSrc; the
// rest read as 0) as 16 words of little-endian elements. `stage` holds the
// tile's bit-packed words (padded) for SRC_BITPACK, bit `sbit` being the
// first field of the tile.
template <int W, int MODE>
__device__ __forceinline__ void npLoad(const NumPipeTask& t, uint64_t j0, uint64_t nSrc, const uint32_t* stage,
                                       uint32_t sbit, uint32_t tileRel, uint32_t (&w)[kNW])
{
    constexpr uint32_t E = kNPBytes / W;
    uint32_t const cs = j0 < nSrc ? uint32_t(umin64(E, nSrc - j0)) : 0u;
    if constexpr (MODE == SRC_PLAIN) {
        if (cs == E) {
            npLdq<kNW / 4>(t.src + j0 * W, w);
        } else {
            const uint8_t* const p = t.src + j0 * W;
#pragma unroll
            for (int m = 0; m < kNW; m++) {
                uint32_t x = 0;
#pragma unroll
                for (int y = 0; y < 4; y++)
                    if (uint32_t(4 * m + y) < cs * W) x |= uint32_t(p[4 * m + y]) << (8 * y);
                w[m] = x;
            }
        }
    } else if constexpr (MODE == SRC_PLANES) {
        constexpr int PW = int(E / 4); // words per plane
        uint32_t raw[kNW];
        if (cs == E) {
#pragma unroll
            for (int b = 0; b < W; b++) {
                if constexpr (PW >= 4) npLdq<PW / 4>(t.planes[b] + j0, raw + PW * b);
                else npLd8(t.planes[b] + j0, raw + PW * b);
            }
        } else {
#pragma unroll
            for (int b = 0; b < W; b++) {
                const uint8_t* const pl = t.planes[b] + j0;
#pragma unroll
                for (int m = 0; m < PW; m++) {
                    uint32_t x = 0;
#pragma unroll
                    for (int y = 0; y < 4; y++)
                        if (uint32_t(4 * m + y) < cs) x |= uint32_t(pl[4 * m + y]) << (8 * y);
                    raw[PW * b + m] = x;
                }
            }
        }
        if constexpr (W == 1) {
#pragma unroll
            for (int m = 0; m < kNW; m++) w[m] = raw[m];
        } else if constexpr (W == 2) {
#pragma unroll
            for (int m = 0; m < kNW; m++) w[m] = __byte_perm(raw[m >> 1], raw[PW + (m >> 1)], (m & 1) ? 0x7362 : 0x5140);
        } else {
            // 4x4 byte transposes of planes 0-3 (and 4-7 for the high words)
#pragma unroll
            for (int h = 0; h < W / 4; h++) {
#pragma unroll
                for (int g = 0; g < PW; g++) {
                    uint32_t const* const pl = raw + PW * (4 * h);
                    uint32_t const p0 = pl[g], p1 = pl[PW + g], p2 = pl[2 * PW + g], p3 = pl[3 * PW + g];
                    uint32_t const t0 = __byte_perm(p0, p1, 0x5140), t1 = __byte_perm(p0, p1, 0x7362);
                    uint32_t const t2 = __byte_perm(p2, p3, 0x5140), t3 = __byte_perm(p2, p3, 0x7362);
                    uint32_t const e[4] = { __byte_perm(t0, t2, 0x5410), __byte_perm(t0, t2, 0x7632),
                                            __byte_perm(t1, t3, 0x5410), __byte_perm(t1, t3, 0x7632) };
#pragma unroll
                    for (int j = 0; j < 4; j++) w[(W / 4) * (4 * g + j) + h] = e[j];
                }
            }
        }
    } else {
        // LSB-first fields of nbBits (1..8W) from the staged words
        uint32_t const nb = t.nbBits;
#pragma unroll
        for (int m = 0; m < kNW; m++) w[m] = 0;
#pragma unroll
        for (uint32_t k = 0; k < E; k++) {
            uint64_t x = 0;
            if (k < cs) {
                uint32_t const bit = sbit + (tileRel + k) * nb;
                uint32_t const q = bit >> 5, r = bit & 31;
                uint32_t const w0 = stage[npPad(q)];
                uint32_t const w1 = (r + nb > 32) ? stage[npPad(q + 1)] : 0u;
                x = __funnelshift_r(w0, w1, r);
                if (r + nb > 64) x |= uint64_t(__funnelshift_r(w1, stage[npPad(q + 2)], r)) << 32;
                else if (nb > 32) x |= uint64_t(w1 >> r) << 32;
                if (nb < 64) x &= (1ull << nb) - 1;
            }
            if constexpr (W == 1) w[k >> 2] |= uint32_t(x) << (8 * (k & 3));
            else if constexpr (W == 2) w[k >> 1] |= uint32_t(x) << (16 * (k & 1));
            else if constexpr (W == 4) w[k] = uint32_t(x);
            else {
                w[2 * k] = uint32_t(x);
                w[2 * k + 1] = uint32_t(x >> 32);
            }
        }
    }
}

template <int W>
__device__ __forceinline__ void npZigzag(uint32_t (&w)[kNW])
{
#pragma unroll
    for (int m = 0; m < kNW; m++) {
        uint32_t const x = w[m];
        if constexpr (W == 1) w[m] = ((x >> 1) & 0x7f7f7f7fu) ^ ((x & 0x01010101u) * 0xffu);
        else if constexpr (W == 2) w[m] = ((x >> 1) & 0x7fff7fffu) ^ ((x & 0x00010001u) * 0xffffu);
        else if constexpr (W == 4) w[m] = (x >> 1) ^ (0u - (x & 1u));
    }
    if constexpr (W == 8) {
#pragma unroll
        for (int m = 0; m < kNW; m += 2) {
            uint64_t const v = uint64_t(w[m]) | (uint64_t(w[m + 1]) << 32);
            uint64_t const z = (v >> 1) ^ (0ull - (v & 1ull));
            w[m] = uint32_t(z);
            w[m + 1] = uint32_t(z >> 32);
        }
    }
}

// sum of the thread's elements (modulo 2^(8W) after masking)
template <int W>
__device__ __forceinline__ uint64_t npSum(const uint32_t (&w)[kNW])
{
    if constexpr (W == 1) {
        uint32_t acc = 0;
#pragma unroll
        for (int m = 0; m < kNW; m++) acc = __vadd4(acc, w[m]);
        return (acc & 0xff) + ((acc >> 8) & 0xff) + ((acc >> 16) & 0xff) + (acc >> 24);
    } else if constexpr (W == 2) {
        uint32_t acc = 0;
#pragma unroll
        for (int m = 0; m < kNW; m++) acc = __vadd2(acc, w[m]);
        return (acc & 0xffff) + (acc >> 16);
    } else if constexpr (W == 4) {
        uint32_t acc = 0;
#pragma unroll
        for (int m = 0; m < kNW; m++) acc += w[m];
        return acc;
    } else {
        uint64_t acc = 0;
#pragma unroll
        for (int m = 0; m < kNW; m += 2) acc += uint64_t(w[m]) | (uint64_t(w[m + 1]) << 32);
        return acc;
    }
}

// exclusive scan of the thread's elements in place
template <int W>
__device__ __forceinline__ void npScan(uint32_t (&w)[kNW])
{
    if constexpr (W == 1) {
        uint32_t c = 0;
#pragma unroll
        for (int m = 0; m < kNW; m++) {
            uint32_t p = __vadd4(w[m], w[m] << 8);
            p = __vadd4(p, p << 16);
            w[m] = __vadd4(p << 8, c * 0x01010101u);
            c = (c + (p >> 24)) & 0xffu;
        }
    } else if constexpr (W == 2) {
        uint32_t c = 0;
#pragma unroll
        for (int m = 0; m < kNW; m++) {
            uint32_t const p = __vadd2(w[m], w[m] << 16);
            w[m] = __vadd2(p << 16, c * 0x00010001u);
            c = (c + (p >> 16)) & 0xffffu;
        }
    } else if constexpr (W == 4) {
        uint32_t c = 0;
#pragma unroll
        for (int m = 0; m < kNW; m++) {
            uint32_t const x = w[m];
            w[m] = c;
            c += x;
        }
    } else {
        uint64_t c = 0;
#pragma unroll
        for (int m = 0; m < kNW; m += 2) {
            uint64_t const x = uint64_t(w[m]) | (uint64_t(w[m + 1]) << 32);
            w[m] = uint32_t(c);
            w[m + 1] = uint32_t(c >> 32);
            c += x;
        }
    }
}

// adds `add` (modulo 2^(8W)) to every element
template <int W>
__device__ __forceinline__ void npAdd(uint32_t (&w)[kNW], uint64_t add)
{
    if constexpr (W == 1) {
        uint32_t const a = uint32_t(add & 0xff) * 0x01010101u;
#pragma unroll
        for (int m = 0; m < kNW; m++) w[m] = __vadd4(w[m], a);
    } else if constexpr (W == 2) {
        uint32_t const a = uint32_t(add & 0xffff) * 0x00010001u;
#pragma unroll
        for (int m = 0; m < kNW; m++) w[m] = __vadd2(w[m], a);
    } else if constexpr (W == 4) {
#pragma unroll
        for (int m = 0; m < kNW; m++) w[m] += uint32_t(add);
    } else {
#pragma unroll
        for (int m = 0; m < kNW; m += 2) {
            uint64_t const v = (uint64_t(w[m]) | (uint64_t(w[m + 1]) << 32)) + add;
            w[m] = uint32_t(v);
            w[m + 1] = uint32_t(v >> 32);
        }
    }
}

// Stages the tile's bit-packed source in shared memory (padded words): the
// 16-byte blocks from the one holding the tile's first field to the one
// holding its last source bit. Returns the bit offset of the first field.
__device__ __forceinline__ uint32_t npStage(const NumPipeTask& t, uint64_t e0, uint64_t nSrc, uint32_t te,
                                            uint32_t* stage)
{
    uint64_t const firstBit = uint64_t(reinterpret_cast<uintptr_t>(t.src) & 15) * 8 + e0 * t.nbBits;
    uintptr_t const a = (reinterpret_cast<uintptr_t>(t.src) & ~uintptr_t(15)) + (firstBit >> 7) * 16;
    uint32_t const sbit = uint32_t(firstBit & 127);
    uint64_t const nFields = e0 < nSrc ? umin64(te, nSrc - e0) : 0;
    uint32_t const nq = nFields ? uint32_t((sbit + nFields * t.nbBits + 127) >> 7) : 0u;
    const uint4* const src = reinterpret_cast<const uint4*>(a);
    for (uint32_t q = threadIdx.x; q < nq; q += kNPThreads) {
        uint4 const u = __ldg(src + q);
        uint32_t const d = npPad(4 * q); // a block never straddles a pad word
        stage[d] = u.x;
        stage[d + 1] = u.y;
        stage[d + 2] = u.z;
        stage[d + 3] = u.w;
    }
    __syncthreads();
    return sbit;
}

// Stores the thread's 64 bytes (w is used up; every lane of the warp calls it).
// A warp whose threads are all full and aligned first exchanges 16-byte quarters
// among four lanes (16 shuffles), so that four lanes' stores are 64 bytes side by
// side: with each thread storing its own quarters, every store instruction
// touched 32 half sectors, which the L2 took as twice the sectors. 256 MiB of
// 8-byte elements: 160 us before, 141 now; numeric pipeline of 4096 mixed frames
// 1.86 and 1.75 ms.
template <int W>
__device__ __forceinline__ void npStore(uint8_t* out, uint32_t cnt, uint32_t (&w)[kNW])
{
    constexpr uint32_t E = kNPBytes / W;
    if (__all_sync(0xffffffffu, cnt == E && !(reinterpret_cast<uintptr_t>(out) & 15))) {
        uint32_t const l = threadIdx.x & 3;
#pragma unroll
        for (int p = 0; p < 16; p += 8)
#pragma unroll
            for (int m = 0; m < 4; m++) {
                uint32_t const x = __shfl_xor_sync(0xffffffffu, l & 1 ? w[p + m] : w[p + 4 + m], 1);
                if (l & 1) w[p + m] = x;
                else w[p + 4 + m] = x;
            }
#pragma unroll
        for (int p = 0; p < 8; p++) {
            uint32_t const x = __shfl_xor_sync(0xffffffffu, l & 2 ? w[p] : w[p + 8], 2);
            if (l & 2) w[p] = x;
            else w[p + 8] = x;
        }
        uint4* const q = reinterpret_cast<uint4*>(out - 64 * l) + l;
#pragma unroll
        for (int i = 0; i < 4; i++) q[4 * i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        return;
    }
    if (cnt == E && !(reinterpret_cast<uintptr_t>(out) & 15)) {
#pragma unroll
        for (int q = 0; q < kNW / 4; q++)
            reinterpret_cast<uint4*>(out)[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < int(kNPBytes); k++)
            if (uint32_t(k) < cnt * W) out[k] = uint8_t(w[k >> 2] >> (8 * (k & 3)));
    }
}

// shared scratch of one tile
struct NPShared {
    uint32_t stage[kNPStagePadded];
    uint64_t warpVal[kNPThreads / 32];
    uint64_t key[24]; // XXH3 secret words at byte offsets 0, 8, ..., 184 (fused block sums)
};

// XXH3 block sums of the output, fused into the output pass. The thread's 64
// bytes (w, little-endian) are stripe tid % 16 of 1 KiB block `blk` of the
// checksummed output; the 16 threads of a block are one half-warp. Each
// thread adds its stripe's increments to 8 accumulators (acc[i ^ 1] +=
// d[i]; acc[i] += lo32(d[i] ^ k[i]) * hi32(d[i] ^ k[i]), k[i] the secret word
// at byte 8 (stripe + i)), then the half-warp reduce-scatters them: after
// four exchanges (4 + 2 + 1 + 1 shuffles) every lane holds the block total of
// accumulator 4 bit3 + 2 bit2 + bit1 of its lane index, and the even lane
// writes it where phase 1 would have. Every lane of the warp takes part; only
// blocks below hashBlocks are written.
__device__ __forceinline__ void npHashStripe(const NumPipeTask& t, const uint32_t* w, uint64_t blk,
                                             const uint64_t* key)
{
    uint32_t const lane = threadIdx.x & 31, s = lane & 15;
    uint64_t acc[8];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint64_t const d = uint64_t(w[2 * i]) | (uint64_t(w[2 * i + 1]) << 32);
        uint64_t const x = d ^ key[s + i];
        acc[i ^ 1] += d;
        acc[i] += uint64_t(uint32_t(x)) * (x >> 32);
    }
    bool const b3 = s & 8, b2 = s & 4, b1 = s & 2;
    uint64_t v4[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        uint64_t const send = b3 ? acc[k] : acc[k + 4];
        uint64_t const keep = b3 ? acc[k + 4] : acc[k];
        v4[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    uint64_t v2[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint64_t const send = b2 ? v4[k] : v4[k + 2];
        uint64_t const keep = b2 ? v4[k + 2] : v4[k];
        v2[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
    uint64_t v = (b1 ? v2[1] : v2[0]) + __shfl_xor_sync(0xffffffffu, b1 ? v2[0] : v2[1], 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (!(s & 1) && blk < t.hashBlocks) t.blockSums[8 * blk + 4 * b3 + 2 * b2 + b1] = v;
}

template <int W, int MODE>
__device__ __forceinline__ void npReduceTile(const NumPipeTask& t, const TileRef& tr, uint64_t* sums, uint32_t g,
                                             NPShared& sh)
{
    constexpr uint32_t TE = kNumTileBytes / W, E = kNPBytes / W;
    uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint64_t const e0 = uint64_t(tr.tile) * TE;
    uint64_t const nSrc = t.n ? t.n - 1 : 0;
    uint64_t acc = 0;
    if (MODE == SRC_PLANES && W > 1 && !t.zigzag && e0 + TE <= nSrc) {
        // the elements' sum is that of the planes' byte sums, shifted to their
        // places: no bytes change places, and a warp's loads are contiguous
        // (a plane of a tile is 16 KiB / W: 16 bytes a thread and round).
        // With this and full-width fields read as plain elements, the numeric
        // pipeline of 4096 mixed frames took 1.91 ms where it took 2.99.
        constexpr uint32_t kPer = TE / 16 < kNPThreads ? TE / 16 : kNPThreads; // threads on a plane at once
        constexpr uint32_t kAtOnce = kNPThreads / kPer;
#pragma unroll
        for (uint32_t b = tid / kPer; b < uint32_t(W); b += kAtOnce) {
            uint32_t s = 0;
            for (uint32_t k = 16 * (tid % kPer); k < TE; k += 16 * kPer) {
                uint32_t x[4];
                npLdq<1>(t.planes[b] + e0 + k, x);
#pragma unroll
                for (int m = 0; m < 4; m++) s = __dp4a(x[m], 0x01010101u, s);
            }
            acc += uint64_t(s) << (8 * b);
        }
    } else {
        uint32_t sbit = 0;
        if constexpr (MODE == SRC_BITPACK) sbit = npStage(t, e0, nSrc, TE, sh.stage);
        uint32_t w[kNW];
        npLoad<W, MODE>(t, e0 + uint64_t(tid) * E, nSrc, sh.stage, sbit, tid * E, w);
        if (t.zigzag) npZigzag<W>(w);
        acc = npSum<W>(w);
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (lane == 0) sh.warpVal[wid] = acc;
    __syncthreads();
    if (tid == 0) {
        uint64_t tot = 0;
#pragma unroll
        for (int w2 = 0; w2 < kNPThreads / 32; w2++) tot += sh.warpVal[w2];
        sums[g] = tot;
    }
}

template <int W, int MODE>
__device__ __forceinline__ void npTile(const NumPipeTask& t, const TileRef& tr, uint32_t g, const uint64_t* prefix,
                                       NPShared& sh)
{
    constexpr uint32_t TE = kNumTileBytes / W, E = kNPBytes / W;
    uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint64_t const e0 = uint64_t(tr.tile) * TE;
    uint64_t const j0 = e0 + uint64_t(tid) * E;
    uint32_t const cnt = j0 < t.n ? uint32_t(umin64(E, t.n - j0)) : 0;
    uint64_t const nSrc = t.delta ? (t.n ? t.n - 1 : 0) : t.n;
    uint32_t sbit = 0;
    if constexpr (MODE == SRC_BITPACK) sbit = npStage(t, e0, nSrc, TE, sh.stage);
    uint32_t w[kNW];
    npLoad<W, MODE>(t, j0, nSrc, sh.stage, sbit, tid * E, w);
    if (t.zigzag) npZigzag<W>(w);
    if (t.delta) {
        uint64_t const tot = npSum<W>(w);
        npScan<W>(w);
        // exclusive scan of thread totals within the warp, then across warps
        uint64_t incl = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t const y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        if (lane == 31) sh.warpVal[wid] = incl;
        __syncthreads();
        uint64_t warpPre = 0;
#pragma unroll
        for (int w2 = 0; w2 < kNPThreads / 32; w2++) warpPre += uint32_t(w2) < wid ? sh.warpVal[w2] : 0;
        npAdd<W>(w, t.first + prefix[g] + warpPre + (incl - tot));
    }
    if (t.blockSums) npHashStripe(t, w, (uint64_t(tr.tile) * kNumTileBytes + uint64_t(tid) * kNPBytes) >> 10, sh.key);
    npStore<W>(t.out + j0 * W, cnt, w);
}

template <int W>
__device__ __forceinline__ void npTileW(const NumPipeTask& t, const TileRef& tr, uint32_t g, const uint64_t* prefix,
                                        NPShared& sh)
{
    switch (t.srcMode) {
        case SRC_PLAIN: npTile<W, SRC_PLAIN>(t, tr, g, prefix, sh); break;
        case SRC_PLANES: npTile<W, SRC_PLANES>(t, tr, g, prefix, sh); break;
        default: npTile<W, SRC_BITPACK>(t, tr, g, prefix, sh); break;
    }
}

template <int W>
__device__ __forceinline__ void npReduceW(const NumPipeTask& t, const TileRef& tr, uint64_t* sums, uint32_t g,
                                          NPShared& sh)
{
    switch (t.srcMode) {
        case SRC_PLAIN: npReduceTile<W, SRC_PLAIN>(t, tr, sums, g, sh); break;
        case SRC_PLANES: npReduceTile<W, SRC_PLANES>(t, tr, sums, g, sh); break;
        default: npReduceTile<W, SRC_BITPACK>(t, tr, sums, g, sh); break;
    }
}

// pass 1 (delta tasks): sum of each tile's sources
__global__ void __launch_bounds__(kNPThreads) kNumReduce(const NumPipeTask* __restrict__ tasks,
                                                         const TileRef* __restrict__ tiles,
                                                         uint64_t* __restrict__ sums)
{
    __shared__ NPShared sh;
    uint32_t const g = blockIdx.x;
    TileRef const tr = tiles[g];
    NumPipeTask const t = tasks[tr.task];
    if (!t.delta) return;
    switch (t.w) {
        case 1: npReduceW<1>(t, tr, sums, g, sh); break;
        case 2: npReduceW<2>(t, tr, sums, g, sh); break;
        case 4: npReduceW<4>(t, tr, sums, g, sh); break;
        default: npReduceW<8>(t, tr, sums, g, sh); break;
    }
}

// pass 2: exclusive scan of tile sums per task, one CTA per task (of up to
// 1,024 threads, eight tiles a thread and round). The 16,384 tiles of a 256
// MiB output took one warp 50 us.
__global__ void __launch_bounds__(1024) kNumPrefix(const NumPipeTask* __restrict__ tasks,
                                                   const uint64_t* __restrict__ sums, uint64_t* __restrict__ prefix)
{
    __shared__ uint64_t warpSum[32];
    NumPipeTask const t = tasks[blockIdx.x];
    if (!t.delta) return;
    uint32_t const lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
    uint32_t const te = kNumTileBytes / t.w;
    uint32_t const nT = uint32_t((t.n + te - 1) / te);
    const uint64_t* const in = sums + t.tileBase;
    uint64_t* const out = prefix + t.tileBase;
    uint64_t running = 0;
    for (uint32_t k0 = 0; k0 < nT; k0 += 8 * blockDim.x) {
        uint32_t const k = k0 + 8 * threadIdx.x;
        uint64_t x[8];
        uint64_t tot = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            x[j] = k + j < nT ? in[k + j] : 0;
            tot += x[j];
        }
        uint64_t incl = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t const y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        __syncthreads(); // the sums of the round before have been read
        if (lane == 31) warpSum[wid] = incl;
        __syncthreads();
        uint64_t run = running + incl - tot;
        for (uint32_t w = 0; w < warps; w++) {
            uint64_t const y = warpSum[w];
            run += w < wid ? y : 0;
            running += y;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (k + j < nT) out[k + j] = run;
            run += x[j];
        }
    }
}

// pass 3: the output. Six CTAs an SM (40 registers, no spills) where the
// compiler's own choice of 48 gave five: 256 MiB of 8-byte elements 141 us with
// five, 133 with six, 130 with seven, which spill and gain nothing in a batch.
__global__ void __launch_bounds__(kNPThreads, 6) kNumPipe(const NumPipeTask* __restrict__ tasks,
                                                       const TileRef* __restrict__ tiles,
                                                       const uint64_t* __restrict__ prefix)
{
    __shared__ NPShared sh;
    uint32_t const g = blockIdx.x;
    TileRef const tr = tiles[g];
    NumPipeTask const t = tasks[tr.task];
    if (t.blockSums) { // the same task for the whole CTA
        if (threadIdx.x < 24) sh.key[threadIdx.x] = kXxhWords.w8[threadIdx.x];
        __syncthreads();
    }
    switch (t.w) {
        case 1: npTileW<1>(t, tr, g, prefix, sh); break;
        case 2: npTileW<2>(t, tr, g, prefix, sh); break;
        case 4: npTileW<4>(t, tr, g, prefix, sh); break;
        default: npTileW<8>(t, tr, g, prefix, sh); break;
    }
}

// ---------------------------------------------------------------------------
// generic transpose (any width)
__global__ void kTranspose(const TransposeTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    TransposeTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kTileElems;
    uint64_t const e1 = umin64(t.n, e0 + kTileElems);
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x)
        for (uint32_t b = 0; b < t.W; b++) t.out[i * t.W + b] = t.planes[b][i];
}

// ---------------------------------------------------------------------------
// tokenize: dictionary gather out[i] = alphabet[idx[i]]
//
// What bounds it: memory, once a thread's loads and stores are whole vectors:
// 16 bytes of output and their indices at a time where both are aligned (a
// tile's first element is; tokenGather), element by element elsewhere. 256 MiB
// of 4-byte elements with 16-bit indices: 181 us element by element, 101 now, 135
// with an unaligned alphabet (193 when its elements were read by bytes).
//
// Elements [e0, e1) of W bytes from IW-byte indices, 16 bytes of output a
// thread and round; returns the first element left over.
template <int W, int IW, bool ALIGNED>
__device__ __forceinline__ uint64_t tokenGather(const TokenizeTask& t, uint64_t e0, uint64_t e1, bool& bad)
{
    constexpr uint32_t E = 16 / W, kIdxBytes = E * IW;
    constexpr uint32_t kAlign = kIdxBytes < 16 ? kIdxBytes : 16; // of the indices
    if ((reinterpret_cast<uintptr_t>(t.out) & 15) || (reinterpret_cast<uintptr_t>(t.idx) & (kAlign - 1))) return e0;
    uint64_t const vectors = (e1 - e0) / E;
#pragma unroll 2
    for (uint64_t v = threadIdx.x; v < vectors; v += blockDim.x) {
        uint64_t const i = e0 + v * E;
        const uint8_t* const at = t.idx + i * IW;
        uint32_t raw[(kIdxBytes + 3) / 4];
        if constexpr (kIdxBytes >= 16) {
#pragma unroll
            for (uint32_t q = 0; q < kIdxBytes / 16; q++)
                *reinterpret_cast<uint4*>(raw + 4 * q) = __ldg(reinterpret_cast<const uint4*>(at) + q);
        } else if constexpr (kIdxBytes == 8) {
            *reinterpret_cast<uint2*>(raw) = __ldg(reinterpret_cast<const uint2*>(at));
        } else if constexpr (kIdxBytes == 4) {
            raw[0] = __ldg(reinterpret_cast<const uint32_t*>(at));
        } else {
            raw[0] = __ldg(reinterpret_cast<const uint16_t*>(at));
        }
        uint32_t o[4] = { 0u, 0u, 0u, 0u };
#pragma unroll
        for (uint32_t j = 0; j < E; j++) {
            uint32_t k = raw[j * IW / 4] >> (8 * (j * IW % 4));
            if (IW < 4) k &= (1u << (8 * (IW & 3))) - 1u;
            if (k >= t.alphabetSize) {
                bad = true;
                k = 0;
            }
            uint64_t x;
            if (!ALIGNED && W >= 4) { // the aligned words that hold the element
                uint32_t const off = uint32_t(reinterpret_cast<uintptr_t>(t.alphabet) & 3);
                const uint32_t* const p = reinterpret_cast<const uint32_t*>(t.alphabet - off) + uint64_t(k) * (W / 4);
                uint32_t const a = __ldg(p), b = W == 8 || off ? __ldg(p + 1) : 0u;
                x = __funnelshift_r(a, b, 8 * off);
                if (W == 8) x |= uint64_t(__funnelshift_r(b, off ? __ldg(p + 2) : 0u, 8 * off)) << 32;
            } else if (!ALIGNED) x = ldElem(t.alphabet + uint64_t(k) * W, W);
            else if (W == 8) x = __ldg(reinterpret_cast<const unsigned long long*>(t.alphabet) + k);
            else if (W == 4) x = __ldg(reinterpret_cast<const uint32_t*>(t.alphabet) + k);
            else if (W == 2) x = __ldg(reinterpret_cast<const uint16_t*>(t.alphabet) + k);
            else x = __ldg(t.alphabet + k);
            o[j * W / 4] |= uint32_t(x) << (8 * (j * W % 4));
            if (W == 8) o[2 * j + 1] = uint32_t(x >> 32);
        }
        *reinterpret_cast<uint4*>(t.out + i * W) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    return e0 + vectors * E;
}
template <int W, bool ALIGNED>
__device__ __forceinline__ uint64_t tokenGatherI(const TokenizeTask& t, uint64_t e0, uint64_t e1, bool& bad)
{
    return t.iw == 1   ? tokenGather<W, 1, ALIGNED>(t, e0, e1, bad)
           : t.iw == 2 ? tokenGather<W, 2, ALIGNED>(t, e0, e1, bad)
           : t.iw == 4 ? tokenGather<W, 4, ALIGNED>(t, e0, e1, bad)
                       : e0;
}
// (an alphabet that was stored lies in the frame at any byte)
template <int W>
__device__ __forceinline__ uint64_t tokenGatherW(const TokenizeTask& t, uint64_t e0, uint64_t e1, bool& bad)
{
    return reinterpret_cast<uintptr_t>(t.alphabet) & (W - 1) ? tokenGatherI<W, false>(t, e0, e1, bad)
                                                             : tokenGatherI<W, true>(t, e0, e1, bad);
}

__global__ void __launch_bounds__(256) kTokenize(const TokenizeTask* __restrict__ tasks, const TileRef* __restrict__ tiles,
                          uint32_t* __restrict__ status)
{
    TileRef const tr = tiles[blockIdx.x];
    TokenizeTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kTileElems;
    uint64_t const e1 = umin64(t.n, e0 + kTileElems);
    bool bad = false;
    uint64_t from = e0;
    if (t.alphabetSize) { // (an empty alphabet has no element to read)
        switch (t.w) {
            case 1: from = tokenGatherW<1>(t, e0, e1, bad); break;
            case 2: from = tokenGatherW<2>(t, e0, e1, bad); break;
            case 4: from = tokenGatherW<4>(t, e0, e1, bad); break;
            case 8: from = tokenGatherW<8>(t, e0, e1, bad); break;
            default: break;
        }
    }
    for (uint64_t i = from + threadIdx.x; i < e1; i += blockDim.x) {
        uint64_t const k = ldElem(t.idx + i * t.iw, t.iw);
        if (k >= t.alphabetSize) { bad = true; continue; }
        if (t.w == 4 || t.w == 2 || t.w == 1 || t.w == 8) stElem(t.out + i * t.w, ldElem(t.alphabet + k * t.w, t.w), t.w);
        else for (uint32_t b = 0; b < t.w; b++) t.out[i * t.w + b] = t.alphabet[k * t.w + b];
    }
    if (bad) reportError(status, DERR_CORRUPTION);
}

// ---------------------------------------------------------------------------
// string lengths to 4 bytes (NUMOP_write32_fromNumerics in
// DI_revert_VSF_separation, decode_conversion_binding.c:245-250)
__global__ void kWiden(const WidenTask* __restrict__ tasks, const TileRef* __restrict__ tiles,
                       uint32_t* __restrict__ status)
{
    TileRef const tr = tiles[blockIdx.x];
    WidenTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kTileElems;
    uint64_t const e1 = umin64(t.n, e0 + kTileElems);
    bool bad = false;
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
        uint64_t const v = ldElem(t.src + i * t.w, t.w);
        bad |= v > 0xffffffffull;
        t.dst[i] = uint32_t(v);
    }
    if (bad) reportError(status, DERR_CORRUPTION);
}

// ---------------------------------------------------------------------------
// float deconstruct (decode_float_deconstruct_kernel.c semantics)
//
// What bounds it: memory, once a thread's loads and stores are vectors: 16
// bytes of output (8 or 4 elements) at a time where they are aligned, element
// by element elsewhere. The sources' vectors are put together from aligned
// words: a stored stream lies in the frame at any byte. 214 M bfloat16
// elements in 18 matrices: 452 us element by element, 172 now.
//
// 4 N bytes at p from the aligned words that hold them
template <int N>
__device__ __forceinline__ void ldBytes(const uint8_t* p, uint32_t (&x)[N])
{
    uint32_t const off = uint32_t(reinterpret_cast<uintptr_t>(p) & 3);
    const uint32_t* const w = reinterpret_cast<const uint32_t*>(p - off);
    uint32_t a = __ldg(w);
#pragma unroll
    for (int k = 0; k < N; k++) {
        uint32_t const b = k + 1 < N || off ? __ldg(w + k + 1) : 0u;
        x[k] = __funnelshift_r(a, b, 8 * off);
        a = b;
    }
}

// Elements [e0, e1), 16 bytes of output a thread and round; returns the first
// element left over. TYPE as eltType.
template <int TYPE>
__device__ __forceinline__ uint64_t floatJoin(const FloatDecTask& t, uint64_t e0, uint64_t e1)
{
    constexpr uint32_t E = TYPE == 0 ? 4 : 8; // elements of 16 bytes
    if (reinterpret_cast<uintptr_t>(t.out) & 15) return e0;
    uint64_t const vectors = (e1 - e0) / E;
#pragma unroll 2
    for (uint64_t v = threadIdx.x; v < vectors; v += blockDim.x) {
        uint64_t const i = e0 + v * E;
        uint32_t o[4];
        if constexpr (TYPE == 0) {
            uint32_t f[3], x[1];
            ldBytes(t.signFrac + 3 * i, f);
            ldBytes(t.exponent + i, x);
            uint32_t const s[4] = { f[0] & 0xffffffu, (f[0] >> 24) | ((f[1] & 0xffffu) << 8),
                                    (f[1] >> 16) | ((f[2] & 0xffu) << 16), f[2] >> 8 };
#pragma unroll
            for (int k = 0; k < 4; k++) o[k] = (((x[0] >> (8 * k)) & 0xffu) << 23) | (s[k] << 31) | (s[k] >> 1);
        } else {
            uint32_t x[2], s[4]; // s: two elements' sign and fraction each, in halves
            ldBytes(t.exponent + i, x);
            if constexpr (TYPE == 1) {
                uint32_t f[2];
                ldBytes(t.signFrac + i, f);
#pragma unroll
                for (int k = 0; k < 4; k++) s[k] = __byte_perm(f[k / 2], 0, k % 2 ? 0x4342 : 0x4140);
            } else {
                ldBytes(t.signFrac + 2 * i, s);
            }
            uint32_t e[4];
#pragma unroll
            for (int k = 0; k < 4; k++) e[k] = __byte_perm(x[k / 2], 0, k % 2 ? 0x4342 : 0x4140);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t const frac = (s[k] >> 1) & 0x7fff7fffu, sign = (s[k] & 0x00010001u) << 15;
                // (an exponent of more than 5 bits runs into the sign, as 16-bit arithmetic has it)
                uint32_t const ex = TYPE == 1 ? e[k] << 7 : (e[k] & 0x003f003fu) << 10;
                o[k] = frac | sign | ex;
            }
        }
        *reinterpret_cast<uint4*>(t.out + i * (16 / E)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    return e0 + vectors * E;
}

__global__ void __launch_bounds__(256) kFloatDec(const FloatDecTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    FloatDecTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kTileElems;
    uint64_t const e1 = umin64(t.n, e0 + kTileElems);
    uint64_t const from = t.eltType == 0   ? floatJoin<0>(t, e0, e1)
                          : t.eltType == 1 ? floatJoin<1>(t, e0, e1)
                                           : floatJoin<2>(t, e0, e1);
    for (uint64_t i = from + threadIdx.x; i < e1; i += blockDim.x) {
        uint32_t const ex = t.exponent[i];
        if (t.eltType == 1) {
            uint32_t const s = t.signFrac[i];
            stElem(t.out + 2 * i, uint16_t((s >> 1) | (s << 15) | (ex << 7)), 2);
        } else if (t.eltType == 2) {
            uint32_t const s = uint32_t(t.signFrac[2 * i]) | (uint32_t(t.signFrac[2 * i + 1]) << 8);
            stElem(t.out + 2 * i, uint16_t((s >> 1) | (s << 15) | (ex << 10)), 2);
        } else {
            uint32_t const s = uint32_t(t.signFrac[3 * i]) | (uint32_t(t.signFrac[3 * i + 1]) << 8)
                    | (uint32_t(t.signFrac[3 * i + 2]) << 16);
            stElem(t.out + 4 * i, (ex << 23) | (s << 31) | (s >> 1), 4);
        }
    }
}

// ---------------------------------------------------------------------------
// flatpack: alphabet + LSB-first indices terminated by a 1 bit
// Flatpack: out[i] = alphabet[field i], fields of nbBits (1..8) LSB-first.
// Each thread decodes 8 consecutive fields from a 64-bit window (three aligned
// words of the packed stream, funnel-shifted) and stores them with one 8-byte
// store. Only words that hold bytes of the packed stream are read (its last
// word holds the terminator).
// What bounds it: the lookups (instructions, and byte loads whose banks
// conflict), so up to 5 bits two fields are one: a table of the symbols of
// every pair of fields, with bit 16 set where one is outside the alphabet.
// Fields of 6 bits and more would take 16 KiB and more for it; they look up the
// alphabet in shared memory. Mixed batch of 4096 frames, all flatpack launches:
// 0.48 ms with a lookup a field, 0.26 ms now.
constexpr uint32_t kFlatPairBits = 5;
__global__ void __launch_bounds__(256) kFlatpack(const FlatpackTask* __restrict__ tasks,
                                                 const TileRef* __restrict__ tiles, uint32_t* __restrict__ status)
{
    __shared__ uint8_t sAlpha[256];
    __shared__ uint32_t sPair[1u << (2 * kFlatPairBits)];
    TileRef const tr = tiles[blockIdx.x];
    FlatpackTask const t = tasks[tr.task];
    uint32_t const as = min(t.alphabetSize, 256u);
    uint32_t const nb = t.nbBits, mask = (1u << nb) - 1u;
    bool const pairs = nb <= kFlatPairBits;
    for (uint32_t i = threadIdx.x; i < as; i += blockDim.x) sAlpha[i] = t.alphabet[i];
    __syncthreads();
    if (pairs) {
        for (uint32_t i = threadIdx.x; i < 1u << (2 * nb); i += blockDim.x) {
            uint32_t const f0 = i & mask, f1 = i >> nb;
            // one field alone may be the last of the stream: each has its own bad mark
            sPair[i] = (f0 < as ? sAlpha[f0] : 0x10000u) | (f1 < as ? uint32_t(sAlpha[f1]) << 8 : 0x20000u);
        }
        __syncthreads();
    }
    const uint32_t* const pw = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(t.packed) & ~uintptr_t(3));
    uint64_t const sb = (reinterpret_cast<uintptr_t>(t.packed) & 3) * 8;
    uint64_t const qLast = (sb + t.n * nb) >> 5;
    uint64_t const e0 = uint64_t(tr.tile) * kTileBytes;
    uint64_t const e1 = umin64(t.n, e0 + kTileBytes);
    bool bad = false;
    for (uint64_t k0 = e0 + 8ull * threadIdx.x; k0 < e1; k0 += 8ull * blockDim.x) {
        uint32_t const cnt = uint32_t(umin64(8, e1 - k0));
        uint64_t const bit = sb + k0 * nb;
        uint64_t const q = bit >> 5;
        uint32_t const r = uint32_t(bit & 31);
        uint32_t const w0 = __ldg(pw + q);
        uint32_t const w1 = q + 1 <= qLast ? __ldg(pw + q + 1) : 0u;
        uint32_t const w2 = q + 2 <= qLast ? __ldg(pw + q + 2) : 0u;
        uint32_t const lo = __funnelshift_r(w0, w1, r), hi = __funnelshift_r(w1, w2, r);
        uint32_t o[2] = { 0u, 0u };
        if (pairs) { // at most 40 bits
            uint32_t const pm = (1u << (2 * nb)) - 1u;
            uint32_t v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                uint32_t const at = 2 * j * nb;
                v[j] = sPair[(at < 32 ? __funnelshift_r(lo, hi, at) : hi >> (at - 32)) & pm];
            }
            o[0] = __byte_perm(v[0], v[1], 0x5410);
            o[1] = __byte_perm(v[2], v[3], 0x5410);
            if (cnt == 8) {
                bad |= ((v[0] | v[1] | v[2] | v[3]) >> 16) != 0;
            } else {
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) bad |= (2 * j < cnt && (v[j] & 0x10000u)) || (2 * j + 1 < cnt && (v[j] & 0x20000u));
            }
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                uint32_t const at = j * nb;
                uint32_t const f = (at < 32 ? __funnelshift_r(lo, hi, at) : hi >> (at - 32)) & mask;
                uint32_t v = 0;
                if (j < cnt) {
                    if (f < as) v = sAlpha[f];
                    else bad = true;
                }
                o[j >> 2] |= v << (8 * (j & 3));
            }
        }
        uint8_t* const dst = t.out + k0;
        if (cnt == 8 && !(reinterpret_cast<uintptr_t>(dst) & 7)) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 8; j++)
                if (j < cnt) dst[j] = uint8_t(o[j >> 2] >> (8 * (j & 3)));
        }
    }
    if (tr.tile == 0 && threadIdx.x == 0) {
        // terminator: the bit after the last index is set and is the last set bit
        uint64_t const endBit = t.n * t.nbBits;
        uint8_t const last = t.packed[endBit >> 3];
        if (!((last >> (endBit & 7)) & 1) || (last >> (endBit & 7)) != 1) bad = true;
    }
    if (bad) reportError(status, DERR_CORRUPTION);
}

// ---------------------------------------------------------------------------
// Backward bit readers (FSE / Huffman bitstreams): fields are read most
// significant bit first from the end of the stream towards its start.
//
// Each lane stages its stream through a small ring of 16-byte chunks in
// shared memory, filled by asynchronous copies (cp.async) issued AHEAD chunks
// before they are needed; the bit window in registers refills from the ring.
__device__ __forceinline__ bool streamStart(const uint8_t* p, uint32_t size, const uint8_t*& g16, int32_t& pos,
                                            int32_t& end)
{
    if (size == 0) return false;
    uint8_t const last = p[size - 1];
    if (last == 0) return false;
    uintptr_t const a = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15);
    g16 = reinterpret_cast<const uint8_t*>(a);
    end = int32_t(reinterpret_cast<uintptr_t>(p) - a) * 8;
    pos = end + int32_t(size - 1) * 8 + (31 - __clz(uint32_t(last)));
    return true;
}

// Backward bit reader by position (FSE and Huffman decoders): `pos` is
// one bit index, window() loads the three stream words at it (one masked
// address) and shifts out the 64 bits below it. The stream's 16-byte chunks
// lie in a ring of RING chunks at byte `ring` of shared memory, from the
// position's down to the one at byte `low` of g16; the ring's last chunk is
// copied to the 16 bytes below the ring too, so that a window's words never
// wrap. Words below the stream are never consumed by a valid stream
// (finished() checks that it ends exactly at its first bit), so the ring's
// stale contents may stand in for them.
// SHIFT: spread() may move positions, so that lanes' windows fall on different
// banks.
template <int RING, int AHEAD, bool SHIFT = false>
struct PosStream {
    static_assert((RING & (RING - 1)) == 0 && AHEAD + 4 <= RING, "ring shape");
    static constexpr uint32_t kBytes = 16 + 16 * RING; // mirror and ring, 16-byte aligned
    const uint8_t *g16, *smem;
    uint32_t ring, ringAddr;
    int32_t pos, end, low;
    int32_t lowest = 0; // byte of the stream's first chunk

    // the next chunk below, unless `low` has reached `goal` (not below 0)
    __device__ __forceinline__ void next(int32_t goal)
    {
        asm volatile("{\n\t.reg .pred p, q;\n\t.reg .u32 s;\n\t.reg .u64 a;\n\t"
                     "setp.gt.s32 p, %0, %1;\n\t"
                     "@p sub.s32 %0, %0, 16;\n\t"
                     "and.b32 s, %0, %4;\n\t"
                     "setp.eq.and.u32 q, s, %4, p;\n\t"
                     "add.u32 s, s, %2;\n\t"
                     "cvt.u64.u32 a, %0;\n\t"
                     "add.u64 a, a, %3;\n\t"
                     "@p cp.async.ca.shared.global.L2::128B [s], [a], 16;\n\t"
                     "@q cp.async.ca.shared.global.L2::128B [s + %5], [a], 16;\n\t}"
                     : "+r"(low) : "r"(goal), "r"(ringAddr), "l"(g16), "n"(16 * RING - 16), "n"(-16 * RING) : "memory");
    }
    // the stream's top bit and its first; `area`: byte of the kBytes of shared memory
    __device__ __forceinline__ bool open(const uint8_t* p, uint32_t size, const uint8_t* sm, uint32_t area)
    {
        smem = sm;
        ring = area + 16;
        ringAddr = uint32_t(__cvta_generic_to_shared(sm + ring));
        return streamStart(p, size, g16, pos, end);
    }
    // goes on from position `to`: fills the ring below it
    __device__ __forceinline__ void seek(int32_t to)
    {
        close(); // a copy in flight may be to the same place
        pos = to;
        int32_t const first = ((pos - 1) >> 7) * 16, goal = max(first - 16 * AHEAD, SHIFT ? lowest : 0);
        low = first + 16;
        while (low > goal) next(goal);
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    }
    // Counts positions from up to RING - 1 chunks before the first one, so that
    // position p falls into the ring's first chunk; returns what it adds to them.
    __device__ __forceinline__ int32_t spread(int32_t p)
    {
        static_assert(SHIFT, "a stream whose positions may move");
        int32_t const k = -((p - 1) >> 7) & (RING - 1);
        lowest = 16 * k;
        g16 -= lowest;
        pos += 128 * k;
        end += 128 * k;
        return 128 * k;
    }
    __device__ __forceinline__ bool init(const uint8_t* p, uint32_t size, const uint8_t* sm, uint32_t area)
    {
        if (!open(p, size, sm, area)) return false;
        seek(pos);
        return true;
    }
    // Keeps AHEAD chunks below the position's in the ring, given that at most
    // N <= 3 of them were read since the last call: N + 1 may be needed until
    // the next call, and were issued at least two calls before it.
    template <int N>
    __device__ __forceinline__ void refill()
    {
        static_assert(3 * N + 1 <= AHEAD, "a chunk is issued two calls before it is read");
        int32_t const goal = max(((pos >> 3) & ~15) - 16 * AHEAD, SHIFT ? lowest : 0);
#pragma unroll
        for (int k = 0; k < N; k++) next(goal);
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 2;" ::: "memory");
    }
    // the 64 bits below pos, most significant first
    __device__ __forceinline__ void window(uint32_t& hi, uint32_t& lo) const
    {
        uint32_t const o = ring + ((uint32_t(pos) & (128 * RING - 32)) >> 3);
        uint32_t const a = *reinterpret_cast<const uint32_t*>(smem + o);
        uint32_t const b = *reinterpret_cast<const uint32_t*>(smem + o - 4);
        uint32_t const c = *reinterpret_cast<const uint32_t*>(smem + o - 8);
        hi = __funnelshift_r(b, a, uint32_t(pos));
        lo = __funnelshift_r(c, b, uint32_t(pos));
    }
    __device__ __forceinline__ bool finished() const { return pos == end; }
    // ends the stream: no copy outlives the lane
    __device__ __forceinline__ void close() { asm volatile("cp.async.wait_all;" ::: "memory"); }
};

// ---------------------------------------------------------------------------
// FSE: one lane per chunk. A CTA keeps its streams' decoding tables in shared
// memory, one cell per decoder state, in one of three forms:
//  - kCells32: a 32-bit cell with nbBits in the low byte, the symbol in the
//    next and newStateBase * 4 above; a transition is one load (8 KiB a stream
//    at tableLog 11, 27 streams per SM);
//  - kCells24: a symbol byte and a 16-bit entry, newStateBase above five bits
//    of nbBits, in two arrays (6 KiB a stream, 36 streams per SM);
//  - kCells24Wide: the same with four bits of nbBits, for tableLog 12.
//
// Table construction restates src/openzl/fse/decompress/fse_decompress.c:
// 73-171; decode order restates fse_decompress.c:255-337 (state i % nbStates
// emits symbol i; the last symbol of each state has no transition).
using FseStream = PosStream<kFseRing, kFseAhead>;
static_assert(FseStream::kBytes == kFseRingBytes, "a lane's ring as fse_shape.h has it");

// Builds the decoding table of task t (cells or entries at tab, newStateBase
// above the low NB bits of an entry; symbols at symOf, for kCells32 in the
// cells themselves) with all 32 lanes of the warp (every lane calls it); `cum`
// and `next` are the warp's build scratch (257 and 256 entries, next 16-byte
// aligned).
//  - Counts: the normalized counts go to the counters; a warp scan of
//    the positive counts gives each symbol's first occurrence (cum), and the
//    count -1 symbols take the top cells in symbol order.
//  - Spread: occurrence k (symbols in order, each repeated count times) goes
//    to the k-th cell of the sequence 0, step, 2 step, ... (mod size) that is
//    not a top cell; 32 sequence positions per round, ranked by a ballot.
//  - Cells, 32 per round in increasing order: a cell's state x is its
//    symbol's counter plus the number of lower lanes of the round holding
//    the same symbol (__match_any_sync); the highest such lane advances the
//    counter.
// The result equals the serial construction of fse_decompress.c:73-171.
template <int CELLS>
__device__ __forceinline__ void fseBuildWarp(const FseTask& t, void* tab, uint8_t* symOf, uint16_t* cum,
                                             uint16_t* next)
{
    constexpr uint32_t SS = CELLS == kCells32 ? 4 : 1; // bytes from one cell's symbol to the next's
    uint32_t const lane = threadIdx.x & 31;
    uint32_t const lt = (1u << lane) - 1u;
    uint32_t const tl = t.tableLog;
    uint32_t const size = 1u << tl, mask = size - 1;
    uint32_t const step = (size >> 1) + (size >> 3) + 3;
    uint32_t const nbSym = t.nbSym;
    // normalized counts (16-byte aligned in the parameter block, which has
    // slack after its end) into the counters: at most 32 16-byte blocks
    uint32_t const nv = (nbSym * 2 + 15) >> 4;
    if (lane < nv) reinterpret_cast<uint4*>(next)[lane] = __ldg(reinterpret_cast<const uint4*>(t.norm) + lane);
    __syncwarp();
    // lane j: symbols 8j .. 8j + 7
    int v[8];
    uint32_t sumC = 0, sumNeg = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        uint32_t const sy = 8 * lane + k;
        v[k] = sy < nbSym ? int(int16_t(next[sy])) : 0;
        sumC += v[k] > 0 ? uint32_t(v[k]) : 0u;
        sumNeg += v[k] == -1 ? 1u : 0u;
    }
    uint32_t inC = sumC, inNeg = sumNeg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t const yc = __shfl_up_sync(0xffffffffu, inC, o), yn = __shfl_up_sync(0xffffffffu, inNeg, o);
        if (lane >= uint32_t(o)) {
            inC += yc;
            inNeg += yn;
        }
    }
    uint32_t const totalNeg = __shfl_sync(0xffffffffu, inNeg, 31);
    uint32_t const high = size - 1 - totalNeg;
    uint32_t c0 = inC - sumC, n0 = inNeg - sumNeg;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        uint32_t const sy = 8 * lane + k;
        cum[sy] = uint16_t(c0);
        c0 += v[k] > 0 ? uint32_t(v[k]) : 0u;
        if (v[k] == -1) {
            symOf[SS * (size - 1 - n0)] = uint8_t(sy);
            next[sy] = 1;
            n0++;
        }
    }
    if (lane == 31) cum[256] = uint16_t(c0);
    __syncwarp();
    // spread
    uint32_t sCur = 0, cumNext = cum[1], occBase = 0;
    for (uint32_t b0 = 0; b0 < size; b0 += 32) {
        uint32_t const pos = ((b0 + lane) * step) & mask;
        bool const valid = totalNeg < size && pos <= high; // all cells are top cells when every count is -1
        uint32_t const bal = __ballot_sync(0xffffffffu, valid);
        if (valid) {
            uint32_t const occ = occBase + __popc(bal & lt);
            while (occ >= cumNext && sCur < 255) cumNext = cum[++sCur + 1];
            symOf[SS * pos] = uint8_t(sCur);
        }
        occBase += __popc(bal);
    }
    __syncwarp();
    // cells
    for (uint32_t b0 = 0; b0 < size; b0 += 32) {
        uint32_t const u = b0 + lane;
        uint32_t const sy = symOf[SS * u];
        uint32_t const m = __match_any_sync(0xffffffffu, sy);
        uint32_t const base = next[sy];
        __syncwarp();
        if (lane == 31u - __clz(m)) next[sy] = uint16_t(base + __popc(m));
        uint32_t const x = base + __popc(m & lt);
        uint32_t const nb = tl - (31 - __clz(x));
        uint32_t const ns = (x << nb) - size;
        if (CELLS == kCells32) static_cast<uint32_t*>(tab)[u] = (ns << 18) | (sy << 8) | nb;
        else static_cast<uint16_t*>(tab)[u] = uint16_t((ns << (CELLS == kCells24 ? 5 : 4)) | nb);
        __syncwarp();
    }
}

// Decodes one stream (kFse's lane). `cell0` is the lane's first cell in the
// CTA's tables, `tabBase` the byte of the entries of cell 0 (kCells24: symbols
// are at byte `cell`), `area` the byte of the lane's stream ring.
//
// What bounds it: a stream is a serial chain and an SM's shared memory holds
// few streams, so a four-symbol step costs its dependent latencies and, with
// one warp a scheduler, its instructions (two cycles each on the integer
// pipe). Both were cut:
//  - The position is one bit index, and each step loads the stream words at it
//    (PosStream). The loads run beside the table lookups; neither waits for
//    the other.
//  - Five bits of nbBits in an entry are its own shift amount (shifts take the
//    low five bits), also summed in pairs (two fields are at most 24 bits).
//  - Ring refills come once per 32 symbols without a branch: up to three
//    predicated 16-byte copies for the at most 48 bytes that the steps read,
//    one commit, and a wait that leaves the last two refills' copies in
//    flight. (A refill per step inside a branch was taken by some lane of the
//    warp at nearly every step; branches around the copies, and copies through
//    registers, measured 10 to 15 cycles a step slower than the predicates.)
//  - Four steps fill one 16-byte store.
// Cycles per step, one stream on an SM: 275 before, 115 with kCells24, 96 with
// kCells32.
// 32 K symbols at tableLog 11: 1.09 ms before, 0.40 ms now. Mixed batch of 4096
// frames, largest FSE launch (beside others): 4.65 ms before, 2.60 ms now.
template <int CELLS, int NST>
__device__ __forceinline__ void fseDecode(const FseTask& t, const uint8_t* smem, uint32_t cell0, uint32_t tabBase,
                                          uint32_t area, uint32_t* status)
{
    FseStream br;
    if (!br.init(t.bits, t.bitsSize, smem, area)) { reportError(status, DERR_CORRUPTION); return; }
    // A state is its cell's index (kCells32: its byte). ent: its cell or
    // entry; to: the state that an entry and its field lead to; amt: the
    // entry's shift amount (low five bits); nbOf: nbBits alone.
    uint32_t const s00 = CELLS == kCells32 ? 4 * cell0 : cell0;
    auto state = [&](uint32_t f) -> uint32_t { return s00 + (CELLS == kCells32 ? 4 * f : f); };
    auto ent = [&](uint32_t st) -> uint32_t {
        if (CELLS == kCells32) return *reinterpret_cast<const uint32_t*>(smem + st);
        return *reinterpret_cast<const uint16_t*>(smem + tabBase + 2 * st);
    };
    auto sym = [&](uint32_t st) -> uint32_t { return CELLS == kCells32 ? smem[st + 1] : smem[st]; };
    auto nbOf = [](uint32_t e) -> uint32_t { return CELLS == kCells24Wide ? e & 15u : e & 31u; };
    auto amt = [&](uint32_t e) -> uint32_t { return CELLS == kCells24Wide ? e & 15u : e; };
    auto to = [&](uint32_t e, uint32_t f) -> uint32_t {
        return CELLS == kCells32 ? s00 + (e >> 16) + 4 * f : s00 + (e >> (CELLS == kCells24 ? 5 : 4)) + f;
    };
    auto top = [](uint32_t x, uint32_t n) -> uint32_t { return __funnelshift_l(x, 0u, n); }; // top n bits
    auto read = [&](uint32_t n) -> uint32_t { // one field
        br.refill<1>();
        uint32_t hi, lo;
        br.window(hi, lo);
        br.pos -= int32_t(n);
        return top(hi, n);
    };
    uint32_t s0 = state(read(t.tableLog)), s1 = state(read(t.tableLog)), s2 = 0, s3 = 0;
    if (NST == 4) {
        s2 = state(read(t.tableLog));
        s3 = state(read(t.tableLog));
    }
    uint32_t const n = t.dstSize;
    uint32_t const lastTr = n > NST ? n - NST : 0; // symbols [0, lastTr) have a transition
    uint8_t* const out = t.out;
    // one symbol from s0, then the states rotate
    auto single = [&](uint32_t i) {
        uint32_t const e = ent(s0);
        out[i] = uint8_t(sym(s0));
        uint32_t ns = s0;
        if (i < lastTr) ns = to(e, read(nbOf(e)));
        if (NST == 4) {
            s0 = s1; s1 = s2; s2 = s3; s3 = ns;
        } else {
            s0 = s1; s1 = ns;
        }
    };
    // four symbols with transitions, as one little-endian word
    auto step = [&]() -> uint32_t {
        uint32_t hi, lo, e0, e1, e2 = 0, e3 = 0, y0 = 0, y1 = 0, y2 = 0, y3 = 0;
        br.window(hi, lo);
        e0 = ent(s0);
        e1 = ent(s1);
        if (NST == 4) {
            e2 = ent(s2);
            e3 = ent(s3);
        }
        if (CELLS != kCells32) {
            y0 = sym(s0);
            y1 = sym(s1);
            if (NST == 4) {
                y2 = sym(s2);
                y3 = sym(s3);
            }
        }
        uint32_t const a0 = amt(e0), a1 = amt(e1), a01 = a0 + a1;
        uint32_t const hi2 = __funnelshift_l(lo, hi, a01); // 32 bits from the second pair's fields on
        s0 = to(e0, top(hi, a0));
        s1 = to(e1, top(__funnelshift_l(0u, hi, a0), a1));
        if (NST == 2) { // the second pair's lookups follow the first pair's
            e2 = ent(s0);
            e3 = ent(s1);
            if (CELLS != kCells32) {
                y2 = sym(s0);
                y3 = sym(s1);
            }
        }
        uint32_t const a2 = amt(e2), a3 = amt(e3), a23 = a2 + a3;
        uint32_t const f2 = top(hi2, a2), f3 = top(__funnelshift_l(0u, hi2, a2), a3);
        if (NST == 4) {
            s2 = to(e2, f2);
            s3 = to(e3, f3);
        } else {
            s0 = to(e2, f2);
            s1 = to(e3, f3);
        }
        br.pos -= int32_t((a01 & 31u) + (a23 & 31u));
        if (CELLS == kCells32) return __byte_perm(__byte_perm(e0, e1, 0x0051), __byte_perm(e2, e3, 0x0051), 0x5410);
        return __byte_perm(__byte_perm(y0, y1, 0x0040), __byte_perm(y2, y3, 0x0040), 0x5410);
    };
    uint32_t i = 0;
    uint32_t const head = min(n, uint32_t((16 - (reinterpret_cast<uintptr_t>(out) & 15)) & 15));
    for (; i < head; i++) single(i);
    for (; i + 32 <= lastTr; i += 32) {
        br.refill<3>();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint4 v;
            v.x = step();
            v.y = step();
            v.z = step();
            v.w = step();
            *reinterpret_cast<uint4*>(out + i + 16 * h) = v;
        }
    }
    for (; i + 4 <= lastTr; i += 4) {
        br.refill<1>();
        *reinterpret_cast<uint32_t*>(out + i) = step();
    }
    for (; i < n; i++) single(i);
    br.close();
    if (!br.finished()) reportError(status, DERR_CORRUPTION);
}

template <int CELLS>
__global__ void __launch_bounds__(96) kFse(const FseTask* __restrict__ tasks, uint32_t nbTasks, uint32_t lanes,
                                           uint32_t tableLogMax, uint32_t* __restrict__ status)
{
    extern __shared__ __align__(16) uint8_t smemFse[];
    uint32_t const wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t const tabBase = CELLS == kCells32 ? 0 : lanes << tableLogMax;
    uint32_t const ringOff = fseRingOff(lanes, tableLogMax, CELLS);
    // every warp builds its share of the CTA's tables, one at a time
    {
        uint16_t* const next = reinterpret_cast<uint16_t*>(smemFse + ringOff + wid * kFseScratch);
        for (uint32_t k = wid; k < lanes; k += blockDim.x >> 5) {
            uint32_t const tk = blockIdx.x * lanes + k;
            if (tk >= nbTasks) break;
            FseTask const tt = tasks[tk];
            uint8_t* const tab = smemFse + tabBase + (k << tableLogMax) * (CELLS == kCells32 ? 4 : 2);
            fseBuildWarp<CELLS>(tt, tab, CELLS == kCells32 ? tab + 1 : smemFse + (k << tableLogMax), next + 256, next);
        }
    }
    __syncthreads();
    uint32_t const ti = blockIdx.x * lanes + lane;
    if (wid != 0 || lane >= lanes || ti >= nbTasks) return;
    FseTask const t = tasks[ti];
    uint32_t const cell0 = lane << tableLogMax, area = ringOff + lane * kFseRingBytes;
    if (t.nbStates == 4) fseDecode<CELLS, 4>(t, smemFse, cell0, tabBase, area, status);
    else fseDecode<CELLS, 2>(t, smemFse, cell0, tabBase, area, status);
}

// FSE with one lane per state: a warp decodes up to eight streams, four lanes
// each (lane k of a group runs state k of its stream, k < nbStates). Symbol
// i uses state i % nbStates, so one step decodes nbStates consecutive
// symbols, one per lane. The lanes of a group keep identical copies of the
// stream's bit window (the same arithmetic on the same words); each looks up
// its own state's cell, a scan over the group's field widths (two shuffles)
// gives its field's offset below the top of the window, and the group's
// total (a third shuffle) advances every copy. The stream's ring is filled by
// the group's first lane; a full-warp __syncwarp() per step makes its
// completed copies visible to the other lanes, so the step loop is
// warp-uniform (streams of a CTA are of similar length: tasks are sorted
// longest first) and ends when no lane of the warp has a symbol left. Tables
// as kFse (one per stream, built by the whole warp).
constexpr uint32_t kFse4Variant = kTuneFseLanePerState; // Launch::tune flag (fse_shape.h)

__global__ void __launch_bounds__(32) kFse4(const FseTask* __restrict__ tasks, uint32_t nbTasks, uint32_t streams,
                                            uint32_t tableLogMax, uint32_t* __restrict__ status)
{
    extern __shared__ __align__(16) uint8_t smemFse[];
    __shared__ uint16_t sCum[260];
    __shared__ __align__(16) uint16_t sNext[256];
    uint32_t const lane = threadIdx.x;
    for (uint32_t q = 0; q < streams; q++) {
        uint32_t const tk = blockIdx.x * streams + q;
        if (tk >= nbTasks) break;
        FseTask const tt = tasks[tk];
        uint8_t* const sl = smemFse + q * fse4SlotBytes(tableLogMax);
        fseBuildWarp<kCells24Wide>(tt, sl, sl + (2u << tableLogMax), sCum, sNext);
    }
    uint32_t const grp = lane >> 2, k = lane & 3;
    uint32_t const ti = blockIdx.x * streams + grp;
    FseTask t{};
    bool ok = grp < streams && ti < nbTasks;
    if (ok) t = tasks[ti];
    uint32_t const slot = grp * fse4SlotBytes(tableLogMax);
    uint32_t* const ring = reinterpret_cast<uint32_t*>(smemFse + slot + (3u << tableLogMax));
    const uint16_t* const tab = reinterpret_cast<const uint16_t*>(smemFse + slot);
    const uint8_t* const symOf = smemFse + slot + (2u << tableLogMax);
    uint32_t const tl = t.tableLog, ns = t.nbStates;
    if (ok && ((ns != 2 && ns != 4) || tl > tableLogMax)) { // the planner admits neither
        if (k == 0) reportError(status, DERR_CORRUPTION);
        ok = false;
    }
    // stream start and ring fill (first lane of the group issues the copies)
    StreamRing<kFseRing, kFseAhead> r;
    int32_t pos = 0, end = 0;
    if (ok && !streamStart(t.bits, t.bitsSize, r.g16, pos, end)) {
        if (k == 0) reportError(status, DERR_CORRUPTION);
        ok = false;
    }
    r.ring = ring;
    r.low = 0;
    if (ok) {
        int32_t const mt = (pos - 1) >> 7;
        if (k == 0) {
            for (int32_t m = mt; m >= mt - kFseAhead; m--) r.issue(m);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        r.low = mt;
    }
    __syncwarp();
    // window: a (bits [cb + 64, cb + 96)), b, c; g = bits of the window read
    uint32_t a = 0, b = 0, c = 0;
    int32_t kb = 0, g = 0;
    if (ok) {
        int32_t const jt = (pos - 1) >> 5;
        a = jt >= 0 ? ring[jt & (4 * kFseRing - 1)] : 0u;
        b = jt - 1 >= 0 ? ring[(jt - 1) & (4 * kFseRing - 1)] : 0u;
        c = jt - 2 >= 0 ? ring[(jt - 2) & (4 * kFseRing - 1)] : 0u;
        kb = jt - 2;
        g = (kb + 3) * 32 - pos;
    }
    // the group's fields of one step: lane k reads nb bits below the k-th
    // lower lanes' fields; returns the field, sets the group's total
    auto fields = [&](uint32_t nb, uint32_t& total) -> uint32_t {
        uint32_t x = nb;
        uint32_t const y1 = __shfl_up_sync(0xffffffffu, x, 1, 4);
        if (k >= 1) x += y1;
        uint32_t const y2 = __shfl_up_sync(0xffffffffu, x, 2, 4);
        if (k >= 2) x += y2;
        total = __shfl_sync(0xffffffffu, x, 3, 4);
        uint32_t const off = x - nb; // <= 36
        uint32_t const hi = __funnelshift_lc(b, a, uint32_t(g));
        uint32_t const lo = __funnelshift_lc(c, b, uint32_t(g));
        uint32_t const w = off < 32 ? __funnelshift_l(lo, hi, off) : (lo << (off - 32));
        return __funnelshift_rc(w, 0u, 32u - nb);
    };
    // drop n bits (n <= 48, g <= 32): one or two words from the ring
    auto advance = [&](uint32_t n) {
        // the next two words below the window must be in the ring
        int32_t const m = (kb - 2) >> 2;
        if (ok && m < r.low) {
            r.low = m;
            if (k == 0) {
                r.issue(m - kFseAhead);
                asm volatile("cp.async.wait_group %0;" ::"n"(kFseAhead) : "memory");
            }
        }
        __syncwarp();
        // a lane without a stream has no ring (its slot may lie past the CTA's memory)
        uint32_t const w1 = ok ? ring[(kb - 1) & (4 * kFseRing - 1)] : 0u;
        uint32_t const w2 = ok ? ring[(kb - 2) & (4 * kFseRing - 1)] : 0u;
        g += int32_t(n);
        bool const one = g > 32, two = g > 64;
        uint32_t const na = two ? c : (one ? b : a);
        uint32_t const nb2 = two ? w1 : (one ? c : b);
        uint32_t const nc = two ? w2 : (one ? w1 : c);
        a = na;
        b = nb2;
        c = nc;
        int32_t const kk = int32_t(one) + int32_t(two);
        kb -= kk;
        g -= 32 * kk;
    };
    // initial states: state k is the k-th field of tableLog bits from the top
    uint32_t st = 0, total = 0;
    {
        bool const mine = ok && k < ns;
        uint32_t const f = fields(mine ? tl : 0u, total);
        st = f;
        advance(total);
    }
    uint32_t const n = ok ? t.dstSize : 0;
    uint32_t const lastTr = n > ns ? n - ns : 0; // symbols [0, lastTr) have a transition
    uint8_t* const out = t.out;
    for (uint32_t i = 0;; i += ns) {
        bool const act = ok && k < ns && i + k < n;
        if (!__any_sync(0xffffffffu, act)) break;
        bool const tr = act && i + k < lastTr;
        uint32_t const e = act ? uint32_t(tab[st]) : 0u;
        uint32_t const y = act ? uint32_t(symOf[st]) : 0u;
        uint32_t const f = fields(tr ? (e & 15u) : 0u, total);
        if (tr) st = (e >> 4) + f;
        if (act) out[i + k] = uint8_t(y);
        advance(total);
    }
    if (k == 0) asm volatile("cp.async.wait_all;" ::: "memory"); // no copy outlives the lane
    if (ok && k == 0 && (kb + 3) * 32 - g != end) reportError(status, DERR_CORRUPTION);
}

// ---------------------------------------------------------------------------
// One Huffman stream on several lanes. A decoder that starts inside a code
// soon meets the true code boundaries, so the stream's bits are cut into S
// runs of about equal length, which start at a multiple of the code lengths'
// common divisor from the top, as every code does (splitStart):
//  1. each lane counts the codes of its run from its first bit, noting its
//     place kMeetBits into the run and where the last code ends;
//  2. a lane whose run truly starts elsewhere (where the run before it ended)
//     counts again from there, up to the noted place if it comes by it, else
//     to the run's end; this repeats until all agree (at worst every run after
//     the one before it, as one lane would);
//  3. the counts give each run's place in the output (the caller decodes again
//     from the true starts, and stores).
// Decoding twice costs less than what it buys: a chunk's streams were four
// chains on four lanes of its table's shared memory, which bounds how many
// tables an SM holds.
// From a first bit at any place, lanes whose codes all had lengths of a common
// divisor never met the boundaries. 256 MiB of bytes, 64 MiB, 256 KiB: codes of
// 2 and 4 bits 1.50, 0.48 and 0.385 ms so, 0.57, 0.17 and 0.062 from multiples
// of 2 (0.94, 0.43 and 0.39 with one lane a stream); 4 and 8 bits 1.70, 0.51,
// 0.386 and 0.69, 0.19, 0.052. Codes nearly all of one length (31 of 5 bits,
// few of 9 to 11) meet late and stay the worst: 1.11, 0.44 and 0.20 ms (one
// lane 1.09, 0.51 and 0.42). More places to meet at (two to four, up to 4,096
// bits into the run) gained nothing.
// Lanes of about equal codes keep their windows' distance in the rings, so each
// lane's positions are moved to begin in a bank group of its own (spread): runs
// of 100 words, as codes of 3.125 bits make in a chunk of 32 K, had all lanes in
// one bank, 1.14 ms for 256 MiB and 0.61 now (geometric bytes 0.83 and 0.81).
constexpr int32_t kMeetBits = 256;
template <int T>
struct SplitShared {
    int32_t pos[T];
    uint32_t count[T];
};
struct SplitRun {
    int32_t start;          // the run's first bit (top)
    uint32_t count, before; // its codes, the codes of the stream's runs before it
    bool ok;                // the stream holds n codes and ends at its first bit
};
// Every thread of the CTA calls it. j < S: the thread's run of its stream
// (br, opened), whose first run is thread tid - j's; run(bound): decodes codes
// until the position is at or below `bound` and returns their number; step:
// lengthStep of the codes.
template <int T, class Stream, class Run>
__device__ __forceinline__ SplitRun splitStream(Stream& br, Run run, uint32_t j, uint32_t S, uint32_t step, uint32_t n,
                                                SplitShared<T>& sh)
{
    uint32_t const tid = threadIdx.x;
    bool const mine = j < S;
    int32_t p = 0, e = 0, c = 0, meet = 0, shift = 0;
    uint32_t upToMeet = 0, count = 0;
    if (mine) {
        int32_t const top = br.pos, bits = top - br.end;
        p = top - splitStart(bits, j, S, step);
        e = top - splitStart(bits, j + 1, S, step);
        shift = br.spread(p);
        p += shift;
        e += shift;
        c = max(p - kMeetBits, e);
        br.seek(p);
        upToMeet = run(c);
        meet = br.pos;
        count = upToMeet + run(e);
        sh.pos[tid] = br.pos - shift;
    }
    __syncthreads();
    int32_t used = p;
    for (;;) {
        int32_t const want = mine && j ? sh.pos[tid - 1] + shift : used;
        bool const differs = want != used;
        if (!__syncthreads_or(differs)) break;
        if (differs) {
            used = want;
            br.seek(want);
            uint32_t const m = run(c);
            if (br.pos == meet) {
                count += m - upToMeet;
            } else {
                meet = br.pos;
                count = m + run(e);
                sh.pos[tid] = br.pos - shift;
            }
            upToMeet = m;
        }
        __syncthreads();
    }
    sh.count[tid] = mine ? count : 0;
    __syncthreads();
    SplitRun r{ used, count, 0, false };
    if (mine) {
        uint32_t total = 0;
        for (uint32_t k = 0; k < S; k++) {
            if (k == j) r.before = total;
            total += sh.count[tid - j + k];
        }
        r.ok = total == n && sh.pos[tid - j + S - 1] == br.end - shift;
    }
    return r;
}

// Huffman: weights -> canonical table (symbols ranked by weight then value;
// weight w spans 2^(w-1) cells, nbBits = tableLog + 1 - w), after
// src/openzl/fse/decompress/huf_decompress.c:342-454. One CTA of T threads per
// chunk: T / 4 lanes for each stream of a 4X chunk, all for a 1X one
// (splitStream). The table (16-bit cells: symbol << 8 | nbBits) has room for
// tableLog 11, the largest the reference's encoder emits
// (encode_entropy_binding.c:222, HUF_TABLELOG_DEFAULT); at tableLog 12 it takes
// the rings' room too, and one lane a stream decodes.
//
// What bounds it: a symbol's code length comes from a table lookup, so a lane
// is a chain of lookups (shift, address, shared-memory load, shift: 43
// cycles). With four lanes a chunk, 48 chunks an SM held six warps, each
// stalled five cycles of six, and a lone chunk left the SM idle. Several lanes
// a stream end both, at two decodes; where chunks fill the GPU the lookups'
// bank conflicts (each of a warp's 32 hits about 3.4 deep) bound it instead.
// What leaves the chain: the window is loaded by position once per four
// symbols (PosStream), a cell's low five bits are the shift amount, refills are
// a predicated copy per eight symbols, 16 symbols share a store.
// A 256 MiB timestamp frame (4,224 chunks of 32 KiB): 0.46 ms with a register
// window and one lane a stream, 0.33 with the present step, 0.32 now; one
// chunk of about 100,000 symbols: 1.12, 0.75 and 0.095 ms.
constexpr uint32_t kHufTableLog = 12;
using HufStream = PosStream<8, 4, true>;
struct HufScratch {
    uint32_t count[16], next[16];
    uint32_t step; // lengthStep of the codes
    uint8_t sorted[256];
};
// table, rings (or a tableLog-12 table and the rings of four lanes), scratch
template <int T>
struct HufSmem {
    static constexpr uint32_t kRings = 2u << 11, kWideRings = 2u << 12;
    static constexpr uint32_t kUsed = kRings + T * HufStream::kBytes, kWide = kWideRings + 4 * HufStream::kBytes;
    static constexpr uint32_t kScratch = kUsed > kWide ? kUsed : kWide, kBytes = kScratch + sizeof(HufScratch);
};

// Ranks the symbols by weight (every lane of the warp calls it): count[w]
// symbols of weight w in `sorted`, from the sum of the counts below w.
// Returns the table log, 0 if the weights are not valid.
__device__ __forceinline__ uint32_t hufRankWarp(const uint8_t* weights, uint32_t nbW, HufScratch& S)
{
    uint32_t const lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    if (nbW > 256) return 0;
    if (lane < 16) S.count[lane] = 0;
    __syncwarp();
    bool bad = false;
    for (uint32_t b = 0; b < nbW; b += 32) {
        uint32_t w = b + lane < nbW ? weights[b + lane] : 0u;
        bad |= w > kHufTableLog;
        w &= 15u;
        uint32_t const m = __match_any_sync(0xffffffffu, w);
        if (lane == 31u - __clz(m)) S.count[w] += __popc(m);
        __syncwarp();
    }
    if (__any_sync(0xffffffffu, bad)) return 0;
    uint32_t const c = lane >= 1 && lane <= kHufTableLog ? S.count[lane] : 0u;
    uint32_t symbols = c, cells = lane ? c << (lane - 1) : 0u;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        uint32_t const ys = __shfl_up_sync(0xffffffffu, symbols, o), yc = __shfl_up_sync(0xffffffffu, cells, o);
        if (lane >= uint32_t(o)) {
            symbols += ys;
            cells += yc;
        }
    }
    if (lane <= kHufTableLog) S.next[lane] = symbols - c;
    __syncwarp();
    uint32_t const sum = __shfl_sync(0xffffffffu, cells, kHufTableLog), nz = __shfl_sync(0xffffffffu, symbols, kHufTableLog);
    if (sum == 0 || (sum & (sum - 1)) || nz < 2) return 0;
    uint32_t const tl = 31 - __clz(sum);
    if (tl > kHufTableLog) return 0;
    // bit w of the ballot is length tl + 1 - w
    uint32_t const used = __ballot_sync(0xffffffffu, c != 0);
    if (lane == 0) S.step = lengthStep(__brev(used) >> (30 - tl));
    for (uint32_t b = 0; b < nbW; b += 32) {
        uint32_t const w = b + lane < nbW ? weights[b + lane] : 0u;
        uint32_t const m = __match_any_sync(0xffffffffu, w);
        uint32_t const at = S.next[w];
        __syncwarp();
        if (w) {
            if (lane == 31u - __clz(m)) S.next[w] = at + __popc(m);
            S.sorted[at + __popc(m & lt)] = uint8_t(b + lane);
        }
        __syncwarp();
    }
    return tl;
}

// Fills the cells of a table from the ranked symbols, one weight after another
// (every thread of the CTA calls it); two cells a store where a symbol has them.
template <int T>
__device__ __forceinline__ void hufFill(const HufScratch& S, uint32_t tl, uint16_t* tab)
{
    uint32_t const lane = threadIdx.x;
    uint32_t base = 0, start = 0;
    for (uint32_t w = 1; w <= tl; w++) {
        uint32_t const c = S.count[w], nb = tl + 1 - w;
        if (w == 1) {
            for (uint32_t j = lane; j < c; j += T) tab[j] = uint16_t((uint32_t(S.sorted[j]) << 8) | nb);
        } else { // the weight's first cell is a multiple of its symbols' spans
            uint32_t* const d = reinterpret_cast<uint32_t*>(tab + start);
            for (uint32_t j = lane; j < c << (w - 2); j += T)
                d[j] = ((uint32_t(S.sorted[base + (j >> (w - 2))]) << 8) | nb) * 0x10001u;
        }
        base += c;
        start += c << (w - 1);
    }
}

template <int T>
__global__ void __launch_bounds__(T) kHuf(const HufTask* __restrict__ tasks, uint32_t* __restrict__ status)
{
    using M = HufSmem<T>;
    __shared__ __align__(16) uint8_t smem[M::kBytes];
    __shared__ SplitShared<T> split;
    __shared__ uint32_t sTl;
    HufTask const t = tasks[blockIdx.x];
    HufScratch& S = *reinterpret_cast<HufScratch*>(smem + M::kScratch);
    uint32_t const tid = threadIdx.x;
    if (tid < 32) {
        uint32_t const r = hufRankWarp(t.weights, t.nbWeights, S);
        if (tid == 0) sTl = r;
    }
    __syncthreads();
    uint32_t const tl = sTl;
    // the streams' places (the whole CTA agrees on them)
    bool ok = tl != 0;
    uint32_t const lanes = t.x4 ? T / 4 : T, sIdx = tid / lanes, j = tid % lanes; // lanes of a stream, stream, run
    uint32_t size = t.bitsSize, off = 0, o0 = 0, n = t.dstSize;
    if (t.x4 && ok) {
        ok = t.bitsSize >= 10;
        if (ok) {
            uint32_t const l1 = t.bits[0] | (t.bits[1] << 8);
            uint32_t const l2 = t.bits[2] | (t.bits[3] << 8);
            uint32_t const l3 = t.bits[4] | (t.bits[5] << 8);
            uint32_t const seg = (t.dstSize + 3) / 4;
            ok = 6ull + l1 + l2 + l3 <= t.bitsSize && 3ull * seg <= t.dstSize;
            off = 6 + (sIdx > 0 ? l1 : 0) + (sIdx > 1 ? l2 : 0) + (sIdx > 2 ? l3 : 0);
            size = sIdx == 0 ? l1 : sIdx == 1 ? l2 : sIdx == 2 ? l3 : t.bitsSize - 6 - l1 - l2 - l3;
            o0 = seg * sIdx;
            n = sIdx == 3 ? t.dstSize - 3 * seg : seg;
        }
    }
    if (!ok) {
        if (tid == 0) reportError(status, DERR_CORRUPTION);
        return;
    }
    hufFill<T>(S, tl, reinterpret_cast<uint16_t*>(smem));
    bool const wide = tl > 11;
    HufStream br;
    uint32_t const area = wide ? M::kWideRings + (sIdx & 3) * HufStream::kBytes : M::kRings + tid * HufStream::kBytes;
    bool const opened = br.open(t.bits + off, size, smem, area);
    uint32_t const runs = !opened ? 0 : wide ? 1 : splitRuns(br.pos - br.end, lanes);
    __syncthreads(); // the table is filled
    uint32_t const sh = 32u - tl;
    // the cell of the code at the top of hi; its low five bits are the shift amount
    auto cell = [&](uint32_t hi) -> uint32_t { return *reinterpret_cast<const uint16_t*>(smem + 2 * (hi >> sh)); };
    auto four = [&]() -> uint32_t {
        uint32_t hi, lo, c[4];
        br.window(hi, lo);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            c[k] = cell(hi);
            if (k < 3) {
                hi = __funnelshift_l(lo, hi, c[k]);
                if (k < 2) lo = __funnelshift_l(0u, lo, c[k]);
            }
        }
        // lengths are at most 12, so four add up within a cell's low byte
        br.pos -= int32_t((c[0] + c[1] + c[2] + c[3]) & 255u);
        return __byte_perm(__byte_perm(c[0], c[1], 0x0051), __byte_perm(c[2], c[3], 0x0051), 0x5410);
    };
    auto one = [&]() -> uint32_t {
        uint32_t hi, lo;
        br.refill<1>();
        br.window(hi, lo);
        uint32_t const c = cell(hi);
        br.pos -= int32_t(c & 31u);
        return c >> 8;
    };
    auto run = [&](int32_t bound) -> uint32_t { // eight codes are at most 96 bits, twelve bytes
        uint32_t m = 0;
        for (; br.pos - bound >= 96; m += 8) {
            br.refill<1>();
            four();
            four();
        }
        if (br.pos - bound >= 48) {
            br.refill<1>();
            four();
            m += 4;
        }
        for (; br.pos > bound; m++) one();
        return m;
    };
    SplitRun const r = splitStream<T>(br, run, j, runs, S.step, n, split);
    if (j >= runs) {
        if (!opened && j == 0) reportError(status, DERR_CORRUPTION);
        return;
    }
    if (!r.ok) {
        if (j == 0) reportError(status, DERR_CORRUPTION);
        br.close();
        return;
    }
    br.seek(r.start);
    uint8_t* const out = t.out + o0 + r.before;
    uint32_t const cnt = r.count, head = min(cnt, uint32_t((16 - (reinterpret_cast<uintptr_t>(out) & 15)) & 15));
    uint32_t i = 0;
    for (; i < head; i++) out[i] = uint8_t(one());
    for (; i + 16 <= cnt; i += 16) {
        uint4 v;
        br.refill<1>();
        v.x = four();
        v.y = four();
        br.refill<1>();
        v.z = four();
        v.w = four();
        *reinterpret_cast<uint4*>(out + i) = v;
    }
    for (; i < cnt; i++) out[i] = uint8_t(one());
    br.close();
}

// ---------------------------------------------------------------------------
// 16-bit-symbol Huffman (huffman_struct_v2), one CTA per chunk. Codes reach 20
// bits, so a cell table of them would take 2^20 cells. The CTA keeps, per
// weight, the first cell and the first index into the symbols sorted by
// (weight, value): the cell range of weight w spans count[w] << (w - 1)
// cells, weight 1 (the longest code) first, and a symbol of weight w spans
// 2^(w-1) consecutive cells and codes on tableLog + 1 - w bits
// (decode_huffman_kernel.c:35-71). The weight of a code is its place among at
// most 20 ranges, so a table over its top kHuf16Log bits knows it but where a
// bucket holds a range's start (at most 20 of 4096 buckets). An entry holds
// the code length and what to add to the code to get its place among the
// sorted symbols (a range's start is a multiple of its symbols' span, since
// the ranges above it fill the rest). Codes of the other buckets find their
// range by binary search. The validity rules of
// decode_entropy_binding.c:349-412 apply: weights at most 20, at least two of
// them non-zero, the sum of 2^(w-1) a power of two. Each of the one or four
// streams is decoded by several lanes (splitStream); a stream that does not
// hold its symbols exactly, which the reference does not refuse, by one, with
// the search.
//
// What bounds it: a lane is a serial chain, a lookup and a shift a symbol
// (four symbols per 64-bit window where codes have at most 16 bits, else
// three). The search and three cached stream loads for every symbol took about
// 550 cycles. A table of whole symbols over 12 bits was no help (5.99 ms):
// 13-bit codes are the ordinary ones of large alphabets. The symbols' loads
// (L1) leave the chain: they are stored a window later.
// 98,304 symbols in four streams, geometric with mean 3000: 7.06 ms with one
// lane a stream and the search, 1.41 with the table, 0.55 now.
constexpr uint32_t kHuf16Log = 12, kHuf16Threads = 128, kHuf16Warps = kHuf16Threads / 32;
using Huf16Stream = PosStream<8, 4, true>;

__global__ void __launch_bounds__(kHuf16Threads) kHuf16(const Huf16Task* __restrict__ tasks, uint32_t* __restrict__ status)
{
    __shared__ uint32_t sCount[kHuf16Warps][32], sStart[32], sBase[32];
    __shared__ uint32_t sTl, sOk, sStep;
    __shared__ uint32_t sTab[1u << kHuf16Log];
    __shared__ __align__(16) uint8_t sRing[kHuf16Threads * Huf16Stream::kBytes];
    __shared__ SplitShared<kHuf16Threads> split;
    Huf16Task const t = tasks[blockIdx.x];
    uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    sCount[wid][lane] = 0;
    if (tid == 0) sOk = 1;
    __syncthreads();
    // every warp takes a run of symbols: counts per weight, then each warp's
    // first place among the symbols of a weight, then the places
    uint32_t const share = ((t.nbWeights + kHuf16Threads - 1) / kHuf16Threads) * 32;
    uint32_t const b0 = min(t.nbWeights, wid * share), b1 = min(t.nbWeights, b0 + share);
    bool bad = false;
    for (uint32_t b = b0; b < b1; b += 32) {
        uint32_t w = b + lane < b1 ? t.weights[b + lane] : 0u;
        if (w > 20) {
            bad = true;
            w = 0;
        }
        uint32_t const m = __match_any_sync(0xffffffffu, w);
        if (lane == 31u - __clz(m)) sCount[wid][w] += __popc(m);
        __syncwarp();
    }
    if (bad) sOk = 0;
    __syncthreads();
    if (tid == 0) {
        uint64_t sum = 0;
        uint32_t nz = 0, total[21];
        for (uint32_t w = 1; w <= 20; w++) {
            total[w] = 0;
            for (uint32_t k = 0; k < kHuf16Warps; k++) total[w] += sCount[k][w];
            nz += total[w];
            sum += uint64_t(total[w]) << (w - 1);
        }
        uint32_t tl = 0;
        while (tl < 63 && (2ull << tl) <= sum) tl++;
        bool const ok = sOk && nz >= 2 && sum != 0 && !(sum & (sum - 1)) && tl <= 20;
        if (ok) {
            uint32_t pos = 0, base = 0, lengths = 0;
            for (uint32_t w = 1; w <= tl; w++) {
                lengths |= uint32_t(total[w] != 0) << (tl + 1 - w);
                sStart[w] = pos;
                sBase[w] = base;
                pos += total[w] << (w - 1);
                for (uint32_t k = 0; k < kHuf16Warps; k++) {
                    uint32_t const c = sCount[k][w];
                    sCount[k][w] = base;
                    base += c;
                }
            }
            sStart[tl + 1] = 1u << tl;
            sStep = lengthStep(lengths);
        }
        sTl = tl;
        sOk = ok ? 1u : 0u;
    }
    __syncthreads();
    if (!sOk) {
        if (tid == 0) reportError(status, DERR_CORRUPTION);
        return;
    }
    uint32_t const tl = sTl;
    for (uint32_t b = b0; b < b1; b += 32) {
        uint32_t const w = b + lane < b1 ? t.weights[b + lane] : 0u;
        uint32_t const m = __match_any_sync(0xffffffffu, w);
        uint32_t const base = sCount[wid][w];
        __syncwarp();
        if (w) {
            if (lane == 31u - __clz(m)) sCount[wid][w] = base + __popc(m);
            t.sorted[base + __popc(m & ((1u << lane) - 1u))] = uint16_t(b + lane);
        }
        __syncwarp();
    }
    __syncthreads();
    // the weight whose cell range holds cell v
    auto weightOf = [&](uint32_t v) -> uint32_t {
        uint32_t a = 1, b = tl;
        while (a < b) {
            uint32_t const mid = (a + b + 1) >> 1;
            if (sStart[mid] <= v) a = mid;
            else b = mid - 1;
        }
        return a;
    };
    // (place - code) << 5 | length of the codes of weight a
    auto entryOf = [&](uint32_t a) -> uint32_t {
        return ((sBase[a] - (sStart[a] >> (a - 1))) << 5) | (tl + 1 - a);
    };
    uint32_t const pl = min(tl, kHuf16Log);
    for (uint32_t j = tid; j < (1u << pl); j += kHuf16Threads) {
        uint32_t const a = weightOf(j << (tl - pl)), b = weightOf(((j + 1) << (tl - pl)) - 1);
        sTab[j] = a == b ? entryOf(a) : 0u;
    }
    __syncthreads();
    uint32_t const lanes = t.nbStreams == 4 ? kHuf16Threads / 4 : kHuf16Threads, sIdx = tid / lanes, j = tid % lanes;
    Huf16Stream br;
    bool const opened = br.open(t.stream[sIdx], t.streamSize[sIdx], sRing, tid * Huf16Stream::kBytes);
    uint32_t const runs = opened ? splitRuns(br.pos - br.end, lanes) : 0, n = t.count[sIdx];
    int32_t const top = br.pos;
    const uint32_t* const words = reinterpret_cast<const uint32_t*>(br.g16);
    auto symbol = [&](uint32_t hi, uint32_t e) -> uint32_t {
        return t.sorted[uint32_t(int32_t(e) >> 5) + __funnelshift_l(hi, 0u, e)];
    };
    // N codes at the position, N times the longest at most 64 bits: first as if
    // the table knew them all (an entry 0 shifts by nothing), with the search
    // only when one was not known, so that a window takes one branch. `get`
    // takes each code's place, top bits and entry.
    auto codes = [&](auto N, auto get) {
        uint32_t hi, lo, used = 0, least = ~0u;
        br.window(hi, lo);
        uint32_t const hi0 = hi, lo0 = lo;
#pragma unroll
        for (int k = 0; k < decltype(N)::value; k++) { // an entry's low five bits are the shift amount
            uint32_t const e = sTab[hi >> (32 - pl)];
            get(k, hi, e);
            used += e & 31u;
            least = min(least, e);
            hi = __funnelshift_l(lo, hi, e);
            lo = __funnelshift_l(0u, lo, e);
        }
        if (least == 0) {
            hi = hi0;
            lo = lo0;
            used = 0;
#pragma unroll
            for (int k = 0; k < decltype(N)::value; k++) {
                uint32_t e = sTab[hi >> (32 - pl)];
                if (e == 0) e = entryOf(weightOf(hi >> (32 - tl)));
                get(k, hi, e);
                used += e & 31u;
                hi = __funnelshift_l(lo, hi, e);
                lo = __funnelshift_l(0u, lo, e);
            }
        }
        br.pos -= int32_t(used);
    };
    using One = std::integral_constant<int, 1>;
    using Three = std::integral_constant<int, 3>;
    using Four = std::integral_constant<int, 4>;
    auto none = [](int, uint32_t, uint32_t) {};
    bool const narrow = tl <= 16; // four codes a window, else three
    // two windows are at most 16 bytes
    auto run = [&](int32_t bound) -> uint32_t {
        uint32_t m = 0;
        while (br.pos - bound >= 128) {
            br.refill<1>();
            if (narrow) {
                codes(Four(), none);
                codes(Four(), none);
                m += 8;
            } else {
                codes(Three(), none);
                codes(Three(), none);
                m += 6;
            }
        }
        for (; br.pos > bound; m++) {
            br.refill<1>();
            codes(One(), none);
        }
        return m;
    };
    SplitRun const r = splitStream<int(kHuf16Threads)>(br, run, j, runs, sStep, n, split);
    if (j >= runs) {
        if (!opened && j == 0 && sIdx < t.nbStreams) reportError(status, DERR_CORRUPTION);
        return;
    }
    uint8_t* const out = t.out + 2ull * (t.dstOff[sIdx] + (r.ok ? r.before : 0));
    auto put = [&](uint32_t k, uint32_t y) {
        if (!(reinterpret_cast<uintptr_t>(out) & 1)) {
            reinterpret_cast<uint16_t*>(out)[k] = uint16_t(y);
        } else {
            out[2 * k] = uint8_t(y);
            out[2 * k + 1] = uint8_t(y >> 8);
        }
    };
    if (!r.ok) { // not exactly n symbols: the first lane decodes n, one by one
        br.close();
        if (j) return;
        // The words come from memory: a stream of too few bits reads below its
        // first 16-byte block, where the ring would hold anything at all. There
        // the block's first word stands in.
        int32_t pos = top;
        for (uint32_t i = 0; i < n; i++) {
            int32_t const k = (pos - 1) >> 5;
            uint32_t const a = __ldg(words + max(k, 0)), b = __ldg(words + max(k - 1, 0));
            uint32_t const hi = __funnelshift_l(b, a, uint32_t(32 * (k + 1) - pos));
            uint32_t const e = entryOf(weightOf(hi >> (32 - tl)));
            put(i, symbol(hi, e));
            pos -= int32_t(e & 31u);
        }
        return;
    }
    br.seek(r.start);
    uint32_t const cnt = r.count;
    uint32_t i = 0;
    auto single = [&]() {
        br.refill<1>();
        uint32_t y = 0;
        codes(One(), [&](int, uint32_t hi, uint32_t e) { y = symbol(hi, e); });
        put(i, y);
    };
    if (narrow && !(reinterpret_cast<uintptr_t>(out) & 1)) {
        uint32_t const head = min(cnt, uint32_t((8 - (reinterpret_cast<uintptr_t>(out) & 7)) & 7) >> 1);
        for (; i < head; i++) single();
        uint32_t y[4] = {}, i0 = i;
        auto store = [&](uint32_t k) {
            *reinterpret_cast<uint2*>(out + 2 * k) = make_uint2(__byte_perm(y[0], y[1], 0x5410), __byte_perm(y[2], y[3], 0x5410));
        };
        for (; i + 8 <= cnt; i += 8) {
            br.refill<1>();
#pragma unroll
            for (uint32_t q = 0; q < 8; q += 4) {
                uint32_t z[4];
                codes(Four(), [&](int k, uint32_t hi, uint32_t e) { z[k] = symbol(hi, e); });
                if (i + q > i0) store(i + q - 4);
#pragma unroll
                for (int k = 0; k < 4; k++) y[k] = z[k];
            }
        }
        if (i > i0) store(i - 4);
    } else {
        uint32_t y[3] = {}, i0 = i;
        auto store = [&](uint32_t k) {
#pragma unroll
            for (int m = 0; m < 3; m++) put(k + m, y[m]);
        };
        for (; i + 6 <= cnt; i += 6) {
            br.refill<1>();
#pragma unroll
            for (uint32_t q = 0; q < 6; q += 3) {
                uint32_t z[3];
                codes(Three(), [&](int k, uint32_t hi, uint32_t e) { z[k] = symbol(hi, e); });
                if (i + q > i0) store(i + q - 3);
#pragma unroll
                for (int k = 0; k < 3; k++) y[k] = z[k];
            }
        }
        if (i > i0) store(i - 3);
    }
    for (; i < cnt; i++) single();
    br.close();
}

// ---------------------------------------------------------------------------
// XXH3-64 checksums. Phase 1: per 1 KiB block, the 16-stripe sum of every
// accumulator lane's increments (they commute within a block). Phase 2: per
// task, the block chain acc = scramble(acc + blockSum) on 8 lanes, then the
// tail stripes and the final merge on one lane (the secret and primes are
// defined above the numeric pipeline). Where the numeric pipeline writes a
// content-checksummed output, it computes that output's block sums itself
// and phase 1 skips those blocks.
__device__ __forceinline__ uint64_t fold128(uint64_t a, uint64_t b)
{
    return (a * b) ^ __umul64hi(a, b);
}
__device__ __forceinline__ uint64_t xAvalanche(uint64_t h)
{
    h ^= h >> 37;
    h *= XPMX1;
    return h ^ (h >> 32);
}
__device__ __forceinline__ uint64_t x64Avalanche(uint64_t h)
{
    h ^= h >> 33;
    h *= XP64_2;
    h ^= h >> 29;
    h *= XP64_3;
    return h ^ (h >> 32);
}
__device__ __forceinline__ uint64_t ldData(const uint8_t* p, bool aligned)
{
    if (aligned && !(reinterpret_cast<uintptr_t>(p) & 7)) return *reinterpret_cast<const uint64_t*>(p);
    uint64_t v = 0;
    for (int b = 0; b < 8; b++) v |= uint64_t(p[b]) << (8 * b);
    return v;
}
__device__ __forceinline__ uint64_t mix16(const uint8_t* in, int soff, bool al)
{
    return fold128(ldData(in, al) ^ secret64(soff), ldData(in + 8, al) ^ secret64(soff + 8));
}

__device__ uint64_t xxh3Short(const uint8_t* in, uint64_t len, bool al)
{
    if (len <= 16) {
        if (len > 8) {
            uint64_t lo = ldData(in, al) ^ (secret64(24) ^ secret64(32));
            uint64_t hi = ldData(in + len - 8, al) ^ (secret64(40) ^ secret64(48));
            uint64_t const swapped = (uint64_t(__byte_perm(uint32_t(lo), 0, 0x0123)) << 32)
                    | __byte_perm(uint32_t(lo >> 32), 0, 0x0123);
            uint64_t acc = len + swapped + hi + fold128(lo, hi);
            return xAvalanche(acc);
        }
        if (len >= 4) {
            uint64_t i1 = 0, i2 = 0;
            for (int b = 0; b < 4; b++) {
                i1 |= uint64_t(in[b]) << (8 * b);
                i2 |= uint64_t(in[len - 4 + b]) << (8 * b);
            }
            uint64_t k = (i2 + (i1 << 32)) ^ (secret64(8) ^ secret64(16));
            k ^= ((k << 49) | (k >> 15)) ^ ((k << 24) | (k >> 40));
            k *= XPMX2;
            k ^= (k >> 35) + len;
            k *= XPMX2;
            return k ^ (k >> 28);
        }
        if (len > 0) {
            uint32_t c = (uint32_t(in[0]) << 16) | (uint32_t(in[len >> 1]) << 24) | in[len - 1] | (uint32_t(len) << 8);
            return x64Avalanche(uint64_t(c) ^ uint64_t(secret32(0) ^ secret32(4)));
        }
        return x64Avalanche(secret64(56) ^ secret64(64));
    }
    if (len <= 128) {
        uint64_t acc = len * XP64_1;
        if (len > 32) {
            if (len > 64) {
                if (len > 96) {
                    acc += mix16(in + 48, 96, al);
                    acc += mix16(in + len - 64, 112, al);
                }
                acc += mix16(in + 32, 64, al);
                acc += mix16(in + len - 48, 80, al);
            }
            acc += mix16(in + 16, 32, al);
            acc += mix16(in + len - 32, 48, al);
        }
        acc += mix16(in, 0, al);
        acc += mix16(in + len - 16, 16, al);
        return xAvalanche(acc);
    }
    uint64_t acc = len * XP64_1;
    uint64_t const rounds = len / 16;
    for (uint64_t i = 0; i < 8; i++) acc += mix16(in + 16 * i, int(16 * i), al);
    acc = xAvalanche(acc);
    for (uint64_t i = 8; i < rounds; i++) acc += mix16(in + 16 * i, int(16 * (i - 8) + 3), al);
    acc += mix16(in + len - 16, 136 - 17, al);
    return xAvalanche(acc);
}

// Phase 1: one warp per 1 KiB block. Lane L holds 16 bytes of each half
// block (stripe L/4 (+8), words 2(L%4) and 2(L%4)+1), read as one aligned
// 16-byte load; for data that is not 16-byte aligned the lane funnels its
// aligned chunk with the next lane's (the last lane loads one more chunk,
// which holds at least one byte of the task's data). Each lane adds both
// words' increments (acc[i] += data[i^1] + lo32(data[i]^key[i]) * hi32(...))
// and the warp reduces over stripes.
__device__ __forceinline__ uint4 funnel16(uint4 c, uint4 n, uint32_t off)
{
    uint32_t const q = off >> 2, r = (off & 3) * 8;
    uint32_t w[4];
    switch (q) {
        case 0:
            w[0] = __funnelshift_r(c.x, c.y, r); w[1] = __funnelshift_r(c.y, c.z, r);
            w[2] = __funnelshift_r(c.z, c.w, r); w[3] = __funnelshift_r(c.w, n.x, r);
            break;
        case 1:
            w[0] = __funnelshift_r(c.y, c.z, r); w[1] = __funnelshift_r(c.z, c.w, r);
            w[2] = __funnelshift_r(c.w, n.x, r); w[3] = __funnelshift_r(n.x, n.y, r);
            break;
        case 2:
            w[0] = __funnelshift_r(c.z, c.w, r); w[1] = __funnelshift_r(c.w, n.x, r);
            w[2] = __funnelshift_r(n.x, n.y, r); w[3] = __funnelshift_r(n.y, n.z, r);
            break;
        default:
            w[0] = __funnelshift_r(c.w, n.x, r); w[1] = __funnelshift_r(n.x, n.y, r);
            w[2] = __funnelshift_r(n.y, n.z, r); w[3] = __funnelshift_r(n.z, n.w, r);
            break;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ void hashBlock(const HashTask* __restrict__ tasks, TileRef const br, const uint64_t* sKey,
                                          uint32_t lane)
{
    HashTask const t = tasks[br.task];
    const uint8_t* const blk = t.data + uint64_t(br.tile) * kHashBlock;
    uintptr_t const base = reinterpret_cast<uintptr_t>(blk) & ~uintptr_t(15);
    uint32_t const off = uint32_t(reinterpret_cast<uintptr_t>(blk) - base);
    const uint4* const A = reinterpret_cast<const uint4*>(base);
    uint32_t const j = lane & 3, sl = lane >> 2;
    uint4 c[2];
    c[0] = __ldg(A + lane);
    c[1] = __ldg(A + 32 + lane);
    if (off) {
        uint4 const ext = lane == 31 ? __ldg(A + 64) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint4 n;
            n.x = __shfl_down_sync(0xffffffffu, c[r].x, 1);
            n.y = __shfl_down_sync(0xffffffffu, c[r].y, 1);
            n.z = __shfl_down_sync(0xffffffffu, c[r].z, 1);
            n.w = __shfl_down_sync(0xffffffffu, c[r].w, 1);
            // lane 31's next chunk: round 0 -> lane 0 of round 1; round 1 -> ext
            uint32_t const x = __shfl_sync(0xffffffffu, c[1].x, 0), y = __shfl_sync(0xffffffffu, c[1].y, 0);
            uint32_t const z = __shfl_sync(0xffffffffu, c[1].z, 0), w = __shfl_sync(0xffffffffu, c[1].w, 0);
            if (lane == 31) n = r == 0 ? make_uint4(x, y, z, w) : ext;
            c[r] = funnel16(c[r], n, off);
        }
    }
    uint64_t a0 = 0, a1 = 0;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        uint32_t const st = sl + 8 * r;
        uint64_t const w0 = uint64_t(c[r].x) | (uint64_t(c[r].y) << 32);
        uint64_t const w1 = uint64_t(c[r].z) | (uint64_t(c[r].w) << 32);
        uint64_t const k0 = w0 ^ sKey[st + 2 * j], k1 = w1 ^ sKey[st + 2 * j + 1];
        a0 += w1 + uint64_t(uint32_t(k0)) * (k0 >> 32);
        a1 += w0 + uint64_t(uint32_t(k1)) * (k1 >> 32);
    }
#pragma unroll
    for (int m = 4; m < 32; m <<= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, m);
        a1 += __shfl_xor_sync(0xffffffffu, a1, m);
    }
    if (lane < 4) {
        t.blockSums[8ull * br.tile + 2 * lane] = a0;
        t.blockSums[8ull * br.tile + 2 * lane + 1] = a1;
    }
}

__global__ void __launch_bounds__(256) kHashBlocks(const HashTask* __restrict__ tasks,
                                                   const TileRef* __restrict__ blocks, uint32_t nbBlocks)
{
    __shared__ uint64_t sKey[24]; // secret words at byte offsets 0, 8, ..., 184
    if (threadIdx.x < 24) sKey[threadIdx.x] = kXxhWords.w8[threadIdx.x];
    __syncthreads();
    uint32_t const lane = threadIdx.x & 31;
    // grid-stride over the blocks, one warp per block at a time: the secret
    // is staged once per CTA
    uint32_t const nw = gridDim.x * (blockDim.x >> 5);
    for (uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); warp < nbBlocks; warp += nw)
        hashBlock(tasks, blocks[warp], sKey, lane);
}


// One step of the block chain acc = scramble(acc + sum), scramble(x) = ((x ^
// (x >> 47)) ^ key) * PRIME32_1, on y = acc + sum of the block about to be
// scrambled, in 32-bit halves; nv: the next block's sum.
//
// The chain is serial, so its latency per block bounds a long input's
// checksum. x >> 47 only reaches the low half, so with t = y.lo ^ (y.hi >> 15)
// ^ key.lo and u = y.hi ^ key.hi the next y is t * P + C with C = next sum +
// ((u * P) << 32). C needs only u and is ready before t, which leaves a shift,
// a xor, the low product (whose addition of C.lo sets the carry) and the high
// product with C.hi and that carry: 4 + 4 + 4 + 9 cycles (dependent-issue
// latencies measured one by one). One 64-bit multiply-add instead of the pair
// measured 27, and the product added to in two steps 23.
__device__ __forceinline__ void xxhChainStep(uint32_t& ylo, uint32_t& yhi, uint32_t klo, uint32_t khi, uint64_t nv)
{
    uint32_t const c = (yhi ^ khi) * XP32_1 + uint32_t(nv >> 32);
    uint32_t const t = ylo ^ (yhi >> 15) ^ klo;
    asm("mad.lo.cc.u32 %0, %2, %3, %4;\n\tmadc.hi.u32 %1, %2, %3, %5;"
        : "=&r"(ylo), "=r"(yhi) : "r"(t), "r"(XP32_1), "r"(uint32_t(nv)), "r"(c));
}

// Phase 2: a CTA of two warps per task. Lane i of the first (and its copies
// i + 8, i + 16, i + 24) runs the block chain of accumulator i, then the
// trailing partial stripes and the final stripe, and lane 0 merges. The second
// warp brings the block sums into a ring of batches of 64 blocks in shared
// memory, three ahead, so that the first does nothing but steps and a barrier
// a batch. (Sums read by the chain's own warp, 48 blocks ahead into registers,
// measured 24.2 cycles a block; staged in shared memory by that warp, 31.)
// 262,144 blocks (a 256 MiB input): 4.71 ms with two dependent multiply-adds
// and the sums staged by the warp, 2.77 ms now (20.9 cycles a block).
// The trailing stripes add to the accumulators without a chain: the four groups
// of 8 lanes take every fourth one (at most 15, and the final stripe as the
// sixteenth), loaded before the chain starts.
constexpr uint32_t kChainBatch = 64, kChainSlots = 4, kFinishThreads = 64;
__global__ void __launch_bounds__(kFinishThreads) kHashFinish(const HashTask* __restrict__ tasks, uint32_t* __restrict__ status)
{
    __shared__ __align__(16) uint64_t ring[kChainSlots][8 * kChainBatch];
    uint32_t const lane = threadIdx.x & 31, i = lane & 7, g = lane >> 3;
    HashTask const t = tasks[blockIdx.x];
    uint32_t const nb = t.len > 240 ? t.nbBlocks : 0;
    // steps that add a next sum (that of block k + 1, step k); the last block's adds none
    uint32_t const m = nb ? nb - 1 : 0, batches = (m + kChainBatch - 1) / kChainBatch;
    if (threadIdx.x >= 32) {
        auto issue = [&](uint32_t b) {
            const uint64_t* const src = t.blockSums + 8 + 8ull * kChainBatch * b;
            uint32_t const words = 8 * min(kChainBatch, b < batches ? m - kChainBatch * b : 0);
#pragma unroll
            for (uint32_t k = 2 * lane; k < 8 * kChainBatch; k += 64)
                if (k < words) {
                    uint32_t const d = uint32_t(__cvta_generic_to_shared(&ring[b % kChainSlots][k]));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + k) : "memory");
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (uint32_t b = 0; b + 1 < kChainSlots; b++) issue(b);
        for (uint32_t b = 0; b < batches; b++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kChainSlots - 2) : "memory");
            __syncthreads(); // batch b is there; batch b - 1 has been read
            issue(b + kChainSlots - 1);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    bool const al = t.aligned8 != 0;
    uint64_t h;
    if (t.len <= 240) {
        if (lane != 0) return;
        h = xxh3Short(t.data, t.len, al);
    } else {
        uint64_t const init = i == 0 ? XP32_3 : i == 1 ? XP64_1 : i == 2 ? XP64_2 : i == 3 ? XP64_3
                            : i == 4 ? XP64_4 : i == 5 ? XP32_2 : i == 6 ? XP64_5 : XP32_1;
        uint64_t const key = kXxhWords.w8[16 + i];
        uint32_t const klo = uint32_t(key), khi = uint32_t(key >> 32);
        uint64_t const len = t.len;
        uint32_t const nbStripes = uint32_t(((len - 1) - uint64_t(kHashBlock) * nb) / 64);
        const uint8_t* const last = t.data + uint64_t(kHashBlock) * nb;
        uint64_t v[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            uint32_t const st = g + 4 * j;
            const uint8_t* const p = st == 15 ? t.data + len - 64 : last + 64 * st;
            v[j] = st < nbStripes || st == 15 ? ldData(p + 8 * i, al) : 0;
        }
        uint64_t const y0 = init + (nb ? t.blockSums[i] : 0); // init + sum of block 0
        uint32_t ylo = uint32_t(y0), yhi = uint32_t(y0 >> 32);
        for (uint32_t b = 0; b < batches; b++) {
            __syncthreads();
            const uint64_t* const s = ring[b % kChainSlots] + i;
            uint32_t const cnt = min(kChainBatch, m - kChainBatch * b);
            if (cnt == kChainBatch) {
#pragma unroll
                for (uint32_t k = 0; k < kChainBatch; k++) xxhChainStep(ylo, yhi, klo, khi, s[8 * k]);
            } else {
                for (uint32_t k = 0; k < cnt; k++) xxhChainStep(ylo, yhi, klo, khi, s[8 * k]);
            }
        }
        if (nb) xxhChainStep(ylo, yhi, klo, khi, 0); // the last block
        uint64_t acc = (uint64_t(yhi) << 32) | ylo;
        uint64_t part = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            uint32_t const st = g + 4 * j;
            uint64_t const vx = __shfl_xor_sync(0xffffffffu, v[j], 1);
            uint64_t const x = v[j] ^ (st == 15 ? kXxhWords.last[i] : kXxhWords.w8[st + i]);
            if (st < nbStripes || st == 15) part += vx + uint64_t(uint32_t(x)) * (x >> 32);
        }
        part += __shfl_xor_sync(0xffffffffu, part, 8);
        part += __shfl_xor_sync(0xffffffffu, part, 16);
        acc += part;
        // merge: pairs (2k, 2k+1) folded with secret words at 11 + 16k
        uint64_t const odd = __shfl_xor_sync(0xffffffffu, acc, 1);
        part = 0;
        if (!(i & 1)) part = fold128(acc ^ kXxhWords.merge[i], odd ^ kXxhWords.merge[i + 1]);
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        part += __shfl_xor_sync(0xffffffffu, part, 4);
        if (lane != 0) return;
        h = xAvalanche(len * XP64_1 + part);
    }
    if (t.hashOut) *t.hashOut = h;
    bool const ok = t.low8 ? ((h & 255) == t.expected) : (uint32_t(h) == t.expected);
    if (!ok && t.errCode) {
        // of a frame's two checksums the compressed one is the first to be
        // verified, so its error stands whichever CTA ends first
        uint32_t const before = atomicCAS(status, 0u, t.errCode);
        if (t.errCode == DERR_COMPRESSED_CK && before == DERR_CONTENT_CK) atomicCAS(status, DERR_CONTENT_CK, DERR_COMPRESSED_CK);
    }
}

} // namespace ozl

// ---------------------------------------------------------------------------
// dispatch
namespace ozl {

namespace {
int smCount()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
            sms = n;
        if (sms <= 0) sms = 152;
    }
    return sms;
}
// Threads per chunk of an untuned Huffman launch: four warps while all chunks
// run at once (eight CTAs an SM by shared memory and threads; a round of
// host-buffer decoding took 0.2 ms where one lane a stream took 0.9), a warp
// from there on, which holds 26 chunks an SM.
uint32_t hufThreads(const Launch& l)
{
    if (l.tune) return l.tune >= 128 ? 128 : 32;
    return l.nbTasks <= 8 * uint32_t(smCount()) ? 128 : 32;
}
// kHashBlocks grid: one warp per block up to eight full CTAs per SM, then
// grid-stride (any grid size is correct)
uint32_t hashGrid(uint32_t nbBlocks)
{
    uint32_t const want = (nbBlocks + 7) / 8;
    uint32_t const cap = uint32_t(smCount()) * 8;
    return want < cap ? (want ? want : 1) : cap;
}
} // namespace

cudaError_t prepareKernels()
{
    cudaError_t e = cudaSuccess;
    for (auto* const k : { kFse<kCells32>, kFse<kCells24>, kFse<kCells24Wide> }) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kFseCtaSmem));
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(kFse4, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kFseCtaSmem));
    if (e != cudaSuccess) return e;
    return cudaSuccess;
}

uint32_t tuneCandidates(const Launch& l, uint32_t* out, uint32_t cap)
{
    uint32_t n = 0;
    if (l.kind == KIND_FSE) {
        n = fseCandidates(l.nbTasks, l.param0, uint32_t(smCount()), out, cap);
    } else if (l.kind == KIND_HUF) {
        for (uint32_t c : { 32u, 128u }) // threads per chunk
            if (n < cap) out[n++] = c;
    }
    return n;
}

long runLaunches(const DeviceLayout& L, uint8_t* dPool, uint8_t* dScratch, uint32_t* dStatus, cudaStream_t s)
{
    long count = 0;
    for (size_t i = 0; i < L.launches.size(); i++) {
        long const n = runOneLaunch(L, i, dPool, dScratch, dStatus, s);
        if (n < 0) return -1;
        count += n;
    }
    return count;
}

long runOneLaunch(const DeviceLayout& L, size_t li, uint8_t* dPool, uint8_t* dScratch, uint32_t* dStatus,
                  cudaStream_t s)
{
    long count = 0;
    {
        const Launch& l = L.launches[li];
        const void* tasks = dPool + l.taskOff;
        const TileRef* tiles = reinterpret_cast<const TileRef*>(dPool + l.tileOff);
        switch (l.kind) {
            case KIND_COPY:
                kCopy<<<l.nbTiles, 256, 0, s>>>(static_cast<const CopyTask*>(tasks), tiles);
                break;
            case KIND_CONST:
                kConst<<<l.nbTiles, 256, 0, s>>>(static_cast<const ConstTask*>(tasks), tiles);
                break;
            case KIND_FSE: {
                uint32_t const maxLanes = fseLanes(l.param0, kCells24);
                if (l.tune & kFse4Variant) { // one lane per state, up to eight streams per warp
                    uint32_t streams = l.tune & 0xFFu;
                    if (streams > 8) streams = 8;
                    if (streams > maxLanes) streams = maxLanes;
                    if (streams == 0) streams = 1;
                    uint32_t const grid = (l.nbTasks + streams - 1) / streams;
                    kFse4<<<grid, 32, streams * fse4SlotBytes(l.param0), s>>>(static_cast<const FseTask*>(tasks), l.nbTasks,
                                                                            streams, l.param0, dStatus);
                    break;
                }
                FseShape const sh(l.nbTasks, l.param0, l.tune, uint32_t(smCount()));
                uint32_t const grid = (l.nbTasks + sh.lanes - 1) / sh.lanes;
                auto* const k = sh.cells == kCells32 ? kFse<kCells32> : sh.cells == kCells24 ? kFse<kCells24>
                                                                                              : kFse<kCells24Wide>;
                k<<<grid, 32 * fseWarps(sh.lanes), fseSmemBytes(sh.lanes, l.param0, sh.cells), s>>>(
                        static_cast<const FseTask*>(tasks), l.nbTasks, sh.lanes, l.param0, dStatus);
                break;
            }
            case KIND_HUF: {
                const HufTask* const huf = static_cast<const HufTask*>(tasks);
                if (hufThreads(l) == 128) kHuf<128><<<l.nbTasks, 128, 0, s>>>(huf, dStatus);
                else kHuf<32><<<l.nbTasks, 32, 0, s>>>(huf, dStatus);
                break;
            }
            case KIND_FLATPACK:
                kFlatpack<<<l.nbTiles, 256, 0, s>>>(static_cast<const FlatpackTask*>(tasks), tiles, dStatus);
                break;
            case KIND_HUF16:
                if (l.nbTasks) kHuf16<<<l.nbTasks, kHuf16Threads, 0, s>>>(static_cast<const Huf16Task*>(tasks), dStatus);
                break;
            case KIND_WIDEN:
                kWiden<<<l.nbTiles, 256, 0, s>>>(static_cast<const WidenTask*>(tasks), tiles, dStatus);
                break;
            case KIND_TOKENIZE:
                kTokenize<<<l.nbTiles, 256, 0, s>>>(static_cast<const TokenizeTask*>(tasks), tiles, dStatus);
                break;
            case KIND_FLOATDEC:
                kFloatDec<<<l.nbTiles, 256, 0, s>>>(static_cast<const FloatDecTask*>(tasks), tiles);
                break;
            case KIND_TRANSPOSE:
                kTranspose<<<l.nbTiles, 256, 0, s>>>(static_cast<const TransposeTask*>(tasks), tiles);
                break;
            case KIND_NUMPIPE: {
                const NumPipeTask* const np = static_cast<const NumPipeTask*>(tasks);
                uint64_t* prefix = nullptr;
                if (l.needsScan) {
                    uint64_t* const sums = reinterpret_cast<uint64_t*>(dScratch + l.statusOff);
                    prefix = sums + l.nbTiles;
                    kNumReduce<<<l.nbTiles, kNPThreads, 0, s>>>(np, tiles, sums);
                    uint32_t threads = 32;
                    while (threads < 1024 && 8 * threads < l.param0) threads *= 2;
                    kNumPrefix<<<l.nbTasks, threads, 0, s>>>(np, sums, prefix);
                    count += 2;
                }
                kNumPipe<<<l.nbTiles, kNPThreads, 0, s>>>(np, tiles, prefix);
                break;
            }
            case KIND_HASH: {
                if (l.nbTiles) {
                    kHashBlocks<<<hashGrid(l.nbTiles), 256, 0, s>>>(static_cast<const HashTask*>(tasks), tiles,
                                                                   l.nbTiles);
                    count++;
                }
                kHashFinish<<<l.nbTasks, kFinishThreads, 0, s>>>(static_cast<const HashTask*>(tasks), dStatus);
                break;
            }
            default:
                return -1;
        }
        count++;
        if (cudaPeekAtLastError() != cudaSuccess) return -1;
    }
    return count;
}

} // namespace ozl

// ---------------------------------------------------------------------------
// standalone XXH3-64 of a device buffer, and launch helpers for the encoder
namespace ozl {
void launchCopy(const CopyTask* tasks, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kCopy<<<nbTiles, 256, 0, s>>>(tasks, tiles);
}

void launchHash(const HashTask* tasks, uint32_t nbTasks, const TileRef* blocks, uint32_t nbBlocks, uint32_t* status,
                cudaStream_t s)
{
    if (nbBlocks) kHashBlocks<<<hashGrid(nbBlocks), 256, 0, s>>>(tasks, blocks, nbBlocks);
    if (nbTasks) kHashFinish<<<nbTasks, kFinishThreads, 0, s>>>(tasks, status);
}

cudaError_t xxh3Device(const uint8_t* data, uint64_t len, uint64_t* dHashOut, uint8_t* dScratch,
                       uint64_t scratchBytes, cudaStream_t s)
{
    uint32_t const nbBlocks = len > 240 ? uint32_t((len - 1) / kHashBlock) : 0;
    size_t const need = 256 + size_t(nbBlocks) * (64 + sizeof(TileRef));
    if (need > scratchBytes) return cudaErrorInvalidValue;
    HashTask t{};
    t.data = data;
    t.len = len;
    t.blockSums = reinterpret_cast<uint64_t*>(dScratch + 256);
    t.nbBlocks = nbBlocks;
    t.aligned8 = (reinterpret_cast<uintptr_t>(data) & 7) == 0;
    t.hashOut = dHashOut;
    HashTask* dTask = reinterpret_cast<HashTask*>(dScratch);
    TileRef* dTiles = reinterpret_cast<TileRef*>(dScratch + 256 + size_t(nbBlocks) * 64);
    cudaError_t e = cudaMemcpyAsync(dTask, &t, sizeof(t), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    if (nbBlocks) {
        std::vector<TileRef> tiles(nbBlocks);
        for (uint32_t k = 0; k < nbBlocks; k++) tiles[k] = TileRef{ 0, k };
        e = cudaMemcpyAsync(dTiles, tiles.data(), nbBlocks * sizeof(TileRef), cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
        kHashBlocks<<<hashGrid(nbBlocks), 256, 0, s>>>(dTask, dTiles, nbBlocks);
    }
    kHashFinish<<<1, kFinishThreads, 0, s>>>(dTask, nullptr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s);
}
} // namespace ozl

// ---------------------------------------------------------------------------
// Allocation-free XXH3 (ozl_gpu_xxh3_64_static): the hash kernels above, fed
// from one file-scope device array instead of allocated scratch.
//
// Array layout: [0, 128) the task, [128, 136) the result, [256, ...) the
// per-block sums (64 bytes per 1 KiB block), then the block list (8 bytes per
// block). Nothing in it has to start at zero: each call writes the task, the
// block list and every block sum it reads, and clears the result word first.
// Calls that overlap on the GPU share the array and race.
#include "../../include/openzl_gb300.h"

namespace {

constexpr uint64_t kStaticMaxLen = OZL_XXH3_STATIC_MAX_LEN;
constexpr uint32_t kStaticMaxBlocks = uint32_t(kStaticMaxLen / ozl::kHashBlock);
constexpr size_t kStaticScratch = OZL_XXH3_STATIC_SCRATCH;
static_assert(kStaticScratch >= 256 + size_t(kStaticMaxBlocks) * (64 + sizeof(ozl::TileRef)), "scratch layout");
static_assert(sizeof(ozl::HashTask) <= 128, "task slot");

static __device__ __align__(256) uint8_t gXxh3Scratch[kStaticScratch];

// Writes the task and the block list into the array (one launch, no host copy).
__global__ void kStageHashStatic(ozl::HashTask t, ozl::HashTask* dTask, ozl::TileRef* dBlocks, uint32_t nbBlocks,
                                 uint64_t* dResult)
{
    uint32_t const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *dTask = t;
        *dResult = 0;
    }
    if (i < nbBlocks) dBlocks[i] = ozl::TileRef{ 0, i };
}

// Device address of the array in the current device's context, looked up on
// every call (no allocation): a cached address would go stale if the host
// application reset the device and the module reloaded elsewhere.
cudaError_t staticScratch(uint8_t** out)
{
    void* p = nullptr;
    cudaError_t const e = cudaGetSymbolAddress(&p, gXxh3Scratch);
    if (e != cudaSuccess) return e;
    *out = static_cast<uint8_t*>(p);
    return cudaSuccess;
}

} // namespace

extern "C" ZL_Report ozl_gpu_xxh3_64_static(const void* d_data, size_t len, void* stream)
{
    if (len > kStaticMaxLen) return ZL_Report{ ZL_ErrorCode_srcSize_tooLarge, 0 };
    if (!d_data && len) return ZL_Report{ ZL_ErrorCode_parameter_invalid, 0 };
    uint8_t* base = nullptr;
    if (staticScratch(&base) != cudaSuccess) return ZL_Report{ ZL_ErrorCode_GENERIC, 0 };
    cudaStream_t const s = static_cast<cudaStream_t>(stream);
    uint32_t const nbBlocks = len > 240 ? uint32_t((len - 1) / ozl::kHashBlock) : 0;
    auto* dTask = reinterpret_cast<ozl::HashTask*>(base);
    auto* dResult = reinterpret_cast<uint64_t*>(base + 128);
    auto* dSums = reinterpret_cast<uint64_t*>(base + 256);
    auto* dBlocks = reinterpret_cast<ozl::TileRef*>(base + 256 + size_t(kStaticMaxBlocks) * 64);
    ozl::HashTask t{};
    t.data = static_cast<const uint8_t*>(d_data);
    t.len = len;
    t.blockSums = dSums;
    t.nbBlocks = nbBlocks;
    t.aligned8 = (reinterpret_cast<uintptr_t>(d_data) & 7) == 0;
    t.hashOut = dResult;
    uint32_t const stageThreads = nbBlocks > 0 ? nbBlocks : 1;
    kStageHashStatic<<<(stageThreads + 255) / 256, 256, 0, s>>>(t, dTask, dBlocks, nbBlocks, dResult);
    if (nbBlocks) ozl::kHashBlocks<<<ozl::hashGrid(nbBlocks), 256, 0, s>>>(dTask, dBlocks, nbBlocks);
    ozl::kHashFinish<<<1, ozl::kFinishThreads, 0, s>>>(dTask, nullptr);
    if (cudaGetLastError() != cudaSuccess) return ZL_Report{ ZL_ErrorCode_GENERIC, 0 };
    uint64_t h = 0;
    if (cudaMemcpyAsync(&h, dResult, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess
        || cudaStreamSynchronize(s) != cudaSuccess)
        return ZL_Report{ ZL_ErrorCode_GENERIC, 0 };
    return ZL_Report{ ZL_ErrorCode_no_error, size_t(h) };
}

