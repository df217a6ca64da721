// sm_103a encode kernels for OpenZL's numeric codec graph.
//
// Data-parallel front ends (delta/zigzag with byte-split or bit packing),
// per-chunk histograms, and the entropy bitstreams (FSE with 2/4 interleaved
// states, Huffman 1X/4X). Bitstream kernels run a CTA or warp per chunk (FSE)
// or a warp per stream (Huffman) with the coding table in shared memory; the
// bit order restates src/openzl/fse/bitstream.h (fields appended LSB-first,
// a final 1 marker bit).
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "enc_exec.h"
#include "enc_tables.h"
#include "fse_norm.h"
#include "fse_segments.h"
#include "huf_tree.h"
#include "enc_tasks.h"
#include "stream_ring.cuh"

namespace ozl {

namespace {

__device__ __forceinline__ uint64_t ldW(const uint8_t* p, uint32_t w)
{
    uint64_t v = 0;
    if (w == 1) return *p;
    if (w == 2 && !(reinterpret_cast<uintptr_t>(p) & 1)) return *reinterpret_cast<const uint16_t*>(p);
    if (w == 4 && !(reinterpret_cast<uintptr_t>(p) & 3)) return *reinterpret_cast<const uint32_t*>(p);
    if (w == 8 && !(reinterpret_cast<uintptr_t>(p) & 7)) return *reinterpret_cast<const uint64_t*>(p);
    for (uint32_t b = 0; b < w; b++) v |= uint64_t(p[b]) << (8 * b);
    return v;
}

__device__ __forceinline__ void stW(uint8_t* p, uint64_t v, uint32_t w)
{
    if (w == 1) { *p = uint8_t(v); return; }
    if (w == 2 && !(reinterpret_cast<uintptr_t>(p) & 1)) { *reinterpret_cast<uint16_t*>(p) = uint16_t(v); return; }
    if (w == 4 && !(reinterpret_cast<uintptr_t>(p) & 3)) { *reinterpret_cast<uint32_t*>(p) = uint32_t(v); return; }
    if (w == 8 && !(reinterpret_cast<uintptr_t>(p) & 7)) { *reinterpret_cast<uint64_t*>(p) = v; return; }
    for (uint32_t b = 0; b < w; b++) p[b] = uint8_t(v >> (8 * b));
}

__device__ __forceinline__ uint64_t transformed(const EncNumTask& t, uint64_t i)
{
    uint64_t const m = t.w >= 8 ? ~0ull : ((1ull << (8 * t.w)) - 1);
    uint64_t v;
    if (t.delta) v = (ldW(t.src + (i + 1) * t.w, t.w) - ldW(t.src + i * t.w, t.w)) & m;
    else v = ldW(t.src + i * t.w, t.w);
    if (t.zigzag) {
        uint64_t const sign = (v >> (8 * t.w - 1)) & 1;
        v = ((v << 1) ^ (0 - sign)) & m;
    }
    return v;
}

// Words of a tile's packed fields in shared memory, one pad word after every
// 32 so that threads a power of two of words apart spread over the banks.
__device__ __forceinline__ uint32_t packPad(uint32_t q) { return q + (q >> 5); }

// Packs fields (LSB-first) into consecutive words from word `q` of `w`.
struct WordPacker {
    uint32_t* w;
    uint32_t q;
    uint64_t acc = 0;
    uint32_t nb = 0;
    __device__ WordPacker(uint32_t* words, uint32_t first) : w(words), q(first) {}
    // bits <= 32 of v, none above them; invariant: nb < 32 between calls
    __device__ __forceinline__ void put32(uint32_t v, uint32_t bits)
    {
        acc |= uint64_t(v) << nb;
        nb += bits;
        if (nb >= 32) {
            w[packPad(q++)] = uint32_t(acc);
            acc >>= 32;
            nb -= 32;
        }
    }
    __device__ __forceinline__ void put(uint64_t v, uint32_t bits)
    {
        if (bits <= 32) {
            put32(uint32_t(v) & uint32_t((1ull << bits) - 1), bits);
        } else {
            put32(uint32_t(v), 32);
            put32(uint32_t(v >> 32) & uint32_t((1ull << (bits - 32)) - 1), bits - 32);
        }
    }
    __device__ __forceinline__ void finish()
    {
        if (nb) w[packPad(q)] = uint32_t(acc);
    }
};

// The CTA writes `bytes` bytes of packed words to out.
__device__ __forceinline__ void storePacked(uint8_t* out, const uint32_t* w, uint32_t bytes)
{
    uint32_t const nv = reinterpret_cast<uintptr_t>(out) & 15 ? 0 : bytes >> 4;
    for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) {
        uint32_t const q = packPad(4 * v); // four words never straddle a pad
        reinterpret_cast<uint4*>(out)[v] = make_uint4(w[q], w[q + 1], w[q + 2], w[q + 3]);
    }
    for (uint32_t b = 16 * nv + threadIdx.x; b < bytes; b += blockDim.x) out[b] = uint8_t(w[packPad(b >> 2)] >> (8 * (b & 3)));
}

} // namespace

// 16 bytes of W-byte elements (u) and the element after them: delta and
// zigzag as the task has them, as little-endian words. Bytes and 16-bit
// elements are subtracted and folded several to a word.
template <int W>
__device__ __forceinline__ void encVec(const EncNumTask& t, uint4 u, uint64_t after, uint32_t (&o)[4])
{
    uint32_t const x[5] = { u.x, u.y, u.z, u.w, uint32_t(after) };
    if constexpr (W == 8) {
        uint64_t const a = uint64_t(u.x) | (uint64_t(u.y) << 32), b = uint64_t(u.z) | (uint64_t(u.w) << 32);
        uint64_t v[2] = { t.delta ? b - a : a, t.delta ? after - b : b };
#pragma unroll
        for (int e = 0; e < 2; e++) {
            if (t.zigzag) v[e] = (v[e] << 1) ^ (0 - (v[e] >> 63));
            o[2 * e] = uint32_t(v[e]);
            o[2 * e + 1] = uint32_t(v[e] >> 32);
        }
    } else {
        constexpr uint32_t hi = W == 1 ? 0x80808080u : W == 2 ? 0x80008000u : 0x80000000u; // the elements' top bits
        constexpr uint32_t ones = hi >> (8 * W - 1), full = uint32_t((1ull << (8 * W)) - 1);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t v = x[k];
            if (t.delta) { // next element minus this one, without borrows between elements
                uint32_t const y = W == 4 ? x[k + 1] : __funnelshift_r(x[k], x[k + 1], 8 * W);
                v = ((y | hi) - (x[k] & ~hi)) ^ ((y ^ ~x[k]) & hi);
            }
            if (t.zigzag) v = ((v & ~hi) << 1) ^ (((v & hi) >> (8 * W - 1) & ones) * full);
            o[k] = v;
        }
    }
}

// The element after 16-byte vector v of the source, when delta needs it: the
// source holds one element more than the outputs.
template <int W>
__device__ __forceinline__ uint64_t encAfter(const EncNumTask& t, uint64_t v)
{
    return t.delta ? ldW(t.src + 16 * (v + 1), W) : 0;
}

// ---------------------------------------------------------------------------
// Per-task OR of the transformed values: its top bit is their maximum's, which
// is the bit width that bitpack_int needs. Elements are read as 16-byte
// vectors; the vectors' elements are only told apart at the end.
template <int W>
__device__ __forceinline__ uint64_t encOr(const EncNumTask& t, uint64_t e0, uint64_t e1)
{
    uint64_t r = 0;
    uint64_t done = e0; // elements covered by whole vectors
    if (!(reinterpret_cast<uintptr_t>(t.src) & 15)) {
        constexpr uint32_t E = 16 / W;
        uint64_t const v0 = e0 / E, v1 = e1 / E; // e0 is a multiple of a tile
        uint32_t acc[4] = { 0, 0, 0, 0 };
        for (uint64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
            uint32_t o[4];
            encVec<W>(t, __ldg(reinterpret_cast<const uint4*>(t.src) + v), encAfter<W>(t, v), o);
#pragma unroll
            for (int k = 0; k < 4; k++) acc[k] |= o[k];
        }
        if constexpr (W == 8) {
            r = uint64_t(acc[0] | acc[2]) | (uint64_t(acc[1] | acc[3]) << 32);
        } else {
            uint32_t a = acc[0] | acc[1] | acc[2] | acc[3];
            if (W < 4) a |= a >> 16;
            if (W < 2) a |= a >> 8;
            r = a & uint32_t((1ull << (8 * W)) - 1);
        }
        done = v1 * E;
    }
    for (uint64_t i = done + threadIdx.x; i < e1; i += blockDim.x) r |= transformed(t, i);
    return r;
}

__global__ void __launch_bounds__(256) kEncMax(const EncNumTask* __restrict__ tasks, const TileRef* __restrict__ tiles,
                                               unsigned long long* __restrict__ maxima)
{
    __shared__ uint64_t warpOr[8];
    TileRef const tr = tiles[blockIdx.x];
    EncNumTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = min(t.n, e0 + kEncTile);
    uint64_t r;
    switch (t.w) {
        case 1: r = encOr<1>(t, e0, e1); break;
        case 2: r = encOr<2>(t, e0, e1); break;
        case 4: r = encOr<4>(t, e0, e1); break;
        default: r = encOr<8>(t, e0, e1); break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r |= __shfl_xor_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0) warpOr[threadIdx.x >> 5] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; k++) r |= warpOr[k];
        atomicOr(&maxima[t.maxSlot], (unsigned long long)r);
    }
}

// Front end: delta/zigzag, then plain elements, byte planes or packed fields,
// a tile of 4,096 elements per CTA of 128 threads. What bounds it is memory:
// each input byte is read once and each output byte written once, so every
// store of a warp should fill whole sectors.
//  - plain (and packed at the full width, which is the same bytes): a 16-byte
//    vector per thread and round;
//  - planes: sixteen elements per thread and round, a 16-byte store a plane;
//  - packed: 32 elements per thread, whose fields fill whole words, staged in
//    shared memory and written 16 bytes a thread. Stored by the threads
//    themselves, word by word, a warp's stores touched 32 sectors each.
// 2,048 mixed frames (1.24 GB): 3.74 ms before, 0.65 now (the maxima,
// kEncMax: 0.79 and 0.24).
template <int W>
__device__ __forceinline__ bool encNumTile(const EncNumTask& t, uint64_t e0, uint64_t e1, uint32_t* words)
{
    uint32_t const tid = threadIdx.x;
    const uint4* const src = reinterpret_cast<const uint4*>(t.src);
    constexpr uint32_t E = 16 / W;
    if (t.mode == EOUT_PLAIN || (t.mode == EOUT_BITPACK && t.nbBits == 8 * W)) {
        if (reinterpret_cast<uintptr_t>(t.out) & 15) return false;
        uint64_t const v1 = e1 / E;
#pragma unroll 2
        for (uint64_t v = e0 / E + tid; v < v1; v += blockDim.x) {
            uint32_t o[4];
            encVec<W>(t, __ldg(src + v), encAfter<W>(t, v), o);
            reinterpret_cast<uint4*>(t.out)[v] = make_uint4(o[0], o[1], o[2], o[3]);
        }
        for (uint64_t i = v1 * E + tid; i < e1; i += blockDim.x) stW(t.out + i * W, transformed(t, i), W);
    } else if (t.mode == EOUT_PLANES) {
        if ((reinterpret_cast<uintptr_t>(t.out) | t.planeStride) & 15) return false;
        uint64_t const whole = e0 + ((e1 - e0) & ~uint64_t(15));
        for (uint64_t i = e0 + 16 * tid; i < whole; i += 16 * blockDim.x) {
            uint32_t o[W][4]; // vector k: elements i + k E ...
            uint64_t const v = i / E;
#pragma unroll
            for (int k = 0; k < W; k++) {
                uint64_t after = 0;
                if (t.delta) after = ldW(t.src + 16 * (v + k + 1), W);
                encVec<W>(t, __ldg(src + v + k), after, o[k]);
            }
            // plane b, word q: byte b of elements 4 q .. 4 q + 3
            const uint32_t* const x = &o[0][0];
#pragma unroll
            for (int b = 0; b < W; b++) {
                uint32_t p[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if constexpr (W == 1) {
                        p[q] = x[q];
                    } else if constexpr (W == 2) {
                        p[q] = __byte_perm(x[2 * q], x[2 * q + 1], b ? 0x7531 : 0x6420);
                    } else {
                        constexpr int S = W / 4; // words an element
                        const uint32_t* const y = x + 4 * S * q + (b >> 2);
                        uint32_t const lo = __byte_perm(y[0], y[S], 0x0040 + (b & 3) * 0x0011);
                        uint32_t const hi = __byte_perm(y[2 * S], y[3 * S], 0x0040 + (b & 3) * 0x0011);
                        p[q] = __byte_perm(lo, hi, 0x5410);
                    }
                }
                *reinterpret_cast<uint4*>(t.out + b * t.planeStride + i) = make_uint4(p[0], p[1], p[2], p[3]);
            }
        }
        for (uint64_t i = whole + tid; i < e1; i += blockDim.x) {
            uint64_t const v = transformed(t, i);
            for (uint32_t b = 0; b < W; b++) t.out[b * t.planeStride + i] = uint8_t(v >> (8 * b));
        }
    } else {
        uint64_t const i0 = e0 + 32 * tid;
        if (i0 < e1) {
            WordPacker wp(words, tid * t.nbBits);
            if (i0 + 32 <= e1) {
#pragma unroll 2
                for (uint32_t k = 0; k < 32 / E; k++) {
                    uint64_t const v = i0 / E + k;
                    uint32_t o[4];
                    encVec<W>(t, __ldg(src + v), encAfter<W>(t, v), o);
#pragma unroll
                    for (uint32_t e = 0; e < E; e++) {
                        if constexpr (W == 8) wp.put(uint64_t(o[2 * e]) | (uint64_t(o[2 * e + 1]) << 32), t.nbBits);
                        else wp.put((o[(e * W) >> 2] >> (8 * ((e * W) & 3))) & uint32_t((1ull << (8 * W)) - 1), t.nbBits);
                    }
                }
            } else {
                for (uint64_t i = i0; i < e1; i++) wp.put(transformed(t, i), t.nbBits);
            }
            wp.finish();
        }
        __syncthreads();
        storePacked(t.out + (e0 >> 3) * t.nbBits, words, uint32_t(((e1 - e0) * t.nbBits + 7) >> 3));
    }
    return true;
}

constexpr uint32_t kPackWords = kEncTile / 32 * 64; // words of a tile's 64-bit fields

__global__ void __launch_bounds__(128) kEncNum(const EncNumTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    __shared__ uint32_t words[kPackWords + kPackWords / 32 + 1];
    TileRef const tr = tiles[blockIdx.x];
    EncNumTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = min(t.n, e0 + kEncTile);
    if (!(reinterpret_cast<uintptr_t>(t.src) & 15)) {
        bool done = false;
        switch (t.w) {
            case 1: done = encNumTile<1>(t, e0, e1, words); break;
            case 2: done = encNumTile<2>(t, e0, e1, words); break;
            case 4: done = encNumTile<4>(t, e0, e1, words); break;
            case 8: done = encNumTile<8>(t, e0, e1, words); break;
            default: break;
        }
        if (done) return;
    }
    if (t.mode == EOUT_BITPACK) { // 32 fields start at a word
        uint64_t const i0 = e0 + 32 * threadIdx.x;
        if (i0 < e1) {
            WordPacker wp(words, threadIdx.x * t.nbBits);
            for (uint64_t i = i0; i < min(e1, i0 + 32); i++) wp.put(transformed(t, i), t.nbBits);
            wp.finish();
        }
        __syncthreads();
        storePacked(t.out + (e0 >> 3) * t.nbBits, words, uint32_t(((e1 - e0) * t.nbBits + 7) >> 3));
        return;
    }
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
        uint64_t const v = transformed(t, i);
        if (t.mode == EOUT_PLAIN) stW(t.out + i * t.w, v, t.w);
        else
            for (uint32_t b = 0; b < t.w; b++) t.out[b * t.planeStride + i] = uint8_t(v >> (8 * b));
    }
}

// Serial bit packing / flatpack indices (fields of at most 8 bits): 32
// elements per thread, read as two vectors and packed into whole words in
// shared memory, the flatpack map there too; written 16 bytes a thread. With
// byte loads, map lookups in global memory and word stores by each thread the
// flatpack streams of 2,048 mixed frames took 1.68 ms, now 0.21.
__global__ void __launch_bounds__(128) kPack(const PackTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    constexpr uint32_t kWords = kEncTile / 32 * 8 + 1; // and the word that a terminator may open
    __shared__ uint32_t words[kWords + kWords / 32 + 1];
    __shared__ uint8_t map[256];
    TileRef const tr = tiles[blockIdx.x];
    PackTask const t = tasks[tr.task];
    uint32_t const tid = threadIdx.x;
    if (t.map)
        for (uint32_t y = tid; y < 256; y += 128) map[y] = t.map[y];
    __syncthreads();
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile, e1 = min(t.n, e0 + kEncTile), i0 = e0 + 32 * tid;
    bool const ends = t.map && e1 == t.n; // the tile holds the terminator
    if (i0 < e1) {
        WordPacker wp(words, tid * t.nbBits);
        uint32_t const cnt = uint32_t(min(uint64_t(32), e1 - i0));
        if (cnt == 32 && !(reinterpret_cast<uintptr_t>(t.src) & 15)) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint4 const u = __ldg(reinterpret_cast<const uint4*>(t.src + i0) + h);
                uint32_t const x[4] = { u.x, u.y, u.z, u.w };
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    uint32_t const y = (x[k >> 2] >> (8 * (k & 3))) & 0xffu;
                    wp.put(t.map ? map[y] : y, t.nbBits);
                }
            }
        } else {
            for (uint32_t k = 0; k < cnt; k++) {
                uint32_t const y = t.src[i0 + k];
                wp.put(t.map ? map[y] : y, t.nbBits);
            }
        }
        if (ends && i0 + cnt == t.n) wp.put(1, 1);
        wp.finish();
    }
    __syncthreads();
    storePacked(t.out + (e0 >> 3) * t.nbBits, words, uint32_t(((e1 - e0) * t.nbBits + (ends ? 1 : 0) + 7) >> 3));
}

// 256-bin histogram of one chunk per CTA: sixteen copies of each bin, one for
// every second lane, side by side (banks differ, so equal bytes in a warp meet
// at most in pairs), read 16 bytes a thread.
// Chunks of 2,048 mixed frames: 0.82 ms with eight copies by thread, 0.32 now.
constexpr uint32_t kHistCopies = 16;
__global__ void __launch_bounds__(256) kHist(const HistTask* __restrict__ tasks, uint32_t* __restrict__ hists)
{
    __shared__ uint32_t h[256 * kHistCopies];
    HistTask const t = tasks[blockIdx.x];
    uint32_t const tid = threadIdx.x;
    for (uint32_t k = tid; k < 256 * kHistCopies; k += 256) h[k] = 0;
    __syncthreads();
    uint32_t* const mine = h + (tid & (kHistCopies - 1));
    uint32_t const n = t.n;
    auto count = [&](uint32_t y) { atomicAdd(mine + y * kHistCopies, 1u); };
    uint32_t const head = min(n, uint32_t(-reinterpret_cast<intptr_t>(t.src) & 15));
    const uint4* const src = reinterpret_cast<const uint4*>(t.src + head);
    uint32_t const nv = (n - head) >> 4;
    for (uint32_t v = tid; v < nv; v += 256) {
        uint4 const u = __ldg(src + v);
        uint32_t const x[4] = { u.x, u.y, u.z, u.w };
#pragma unroll
        for (int k = 0; k < 16; k++) count((x[k >> 2] >> (8 * (k & 3))) & 0xffu);
    }
    if (tid < head) count(t.src[tid]);
    for (uint32_t i = head + 16 * nv + tid; i < n; i += 256) count(t.src[i]);
    __syncthreads();
    uint32_t s = 0;
#pragma unroll
    for (uint32_t r = 0; r < kHistCopies; r++) s += h[tid * kHistCopies + ((r + tid) & (kHistCopies - 1))];
    hists[uint64_t(t.outIndex) * 256 + tid] = s;
}

// FSE coding tables on the device, a warp or a CTA of four per chunk: the
// histogram is normalized (fse_norm.h; a lane has eight symbols, a sum and a
// maximum over the warp give the remainder and the symbol that takes it, sums
// and a scan the second method), the encoding table is built
// (FSE_buildCTable_wksp, fse_compress.c:69-207) and the normalized-count
// header written (fseHeader). Cells: the count -1 symbols take the top cells in
// symbol order; occurrence k of the other symbols (in symbol order, each
// repeated count times) goes to the k-th cell of the sequence 0, step,
// 2 step, ... (mod size) below the top cells, 32 positions per round ranked
// by a ballot. States: a symbol's state slots, from its cumulative count,
// take its cells in increasing order, ranked within the round by
// __match_any_sync; with four warps, each takes a quarter of the rounds, from
// the occurrences before it (counted) and from the symbols' cells in the
// quarters before it (a count in shared memory first). The result equals the
// serial construction.
//
// What bounds it: the chain of rounds, each a ballot or match and dependent
// shared loads (64 and 64 at table log 11). With normalization and header on
// one lane a chunk took 72 us, a quarter of a small encode call; on 32 lanes
// 35 us, with four warps 15.7 us. 64 messages, some for the second method: 84 us
// while that ran on one lane, now 24.
constexpr int kFseTabWarps = 4;
// Up to this many chunks take a CTA each, beyond it a warp each (chunks of 32 K
// symbols; a warp and a CTA each): 4 chunks 37 and 18 us, 1,024 44 and 35, 2,048
// 60 and 60, 4,096 91 and 106, where the repeated normalization costs more
// than the shorter rounds give.
constexpr uint32_t kFseTabWide = 2048;
struct FseBuildSmem {
    uint32_t count[256];
    int16_t norm[256];
    uint16_t posCum[260];  // occurrences before each symbol (positive counts)
    uint16_t cumul[260];   // state slots before each symbol (count -1 takes one)
    uint32_t header[132]; // at most 2 + 2 * 256 + 2 bytes
    uint8_t symbolAt[2048];
};

// The normalized-count header (fseWriteNCountTo) by a whole warp: lane j holds
// the normalized counts v of symbols 8j .. 8j + 7 and `slots`, the table's
// cells before them. What a symbol writes depends on those before it by that
// sum alone: the field's width follows from the cells that remain, and the
// first zero of a run writes the run. Returns the bytes.
__device__ __forceinline__ uint32_t fseHeader(uint32_t* header, const int (&v)[8], uint32_t slots, uint32_t maxSym,
                                              uint32_t tl)
{
    uint32_t const lane = threadIdx.x & 31;
    for (uint32_t i = lane; i < 132; i += 32) header[i] = i == 0 ? tl - 5 : 0u;
    // the first symbol from the lane's last on that is not zero
    int next = 512;
#pragma unroll
    for (int k = 7; k >= 0; k--) next = v[k] ? int(8 * lane + k) : next;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { // the least of the lane's and those above
        int const y = __shfl_down_sync(0xffffffffu, next, o);
        if (lane + o < 32) next = min(next, y);
    }
    next = __shfl_down_sync(0xffffffffu, next, 1);
    if (lane == 31) next = 512;
    bool zero = __shfl_up_sync(0xffffffffu, v[7], 1) == 0 && lane > 0; // the symbol before is zero
    // fields (bits 0-11), their widths (12-16), and for a run's first zero the zeros that follow, plus 1 (17 on)
    uint32_t f[8], bits = 0;
    int remaining = int((1u << tl) + 1 - slots);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        f[k] = 0;
        uint32_t const sy = 8 * lane + k;
        if (sy <= maxSym && remaining > 1 && (v[k] || !zero)) {
            int const lg = ent::highbit32v(uint32_t(remaining)), threshold = 1 << lg, most = 2 * threshold - 1 - remaining;
            int c = v[k] + 1;
            if (c >= threshold) c += most;
            uint32_t const w = uint32_t(lg) + 1 - uint32_t(c < most);
            f[k] = uint32_t(c) | (w << 12);
            bits += w;
            if (!v[k]) {
                int to = next;
#pragma unroll
                for (int j = 7; j > 0; j--)
                    if (j > k && v[j]) to = int(8 * lane + j);
                if (to == 512) to = int(sy) + 1; // (no symbol at all)
                uint32_t const run = uint32_t(to) - sy - 1;
                f[k] |= (run + 1) << 17;
                bits += 16 * (run / 24) + 2 * (run % 24 / 3) + 2;
            }
        }
        zero = v[k] == 0;
        remaining -= v[k] < 0 ? 1 : v[k];
    }
    uint32_t at = bits;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t const y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= uint32_t(o)) at += y;
    }
    uint32_t const total = 4 + __shfl_sync(0xffffffffu, at, 31);
    at += 4 - bits;
    __syncwarp();
    auto put = [&](uint32_t x, uint32_t n) {
        atomicOr(&header[at >> 5], x << (at & 31));
        if ((at & 31) + n > 32) atomicOr(&header[(at >> 5) + 1], x >> (32 - (at & 31)));
        at += n;
    };
#pragma unroll
    for (int k = 0; k < 8; k++) {
        uint32_t const w = (f[k] >> 12) & 31u;
        if (w) put(f[k] & 0xfffu, w);
        if (f[k] >> 17) {
            uint32_t const run = (f[k] >> 17) - 1;
            for (uint32_t i = 0; i < run / 24; i++) put(0xffffu, 16);
            uint32_t const threes = run % 24 / 3;
            put((1u << (2 * threes)) - 1 + ((run % 3) << (2 * threes)), 2 * threes + 2);
        }
    }
    __syncwarp();
    return (total + 7) >> 3;
}

// fseNormalizeM2 by a whole warp: lane j holds the counts c of symbols
// 8j .. 8j + 7 (0 from maxSym + 1 on) and gets their normalized counts v. False
// where the distribution cannot be normalized.
__device__ __forceinline__ bool fseNormalizeSecond(int (&v)[8], const uint32_t (&c)[8], uint32_t tl, uint32_t total,
                                                   uint32_t maxSym)
{
    uint32_t const lane = threadIdx.x & 31, size = 1u << tl, low = total >> tl;
    uint32_t lowOne = uint32_t((uint64_t(total) * 3) >> (tl + 1));
    uint32_t some = 0, used = 0; // symbols with their final count, and their occurrences
#pragma unroll
    for (int k = 0; k < 8; k++) {
        v[k] = c[k] == 0 ? 0 : c[k] <= low ? -1 : c[k] <= lowOne ? 1 : -2; // -2: not known yet
        if (v[k] == 1 || v[k] == -1) {
            some++;
            used += c[k];
        }
    }
    uint32_t distributed = __reduce_add_sync(0xffffffffu, some);
    total -= __reduce_add_sync(0xffffffffu, used);
    uint32_t left = size - distributed;
    if (left == 0) return true;
    if (total / left > lowOne) {
        lowOne = uint32_t((uint64_t(total) * 3) / (left * 2));
        some = used = 0;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (v[k] == -2 && c[k] <= lowOne) {
                v[k] = 1;
                some++;
                used += c[k];
            }
        distributed += __reduce_add_sync(0xffffffffu, some);
        total -= __reduce_add_sync(0xffffffffu, used);
        left = size - distributed;
    }
    if (distributed == maxSym + 1) { // the rest goes to the first of the most frequent symbols
        uint32_t most = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) most = max(most, c[k]);
        most = __reduce_max_sync(0xffffffffu, most);
        uint32_t first = 256;
#pragma unroll
        for (int k = 7; k >= 0; k--) first = c[k] == most ? 8 * lane + k : first;
        first = __reduce_min_sync(0xffffffffu, first);
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (8 * lane + k == first) v[k] = int16_t(v[k] + int16_t(left));
        return true;
    }
    if (total == 0) { // one each in turn to the symbols with a positive count
        uint32_t mine = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) mine += v[k] > 0;
        uint32_t at = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t const y = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= uint32_t(o)) at += y;
        }
        uint32_t const all = __shfl_sync(0xffffffffu, at, 31);
        if (all == 0) return false;
        at -= mine;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (v[k] > 0) v[k] += int(left / all + (at++ < left % all ? 1u : 0u));
        return true;
    }
    uint32_t const stepLog = 62 - tl;
    uint64_t const mid = (uint64_t(1) << (stepLog - 1)) - 1, step = ((uint64_t(1) << stepLog) * left + mid) / total;
    uint64_t sum = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (v[k] == -2) sum += c[k] * step;
    uint64_t at = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t const y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= uint32_t(o)) at += y;
    }
    at += mid - sum;
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (v[k] == -2) {
            uint64_t const end = at + c[k] * step;
            uint32_t const w = uint32_t(end >> stepLog) - uint32_t(at >> stepLog);
            bad |= w < 1;
            v[k] = int16_t(w);
            at = end;
        }
    return !__any_sync(0xffffffffu, bad);
}

template <int W>
__global__ void __launch_bounds__(32 * kFseTabWarps) kFseTables(const FseTableTask* __restrict__ tasks, uint32_t nbTasks,
                                                                uint32_t* __restrict__ sizes,
                                                                uint32_t* __restrict__ errors)
{
    static_assert(W == 1 || W == kFseTabWarps, "warps of a chunk: one, or the CTA");
    __shared__ FseBuildSmem sm[kFseTabWarps / W];
    __shared__ uint32_t nextSlot[kFseTabWarps][256];
    uint32_t const wid = threadIdx.x >> 5, lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    uint32_t const part = W == 1 ? 0 : wid; // the chunk's warp, which takes its share of the table's cells
    uint32_t const ti = W == 1 ? blockIdx.x * kFseTabWarps + wid : blockIdx.x;
    if (ti >= nbTasks) return; // the whole warp
    auto sync = [] {
        if (W == 1) __syncwarp();
        else __syncthreads();
    };
    FseTableTask const t = tasks[ti];
    FseBuildSmem& S = sm[W == 1 ? wid : 0];
    uint32_t* const next = nextSlot[wid];
    uint32_t const tl = t.tableLog, maxSym = t.maxSym;
    uint32_t const size = 1u << tl, mask = size - 1, step = (size >> 1) + (size >> 3) + 3;
    if (tl < 5 || tl > 11 || maxSym > 255) { // outside what the encoder emits
        if (lane == 0) atomicOr(errors, 1u);
        return;
    }
    for (uint32_t k = part * 32 + lane; k < 256; k += 32 * W) {
        S.count[k] = t.hist[k];
    }
    sync();
    // (every warp of the chunk computes the same, the first one writes)
    // lane j: symbols 8j .. 8j + 7
    int v[8];
    {
        ent::FseNormScale const normOf(tl, t.n);
        uint32_t const low = uint32_t(t.n >> tl);
        uint32_t c[8];
        int still = 0, largest = 0; // largest: value, then 255 - symbol
        bool one = false;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            uint32_t const sy = 8 * lane + k;
            c[k] = sy <= maxSym ? S.count[sy] : 0u;
            one |= c[k] && c[k] == t.n;
            v[k] = c[k] == 0 ? 0 : c[k] <= low ? -1 : int(normOf(c[k]));
            still -= v[k] < 0 ? 1 : v[k];
            if (v[k] > 0) largest = max(largest, (v[k] << 8) | int(255 - sy));
        }
        still = __reduce_add_sync(0xffffffffu, still) + int(size);
        largest = __reduce_max_sync(0xffffffffu, largest);
        one = __any_sync(0xffffffffu, one);
        uint32_t const ls = largest ? 255u - uint32_t(largest & 255) : 0u;
        if (one) { // (one symbol: no counts, as there)
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = 0;
        } else if (-still >= (largest >> 9)) {
            if (!fseNormalizeSecond(v, c, tl, uint32_t(t.n), maxSym) && part == 0 && lane == 0) atomicOr(errors, 1u);
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (8 * lane + k == ls) v[k] += still;
        }
        if (part == 0) {
#pragma unroll
            for (int k = 0; k < 8; k++) S.norm[8 * lane + k] = int16_t(v[k]);
        }
    }
    // scans of occurrences, state slots and top cells
    uint32_t sp = 0, sc = 0, sn = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        sp += v[k] > 0 ? uint32_t(v[k]) : 0u;
        sc += v[k] == -1 ? 1u : (v[k] > 0 ? uint32_t(v[k]) : 0u);
        sn += v[k] == -1 ? 1u : 0u;
    }
    uint32_t ip = sp, ic = sc, in = sn;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t const yp = __shfl_up_sync(0xffffffffu, ip, o), yc = __shfl_up_sync(0xffffffffu, ic, o),
                       yn = __shfl_up_sync(0xffffffffu, in, o);
        if (lane >= uint32_t(o)) {
            ip += yp;
            ic += yc;
            in += yn;
        }
    }
    uint32_t const totalNeg = __shfl_sync(0xffffffffu, in, 31);
    uint32_t const high = size - 1 - totalNeg;
    uint32_t p0 = ip - sp, c0 = ic - sc, n0 = in - sn;
    if (part == 0) {
#pragma unroll
        for (int k = 0; k < 8; k++) {
            uint32_t const sy = 8 * lane + k;
            S.posCum[sy] = uint16_t(p0);
            S.cumul[sy] = uint16_t(c0);
            if (W == 1) next[sy] = c0;
            p0 += v[k] > 0 ? uint32_t(v[k]) : 0u;
            c0 += v[k] == -1 ? 1u : (v[k] > 0 ? uint32_t(v[k]) : 0u);
            if (v[k] == -1) {
                S.symbolAt[size - 1 - n0] = uint8_t(sy);
                n0++;
            }
        }
        if (lane == 31) {
            S.posCum[256] = uint16_t(p0);
            S.cumul[256] = uint16_t(c0);
        }
    }
    if (W > 1)
        for (uint32_t sy = lane; sy < 256; sy += 32) next[sy] = 0;
    sync();
    // spread: the warp's rounds of 32 positions
    uint32_t const rounds = size / 32, r0 = rounds * part / W, r1 = rounds * (part + 1) / W;
    bool const any = totalNeg < size;
    uint32_t occBase = 0; // occurrences before the round
    if (any)
        for (uint32_t r = 0; r < r0; r++)
            occBase += totalNeg ? __popc(__ballot_sync(0xffffffffu, (((32 * r + lane) * step) & mask) <= high)) : 32u;
    uint32_t sCur = 0;
    if (r0) { // the symbol of the warp's first occurrence
#pragma unroll
        for (uint32_t h = 128; h; h >>= 1)
            if (S.posCum[sCur + h] <= occBase) sCur += h;
    }
    uint32_t cumNext = S.posCum[sCur + 1];
    for (uint32_t r = r0; r < r1; r++) {
        uint32_t const pos = ((32 * r + lane) * step) & mask;
        bool const valid = any && pos <= high;
        uint32_t const bal = __ballot_sync(0xffffffffu, valid);
        if (valid) {
            uint32_t const occ = occBase + __popc(bal & lt);
            while (occ >= cumNext && sCur < 255) cumNext = S.posCum[++sCur + 1];
            S.symbolAt[pos] = uint8_t(sCur);
        }
        occBase += __popc(bal);
    }
    sync();
    // state table; with several warps, each symbol's cells of each warp first
    if (W > 1) {
        for (uint32_t r = r0; r < r1; r++) atomicAdd(&next[S.symbolAt[32 * r + lane]], 1u);
        sync();
        for (uint32_t sy = threadIdx.x; sy < 256; sy += 32 * W) {
            uint32_t slot = S.cumul[sy];
#pragma unroll
            for (int w = 0; w < W; w++) {
                uint32_t const c = nextSlot[w][sy];
                nextSlot[w][sy] = slot;
                slot += c;
            }
        }
        sync();
    }
    ent::FseCTable* const ct = reinterpret_cast<ent::FseCTable*>(t.ctable);
    for (uint32_t r = r0; r < r1; r++) {
        uint32_t const u = 32 * r + lane;
        uint32_t const sy = S.symbolAt[u];
        uint32_t const m = __match_any_sync(0xffffffffu, sy);
        uint32_t const base = next[sy];
        __syncwarp();
        if (lane == 31u - __clz(m)) next[sy] = base + __popc(m);
        ct->state[base + __popc(m & lt)] = uint16_t(size + u);
        __syncwarp();
    }
    for (uint32_t sy = part * 32 + lane; sy < 256; sy += 32 * W) {
        int const c = sy <= maxSym ? int(S.norm[sy]) : 0;
        ent::fseSymbolDeltas(c, tl, S.cumul[sy], ct->deltaNbBits[sy], ct->deltaFindState[sy]);
        if (sy <= maxSym) t.norm[sy] = S.norm[sy];
    }
    if (part != W - 1) return;
    uint32_t const headerBytes = fseHeader(S.header, v, ic - sc, maxSym, tl);
    for (uint32_t i = lane; i < headerBytes; i += 32) t.ncount[i] = uint8_t(S.header[i >> 2] >> (8 * (i & 3)));
    if (lane == 0) {
        ct->tableLog = uint16_t(tl);
        ct->maxSym = uint16_t(maxSym);
        sizes[t.sizeSlot] = headerBytes;
    }
}

// Huffman code lengths and codes on the device, one warp per chunk
// (huf_tree.h, as the reference's HUF_buildCTable, has the serial form of every
// step). The buckets are counted and filled 32 symbols a round, ranked by
// __match_any_sync; each lane sorts a bucket of large counts of its own (the
// quicksort's order of equal counts is part of the result, so a bucket is one
// lane's); lane 0 joins the tree, with the two candidates' counts in registers,
// and repairs its height; the depths follow by doubling the way to the root; the
// codes are counted off by length as the buckets were.
//
// What bounds it: the join (two dependent shared loads a node) and the largest
// bucket's quicksort, each one lane's chain. With every step on lane 0 the
// launch over the 529 chunks of a 256 MiB timestamp array's tables took 220 us,
// now 54 (64 messages: 155 and 54).
constexpr int kHufTabWarps = 4;
struct HufBuildSmem {
    ent::HufNode nodes[ent::kHufNodes];
    uint32_t count[256];
    uint16_t base[192], curr[192]; // symbols in bucket r or above; the next place of bucket r - 1
    uint16_t rank[16], code[16];   // codes of a length; the next one
    uint16_t up[256];              // inner nodes: the way to the root
    uint8_t depth[256], nbBits[256];
};

// hufBuildCodes by the whole warp
__device__ __forceinline__ uint32_t hufBuildWarp(HufBuildSmem& S, uint16_t* value, uint32_t maxSym, uint32_t maxNbBits)
{
    uint32_t const lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    ent::HufNode* const node = S.nodes + 1;
    for (int k = lane; k < ent::kHufNodes; k += 32) S.nodes[k] = ent::HufNode{ 0, 0, 0, 0 };
    for (uint32_t k = lane; k < 192; k += 32) S.base[k] = 0;
    for (uint32_t k = lane; k < 256; k += 32) S.nbBits[k] = 0;
    if (lane < 16) S.rank[lane] = 0;
    __syncwarp();
    // buckets: counts, then the symbols of higher buckets before each
    for (uint32_t n0 = 0; n0 <= maxSym; n0 += 32) {
        uint32_t const n = n0 + lane, bk = n <= maxSym ? ent::hufBucketOf(S.count[n]) : 192u;
        uint32_t const m = __match_any_sync(0xffffffffu, bk);
        if (bk < 192 && lane == 31u - __clz(m)) S.base[bk] = uint16_t(S.base[bk] + __popc(m));
        __syncwarp();
    }
    {
        uint32_t v[6], sum = 0; // lane j: buckets 6j .. 6j + 5
#pragma unroll
        for (int k = 5; k >= 0; k--) {
            sum += S.base[6 * lane + k];
            v[k] = sum;
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t const y = __shfl_down_sync(0xffffffffu, incl, o);
            if (lane + o < 32) incl += y;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 6; k++) S.base[6 * lane + k] = S.curr[6 * lane + k] = uint16_t(v[k] + incl - sum);
    }
    __syncwarp();
    for (uint32_t n0 = 0; n0 <= maxSym; n0 += 32) {
        uint32_t const n = n0 + lane, bk = n <= maxSym ? ent::hufBucketOf(S.count[n]) : 191u;
        uint32_t const m = __match_any_sync(0xffffffffu, bk);
        uint32_t const at = bk < 191 ? S.curr[bk + 1] : 0u;
        __syncwarp();
        if (bk < 191) {
            uint32_t const pos = at + __popc(m & lt);
            node[pos].count = S.count[n];
            node[pos].byte = uint8_t(n);
            if (lane == 31u - __clz(m)) S.curr[bk + 1] = uint16_t(at + __popc(m));
        }
        __syncwarp();
    }
    if (ent::kHufDistinctCutoff + lane < 191) {
        uint32_t const r = ent::kHufDistinctCutoff + lane;
        int const size = int(S.curr[r]) - int(S.base[r]);
        if (size > 1) ent::hufQuickSortDesc(node + S.base[r], 0, size - 1);
    }
    __syncwarp();
    // leaves 0 .. nonNull by decreasing count, inner nodes 256 .. root
    uint32_t present = 0;
    for (uint32_t n = lane; n <= maxSym; n += 32) present += node[n].count != 0;
    present = __reduce_add_sync(0xffffffffu, present);
    int const start = 256, nonNull = int(present) - 1, root = start + nonNull - 1;
    if (lane == 0) {
        int lowS = nonNull, nodeNb = start, lowN = start;
        S.nodes[0].count = 1u << 31; // node[-1]: above every count
        uint32_t cN = node[lowS].count + node[lowS - 1].count;
        node[nodeNb].count = cN;
        node[lowS].parent = node[lowS - 1].parent = uint16_t(nodeNb);
        nodeNb++;
        lowS -= 2;
        uint32_t cS = node[lowS].count;
        // the lesser of the next leaf and the next inner node; one not made yet
        // counts 2^30, as there
        auto take = [&](uint32_t& c) -> int {
            int n;
            if (cS < cN) {
                c = cS;
                n = lowS--;
                cS = node[lowS].count;
            } else {
                c = cN;
                n = lowN++;
                cN = lowN < nodeNb ? node[lowN].count : 1u << 30;
            }
            return n;
        };
        while (nodeNb <= root) {
            uint32_t c1, c2;
            int const n1 = take(c1), n2 = take(c2);
            node[nodeNb].count = c1 + c2;
            node[n1].parent = node[n2].parent = uint16_t(nodeNb);
            if (lowN == nodeNb) cN = c1 + c2;
            nodeNb++;
        }
    }
    __syncwarp();
    for (int n = start + int(lane); n <= root; n += 32) {
        S.up[n - start] = uint16_t(n == root ? root : node[n].parent);
        S.depth[n - start] = n == root ? 0 : 1;
    }
    __syncwarp();
    for (bool far = true; far;) { // (every way doubles: at most eight rounds)
        uint32_t to[8], d[8];
        far = false;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            int const n = 32 * k + int(lane);
            if (start + n > root) continue;
            uint32_t const u = S.up[n] - start;
            d[k] = S.depth[n] + S.depth[u];
            to[k] = S.up[u];
            far |= int(to[k]) != root;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; k++) {
            int const n = 32 * k + int(lane);
            if (start + n > root) continue;
            S.depth[n] = uint8_t(d[k]);
            S.up[n] = uint16_t(to[k]);
        }
        far = __any_sync(0xffffffffu, far);
        __syncwarp();
    }
    for (int n = lane; n <= nonNull; n += 32) node[n].nbBits = uint8_t(S.depth[node[n].parent - start] + 1);
    __syncwarp();
    uint32_t maxBits = 0;
    if (lane == 0) maxBits = ent::hufLimitHeight(node, uint32_t(nonNull), maxNbBits);
    maxBits = __shfl_sync(0xffffffffu, maxBits, 0);
    __syncwarp();
    // codes of each length, in symbol order
    for (uint32_t n0 = 0; n0 <= maxSym; n0 += 32) {
        uint32_t const n = n0 + lane, nb = n <= maxSym ? node[n].nbBits : 0u;
        uint32_t const m = __match_any_sync(0xffffffffu, nb);
        if (nb && lane == 31u - __clz(m)) S.rank[nb] = uint16_t(S.rank[nb] + __popc(m));
        if (n <= maxSym) S.nbBits[node[n].byte] = uint8_t(nb);
        __syncwarp();
    }
    if (lane == 0) {
        uint16_t mn = 0;
        for (int n = int(maxBits); n > 0; n--) {
            S.code[n] = mn;
            mn = uint16_t((mn + S.rank[n]) >> 1);
        }
        S.code[0] = 0;
    }
    __syncwarp();
    for (uint32_t n0 = 0; n0 < 256; n0 += 32) {
        uint32_t const n = n0 + lane, nb = S.nbBits[n];
        uint32_t const m = __match_any_sync(0xffffffffu, n <= maxSym ? nb : 16u);
        uint32_t const at = S.code[nb];
        __syncwarp();
        // (absent symbols count off length 0's, as there)
        value[n] = n <= maxSym ? uint16_t(at + __popc(m & lt)) : uint16_t(0);
        if (n <= maxSym && lane == 31u - __clz(m)) S.code[nb] = uint16_t(at + __popc(m));
        __syncwarp();
    }
    return maxBits;
}

__global__ void __launch_bounds__(32 * kHufTabWarps) kHufTables(const HufTableTask* __restrict__ tasks, uint32_t nbTasks)
{
    __shared__ HufBuildSmem sm[kHufTabWarps];
    uint32_t const wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t const ti = blockIdx.x * kHufTabWarps + wid;
    if (ti >= nbTasks) return; // the whole warp
    HufTableTask const t = tasks[ti];
    HufBuildSmem& S = sm[wid];
    for (uint32_t k = lane; k < 256; k += 32) S.count[k] = t.hist[k];
    __syncwarp();
    ent::HufCTable* const ct = reinterpret_cast<ent::HufCTable*>(t.ctable);
    uint32_t const tl = hufBuildWarp(S, ct->value, t.maxSym, t.maxNbBits);
    if (lane == 0) ct->tableLog = tl;
    for (uint32_t k = lane; k < 256; k += 32) {
        uint32_t const nb = S.nbBits[k];
        ct->nbBits[k] = uint8_t(nb);
        if (k <= t.maxSym) t.weights[k] = uint8_t(nb ? tl + 1 - nb : 0);
    }
}

// A bitstream written by a whole warp: each round the lanes bring two runs of
// bits (at most 48 each), a scan of their lengths places them, they are ORed
// into a window of words in shared memory and the complete words go out. What
// does not fit the capacity is dropped and shows in the returned size (> cap).
struct WarpBits {
    static constexpr uint32_t kWindow = 128; // words: a round adds at most 96 to the partial one
    uint32_t* w;
    uint8_t* out; // 4-byte aligned
    uint32_t cap, lane, B = 0, wb = 0; // bits placed; first word not written yet
    __device__ WarpBits(uint32_t* window, uint8_t* o, uint32_t c) : w(window), out(o), cap(c), lane(threadIdx.x & 31u)
    {
        for (uint32_t q = lane; q < kWindow; q += 32) w[q] = 0;
        __syncwarp();
    }
    // bits f (nb of them, none above) at bit p
    __device__ __forceinline__ void place(uint64_t f, uint32_t nb, uint32_t p)
    {
        if (!nb) return;
        uint32_t const q = p >> 5, sh = p & 31u;
        uint64_t const lo = f << sh;
        atomicOr(&w[q & (kWindow - 1)], uint32_t(lo));
        if (sh + nb > 32) atomicOr(&w[(q + 1) & (kWindow - 1)], uint32_t(lo >> 32));
        if (sh + nb > 64) atomicOr(&w[(q + 2) & (kWindow - 1)], uint32_t(f >> (64 - sh)));
    }
    __device__ __forceinline__ void flush()
    {
        uint32_t const upTo = B >> 5;
        for (uint32_t q = wb + lane; q < upTo; q += 32) {
            uint32_t const x = w[q & (kWindow - 1)];
            w[q & (kWindow - 1)] = 0;
            if (4 * q + 4 <= cap) *reinterpret_cast<uint32_t*>(out + 4 * q) = x;
        }
        __syncwarp();
        wb = upTo;
    }
    // every lane of the warp calls it
    __device__ __forceinline__ void add(uint64_t f0, uint32_t n0, uint64_t f1, uint32_t n1)
    {
        uint32_t inc = n0 + n1;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            uint32_t const y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        uint32_t const p = B + inc - n0 - n1;
        place(f0, n0, p);
        place(f1, n1, p + n0);
        B += __shfl_sync(0xffffffffu, inc, 31);
        __syncwarp();
        flush();
    }
    // the end mark and the last bytes; returns the stream's size
    __device__ __forceinline__ uint32_t close()
    {
        if (lane == 0) w[(B >> 5) & (kWindow - 1)] |= 1u << (B & 31u);
        B += 1;
        __syncwarp();
        flush();
        uint32_t const bytes = (B + 7) >> 3;
        for (uint32_t b = 4 * wb + lane; b < bytes; b += 32)
            if (b < cap) out[b] = uint8_t(w[(b >> 2) & (kWindow - 1)] >> (8 * (b & 3u)));
        return bytes;
    }
};

// FSE, short chunks (below kFseLongMin symbols, two states), one warp each:
// the warp brings the coding table and the source into shared memory, lanes 0
// and 1 run a state each (the c-th symbol from the end belongs to state
// (s0 + c) % 2; the last two symbols start the states and emit nothing) and
// leave a 16-bit entry per transition (the field in bits 0-11, its width
// above) in append order, the states' flushes last; then the warp appends
// them, eight entries a lane. With sixteen lanes of a warp each loading its
// table alone and encoding alone, the tables took longer than the chunks: the
// 4,224 weights streams of a 128 MiB timestamp frame 0.060 ms, now 0.015.
__global__ void __launch_bounds__(32) kFseEnc(const FseEncTask* __restrict__ tasks, uint32_t* __restrict__ sizes)
{
    __shared__ uint2 tt[256]; // per symbol: deltaNbBits, deltaFindState
    __shared__ uint16_t st[2048], entry[1024];
    __shared__ uint8_t src[kFseLongMin];
    __shared__ uint32_t window[WarpBits::kWindow];
    FseEncTask const t = tasks[blockIdx.x];
    uint32_t const lane = threadIdx.x, n = t.n, size = 1u << t.tableLog;
    const ent::FseCTable* const ct = reinterpret_cast<const ent::FseCTable*>(t.ctable);
    for (uint32_t y = lane; y < 256; y += 32) tt[y] = make_uint2(ct->deltaNbBits[y], uint32_t(ct->deltaFindState[y]));
    for (uint32_t u = lane; u < size; u += 32) st[u] = ct->state[u];
    for (uint32_t i = lane; i < n; i += 32) src[i] = t.src[i];
    __syncwarp();
    if (lane < 2) {
        uint32_t c = (lane + n) & 1u; // s0 = 2 - n % 2
        uint2 d = tt[src[n - 1 - c]];
        uint32_t const nb0 = (d.x + (1u << 15)) >> 16, x = (nb0 << 16) - d.x;
        uint32_t v = st[(x >> nb0) + d.y];
        for (c += 2; c < n; c += 2) {
            d = tt[src[n - 1 - c]];
            uint32_t const nb = (v + d.x) >> 16, q = v >> nb;
            entry[c - 2] = uint16_t((v - (q << nb)) + (nb << 12));
            v = st[q + d.y];
        }
        entry[n - 2 + lane] = uint16_t((v & (size - 1u)) | (t.tableLog << 12));
    }
    __syncwarp();
    WarpBits wb(window, t.out, n + n / 128 + 512);
    for (uint32_t j0 = 0; j0 < n; j0 += 256) {
        uint64_t f[2];
        uint32_t w[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            f[h] = w[h] = 0;
#pragma unroll
            for (uint32_t m = 0; m < 4; m++) {
                uint32_t const j = j0 + 8 * lane + 4 * h + m, e = j < n ? entry[j] : 0u;
                f[h] |= uint64_t(e & 0xfffu) << w[h];
                w[h] += e >> 12;
            }
        }
        wb.add(f[0], w[0], f[1], w[1]);
    }
    uint32_t const bytes = wb.close();
    if (lane == 0) sizes[t.sizeSlot] = bytes;
}

// FSE, long chunks (four states, kFseLongMin symbols or more), one CTA each.
// The four states' chains are independent (only the order in which their
// fields are appended couples them), and a chain forgets where it came from,
// so each is cut into up to 32 segments run at once, lane k of a group of four
// running state k:
//  1. A segment starts some steps early from an arbitrary state (from the true
//     state where that reaches the chain's start) and records, for each batch
//     of four steps, the state that enters it.
//  2. A segment whose entry state is not the end state of the segment before
//     it runs again from that state, until it meets its own earlier state at a
//     quarter of the segment, or its end; this repeats until all agree.
//  3. All threads replay the batches from their recorded states and write one
//     16-bit entry per transition (the field in bits 0-11, its width in bits
//     12-15) at the field's index in append order.
//  4. The entries are then the chunk's fields in order. Their widths give each
//     warp's first bit; a warp appends its quarter of the batches, 128 entries
//     a round (a scan of the lanes' widths places them, they are ORed into a
//     window of words in shared memory, complete words go out; only those that
//     fit the capacity are written, as in the one-lane encoder). The words that
//     two warps share meet in shared memory.
//
// The run-up, and the shortest segment, is four times the mean number of steps
// in which two unlike states meet. A symbol that holds c of the table's cells
// maps a state's logarithm by a rotation and rounds it to c values, so two
// states drift apart or together only by that rounding: the mean is about
// 300 / (sum of 1 / c) plus (table size) / (symbols present) (simulated for 36
// distributions of 2 to 200 symbols; within a factor of two of the former term
// or their sum). With few symbols that is longer than the chunk and one
// segment is left; a run-up too short for them cost twelve repeats of step 2.
//
// What bounds it: a transition's chain (two adds, two shifts and a shared
// load, 47 cycles; 57 in step 1, whose loads run three batches ahead and
// lookups one). With one lane a chain it was 8,192 of them for a chunk of 32 K
// symbols, at 290 cycles, in 24 lanes per SM. Writing the entries inside the
// chain (as before step 3 was split off) took 115 cycles a transition. 32 K
// symbols, a plane of about 200 symbols: 1.19 ms and 0.11 ms of packing with
// one lane a chain, 0.062 ms with entries in the chain, 0.056 ms now; two
// symbols (one segment) 1.3, 0.58 and 0.27 ms. Encoder batch of 64 messages,
// this launch: 0.59 ms before the split, 0.39 now; of 2048 mixed frames, in
// one part: 3.3 and 2.5 ms.
constexpr uint32_t kFseSegs = 32, kFseLongThreads = 4 * kFseSegs, kFseLongWarps = kFseLongThreads / 32;
constexpr uint32_t kFseSegBatches = 16; // fewest batches in a segment, if there are several

__global__ void __launch_bounds__(kFseLongThreads) kFseEncLong(const FseEncTask* __restrict__ tasks,
                                                               uint32_t* __restrict__ sizes)
{
    __shared__ uint2 tt[256];      // per symbol: deltaNbBits, deltaFindState
    __shared__ uint16_t st[2048];
    __shared__ uint32_t endState[kFseSegs][4], warpBits[kFseLongWarps];
    __shared__ uint16_t check[4][kFseLongThreads]; // per thread and quarter of its segment: the state after it
    __shared__ uint32_t win[kFseLongWarps][64];
    __shared__ uint32_t edgeWord[kFseLongWarps][2], edgeAt[kFseLongWarps][2]; // first and last word of each warp
    __shared__ float warpInv[kFseLongWarps];
    FseEncTask const t = tasks[blockIdx.x];
    uint32_t const tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5, k = tid & 3u;
    // the first segments are not those of the first warp in every CTA: with few
    // segments the SM's CTAs would all run them on one of its schedulers
    uint32_t const g = (tid / 4 + 8 * (blockIdx.x * 0x9E3779B1u >> 30)) & (kFseSegs - 1);
    const ent::FseCTable* const ct = reinterpret_cast<const ent::FseCTable*>(t.ctable);
    uint32_t const size = 1u << t.tableLog;
    if (tid < kFseLongWarps) warpBits[tid] = 0;
    for (uint32_t y = tid; y < 256; y += kFseLongThreads) tt[y] = make_uint2(ct->deltaNbBits[y], uint32_t(ct->deltaFindState[y]));
    for (uint32_t u = tid; u < size; u += kFseLongThreads) st[u] = ct->state[u];
    // symbols present and the sum over them of 1 / cells, each thread from the
    // pairs that it put in place itself (the others' are not there yet)
    float inv = 0;
    uint32_t const own = fseSymbolShare(tid, kFseLongThreads, t.tableLog, [&](uint32_t y) { return tt[y].x; }, inv);
    static_assert(2 * kFseLongThreads == 256, "two symbols a thread");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) inv += __shfl_xor_sync(0xffffffffu, inv, o);
    if (lane == 0) warpInv[wid] = inv;
    uint32_t const symbols = __syncthreads_count(own > 0) + __syncthreads_count(own > 1);
    inv = warpInv[0] + warpInv[1] + warpInv[2] + warpInv[3];

    // The c-th symbol from the end belongs to state (s0 + c) % 4; the last
    // four symbols start the states and emit nothing. Then the r = n % 4
    // single symbols (fields 0 .. r - 1), then steps of four symbols: step i
    // takes the bytes [ip - 4 i - 4, ip - 4 i), the top one for state 0, and
    // state k's field is r + 4 i + k.
    uint32_t const n = t.n, r = n & 3u, s0 = 4u - r, ip = n - 4 - r;
    uint32_t const pad = (4u - r) & 3u; // entries start here, so that steps start at multiples of four
    uint16_t* const fo = t.fields + pad;
    uint32_t const steps = ip >> 2;
    // batches of four steps: 16 bytes of the source, the first ones after so
    // many single steps (i1) that they start in a block's first word
    uint32_t const i1 = uint32_t(reinterpret_cast<uintptr_t>(t.src + ip) & 15) >> 2, r1 = r + 4 * i1;
    uint32_t const batches = (steps - i1) >> 2;
    uintptr_t const top = reinterpret_cast<uintptr_t>(t.src) + ip - 4 * i1;
    uint32_t const off = uint32_t(top & 3);
    uint32_t const warm = fseRunUp(kFseSegBatches, size, symbols, inv);
    uint32_t const segs = min(kFseSegs, max(1u, batches / warm));
    uint32_t v;
    {
        uint32_t const y = t.src[n - 1 - ((k + 4u - (s0 & 3u)) & 3u)];
        uint32_t const nb = (tt[y].x + (1u << 15)) >> 16, x = (nb << 16) - tt[y].x;
        v = st[(x >> nb) + tt[y].y];
    }
    // one transition of state x with the symbol's pair; the entry of one
    auto trans = [&](uint32_t x, uint2 d) -> uint32_t { return st[(x >> ((x + d.x) >> 16)) + d.y]; };
    auto entryOf = [&](uint32_t x, uint2 d) -> uint32_t {
        uint32_t const nb = (x + d.x) >> 16;
        return (x & ((1u << nb) - 1u)) + (nb << 12);
    };
    uint32_t head = 0, tail = 0; // bits of the fields that this thread writes here
    for (uint32_t c = 4; c < 4 + r; c++)
        if (((s0 + c) & 3u) == k) {
            uint2 const d = tt[t.src[n - 1 - c]];
            if (g == 0) {
                uint32_t const e = entryOf(v, d);
                fo[c - 4] = uint16_t(e);
                head += e >> 12;
            }
            v = trans(v, d);
        }
    for (uint32_t i = 0; i < i1; i++) {
        uint2 const d = tt[t.src[ip - 4 * i - 1 - k]];
        if (g == 0) {
            uint32_t const e = entryOf(v, d);
            fo[r + 4 * i + k] = uint16_t(e);
            head += e >> 12;
        }
        v = trans(v, d);
    }

    // Batches [from, to) from state v. A batch's 16 source bytes are loaded
    // three batches ahead and its pairs one ahead, in between the transitions,
    // so that only the chain itself is left between two states. `record`: the
    // states that enter a batch go to its first four entries.
    uint4 const zero = make_uint4(0, 0, 0, 0);
    // the 16 bytes from byte `off` (0 to 3) of block lo on, up the block above it
    auto window = [&](const uint4& lo, uint32_t up) -> uint4 {
        return make_uint4(__funnelshift_r(lo.x, lo.y, 8 * off), __funnelshift_r(lo.y, lo.z, 8 * off),
                          __funnelshift_r(lo.z, lo.w, 8 * off), __funnelshift_r(lo.w, up, 8 * off));
    };
    auto fetch = [](const uint4* p) -> uint4 {
        uint4 x;
        asm volatile("ld.global.nc.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "l"(p));
        return x;
    };
    auto run = [&](uint32_t from, uint32_t to, bool record) {
        if (from >= to) return;
        uint32_t left = to - from; // batches from the one that p is at on
        const uint4* p = reinterpret_cast<const uint4*>(top - off) - (from + 1);
        auto down = [&] { // past the last batch, its block is loaded again
            if (left > 1) {
                left--;
                p--;
            }
        };
        uint32_t const sel = 0x4443u - k;
        uint4 cur = __ldg(p), w = window(cur, off ? __ldg(reinterpret_cast<const uint32_t*>(p + 1)) : 0u);
        uint32_t up = cur.x;
        uint2 d[4] = { tt[__byte_perm(w.w, 0, sel)], tt[__byte_perm(w.z, 0, sel)], tt[__byte_perm(w.y, 0, sel)],
                       tt[__byte_perm(w.x, 0, sel)] };
        down();
        uint4 n1 = fetch(p);
        down();
        uint4 n2 = fetch(p);
        down();
        uint4 n3 = fetch(p);
        down();
        uint4 n4 = fetch(p);
        uint16_t* f = fo + r1 + 16 * from + k;
        for (uint32_t b = from; b < to; b++, f += 16) {
            if (record) *f = uint16_t(v);
            down();
            uint4 const n5 = fetch(p);
            w = window(n1, up);
            v = trans(v, d[0]);
            d[0] = tt[__byte_perm(w.w, 0, sel)];
            v = trans(v, d[1]);
            d[1] = tt[__byte_perm(w.z, 0, sel)];
            v = trans(v, d[2]);
            d[2] = tt[__byte_perm(w.y, 0, sel)];
            v = trans(v, d[3]);
            d[3] = tt[__byte_perm(w.x, 0, sel)];
            up = n1.x;
            n1 = n2;
            n2 = n3;
            n3 = n4;
            n4 = n5;
        }
    };
    uint32_t const b0 = g < segs ? batches * g / segs : 0, b1 = g < segs ? batches * (g + 1) / segs : 0;
    if (g && g < segs) {
        uint32_t const w0 = b0 > warm ? b0 - warm : 0;
        if (w0) v = size;
        run(w0, b0, false);
    }
    uint32_t entry = 0; // the state that the recorded ones follow from
    for (uint32_t want = v;;) {
        bool const bad = g < segs && want != entry;
        if (!__syncthreads_or(bad)) break;
        if (bad) {
            bool met = false;
            v = want;
            for (uint32_t q = 0; q < 4 && !met; q++) {
                run(b0 + (b1 - b0) * q / 4, b0 + (b1 - b0) * (q + 1) / 4, true);
                met = entry && v == check[q][tid];
                check[q][tid] = uint16_t(v);
            }
            entry = want;
            endState[g][k] = check[3][tid];
        }
        __syncthreads();
        if (g && g < segs) want = endState[g - 1][k];
    }
    if (g == segs - 1) { // the steps past the last batch, then the state's flush
        v = check[3][tid];
        for (uint32_t i = i1 + 4 * batches; i < steps; i++) {
            uint2 const d = tt[t.src[ip - 4 * i - 1 - k]];
            uint32_t const e = entryOf(v, d);
            fo[r + 4 * i + k] = uint16_t(e);
            tail += e >> 12;
            v = trans(v, d);
        }
        fo[n - 4 + k] = uint16_t((v & (size - 1u)) | (t.tableLog << 12));
        tail += t.tableLog;
    }
    if (head) atomicAdd(&warpBits[0], head);
    if (tail) atomicAdd(&warpBits[kFseLongWarps - 1], tail);

    // 2. the warp's quarter of the batches, one per lane: four steps from the
    // recorded states, whose entries take their place
    uint32_t const B0 = batches * wid / kFseLongWarps, B1 = batches * (wid + 1) / kFseLongWarps;
    uint32_t bits = 0;
    for (uint32_t b = B0 + lane; b < B1; b += 32) {
        const uint4* const a = reinterpret_cast<const uint4*>(top - off) - (b + 1);
        uint4 const lo = __ldg(a);
        uint4 const w = window(lo, off ? __ldg(reinterpret_cast<const uint32_t*>(a + 1)) : 0u);
        uint2* const f = reinterpret_cast<uint2*>(fo + r1 + 16 * b);
        uint2 const in = *f;
        uint32_t x[4] = { in.x & 0xffffu, in.x >> 16, in.y & 0xffffu, in.y >> 16 };
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            uint32_t const y = i == 0 ? w.w : i == 1 ? w.z : i == 2 ? w.y : w.x;
            uint32_t e[4];
#pragma unroll
            for (uint32_t m = 0; m < 4; m++) {
                uint2 const d = tt[__byte_perm(y, 0, 0x4443u - m)];
                e[m] = entryOf(x[m], d);
                bits += e[m] >> 12;
                if (i < 3) x[m] = trans(x[m], d);
            }
            f[i] = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bits += __shfl_xor_sync(0xffffffffu, bits, o);
    if (lane == 0) atomicAdd(&warpBits[wid], bits);
    __syncthreads();

    // 3. the warp's entries [j0, j1) from `fields` on
    uint32_t const cap = n + n / 128 + 512;
    uint8_t* const out = t.out;
    uint32_t* const w = win[wid];
    w[lane] = 0;
    w[lane + 32] = 0;
    __syncwarp();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t q = 0; q < kFseLongWarps; q++) {
        before += q < wid ? warpBits[q] : 0u;
        total += warpBits[q];
    }
    uint32_t B = before, wb = before >> 5; // bits placed; first word not written yet
    uint32_t const j0 = wid == 0 ? 0u : pad + r1 + 16 * B0,
                   j1 = wid == kFseLongWarps - 1 ? pad + n : pad + r1 + 16 * B1;
    if (lane == 0) {
        edgeAt[wid][0] = edgeAt[wid][1] = before >> 5;
        edgeWord[wid][0] = edgeWord[wid][1] = 0;
    }
    auto flushWords = [&](uint32_t upTo) { // words [wb, upTo) are complete but for the warp's first one
        for (uint32_t q = wb + lane; q < upTo; q += 32) {
            uint32_t const x = w[q & 63u];
            w[q & 63u] = 0;
            if (q == before >> 5) edgeWord[wid][0] = x;
            else if (4 * q + 4 <= cap) *reinterpret_cast<uint32_t*>(out + 4 * q) = x;
        }
        __syncwarp();
        wb = upTo;
    };
    const uint2* const src = reinterpret_cast<const uint2*>(t.fields);
    uint32_t const g1 = (j1 + 3) >> 2; // entries in groups of four (j0 is a multiple of four)
    uint32_t gi = (j0 >> 2) + lane;
    uint2 d = gi < g1 ? src[gi] : make_uint2(0u, 0u);
    for (uint32_t i0 = j0 >> 2; i0 < g1; i0 += 32) {
        uint2 const cur = d;
        uint32_t const j = 4 * (i0 + lane);
        gi = i0 + 32 + lane;
        d = gi < g1 ? src[gi] : make_uint2(0u, 0u); // the next round's entries, in flight
        uint32_t e0 = cur.x & 0xffffu, e1 = cur.x >> 16, e2 = cur.y & 0xffffu, e3 = cur.y >> 16;
        if (j < pad || j + 4 > pad + n) { // entries outside the chunk's
            if (j + 0 < pad || j + 0 >= pad + n) e0 = 0;
            if (j + 1 < pad || j + 1 >= pad + n) e1 = 0;
            if (j + 2 < pad || j + 2 >= pad + n) e2 = 0;
            if (j + 3 < pad || j + 3 >= pad + n) e3 = 0;
        }
        uint32_t const n0 = e0 >> 12, n01 = n0 + (e1 >> 12), n012 = n01 + (e2 >> 12), sum = n012 + (e3 >> 12);
        uint32_t inc = sum;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            uint32_t const y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        uint32_t const p = B + inc - sum, q = p >> 5, sh = p & 31u;
        if (sum) { // at most 48 bits, from bit sh of word q
            uint64_t const f = uint64_t(e0 & 0xfffu) | (uint64_t(e1 & 0xfffu) << n0) | (uint64_t(e2 & 0xfffu) << n01)
                               | (uint64_t(e3 & 0xfffu) << n012);
            uint64_t const lo = f << sh;
            atomicOr(&w[q & 63u], uint32_t(lo));
            if (sh + sum > 32) atomicOr(&w[(q + 1) & 63u], uint32_t(lo >> 32));
            if (sh + sum > 64) atomicOr(&w[(q + 2) & 63u], uint32_t(f >> (64 - sh)));
        }
        B += __shfl_sync(0xffffffffu, inc, 31);
        __syncwarp();
        flushWords(B >> 5);
    }
    if (lane == 0 && j0 < j1) {
        edgeAt[wid][1] = B >> 5;
        edgeWord[wid][1] = w[(B >> 5) & 63u]; // the warp's last word, not complete (its first one, if it has no other)
    }
    __syncthreads();
    // the words at the warps' edges, then the end mark: the word it completes
    // goes out as a word, then the bytes
    if (tid == 0) {
        uint32_t at = 0, x = 0;
        auto put = [&](uint32_t pos, uint32_t word) {
            if (pos != at) {
                if (4 * at + 4 <= cap) *reinterpret_cast<uint32_t*>(out + 4 * at) = x;
                at = pos;
                x = 0;
            }
            x |= word;
        };
        for (uint32_t q = 0; q < kFseLongWarps; q++) {
            put(edgeAt[q][0], edgeWord[q][0]);
            put(edgeAt[q][1], edgeWord[q][1]);
        }
        put(total >> 5, 1u << (total & 31u));
        uint32_t const bytes = (total + 1 + 7) >> 3;
        if (((total + 1) & 31u) == 0) {
            put(at + 1, 0);
        } else {
            for (uint32_t b = 4 * at; b < bytes; b++)
                if (b < cap) out[b] = uint8_t(x >> (8 * (b & 3u)));
        }
        sizes[t.sizeSlot] = bytes;
    }
}

// Huffman: one warp per stream (4 per chunk for 4X, else the first); symbols
// are appended from the end of the stream to its start, a lane's eight at a
// time (codes of at most 11 bits, four joined to a run of WarpBits). Each
// stream writes at its own offset of the chunk buffer; the frame assembly
// joins them.
// The codes of a stream do not depend on one another; with one lane a stream
// the launch waited for serial writers: 4,224 chunks of a 128 MiB timestamp
// frame took 0.56 ms, now 0.084.
constexpr uint32_t kHufEncThreads = 128;

__device__ __forceinline__ uint32_t hufStreamCap(uint32_t seg) { return ((seg + (seg >> 3) + 64) + 15) & ~15u; }

// the 8 bytes below p of which cnt (1..8) belong to the caller's range, the
// highest in bits 56-63; reads only 8-byte words that hold bytes of the range
__device__ __forceinline__ uint64_t ldBelow8(const uint8_t* p, uint32_t cnt)
{
    uintptr_t const top = reinterpret_cast<uintptr_t>(p);
    uint32_t const off = uint32_t(top & 7); // bytes of the upper word
    const uint64_t* const a = reinterpret_cast<const uint64_t*>(top - off);
    uint64_t const lo = off < cnt ? __ldg(a - 1) : 0;
    if (off == 0) return lo;
    return (__ldg(a) << (64 - 8 * off)) | (lo >> (8 * off));
}

__global__ void __launch_bounds__(kHufEncThreads) kHufEnc(const HufEncTask* __restrict__ tasks, uint32_t* __restrict__ sizes)
{
    __shared__ uint32_t code[256]; // value, length above
    __shared__ uint32_t window[kHufEncThreads / 32][WarpBits::kWindow];
    HufEncTask const t = tasks[blockIdx.x];
    const ent::HufCTable* const ct = reinterpret_cast<const ent::HufCTable*>(t.ctable);
    for (uint32_t y = threadIdx.x; y < 256; y += kHufEncThreads) code[y] = ct->value[y] | (uint32_t(ct->nbBits[y]) << 16);
    __syncthreads();
    uint32_t const k = threadIdx.x >> 5, lane = threadIdx.x & 31u, seg = (t.n + 3) / 4;
    if (!t.x4 && k) return;
    uint32_t const start = t.x4 ? seg * k : 0, len = t.x4 ? (k < 3 ? seg : t.n - 3 * seg) : t.n;
    WarpBits wb(window[k], t.out + (t.x4 ? 16 + k * hufStreamCap(seg) : 0), t.x4 ? hufStreamCap(seg) : t.n + t.n / 8 + 64);
    const uint8_t* const end = t.src + start + len;
    // lane L's symbols of a round: the eight below end - (j + 8 L)
    uint32_t cnt = 8 * lane < len ? min(8u, len - 8 * lane) : 0;
    uint64_t y = cnt ? ldBelow8(end - 8 * lane, cnt) : 0;
    for (uint32_t j = 0; j < len; j += 256) {
        uint64_t const cur = y;
        uint32_t const c = cnt, jn = j + 256 + 8 * lane;
        cnt = jn < len ? min(8u, len - jn) : 0; // the next round's symbols, in flight
        y = cnt ? ldBelow8(end - jn, cnt) : 0;
        uint64_t f[2];
        uint32_t n[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            uint32_t const x = uint32_t(cur >> (32 - 32 * h));
            f[h] = n[h] = 0;
#pragma unroll
            for (uint32_t m = 0; m < 4; m++) {
                uint32_t const e = 4 * h + m < c ? code[(x >> (24 - 8 * m)) & 0xffu] : 0;
                f[h] |= uint64_t(e & 0xffffu) << n[h];
                n[h] += e >> 16;
            }
        }
        wb.add(f[0], n[0], f[1], n[1]);
    }
    uint32_t const size = wb.close();
    if (lane == 0) sizes[t.sizeSlot + k] = size;
}

// 16-bit chunk statistics (the counts ZS_Histogram_count16 takes,
// src/openzl/shared/histogram.c:37-80, plus first occurrences for tokenize):
// one tile of kEncTile values per CTA, global atomics per value; the maximum
// is reduced per warp first.
__global__ void __launch_bounds__(256) kHist16(const Hist16Task* __restrict__ tasks,
                                               const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    Hist16Task const t = tasks[tr.task];
    uint32_t const i0 = tr.tile * kEncTile;
    uint32_t mx = 0;
    for (uint32_t k = threadIdx.x; k < kEncTile; k += 256) {
        uint32_t const i = i0 + k;
        if (i >= t.n) break;
        uint32_t const v = uint32_t(t.src[2 * i]) | (uint32_t(t.src[2 * i + 1]) << 8);
        atomicAdd(&t.count[v], 1u);
        atomicMin(&t.first[v], i);
        mx = max(mx, v);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(t.maxOut, mx);
}

// tokenize indices: binary search of each value among the chunk's sorted
// distinct values (fewer than 256, staged in shared memory)
__global__ void __launch_bounds__(256) kTok16(const Tok16Task* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    __shared__ uint16_t keys[256];
    __shared__ uint8_t ids[256];
    TileRef const tr = tiles[blockIdx.x];
    Tok16Task const t = tasks[tr.task];
    for (uint32_t k = threadIdx.x; k < t.na; k += 256) {
        keys[k] = t.keys[k];
        ids[k] = t.ids[k];
    }
    __syncthreads();
    uint32_t const i0 = tr.tile * kEncTile;
    for (uint32_t k = threadIdx.x; k < kEncTile; k += 256) {
        uint32_t const i = i0 + k;
        if (i >= t.n) break;
        uint32_t const v = uint32_t(t.src[2 * i]) | (uint32_t(t.src[2 * i + 1]) << 8);
        uint32_t lo = 0, hi = t.na; // first key >= v
        while (lo < hi) {
            uint32_t const mid = (lo + hi) >> 1;
            if (keys[mid] < v) lo = mid + 1;
            else hi = mid;
        }
        t.idx[i] = ids[lo < t.na ? lo : 0];
    }
}

// 16-bit-symbol Huffman streams (ZS_largeHuffmanEncodeUsingCTable and its 4X
// split, src/openzl/codecs/entropy/encode_huffman_kernel.c:413-508): stream k
// of a 4X chunk holds size/4 + 1 symbols, the last one the rest; symbols are
// appended from the end of the stream to its start, then a 1 bit closes it.
// sizes[sizeSlot + k] gets the bitstream's size, sizes[sizeSlot + 4 + k] its
// whole bytes (the reference's writer fails once these reach its capacity
// less 8 bytes).
// One warp per stream, four symbols a lane and round (codes of at most 20
// bits, two joined to a run of WarpBits). One thread a stream read and looked
// up symbol after symbol: 98,304 symbols in four streams took 6.2 ms, now
// 0.16.
constexpr uint32_t kHuf16EncThreads = 128;
__global__ void __launch_bounds__(kHuf16EncThreads) kHuf16Enc(const Huf16EncTask* __restrict__ tasks,
                                                              uint32_t* __restrict__ sizes)
{
    __shared__ uint32_t window[kHuf16EncThreads / 32][WarpBits::kWindow];
    Huf16EncTask const t = tasks[blockIdx.x];
    uint32_t const k = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (!t.x4 && k) return;
    uint32_t const chunk = t.x4 ? t.n / 4 + 1 : t.n;
    uint32_t const start = min(t.n, k * chunk);
    uint32_t const len = min(chunk, t.n - start);
    uint8_t* const out = t.out + uint64_t(k) * t.streamCap;
    WarpBits wb(window[k], out + 8, t.streamCap - 8);
    const uint8_t* const end = t.src + 2ull * (start + len);
    uint32_t cnt = 4 * lane < len ? min(4u, len - 4 * lane) : 0;
    uint64_t y = cnt ? ldBelow8(end - 8 * lane, 2 * cnt) : 0;
    for (uint32_t j = 0; j < len; j += 128) {
        uint64_t const cur = y;
        uint32_t const c = cnt, jn = j + 128 + 4 * lane;
        cnt = jn < len ? min(4u, len - jn) : 0; // the next round's symbols, in flight
        y = cnt ? ldBelow8(end - 2 * jn, 2 * cnt) : 0;
        uint64_t f[2];
        uint32_t n[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            f[h] = n[h] = 0;
#pragma unroll
            for (uint32_t m = 0; m < 2; m++)
                if (2 * h + m < c) {
                    uint32_t const v = uint32_t(cur >> (48 - 32 * h - 16 * m)) & 0xffffu;
                    uint32_t const nb = __ldg(t.nbBits + v);
                    f[h] |= uint64_t(__ldg(t.code + v) & ((1u << nb) - 1u)) << n[h];
                    n[h] += nb;
                }
        }
        wb.add(f[0], n[0], f[1], n[1]);
    }
    uint32_t const size = wb.close();
    if (lane == 0) {
        *reinterpret_cast<uint32_t*>(out) = len;
        *reinterpret_cast<uint32_t*>(out + 4) = size;
        sizes[t.sizeSlot + k] = size;
        sizes[t.sizeSlot + 4 + k] = wb.B / 8; // with the end mark
    }
}

__global__ void __launch_bounds__(256) kRemap(const RemapTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    RemapTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = min(t.n, e0 + kEncTile);
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x)
        stW(t.idx + i * t.iw, t.rankOf[ldW(t.idx + i * t.iw, t.iw)], t.iw);
}

__global__ void kPut(const PutTask* __restrict__ tasks, uint32_t n)
{
    uint32_t const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    PutTask const t = tasks[i];
    uint64_t const h = *t.hash;
    for (uint32_t b = 0; b < t.bytes; b++) t.dst[b] = uint8_t(h >> (8 * b));
}

// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// bf16 deconstruct: 4096 elements per tile
__global__ void __launch_bounds__(256) kBf16(const Bf16Task* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    Bf16Task const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = e0 + kEncTile < t.n ? e0 + kEncTile : t.n;
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
        uint32_t const x = uint32_t(t.src[2 * i]) | (uint32_t(t.src[2 * i + 1]) << 8);
        t.signFrac[i] = uint8_t(((x >> 15) & 1) | ((x & 0x7f) << 1));
        t.exponent[i] = uint8_t(x >> 7);
    }
}

// ---------------------------------------------------------------------------
// tokenize: open-addressing table of distinct values with their first index
__device__ __forceinline__ uint64_t tokHash(uint64_t k)
{
    // splitmix64 finalizer
    k ^= k >> 30;
    k *= 0xbf58476d1ce4e5b9ull;
    k ^= k >> 27;
    k *= 0x94d049bb133111ebull;
    return k ^ (k >> 31);
}

__global__ void __launch_bounds__(256) kTokInsert(const TokTask* __restrict__ tasks, const TileRef* __restrict__ tiles,
                                                  uint32_t* __restrict__ errors)
{
    TileRef const tr = tiles[blockIdx.x];
    TokTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = e0 + kEncTile < t.n ? e0 + kEncTile : t.n;
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
        uint64_t const k = ldW(t.src + i * t.w, t.w);
        uint64_t h = tokHash(k) & t.capMask;
        bool placed = false;
        for (uint64_t probe = 0; probe <= t.capMask && !placed; probe++) {
            volatile uint32_t* const st = t.state + h;
            uint32_t s = *st;
            if (s == 0) {
                if (atomicCAS(t.state + h, 0u, 1u) == 0u) {
                    t.key[h] = k;
                    __threadfence();
                    atomicExch(t.state + h, 2u);
                    atomicMin(t.first + h, uint32_t(i));
                    placed = true;
                    break;
                }
                s = *st;
            }
            // another element is writing this slot: wait (bounded) for its key
            uint32_t spins = 0;
            while (s == 1 && spins < (1u << 22)) {
                s = *st;
                spins++;
            }
            if (s != 2) break;
            __threadfence();
            if (*reinterpret_cast<volatile uint64_t*>(t.key + h) == k) {
                atomicMin(t.first + h, uint32_t(i));
                placed = true;
                break;
            }
            h = (h + 1) & t.capMask;
        }
        if (!placed) atomicAdd(errors, 1u);
    }
}

// Marks first occurrences (rank[i] = 1) and records each element's slot;
// per-tile mark counts go to tileSums.
__global__ void __launch_bounds__(256) kTokMark(const TokTask* __restrict__ tasks, const TileRef* __restrict__ tiles,
                                                uint64_t* __restrict__ tileSums, uint32_t* __restrict__ errors)
{
    __shared__ uint32_t warpCnt[8];
    TileRef const tr = tiles[blockIdx.x];
    TokTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = e0 + kEncTile < t.n ? e0 + kEncTile : t.n;
    uint32_t cnt = 0;
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
        uint64_t const k = ldW(t.src + i * t.w, t.w);
        uint64_t h = tokHash(k) & t.capMask;
        uint64_t probe = 0;
        while (probe <= t.capMask && !(t.state[h] == 2 && t.key[h] == k)) {
            h = (h + 1) & t.capMask;
            probe++;
        }
        if (probe > t.capMask) {
            atomicAdd(errors, 1u);
            t.slotOf[i] = 0;
            t.rank[i] = 0;
            continue;
        }
        t.slotOf[i] = uint32_t(h);
        uint32_t const m = t.first[h] == uint32_t(i) ? 1u : 0u;
        t.rank[i] = m;
        cnt += m;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) warpCnt[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint64_t tot = 0;
        for (int w = 0; w < 8; w++) tot += warpCnt[w];
        tileSums[blockIdx.x] = tot;
    }
}

// one warp per task: exclusive scan of its tiles' mark counts; the total is
// the alphabet size
__global__ void __launch_bounds__(256) kTokPrefix(const TokTask* __restrict__ tasks, uint32_t nbTasks,
                                                  const uint64_t* __restrict__ tileSums,
                                                  uint64_t* __restrict__ tilePrefix, uint32_t* __restrict__ counts)
{
    uint32_t const ti = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t const lane = threadIdx.x & 31;
    if (ti >= nbTasks) return;
    TokTask const t = tasks[ti];
    uint32_t const nT = uint32_t((t.n + kEncTile - 1) / kEncTile);
    uint64_t running = 0;
    for (uint32_t k0 = 0; k0 < nT; k0 += 32) {
        uint32_t const k = k0 + lane;
        uint64_t const x = k < nT ? tileSums[t.tileBase + k] : 0;
        uint64_t incl = x;
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t const y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        if (k < nT) tilePrefix[t.tileBase + k] = running + incl - x;
        running += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) counts[ti] = uint32_t(running);
}

// marks -> exclusive ranks, 16 consecutive elements per thread
__global__ void __launch_bounds__(256) kTokRank(const TokTask* __restrict__ tasks, const TileRef* __restrict__ tiles,
                                                const uint64_t* __restrict__ tilePrefix)
{
    __shared__ uint32_t warpTot[8];
    TileRef const tr = tiles[blockIdx.x];
    TokTask const t = tasks[tr.task];
    uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint64_t const base = uint64_t(tr.tile) * kEncTile + uint64_t(tid) * 16;
    uint32_t v[16];
    uint32_t acc = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        uint32_t const m = base + k < t.n ? t.rank[base + k] : 0u;
        v[k] = acc;
        acc += m;
    }
    uint32_t incl = acc;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t const y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= uint32_t(o)) incl += y;
    }
    if (lane == 31) warpTot[wid] = incl;
    __syncthreads();
    uint32_t pre = 0;
    for (uint32_t w = 0; w < wid; w++) pre += warpTot[w];
    uint32_t const add = uint32_t(tilePrefix[blockIdx.x]) + pre + (incl - acc);
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (base + k < t.n) t.rank[base + k] = v[k] + add;
}

// indices and alphabet
__global__ void __launch_bounds__(256) kTokEmit(const TokTask* __restrict__ tasks, const TileRef* __restrict__ tiles)
{
    TileRef const tr = tiles[blockIdx.x];
    TokTask const t = tasks[tr.task];
    uint64_t const e0 = uint64_t(tr.tile) * kEncTile;
    uint64_t const e1 = e0 + kEncTile < t.n ? e0 + kEncTile : t.n;
    for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
        uint32_t const f = t.first[t.slotOf[i]];
        uint32_t const r = t.rank[f];
        stW(t.idx + i * t.iw, r, t.iw);
        if (f == uint32_t(i)) stW(t.alphabet + uint64_t(r) * t.w, ldW(t.src + i * t.w, t.w), t.w);
    }
}


uint32_t hufEncStreamCap(uint32_t seg) { return ((seg + (seg >> 3) + 64) + 15) & ~15u; }

void launchEncMax(const EncNumTask* t, const TileRef* tiles, uint32_t nbTiles, unsigned long long* maxima,
                  cudaStream_t s)
{
    if (nbTiles) kEncMax<<<nbTiles, 256, 0, s>>>(t, tiles, maxima);
}
void launchEncNum(const EncNumTask* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kEncNum<<<nbTiles, 128, 0, s>>>(t, tiles);
}
void launchPack(const PackTask* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kPack<<<nbTiles, 128, 0, s>>>(t, tiles);
}
void launchHist(const HistTask* t, uint32_t n, uint32_t* hists, cudaStream_t s)
{
    if (n) kHist<<<n, 256, 0, s>>>(t, hists);
}
void launchFseTables(const FseTableTask* t, uint32_t n, uint32_t* sizes, uint32_t* errors, cudaStream_t s)
{
    if (!n) return;
    if (n <= kFseTabWide) kFseTables<kFseTabWarps><<<n, 32 * kFseTabWarps, 0, s>>>(t, n, sizes, errors);
    else kFseTables<1><<<(n + kFseTabWarps - 1) / kFseTabWarps, 32 * kFseTabWarps, 0, s>>>(t, n, sizes, errors);
}

void launchHufTables(const HufTableTask* t, uint32_t n, cudaStream_t s)
{
    if (n) kHufTables<<<(n + kHufTabWarps - 1) / kHufTabWarps, 32 * kHufTabWarps, 0, s>>>(t, n);
}

void launchFseEnc(const FseEncTask* t, uint32_t n, uint32_t* sizes, cudaStream_t s)
{
    if (n) kFseEnc<<<n, 32, 0, s>>>(t, sizes);
}
void launchFseEncLong(const FseEncTask* t, uint32_t n, uint32_t* sizes, cudaStream_t s)
{
    if (n) kFseEncLong<<<n, kFseLongThreads, 0, s>>>(t, sizes);
}
void launchHufEnc(const HufEncTask* t, uint32_t n, uint32_t* sizes, cudaStream_t s)
{
    if (n) kHufEnc<<<n, kHufEncThreads, 0, s>>>(t, sizes);
}
void launchPut(const PutTask* t, uint32_t n, cudaStream_t s)
{
    if (n) kPut<<<(n + 127) / 128, 128, 0, s>>>(t, n);
}


void launchBf16(const Bf16Task* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kBf16<<<nbTiles, 256, 0, s>>>(t, tiles);
}

void launchTokCount(const TokTask* t, uint32_t nbTasks, const TileRef* tiles, uint32_t nbTiles, uint64_t* tileSums,
                    uint64_t* tilePrefix, uint32_t* counts, uint32_t* errors, cudaStream_t s)
{
    if (!nbTiles) return;
    kTokInsert<<<nbTiles, 256, 0, s>>>(t, tiles, errors);
    kTokMark<<<nbTiles, 256, 0, s>>>(t, tiles, tileSums, errors);
    kTokPrefix<<<(nbTasks * 32 + 255) / 256, 256, 0, s>>>(t, nbTasks, tileSums, tilePrefix, counts);
    kTokRank<<<nbTiles, 256, 0, s>>>(t, tiles, tilePrefix);
}

void launchHist16(const Hist16Task* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kHist16<<<nbTiles, 256, 0, s>>>(t, tiles);
}
void launchTok16(const Tok16Task* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kTok16<<<nbTiles, 256, 0, s>>>(t, tiles);
}
void launchHuf16Enc(const Huf16EncTask* t, uint32_t n, uint32_t* sizes, cudaStream_t s)
{
    if (n) kHuf16Enc<<<n, kHuf16EncThreads, 0, s>>>(t, sizes);
}

void launchRemap(const RemapTask* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kRemap<<<nbTiles, 256, 0, s>>>(t, tiles);
}

void launchTokEmit(const TokTask* t, const TileRef* tiles, uint32_t nbTiles, cudaStream_t s)
{
    if (nbTiles) kTokEmit<<<nbTiles, 256, 0, s>>>(t, tiles);
}

} // namespace ozl
