// qssb_decode.cu - HDF5 bitshuffle + LZ4 chunks of u16 detector frames <-> device frames.
//
// The step before the SSB path: the reference reads 4D-STEM acquisitions as
// HDF5 chunks (one detector frame each) compressed by the bitshuffle filter
// with LZ4 (io/load.py:3271-3320, io/backends/cuda/decoder.py:258-403 of
// bobleesj/quantem.gpu) and writes them the same way (io/save.py,
// decoder.py:496-1003). Chunk format: big-endian uint64 uncompressed bytes,
// big-endian uint32 block bytes (8192), then per block a big-endian uint32
// compressed size and an LZ4 block of the bit-shuffled elements (bit plane b
// = bit b of every element, byte k of a plane = elements 8k..8k+7, element
// 8k+j in bit j); the last block holds the rest rounded down to 8 elements;
// the remaining < 8 elements follow raw.
//
// Decode: one CTA per chunk. Each warp walks the block chain (every offset
// checked against the chunk's end) and decodes its blocks' LZ4
// sequences into shared memory (every lane parses the token stream through
// L1, all lanes copy literals and matches - a match byte j reads
// out[op - off + j mod off], so overlapping matches need no serial copy) and
// bit-unshuffles the block with 8x8 bit transposes straight into the u16
// frame (32-byte stores where the frames allow it). A malformed chunk sets status[c] (the block is
// zero-filled); nothing traps.
// Encode: a warp per block makes the same transposes forward and the greedy
// LZ4 of a serial search (32 positions a step, a 4096-entry hash table in
// shared memory) into fixed-stride slots, then a pack kernel lays out the
// chunks at caller offsets.
#include <limits.h>

#include "qssb_internal.h"

namespace qssb {

constexpr int kDecWarps = 4;
constexpr int kBlockBytes = 8192;                         // bytes per shuffled block
constexpr int kBlockElems = kBlockBytes / 2;
constexpr int kLz4Bound = kBlockBytes + kBlockBytes / 255 + 16;  // LZ4 worst case
constexpr int kMaxBlocks = 512;                           // 4 MB frames
constexpr int kEncHash = 4096;

// Status codes written per chunk.
constexpr int kStOk = 0;
constexpr int kStHeader = 1;    // header size / block size / chunk too short
constexpr int kStChain = 2;     // a block extends past the chunk's end
constexpr int kStLz4 = 3;       // malformed LZ4 sequence or wrong decoded size

__device__ __forceinline__ uint32_t be32(const uint8_t* p) {
    return ((uint32_t)p[0] << 24) | ((uint32_t)p[1] << 16) | ((uint32_t)p[2] << 8) | (uint32_t)p[3];
}

// 8x8 bit transpose (byte i = row i, bit j = column j), three delta swaps.
__device__ __forceinline__ uint64_t transpose8(uint64_t x) {
    uint64_t t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAull;
    x = x ^ t ^ (t << 7);
    t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCull;
    x = x ^ t ^ (t << 14);
    t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ull;
    x = x ^ t ^ (t << 28);
    return x;
}

// Four bytes at any byte position of a 4-aligned shared buffer. The second
// word of an aligned position is read too (inside the kernel's shared memory
// in every use) and shifted out.
__device__ __forceinline__ uint32_t rd32(const uint8_t* base, int pos) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(base) + (pos >> 2);
    return __funnelshift_r(w[0], w[1], 8 * (pos & 3));
}

// out[op + j] = out[op - off + j], j < ml, by the whole warp, as if byte by
// byte (off < ml repeats the last off bytes). Up to 32 bytes in one step.
// Longer: the output has period off, so it may be read from any multiple of
// off back that lies behind op - off; bytes fill the first multiple D >= 128,
// then words copy from D back, 128 bytes a step and, once D has doubled to
// 512, 512 a step (the runs of zero planes: 8 KB in ~25 steps).
__device__ __forceinline__ void copy_match(uint8_t* out, int op, int off, int ml, int lane) {
    // lane mod off: (lane + 1/2) / off is never within 1/64 of an integer
    const int r0 = off > 31 ? lane : lane - off * (int)__fdividef((float)lane + 0.5f, (float)off);
    if (ml <= 32) {
        if (lane < ml) out[op + lane] = out[op - off + r0];
        return;
    }
    int d = off;
    if (d < 128) d *= (127 + off) / off;
    const int n0 = min(ml, (off < 128 ? d : 0) + ((4 - ((op + (off < 128 ? d : 0)) & 3)) & 3));
    if (off < 32) {
        int r = r0;
        const int step = 32 % off;
        for (int j = lane; j < n0; j += 32) {
            out[op + j] = out[op - off + r];
            r += step;
            if (r >= off) r -= off;
        }
    } else {  // 32 <= off: a step reads behind what it writes
        for (int j0 = 0; j0 < n0; j0 += 32) {
            if (j0 + lane < n0) out[op + j0 + lane] = out[op - off + j0 + lane];
            __syncwarp();
        }
    }
    __syncwarp();
    int p = op + n0;  // a multiple of 4 while words remain
    int words = (ml - n0) >> 2;
    while (words > 0) {
        while (d < 512 && p - 2 * d >= op - off) d *= 2;
        if (d >= 512) {
            uint32_t w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (lane + 32 * u < words) w[u] = rd32(out, p - d + 4 * (lane + 32 * u));
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (lane + 32 * u < words)
                    *reinterpret_cast<uint32_t*>(out + p + 4 * (lane + 32 * u)) = w[u];
            const int n = min(words, 128);
            p += 4 * n;
            words -= n;
        } else {
            if (lane < words)
                *reinterpret_cast<uint32_t*>(out + p + 4 * lane) = rd32(out, p - d + 4 * lane);
            const int n = min(words, 32);
            p += 4 * n;
            words -= n;
        }
        __syncwarp();
    }
    const int rest = op + ml - p;
    if (lane < rest) out[p + lane] = out[p - d + lane];
}

// Decode one LZ4 block from in[0, csz) (global memory, read through L1) into
// out[0, cap) (shared memory) by the whole warp. A window of 32 input bytes is
// parsed at once, every lane taking its byte for a token: literal and match
// lengths and the offset behind them. The chain of actual tokens is then
// followed by shuffles, one a sequence, with the next sequence's literals
// fetched before this one's match is copied. A token with extended lengths,
// the last sequence and anything malformed go through the checked path, one
// sequence parsed by all lanes in step. Returns true when the stream is well
// formed and fills exactly cap bytes.
__device__ bool lz4_block_warp(const uint8_t* __restrict__ in, int csz, uint8_t* out, int cap,
                               int lane) {
    int ip = 0, op = 0;
    while (ip < csz) {
        const int p = ip + lane;
        uint32_t seq = 0;  // literals | match code << 4 | plain << 8 | offset << 16
        if (p < csz) {
            const uint32_t token = __ldg(in + p);
            const int at = p + 1 + (int)(token >> 4);
            if (token < 0xf0 && (token & 15) != 15 && at + 2 <= csz)
                seq = (token >> 4) | ((token & 15) << 4) | 0x100u |
                      ((uint32_t)__ldg(in + at) << 16) | ((uint32_t)__ldg(in + at + 1) << 24);
        }
        int cur = 0;
        uint32_t w = __shfl_sync(0xffffffffu, seq, 0);
        uint8_t byte = __ldg(in + min(ip + 1 + lane, csz - 1));
        while (w & 0x100u) {
            const int lit = w & 15, ml = ((w >> 4) & 15) + 4, off = w >> 16;
            if (lit + ml > cap - op || (unsigned)(off - 1) >= (unsigned)(op + lit)) return false;
            if (lane < lit) out[op + lane] = byte;
            op += lit;
            cur += 3 + lit;
            w = cur < 32 ? __shfl_sync(0xffffffffu, seq, cur) : 0u;
            byte = __ldg(in + min(ip + cur + 1 + lane, csz - 1));
            __syncwarp();  // these literals and the last match, before the match reads them
            // ml <= 18, one step; lane mod off as in copy_match
            const int r = off >= ml ? lane
                                    : lane - off * (int)__fdividef((float)lane + 0.5f, (float)off);
            if (lane < ml) out[op + lane] = out[op - off + r];
            op += ml;
        }
        ip += cur;
        if (cur >= 32) continue;  // the next window
        __syncwarp();
        // one sequence, every length and bound checked
        if (ip >= csz) return false;
        const int token = __ldg(in + ip++);
        int lit = token >> 4;
        if (lit == 15) {
            int b;
            do {
                if (ip >= csz) return false;
                b = __ldg(in + ip++);
                lit += b;
            } while (b == 255 && lit <= cap);
        }
        if (lit > cap - op || lit > csz - ip) return false;
#pragma unroll 4
        for (int j = lane; j < lit; j += 32) out[op + j] = __ldg(in + ip + j);
        ip += lit;
        op += lit;
        if (ip == csz) {
            __syncwarp();
            return op == cap;
        }
        if (ip + 2 > csz) return false;
        const int off = __ldg(in + ip) | (__ldg(in + ip + 1) << 8);
        ip += 2;
        int ml = (token & 15) + 4;
        if ((token & 15) == 15) {
            int b;
            do {
                if (ip >= csz) return false;
                b = __ldg(in + ip++);
                ml += b;
            } while (b == 255 && ml <= cap);
        }
        if (off == 0 || off > op || ml > cap - op) return false;
        __syncwarp();  // literals (and earlier matches) visible to the match reads
        copy_match(out, op, off, ml, lane);
        op += ml;
        __syncwarp();
    }
    return false;
}

// Bytes g of the eight words w, g = 0..3, as 8-byte values m[g] (byte b from w[b]).
__device__ __forceinline__ void byte_columns(const uint32_t* w, uint64_t* m) {
    uint32_t h[2][4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t* x = w + 4 * k;
        const uint32_t a = __byte_perm(x[0], x[1], 0x5140), b = __byte_perm(x[2], x[3], 0x5140);
        const uint32_t c = __byte_perm(x[0], x[1], 0x7362), d = __byte_perm(x[2], x[3], 0x7362);
        h[k][0] = __byte_perm(a, b, 0x5410);
        h[k][1] = __byte_perm(a, b, 0x7632);
        h[k][2] = __byte_perm(c, d, 0x5410);
        h[k][3] = __byte_perm(c, d, 0x7632);
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) m[g] = (uint64_t)h[0][g] | ((uint64_t)h[1][g] << 32);
}

// Eight u16 elements from their low and high bytes.
__device__ __forceinline__ uint4 join_bytes(uint64_t lo, uint64_t hi) {
    const uint32_t l0 = (uint32_t)lo, l1 = (uint32_t)(lo >> 32);
    const uint32_t h0 = (uint32_t)hi, h1 = (uint32_t)(hi >> 32);
    return make_uint4(__byte_perm(l0, h0, 0x5140), __byte_perm(l0, h0, 0x7362),
                      __byte_perm(l1, h1, 0x5140), __byte_perm(l1, h1, 0x7362));
}

// Bit-unshuffle cnt (a multiple of 8) elements from a block's planes into dst.
// wide: dst is 32-byte aligned; a lane then takes a word of every plane (32
// elements, the high planes skipped where they are zero) and stores whole
// 32-byte sectors. Otherwise (and where a plane is not whole words) a byte of
// every plane, 8 elements.
__device__ __forceinline__ void unshuffle_store(const uint8_t* planes, int cnt, uint16_t* dst,
                                                bool vec, bool wide, int lane) {
    const int P = cnt / 8;
    if (wide && (P & 3) == 0) {
        const uint32_t* words = reinterpret_cast<const uint32_t*>(planes);
        for (int q = lane; q < P / 4; q += 32) {
            uint32_t w[16];
            uint32_t high = 0;
#pragma unroll
            for (int b = 0; b < 16; ++b) {
                w[b] = words[b * (P / 4) + q];
                if (b >= 8) high |= w[b];
            }
            uint64_t lo[4], hi[4] = {0, 0, 0, 0};
            byte_columns(w, lo);
            if (high) {
                byte_columns(w + 8, hi);
#pragma unroll
                for (int g = 0; g < 4; ++g) hi[g] = transpose8(hi[g]);
            }
#pragma unroll
            for (int g = 0; g < 4; g += 2) {
                const uint4 a = join_bytes(transpose8(lo[g]), hi[g]);
                const uint4 b = join_bytes(transpose8(lo[g + 1]), hi[g + 1]);
                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                             :: "l"(dst + 32 * q + 8 * g), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                                "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
            }
        }
        return;
    }
    for (int p = lane; p < P; p += 32) {
        uint64_t lo = 0, hi = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            lo |= (uint64_t)planes[b * P + p] << (8 * b);
            hi |= (uint64_t)planes[(8 + b) * P + p] << (8 * b);
        }
        // transposed: byte j of lo (hi) holds bits 0..7 (8..15) of element 8p + j
        const uint4 w = join_bytes(transpose8(lo), transpose8(hi));
        uint16_t* o = dst + 8 * p;
        if (vec) {
            *reinterpret_cast<uint4*>(o) = w;
        } else {
            const uint32_t e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                o[2 * q] = (uint16_t)(e[q] & 0xffff);
                o[2 * q + 1] = (uint16_t)(e[q] >> 16);
            }
        }
    }
}

// W warps per chunk, which share nothing: each walks the block chain itself
// (every lane reads the same words, prefetched into L1), first to the end to
// check it, then along the blocks it takes. W = 1 where the chunks fill the
// chip (decode_one_warp): a frame's blocks differ widely in cost, and the warps
// of a larger CTA hold their shared memory until its slowest is done. Bound by the latency
// and issue of the per-sequence chain. 16384 frames of 128 x 128 counts: the
// call 0.49 ms, against 1.09 with four warps a chunk, one thread's chain
// walk, one sequence parsed at a time, matches copied and planes read by bytes.
template <int W>
__global__ void __launch_bounds__(32 * W) k_decode_bslz4_u16(
    const uint8_t* __restrict__ comp, long long comp_bytes, const long long* __restrict__ offsets,
    int n_chunks, long long chunk_bytes, uint16_t* __restrict__ out, int* __restrict__ status) {
    __shared__ uint4 planes4[W * kBlockBytes / 16 + 1];  // + a word that unaligned reads may touch
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    uint8_t* planes = reinterpret_cast<uint8_t*>(planes4) + (size_t)warp * kBlockBytes;
    const int c = blockIdx.x;
    const long long n_elem = chunk_bytes / 2;
    const long long n8 = n_elem & ~7LL;
    const int n_blocks = (int)((n8 + kBlockElems - 1) / kBlockElems);
    const long long c0 = offsets[c];
    const long long c1 = c + 1 < n_chunks ? offsets[c + 1] : comp_bytes;
    const uint8_t* ch = comp + c0;
    const long long len = c1 - c0;
    int st = kStOk;
    if (c0 < 0 || c1 > comp_bytes || len < 12) {
        st = kStHeader;
    } else {
        // the chunk's bytes into L1 (one prefetch per 128-byte line)
        for (long long i = (long long)tid * 128; i < len; i += 128LL * 32 * W)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(ch + i));
        unsigned long long total = 0;
        for (int i = 0; i < 8; ++i) total = (total << 8) | ch[i];
        if ((long long)total != chunk_bytes || be32(ch + 8) != (uint32_t)kBlockBytes) st = kStHeader;
    }
    long long pos = 12;
    for (int i = 0; i < n_blocks && st == kStOk; ++i) {
        if (pos + 4 > len) { st = kStChain; break; }
        const long long csz = be32(ch + pos);
        if (csz > kLz4Bound || pos + 4 + csz > len) { st = kStChain; break; }
        pos += 4 + csz;
    }
    if (st == kStOk && pos + (n_elem - n8) * 2 > len) st = kStChain;
    uint16_t* frame = out + (size_t)c * n_elem;
    if (W > 1) {  // blocks that fail raise the status below
        if (tid == 0 && status) status[c] = st;
        __syncthreads();
    } else if (lane == 0 && status) {
        status[c] = st;
    }
    if (st != kStOk) {  // the same in every warp
        for (long long i = tid; i < n_elem; i += 32 * W) frame[i] = 0;
        return;
    }
    const bool vec = (n_elem & 7) == 0 && ((uintptr_t)out & 15u) == 0;
    const bool wide = (n_elem & 15) == 0 && ((uintptr_t)out & 31u) == 0;
    if (warp == 0) {  // raw leftover elements
        const uint8_t* raw = ch + pos;
        for (long long j = n8 + lane; j < n_elem; j += 32) {
            const long long b = (j - n8) * 2;
            frame[j] = (uint16_t)(raw[b] | (raw[b + 1] << 8));
        }
    }
    pos = 12;
    for (int i = 0; i < n_blocks; ++i) {
        const int csz = (int)be32(ch + pos);
        const uint8_t* in = ch + pos + 4;
        pos += 4 + csz;
        if (W > 1 && i % W != warp) continue;
        const long long e0 = (long long)i * kBlockElems;
        const int cnt = (int)min((long long)kBlockElems, n8 - e0);
        const bool good = lz4_block_warp(in, csz, planes, 2 * cnt, lane);
        if (good) {
            unshuffle_store(planes, cnt, frame + e0, vec, wide, lane);
        } else {
            for (int j = lane; j < cnt; j += 32) frame[e0 + j] = 0;
            if (lane == 0 && status) atomicMax(status + c, kStLz4);
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ encode
// Scratch layout: per (chunk, block) a slot of kEncSlot bytes holding the
// big-endian compressed size followed by the LZ4 block.
constexpr int kEncSlot = (4 + kLz4Bound + 15) & ~15;
// one warp per CTA: a block of zeros leaves its 16 KB to the next one at once
// (with four, the blocks of one frame kept the slowest one's time: 645 us
// at 4096 frames in the kernel)
constexpr int kEncWarps = 1;
// planes | hash table
constexpr int kEncWarpBytes = kBlockBytes + 2 * kEncHash;

// LZ4 length extension: x / 255 bytes of 255, then the rest. Returns the bytes written.
__device__ __forceinline__ int put_length(uint8_t* o, int x, int lane) {
    const int q = x / 255;
    for (int k = lane; k <= q; k += 32) o[k] = (uint8_t)(k < q ? 255 : x - 255 * q);
    return q + 1;
}

// The greedy LZ4 of one block in shared memory by a whole warp, with the
// bytes of the serial search: every position from ip on looks up the last
// position of its 12-bit hash and enters itself, until the first whose four
// bytes match. The 32 lanes take positions ip .. ip + 31 at once: a lane's
// candidate is the nearest lower lane of the same hash (__match_any_sync) or
// the table's entry, the first hit is the lowest set bit of a ballot, and
// only lanes up to it enter the table (the highest of each hash). Matches are
// extended 128 bytes a step, literals copied 32 bytes a step.
__device__ int lz4_encode_block_warp(const uint8_t* planes, int n, uint16_t* table, uint8_t* o,
                                     int lane) {
    int op = 0, anchor = 0, ip = 0;
    const int last = n - 12;  // no match starts in the last 12 bytes
    while (ip < last) {
        const int pos = ip + lane;
        const bool on = pos < last;
        const uint32_t v = rd32(planes, on ? pos : ip);
        const uint32_t h = on ? (v * 2654435761u) >> 20 : kEncHash;  // idle lanes: a hash of their own
        const unsigned same = __match_any_sync(0xffffffffu, h);
        const unsigned below = same & ((1u << lane) - 1u);
        int cand = 0xffff;
        if (on) cand = below ? ip + 31 - __clz(below) : (int)table[h];
        const bool hit = cand != 0xffff && rd32(planes, cand) == v;
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        const int first = hits ? __ffs(hits) - 1 : 31;
        // a lane at or before the first hit enters its position unless a later
        // such lane has its hash (lanes beyond `last` have none)
        if (on && lane <= first && (same & (0xffffffffu >> (31 - first))) >> lane == 1u)
            table[h] = (uint16_t)pos;
        __syncwarp();
        if (!hits) {
            ip += 32;
            continue;
        }
        ip += first;
        cand = __shfl_sync(0xffffffffu, cand, first);
        int m = 4;
        const int room = n - 5 - ip;  // the last 5 bytes stay literal
        for (;;) {
            const int at = m + 4 * lane;
            int eq = 0;  // equal bytes of this lane's four
            if (at < room) {
                const uint32_t x = rd32(planes, ip + at) ^ rd32(planes, cand + at);
                eq = min(x ? (__ffs(x) - 1) >> 3 : 4, room - at);
            }
            const unsigned stop = __ballot_sync(0xffffffffu, eq < 4);
            if (stop) {
                const int l = __ffs(stop) - 1;
                m += 4 * l + __shfl_sync(0xffffffffu, eq, l);
                break;
            }
            m += 128;
        }
        const int lit = ip - anchor;
        if (lane == 0) o[op] = (uint8_t)((min(lit, 15) << 4) | min(m - 4, 15));
        ++op;
        if (lit >= 15) op += put_length(o + op, lit - 15, lane);
        for (int k = lane; k < lit; k += 32) o[op + k] = planes[anchor + k];
        op += lit;
        const int off = ip - cand;
        if (lane < 2) o[op + lane] = (uint8_t)(off >> (8 * lane));
        op += 2;
        if (m - 4 >= 15) op += put_length(o + op, m - 4 - 15, lane);
        ip += m;
        anchor = ip;
    }
    const int lit = n - anchor;
    if (lane == 0) o[op] = (uint8_t)(min(lit, 15) << 4);
    ++op;
    if (lit >= 15) op += put_length(o + op, lit - 15, lane);
    for (int k = lane; k < lit; k += 32) o[op + k] = planes[anchor + k];
    return op + lit;
}

// One warp per (chunk, block), blocks of one chunk in consecutive warps.
// Bound by the latency of a window's shared-memory chain (hash, table,
// candidate bytes, ballots) times the windows of a block, so the launch is as
// many warps as the 16 KB of planes and table of each allow (13 an SM). 4096
// frames of 128 x 128 counts: the whole call 0.46 ms against 4.00 ms with one
// lane searching byte by byte and copying (the same bytes).
__global__ void __launch_bounds__(32 * kEncWarps) k_encode_bslz4_u16(
    const uint16_t* __restrict__ frames, long long n_slots, int n_blocks, long long chunk_bytes,
    uint8_t* __restrict__ scratch) {
    extern __shared__ uint4 enc_smem4[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const long long item = (long long)blockIdx.x * kEncWarps + warp;
    if (item >= n_slots) return;
    const long long c = item / n_blocks;
    const int i = (int)(item - c * n_blocks);
    const long long n_elem = chunk_bytes / 2;
    const long long n8 = n_elem & ~7LL;
    uint8_t* planes = reinterpret_cast<uint8_t*>(enc_smem4) + (size_t)warp * kEncWarpBytes;
    uint16_t* table = reinterpret_cast<uint16_t*>(planes + kBlockBytes);
    const long long e0 = (long long)i * kBlockElems;
    const uint16_t* src = frames + (size_t)c * n_elem + e0;
    const int cnt = (int)min((long long)kBlockElems, n8 - e0);
    const int P = cnt / 8;
    const bool vec = ((uintptr_t)src & 15u) == 0;
    for (int p = lane; p < P; p += 32) {  // forward bit shuffle
        uint32_t w[4];
        if (vec) {
            const uint4 q = __ldcs(reinterpret_cast<const uint4*>(src) + p);
            w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                w[j] = (uint32_t)src[8 * p + 2 * j] | ((uint32_t)src[8 * p + 2 * j + 1] << 16);
        }
        // low and high bytes of the 8 elements
        const uint64_t lo = transpose8((uint64_t)__byte_perm(w[0], w[1], 0x6420) |
                                       ((uint64_t)__byte_perm(w[2], w[3], 0x6420) << 32));
        const uint64_t hi = transpose8((uint64_t)__byte_perm(w[0], w[1], 0x7531) |
                                       ((uint64_t)__byte_perm(w[2], w[3], 0x7531) << 32));
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            planes[b * P + p] = (uint8_t)(lo >> (8 * b));
            planes[(8 + b) * P + p] = (uint8_t)(hi >> (8 * b));
        }
    }
    uint4* t4 = reinterpret_cast<uint4*>(table);
    for (int h = lane; h < kEncHash / 8; h += 32) t4[h] = make_uint4(~0u, ~0u, ~0u, ~0u);
    __syncwarp();
    uint8_t* slot = scratch + (size_t)item * kEncSlot;
    const int op = lz4_encode_block_warp(planes, 2 * cnt, table, slot + 4, lane);
    if (lane < 4) slot[lane] = (uint8_t)(op >> (24 - 8 * lane));
}

// sizes[c] = bytes of chunk c: header, the blocks with their size words, raw leftovers.
__global__ void k_bslz4_chunk_sizes(const uint8_t* __restrict__ scratch, int n_chunks,
                                    long long chunk_bytes, long long* __restrict__ sizes) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_chunks) return;
    const long long n_elem = chunk_bytes / 2;
    const long long n8 = n_elem & ~7LL;
    const int n_blocks = (int)((n8 + kBlockElems - 1) / kBlockElems);
    long long total = 12 + (n_elem - n8) * 2;
    for (int i = 0; i < n_blocks; ++i) total += 4 + be32(scratch + ((size_t)c * n_blocks + i) * kEncSlot);
    sizes[c] = total;
}

// One warp per (chunk, block): the block's slot to its place in the chunk
// (the sizes of the chunk's earlier blocks summed by the lanes), 16 bytes a
// lane on the destination's alignment, the source words funnel-shifted (by
// bytes where a caller's scratch does not start on a word). The first block's
// warp writes the chunk header, the last one's the raw leftovers.
constexpr int kPackWarps = 8;
__global__ void __launch_bounds__(32 * kPackWarps) k_bslz4_pack(
    const uint8_t* __restrict__ scratch, const uint16_t* __restrict__ frames, long long n_items,
    int n_blocks, long long chunk_bytes, const long long* __restrict__ offsets,
    uint8_t* __restrict__ packed) {
    const int lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * kPackWarps + (threadIdx.x >> 5);
    if (item >= n_items) return;
    const int per = max(n_blocks, 1);  // a chunk of fewer than 8 elements has no block
    const long long c = item / per;
    const int i = (int)(item - c * per);
    const long long n_elem = chunk_bytes / 2;
    const long long n8 = n_elem & ~7LL;
    uint8_t* dst = packed + offsets[c];
    if (i == 0 && lane < 12) {
        dst[lane] = lane < 8 ? (uint8_t)((unsigned long long)chunk_bytes >> (8 * (7 - lane)))
                             : (uint8_t)((uint32_t)kBlockBytes >> (8 * (11 - lane)));
    }
    const uint8_t* first = scratch + (size_t)c * n_blocks * kEncSlot;
    int before = 0;
    for (int j = lane; j < i; j += 32) before += 4 + (int)be32(first + (size_t)j * kEncSlot);
    dst += 12 + __reduce_add_sync(0xffffffffu, before);
    const uint8_t* slot = first + (size_t)i * kEncSlot;
    const int len = n_blocks ? 4 + (int)be32(slot) : 0;
    const int head = min(len, (int)((16u - ((uintptr_t)dst & 15u)) & 15u));
    if (lane < head) dst[lane] = slot[lane];
    const int n_vec = ((uintptr_t)slot & 3u) == 0 ? (len - head) >> 4 : 0;
    const int shift = 8 * (head & 3);
    const uint32_t* words = reinterpret_cast<const uint32_t*>(slot) + (head >> 2);
    uint4* out = reinterpret_cast<uint4*>(dst + head);
    for (int t = lane; t < n_vec; t += 32) {
        const uint32_t* w = words + 4 * t;
        const uint32_t w4 = shift ? w[4] : 0u;  // within the slot: it holds needed bytes
        const uint32_t w1 = w[1], w2 = w[2], w3 = w[3];
        out[t] = make_uint4(__funnelshift_r(w[0], w1, shift), __funnelshift_r(w1, w2, shift),
                            __funnelshift_r(w2, w3, shift), __funnelshift_r(w3, w4, shift));
    }
    for (int j = head + 16 * n_vec + lane; j < len; j += 32) dst[j] = slot[j];
    if (i + 1 < n_blocks) return;
    const uint16_t* frame = frames + (size_t)c * n_elem;
    for (long long j = n8 + lane; j < n_elem; j += 32) {
        const uint16_t v = frame[j];
        dst[len + 2 * (j - n8)] = (uint8_t)(v & 0xff);
        dst[len + 2 * (j - n8) + 1] = (uint8_t)(v >> 8);
    }
}

// The shuffled blocks of one chunk.
static int chunk_blocks(long long chunk_bytes) {
    const long long n8 = (chunk_bytes / 2) & ~7LL;
    return (int)((n8 + kBlockElems - 1) / kBlockElems);
}

// One warp per chunk or four. An SM holds 24 one-warp CTAs (8 KB, and 1 KB of
// the system's, each) or 6 four-warp CTAs, the same 24 blocks, so the choice is
// between idle warps and chunks left waiting. Four warps a chunk against one,
// call, us (counts of dose 1000):
//   1 block (64 x 64):    900 chunks  51.3 / 30.7, 128 to 512 chunks equal;
//   3 blocks (110 x 110): 888 chunks  47.2 / 64.7, 900 (a second wave of
//                         four-warp CTAs) 67.4 / 65.5, 1860  105 / 84;
//   4 blocks (128 x 128): 1776 chunks 69.8 / 76.1, 1924 86.4 / 83.8,
//                         8192  295 / 243;
//   6 blocks (144 x 144): 1924 chunks 95 / 101, 4096 176 / 184; sparser counts
//                         up to 14% for four warps, denser ones 7% for one;
//   7 blocks (160 x 160): 1924 chunks 103 / 121, 4096 189 / 217; 16 blocks
//                         4096 chunks 442 / 545: one warp's chain through many
//                         blocks of a chunk outlasts the others.
static bool decode_one_warp(int n_chunks, int n_blocks) {
    const int sms = device_sm_count();
    if (n_blocks <= 1) return true;
    if (n_blocks <= 3) return n_chunks > 6 * sms;
    return n_blocks <= 6 && n_chunks >= 13 * sms;
}

static int check_chunk_bytes(long long chunk_bytes, const char* who) {
    if (chunk_bytes < 2 || (chunk_bytes & 1) || chunk_bytes / 2 / kBlockElems >= kMaxBlocks)
        return set_error(QSSB_ERR_INVALID, who);
    return QSSB_OK;
}

}  // namespace qssb

using namespace qssb;

extern "C" int qssb_decode_bslz4_u16(const uint8_t* compressed, int64_t compressed_bytes,
                                     const int64_t* chunk_offsets, int32_t n_chunks,
                                     int64_t chunk_bytes, uint16_t* out, int32_t* status,
                                     void* stream) {
    if (!compressed || !chunk_offsets || !out || n_chunks <= 0 || compressed_bytes <= 0)
        return set_error(QSSB_ERR_INVALID, "qssb_decode_bslz4_u16: null pointer or empty input");
    int rc = check_chunk_bytes(chunk_bytes, "qssb_decode_bslz4_u16: chunk_bytes must be even, "
                                            "at most 4 MB");
    if (rc) return rc;
    auto launch = [&](auto kern, int warps) {
        kern<<<n_chunks, 32 * warps, 0, (cudaStream_t)stream>>>(
            compressed, compressed_bytes, reinterpret_cast<const long long*>(chunk_offsets), n_chunks,
            chunk_bytes, out, status);
        note_launch();
    };
    if (decode_one_warp(n_chunks, chunk_blocks(chunk_bytes)))
        launch(k_decode_bslz4_u16<1>, 1);
    else
        launch(k_decode_bslz4_u16<kDecWarps>, kDecWarps);
    CUDA_TRY(cudaGetLastError());
    return QSSB_OK;
}

extern "C" int qssb_encode_bslz4_scratch_bytes(int32_t n_chunks, int64_t chunk_bytes,
                                               size_t* bytes) {
    if (!bytes || n_chunks <= 0)
        return set_error(QSSB_ERR_INVALID, "qssb_encode_bslz4_scratch_bytes: bad arguments");
    int rc = check_chunk_bytes(chunk_bytes, "qssb_encode_bslz4_scratch_bytes: chunk_bytes must be "
                                            "even, at most 4 MB");
    if (rc) return rc;
    *bytes = (size_t)n_chunks * (size_t)chunk_blocks(chunk_bytes) * kEncSlot;
    return QSSB_OK;
}

extern "C" int qssb_encode_bslz4_u16(const uint16_t* frames, int32_t n_chunks, int64_t chunk_bytes,
                                     uint8_t* scratch, int64_t* chunk_sizes, void* stream) {
    if (!frames || !scratch || !chunk_sizes || n_chunks <= 0)
        return set_error(QSSB_ERR_INVALID, "qssb_encode_bslz4_u16: null pointer or empty input");
    int rc = check_chunk_bytes(chunk_bytes, "qssb_encode_bslz4_u16: chunk_bytes must be even, "
                                            "at most 4 MB");
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int n_blocks = chunk_blocks(chunk_bytes);
    const long long n_slots = (long long)n_chunks * n_blocks;
    if (n_slots > 0) {
        const int smem = kEncWarps * kEncWarpBytes;
        const long long grid = (n_slots + kEncWarps - 1) / kEncWarps;
        if (grid > INT_MAX) return set_error(QSSB_ERR_INVALID, "qssb_encode_bslz4_u16: too many blocks");
        CUDA_TRY(cudaFuncSetAttribute(k_encode_bslz4_u16, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        { k_encode_bslz4_u16<<<(unsigned)grid, 32 * kEncWarps, smem, s>>>(frames, n_slots, n_blocks, chunk_bytes, scratch); note_launch(); }
        CUDA_TRY(cudaGetLastError());
    }
    { k_bslz4_chunk_sizes<<<(n_chunks + 255) / 256, 256, 0, s>>>(
        scratch, n_chunks, chunk_bytes, reinterpret_cast<long long*>(chunk_sizes)); note_launch(); }
    CUDA_TRY(cudaGetLastError());
    return QSSB_OK;
}

extern "C" int qssb_pack_bslz4(const uint8_t* scratch, const uint16_t* frames, int32_t n_chunks,
                               int64_t chunk_bytes, const int64_t* chunk_offsets, uint8_t* packed,
                               void* stream) {
    if (!scratch || !frames || !chunk_offsets || !packed || n_chunks <= 0)
        return set_error(QSSB_ERR_INVALID, "qssb_pack_bslz4: null pointer or empty input");
    int rc = check_chunk_bytes(chunk_bytes, "qssb_pack_bslz4: chunk_bytes must be even, at most 4 MB");
    if (rc) return rc;
    const int n_blocks = chunk_blocks(chunk_bytes);
    const long long n_items = (long long)n_chunks * (n_blocks > 0 ? n_blocks : 1);
    const long long grid = (n_items + kPackWarps - 1) / kPackWarps;
    if (grid > INT_MAX) return set_error(QSSB_ERR_INVALID, "qssb_pack_bslz4: too many blocks");
    { k_bslz4_pack<<<(unsigned)grid, 32 * kPackWarps, 0, (cudaStream_t)stream>>>(
        scratch, frames, n_items, n_blocks, chunk_bytes,
        reinterpret_cast<const long long*>(chunk_offsets), packed); note_launch(); }
    CUDA_TRY(cudaGetLastError());
    return QSSB_OK;
}
