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
// Decode: one CTA per chunk. Thread 0 walks the block chain (every offset
// checked against the chunk's end); each warp decodes a block's LZ4
// sequences into shared memory (every lane parses the token stream through
// L1, all lanes copy literals and matches - a match byte j reads
// out[op - off + j mod off], so overlapping matches need no serial copy) and
// bit-unshuffles the block with 8x8 bit transposes straight into the u16
// frame (16-byte stores). A malformed chunk sets status[c] (the block is
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

// Decode one LZ4 block from in[0, csz) (global memory, read through L1) into
// out[0, cap) (shared memory) by the whole warp. Every lane parses the token
// stream itself (the same bytes: broadcast reads, uniform control flow, no
// shuffles); literal and match bytes are copied lane-parallel. Returns true
// when the stream is well formed and fills exactly cap bytes.
__device__ bool lz4_block_warp(const uint8_t* __restrict__ in, int csz, uint8_t* out, int cap,
                               int lane) {
    int ip = 0, op = 0;
    for (int guard = 0; guard < kBlockBytes + 1; ++guard) {
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
        if (off >= ml) {  // no self-overlap: a plain copy
            for (int j = lane; j < ml; j += 32) out[op + j] = out[op - off + j];
        } else {
            // out[op + j] = out[op - off + (j mod off)]: reads only bytes before op
            int r = lane % off;
            const int step = 32 % off;
            for (int j = lane; j < ml; j += 32) {
                out[op + j] = out[op - off + r];
                r += step;
                if (r >= off) r -= off;
            }
        }
        op += ml;
        __syncwarp();
    }
    return false;
}

// Bit-unshuffle cnt (a multiple of 8) elements from a block's planes into dst.
__device__ __forceinline__ void unshuffle_store(const uint8_t* planes, int cnt, uint16_t* dst,
                                                bool vec, int lane) {
    const int P = cnt / 8;
    for (int p = lane; p < P; p += 32) {
        uint64_t lo = 0, hi = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            lo |= (uint64_t)planes[b * P + p] << (8 * b);
            hi |= (uint64_t)planes[(8 + b) * P + p] << (8 * b);
        }
        lo = transpose8(lo);  // byte j: bits 0..7 of element 8p + j
        hi = transpose8(hi);  // byte j: bits 8..15
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t e0 = (uint32_t)((lo >> (16 * q)) & 0xff) | ((uint32_t)((hi >> (16 * q)) & 0xff) << 8);
            const uint32_t e1 = (uint32_t)((lo >> (16 * q + 8)) & 0xff) | ((uint32_t)((hi >> (16 * q + 8)) & 0xff) << 8);
            w[q] = e0 | (e1 << 16);
        }
        uint16_t* o = dst + 8 * p;
        if (vec) {
            *reinterpret_cast<uint4*>(o) = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                o[2 * q] = (uint16_t)(w[q] & 0xffff);
                o[2 * q + 1] = (uint16_t)(w[q] >> 16);
            }
        }
    }
}

struct DecSmem {
    int start[kMaxBlocks];  // block's LZ4 data offset within the chunk
    int size[kMaxBlocks];
    int tail_at;            // raw leftover elements' offset
    int status;
};

__global__ void __launch_bounds__(32 * kDecWarps) k_decode_bslz4_u16(
    const uint8_t* __restrict__ comp, long long comp_bytes, const long long* __restrict__ offsets,
    int n_chunks, long long chunk_bytes, uint16_t* __restrict__ out, int* __restrict__ status) {
    extern __shared__ uint4 dec_smem4[];
    uint8_t* wbuf = reinterpret_cast<uint8_t*>(dec_smem4);  // per warp: one decoded block
    __shared__ DecSmem sh;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int c = blockIdx.x;
    const long long n_elem = chunk_bytes / 2;
    const long long n8 = n_elem & ~7LL;
    const int n_blocks = (int)((n8 + kBlockElems - 1) / kBlockElems);
    const long long c0 = offsets[c];
    const long long c1 = c + 1 < n_chunks ? offsets[c + 1] : comp_bytes;
    const uint8_t* ch = comp + c0;
    const long long len = c1 - c0;
    if (c0 >= 0 && c1 <= comp_bytes) {
        // the chunk's bytes into L1 (one prefetch per 128-byte line) before the
        // serial block-chain walk and the parses read them
        for (long long i = (long long)tid * 128; i < len; i += 128LL * 32 * kDecWarps)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(ch + i));
    }
    __syncthreads();
    if (tid == 0) {
        int st = kStOk;
        if (c0 < 0 || c1 > comp_bytes || len < 12) {
            st = kStHeader;
        } else {
            unsigned long long total = 0;
            for (int i = 0; i < 8; ++i) total = (total << 8) | ch[i];
            if ((long long)total != chunk_bytes || be32(ch + 8) != (uint32_t)kBlockBytes) st = kStHeader;
        }
        long long pos = 12;
        for (int i = 0; i < n_blocks && st == kStOk; ++i) {
            if (pos + 4 > len) { st = kStChain; break; }
            const long long csz = be32(ch + pos);
            if (csz > kLz4Bound || pos + 4 + csz > len) { st = kStChain; break; }
            sh.start[i] = (int)(pos + 4);
            sh.size[i] = (int)csz;
            pos += 4 + csz;
        }
        if (st == kStOk && pos + (n_elem - n8) * 2 > len) st = kStChain;
        sh.tail_at = (int)pos;
        sh.status = st;
        if (status) status[c] = st;  // blocks that fail raise it below
    }
    __syncthreads();
    uint16_t* frame = out + (size_t)c * n_elem;
    const bool vec = (n_elem & 7) == 0 && ((uintptr_t)out & 15u) == 0;
    if (sh.status != kStOk) {
        for (long long i = tid; i < n_elem; i += 32 * kDecWarps) frame[i] = 0;
        return;
    }
    uint8_t* out_buf = wbuf + (size_t)warp * kBlockBytes;
    for (int i = warp; i < n_blocks; i += kDecWarps) {
        const long long e0 = (long long)i * kBlockElems;
        const int cnt = (int)min((long long)kBlockElems, n8 - e0);
        const bool good = lz4_block_warp(ch + sh.start[i], sh.size[i], out_buf, 2 * cnt, lane);
        if (good) {
            unshuffle_store(out_buf, cnt, frame + e0, vec, lane);
        } else {
            for (int j = lane; j < cnt; j += 32) frame[e0 + j] = 0;
            if (lane == 0 && status) atomicMax(status + c, kStLz4);
        }
        __syncwarp();
    }
    if (warp == 0) {  // raw leftover elements
        const uint8_t* raw = ch + sh.tail_at;
        for (long long j = n8 + lane; j < n_elem; j += 32) {
            const long long b = (j - n8) * 2;
            frame[j] = (uint16_t)(raw[b] | (raw[b + 1] << 8));
        }
    }
}

// ------------------------------------------------------------------ encode
// Scratch layout: per (chunk, block) a slot of kEncSlot bytes holding the
// big-endian compressed size followed by the LZ4 block.
constexpr int kEncSlot = (4 + kLz4Bound + 15) & ~15;
constexpr int kEncWarps = 4;
// planes | hash table; the warps of a CTA share nothing
constexpr int kEncWarpBytes = kBlockBytes + 2 * kEncHash;

// Four bytes at any byte position of a 4-aligned shared buffer. The second
// word of an aligned position is read (it may be the first word of the hash
// table) and shifted out.
__device__ __forceinline__ uint32_t rd32(const uint8_t* base, int pos) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(base) + (pos >> 2);
    return __funnelshift_r(w[0], w[1], 8 * (pos & 3));
}

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
// many warps as the 16 KB of planes and table of each allow. 4096 frames of
// 128 x 128 counts: the whole call 0.73 ms against 4.00 ms with one lane
// searching byte by byte and copying (the same bytes).
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
// lane on the destination's alignment, the source words funnel-shifted. The
// first block's warp writes the chunk header, the last one's the raw leftovers.
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
    const int n_vec = (len - head) >> 4;
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
    const int done = head + 16 * n_vec;
    if (done + lane < len) dst[done + lane] = slot[done + lane];
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
    const size_t smem = (size_t)kDecWarps * kBlockBytes;
    CUDA_TRY(cudaFuncSetAttribute(k_decode_bslz4_u16, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
    { k_decode_bslz4_u16<<<n_chunks, 32 * kDecWarps, smem, (cudaStream_t)stream>>>(
        compressed, compressed_bytes, reinterpret_cast<const long long*>(chunk_offsets), n_chunks,
        chunk_bytes, out, status); note_launch(); }
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
