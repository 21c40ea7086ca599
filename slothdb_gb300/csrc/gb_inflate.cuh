// gb_inflate.cuh — page decompression (SNAPPY, ZSTD) with a block of threads
// per page.
//
// Both formats describe a page as a list of elements: literal bytes taken
// from the compressed stream and copies of earlier output.  Decoding it byte
// after byte is one long dependent chain, so the work is split into finding
// the elements (serial by nature, made short or spread over lanes) and
// producing the bytes, which a block does in windows of XW output bytes:
// every byte of a window gets its source in a shared map (a literal byte, or
// an earlier output byte); a source inside the window is followed through the
// map to one before the window or to a literal; then all bytes of the window
// are independent and are loaded and stored together.
#pragma once

#include "gb_kernels.cuh"
#include "gb_zstd.h"

namespace gb {

constexpr int XT = 512;              // threads of a block
constexpr int XW = 8192;             // output bytes of a window
constexpr int XPER = XW / XT;        // consecutive map entries one thread fills
constexpr int X_MAP = XW + XW / 16;  // map words, one pad word per 16 (a thread's 16 entries start in other banks)
constexpr u32 X_LIT = 0x80000000u;   // source: a literal (index in the low bits), else an output position

__device__ __forceinline__ u32 x_at(u32 b) { return b + (b >> 4); }

// dst[0, n) = src[0, n) by the whole block: words stored aligned, each from
// the two aligned source words it spans (an aligned word that holds a byte
// of the source can be read).
__device__ __forceinline__ void x_copy(uint8_t *dst, const uint8_t *src, u32 n) {
    const u32 head = min(n, (u32)(-(uintptr_t)dst & 3));
    if (threadIdx.x < head) dst[threadIdx.x] = src[threadIdx.x];
    const u32 nw = (n - head) >> 2, tail = head + 4 * nw;
    const uint8_t *s = src + head;
    const u32 sh = 8 * (u32)((uintptr_t)s & 3);
    const u32 *sw = (const u32 *)((uintptr_t)s & ~(uintptr_t)3);
    u32 *dw = (u32 *)(dst + head);
    for (u32 i = threadIdx.x; i < nw; i += XT) {
        const u32 lo = __ldg(sw + i);
        dw[i] = sh ? __funnelshift_r(lo, __ldg(sw + i + 1), sh) : lo;
    }
    if (threadIdx.x < n - tail) dst[tail + threadIdx.x] = src[tail + threadIdx.x];
}

// The n bytes of a window that starts at output position w0: sources in
// `map`, literals at lit.  A source is an earlier position than the byte it
// feeds, so following it ends; entries are replaced by what they lead to,
// which shortens the chains of the bytes behind (any value another thread
// reads meanwhile leads to the same byte).
__device__ __forceinline__ void x_write(volatile u32 *map, u32 n, u32 w0, uint8_t *dst, const uint8_t *lit) {
    for (u32 b0 = threadIdx.x; b0 < n; b0 += 4 * XT) {
        u32 s[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const u32 b = b0 + j * XT;
            s[j] = X_LIT;
            if (b < n) {
                u32 x = map[x_at(b)];
                if (!(x & X_LIT) && x >= w0) {
                    do {
                        x = map[x_at(x - w0)];
                    } while (!(x & X_LIT) && x >= w0);
                    map[x_at(b)] = x;
                }
                s[j] = x;
            }
        }
        uint8_t v[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (b0 + j * XT < n) v[j] = (s[j] & X_LIT) ? __ldg(lit + (s[j] & ~X_LIT)) : dst[s[j]];
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (b0 + j * XT < n) dst[w0 + b0 + j * XT] = v[j];
    }
}

// Exclusive scan of one value per thread over the block; *total gets the sum.
template <class T>
__device__ __forceinline__ T x_scan(T v, T *warp_sums, T *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    T before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < XT / 32; w++) {
        const T y = warp_sums[w];
        before += w < warp ? y : 0;
        all += y;
    }
    *total = all;
    __syncthreads();  // warp_sums is used again
    return before + x - v;
}

// One piece of a batch's decompressed image: `src_len` bytes at file offset
// `src` copied (mode 0), inflated from a raw Snappy block (mode 1, the codec
// of parquet.cpp:44-90, the vendored snappy 1.2.1) or from ZSTD frames (mode
// 2, parquet.cpp:693-736) into `dst_len` bytes at image offset `dst`.  lvl_slot != ~0: the piece is a page v1 of an
// OPTIONAL column, whose first 4 bytes (the level length) go to lvl[slot].
struct InflateJob {
    uint64_t src, dst;
    uint32_t src_len, dst_len;
    uint32_t mode, lvl_slot;
    uint64_t aux;          // ZSTD: the piece's place in the launch's literal and sequence scratch
    uint32_t blk, blk_cap; // ZSTD: first block descriptor, and how many it has
};

__device__ __forceinline__ void x_level(const InflateJob &J, const uint8_t *dst, bool bad, uint32_t *lvl) {
    if (J.lvl_slot == ~0u) return;
    uint32_t l4 = ~0u;  // too short to hold a level length: corrupt
    if (!bad && J.dst_len >= 4)
        l4 = (uint32_t)dst[0] | ((uint32_t)dst[1] << 8) | ((uint32_t)dst[2] << 16) | ((uint32_t)dst[3] << 24);
    lvl[J.lvl_slot] = l4;
}

// ------------------------------------------------------------------ Snappy
// The published format: a varint with the uncompressed length, then elements
// whose tag's low 2 bits say literal (00: length in the tag or in 1-4
// following bytes), or copy with a 1-, 2- or 4-byte offset (01/10/11) of an
// earlier output position, possibly overlapping the bytes it writes.
//
// Where an element starts is known only from the one before it.  The block
// takes SN_C compressed bytes at a time, computes for every position where
// the element that a tag there would be ends, and follows these jumps in
// three steps that all positions take at once: to the end of the position's
// 32 bytes, then of its 256 bytes, then (one thread, 16 hops) through the
// SN_C bytes; on the way back 16 threads enter the 32-byte pieces and 128
// threads mark the real starts in them.  A scan of the starts' output
// lengths places them.
constexpr int SN_C = 4096;  // compressed bytes parsed at a time
constexpr int SN_PER = SN_C / XT;

struct SnapShared {
    u32 map[X_MAP];
    union {
        struct {
            uint16_t j[SN_C], j32[SN_C], j256[SN_C];
        } jump;
        u32 o[SN_C];  // output place of each position's element (of the next one, where none starts)
    };
    u32 words[SN_C / 4 + 4];  // the compressed bytes, as aligned words
    u32 mask[SN_C / 32];
    uint16_t ent32[SN_C / 32], ent256[SN_C / 256];
    u32 sums[XT / 32];
    u32 next, job, ip, bad;
};

struct SnapElem {
    u32 lit, hdr, len, off, cs;
};

__device__ __forceinline__ SnapElem sn_decode(const uint8_t *c) {
    SnapElem e;
    const u32 tag = c[0], t = tag & 3u, l6 = tag >> 2;
    e.lit = t == 0;
    e.off = 0;
    if (t == 0) {
        u32 lraw = l6;
        e.hdr = 1;
        if (l6 >= 60) {
            const u32 nb = l6 - 59;
            lraw = 0;
            for (u32 k = 0; k < nb; k++) lraw |= (u32)c[1 + k] << (8 * k);
            e.hdr = 1 + nb;
        }
        e.len = lraw + 1;  // 0 after a wrap
        e.cs = lraw >= 0x7fff0000u ? 0x7fffffffu : e.hdr + lraw + 1;
    } else if (t == 1) {
        e.hdr = e.cs = 2;
        e.len = 4 + (l6 & 7u);
        e.off = ((tag >> 5) << 8) | c[1];
    } else {
        e.hdr = e.cs = t == 2 ? 3 : 5;
        e.len = l6 + 1;
        e.off = (u32)c[1] | ((u32)c[2] << 8);
        if (t == 3) e.off |= ((u32)c[3] << 16) | ((u32)c[4] << 24);
    }
    return e;
}

__device__ __forceinline__ bool sn_piece(const uint8_t *src, const u32 slen, uint8_t *dst, const u32 dlen,
                                         SnapShared &S) {
    const u32 t = threadIdx.x;
    if (t == 0) {  // the preamble: the uncompressed length
        u64 ulen = 0;
        u32 at = 0, bad = 0;
        int sh = 0;
        for (;;) {
            if (at >= slen || sh > 28) {
                bad = 1;
                break;
            }
            const uint8_t b = src[at++];
            ulen |= (u64)(b & 0x7f) << sh;
            if (!(b & 0x80)) break;
            sh += 7;
        }
        S.ip = at;
        S.bad = bad || ulen != dlen;
    }
    __syncthreads();
    u32 ip = S.ip, op = 0;
    if (S.bad) return false;
    while (op < dlen) {
        if (ip >= slen) return false;
        const u32 a = (u32)((uintptr_t)(src + ip) & 3);
        const u32 *blk = (const u32 *)(src + ip - a);
        // words with a byte of [ip, slen), up to SN_C + 8 bytes from ip
        for (u32 k = t; k < SN_C / 4 + 3; k += XT) S.words[k] = 4 * (u64)k < (u64)(slen - ip) + a ? __ldg(blk + k) : 0u;
        if (t < SN_C / 32) S.ent32[t] = 0xffff;
        if (t < SN_C / 256) S.ent256[t] = 0xffff;
        if (t == 0) S.next = 0;
        __syncthreads();
        const uint8_t *c = (const uint8_t *)S.words + a;
        const u32 avail = min((u32)SN_C, slen - ip);
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            const u32 i = t + k * XT;
            const u32 tag = c[i], ty = tag & 3u, l6 = tag >> 2;
            u32 cs = ty == 0 ? l6 + 2 : (ty == 1 ? 2u : (ty == 2 ? 3u : 5u));
            if (ty == 0 && l6 >= 60) cs = min(sn_decode(c + i).cs, 0x10000u);
            S.jump.j[i] = (uint16_t)min(i + cs, 0xffffu);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            const u32 i = t + k * XT, end = (i | 31) + 1;
            u32 e = S.jump.j[i];
            while (e < end) e = S.jump.j[e];
            S.jump.j32[i] = (uint16_t)e;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            const u32 i = t + k * XT, end = (i | 255) + 1;
            u32 e = S.jump.j32[i];
            while (e < end) e = S.jump.j32[e];
            S.jump.j256[i] = (uint16_t)e;
        }
        __syncthreads();
        if (t == 0)
            for (u32 e = 0; e < SN_C; e = S.jump.j256[e]) S.ent256[e >> 8] = (uint16_t)e;
        __syncthreads();
        if (t < SN_C / 256)
            for (u32 e = S.ent256[t]; e < (t + 1) * 256; e = S.jump.j32[e]) S.ent32[e >> 5] = (uint16_t)e;
        __syncthreads();
        if (t < SN_C / 32) {
            u32 m = 0;
            for (u32 e = S.ent32[t]; e < (t + 1) * 32; e = S.jump.j[e]) m |= 1u << (e & 31);
            S.mask[t] = m;
        }
        __syncthreads();
        // this thread's SN_PER positions: the starts' lengths and their checks.  Only the last start can be longer
        // than the compressed bytes it lies in: lengths are clamped for the scan.
        const u32 i0 = t * SN_PER, bits = (S.mask[i0 >> 5] >> (i0 & 31)) & ((1u << SN_PER) - 1);
        u32 sum = 0, end = 0;
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            if (((bits >> k) & 1u) && i0 + k < avail) {
                const SnapElem e = sn_decode(c + i0 + k);
                sum += min(e.len, 1u << 30);
                end = i0 + k + e.cs;
            }
        }
        u32 total, o = x_scan(sum, S.sums, &total);
        bool mybad = false;
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            S.o[i0 + k] = o;
            if (((bits >> k) & 1u) && i0 + k < avail) {
                const SnapElem e = sn_decode(c + i0 + k);
                const u64 at = (u64)op + o;
                // elements after the last output byte are ignored
                if (at < dlen && ((u64)ip + i0 + k + e.cs > slen || e.len == 0 || at + e.len > dlen ||
                                  (!e.lit && (e.off == 0 || e.off > at))))
                    mybad = true;
                o += min(e.len, 1u << 30);
            }
        }
        end = __reduce_max_sync(FULL, end);
        if ((t & 31) == 0) atomicMax(&S.next, end);
        if (__syncthreads_or(mybad)) return false;
        total = min(total, dlen - op);
        for (u32 w = 0; w < total; w += XW) {
            const u32 n = min((u32)XW, total - w);
            const u32 first = w + t * XPER;
            bool whole = true;  // one literal covers the window
            u32 from = 0;
            if (t * XPER < n) {
                u32 lo = 0, hi = SN_C;
                while (hi - lo > 1) {
                    const u32 mid = (lo + hi) >> 1;
                    if (S.o[mid] <= first) lo = mid;
                    else hi = mid;
                }
                u32 i = lo, e0 = S.o[i], b = first;
                SnapElem e = sn_decode(c + i);
                from = i + e.hdr;
                whole = e.lit && e0 <= w && (u64)e0 + e.len >= w + n;
                if (whole) {
                    from += w - e0;
                } else {
                    const u32 stop_all = min(first + XPER, w + n);
                    for (;;) {
                        const u32 stop = min(stop_all, e0 + min(e.len, 1u << 30));
                        if (e.lit) {
                            u32 s = X_LIT | (ip + i + e.hdr + (b - e0));
                            for (; b < stop; b++) S.map[x_at(b - w)] = s++;
                        } else {
                            const u32 m = b - e0, base = op + e0 - e.off;
                            u32 r = m < e.off ? m : m % e.off;
                            for (; b < stop; b++) {
                                S.map[x_at(b - w)] = base + r;
                                r = r + 1 == e.off ? 0 : r + 1;
                            }
                        }
                        if (b >= stop_all) break;
                        i += e.cs;
                        e0 = S.o[i];
                        e = sn_decode(c + i);
                    }
                }
            }
            if (__syncthreads_and(whole)) {
                if (t == 0) S.ip = from;
                __syncthreads();
                x_copy(dst + op + w, src + ip + S.ip, n);
            } else {
                x_write(S.map, n, op + w, dst, src);
            }
            __syncthreads();
        }
        op += total;
        ip += S.next;
        __syncthreads();
    }
    return true;
}

// Stored and SNAPPY pieces: a block claims pieces from a counter (the word
// after the last job, zero at launch), longest first, until none is left.
__global__ void __launch_bounds__(XT, 3) k_pq_inflate(const uint8_t *__restrict__ file, InflateJob *jobs, uint32_t n,
                                                      uint8_t *img, uint32_t *lvl, Ctl *ctl) {
    extern __shared__ __align__(16) unsigned char x_smem[];
    SnapShared &S = *(SnapShared *)x_smem;
    uint32_t *next = (uint32_t *)(jobs + n);
    for (;;) {
        if (threadIdx.x == 0) S.job = atomicAdd(next, 1u);
        __syncthreads();
        const u32 j = S.job;
        if (j >= n) return;
        const InflateJob J = jobs[j];
        uint8_t *dst = img + J.dst;
        bool ok = true;
        if (J.mode == 0) x_copy(dst, file + J.src, J.src_len);
        else ok = sn_piece(file + J.src, J.src_len, dst, J.dst_len, S);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (!ok) atomicOr(&ctl->err, (u32)ERR_CORRUPT);
            x_level(J, dst, !ok, lvl);
        }
        __syncthreads();  // S.job is written again
    }
}

// -------------------------------------------------------------------- ZSTD
// A frame (RFC 8878) is a chain of blocks of at most 128 KB; a block's
// literals and its sequences (literal length, match length, offset) are
// entropy-coded on their own, given the tables, so that all blocks of all
// pages decode at once:
//   k_pz_blocks   one thread per page walks the block headers into
//                 descriptors: where the literals and sequences lie, which
//                 earlier block described a table that this one repeats,
//                 where its decoded literals and sequences go in the scratch
//   k_pz_entropy  one warp per compressed block decodes its literals and its
//                 sequences.  Repeat offsets that reach back before the block
//                 stay symbolic (which of the three, less how much)
//   k_pz_bytes    one thread block per page, in order over its blocks:
//                 resolves the offsets and produces the bytes by windows
// A page that any step finds odd (several frames, more blocks than its
// descriptors, anything malformed) goes to a list and is decoded from the
// start by the serial decoder (k_pz_serial), whose verdict counts.
struct ZBlk {
    u64 src;                 // file offset of the block's content
    u32 size, type;          // 0 raw, 1 RLE, 2 compressed
    u32 piece;
    u32 lit_kind;            // 0 raw in the file, 1 RLE, 2 Huffman, 3 Huffman with an earlier table
    u32 lit_hdr, lit_csize, lsize, four;
    u32 seq_at, nseq;        // offset of the modes byte in the block, sequences
    u32 lit_off, seq_off;    // places in the piece's scratch
    u32 first;               // first block of its frame: the repeat offsets start as 1, 4, 8
    u32 def_huf, def_tab[3]; // descriptors of the blocks that describe this one's tables (LL, OF, ML)
    u32 bad, used, rep[3];   // k_pz_entropy: malformed, literals its sequences take, repeat offsets after it
    u32 pad;
};

struct ZWork {
    u32 n_list, claim_entropy, claim_bytes, n_odd;
};

struct ZArgs {
    const uint8_t *file;
    InflateJob *jobs;
    u32 n, pad;
    uint8_t *img;
    u32 *lvl;
    Ctl *ctl;
    ZBlk *blk;
    u32 *n_blk;     // per piece
    u32 *list;      // compressed blocks
    u32 *odd;       // pieces for the serial decoder
    ZWork *work;
    uint8_t *lits;
    u32 *seq_ll, *seq_ml, *seq_off;
};

constexpr u32 Z_SYM = 0x80000000u;  // a symbolic offset: bits 29, 30 which repeat offset, below them how much less

__device__ __forceinline__ u32 z_le(const uint8_t *p, int n) {
    u32 v = 0;
    for (int k = 0; k < n; k++) v |= (u32)p[k] << (8 * k);
    return v;
}

// The blocks of one page into descriptors; false: for the serial decoder.
__device__ __forceinline__ bool pz_walk(const ZArgs &A, u32 piece, const InflateJob &J, u32 *n_blocks) {
    const uint8_t *src = A.file + J.src;
    const int64_t n = J.src_len;
    if (n < 6 || z_le(src, 4) != 0xFD2FB528u) return false;
    const u32 fhd = src[4];
    if (fhd & 8) return false;
    const u32 single = (fhd >> 5) & 1, did = fhd & 3, fcs = fhd >> 6;
    if (did) return false;
    int64_t ip = 5 + (single ? 0 : 1) + (fcs == 0 ? (single ? 1 : 0) : (1 << fcs));
    ZBlk *B = A.blk + J.blk;
    u32 k = 0, lit = 0, seq = 0, def_huf = ~0u, def[3] = {~0u, ~0u, ~0u};
    for (;;) {
        if (n - ip < 3 || k >= J.blk_cap) return false;
        const u32 bh = z_le(src + ip, 3), type = (bh >> 1) & 3, size = bh >> 3;
        ip += 3;
        const u32 in_file = type == 1 ? 1 : size;
        if (type == 3 || (int64_t)in_file > n - ip) return false;
        ZBlk D;
        memset(&D, 0, sizeof D);
        D.src = J.src + (u64)ip;
        D.size = size;
        D.type = type;
        D.piece = piece;
        D.first = k == 0;
        if (type == 2) {
            if (size > gbz::ZS_BLOCK_MAX || size < 2) return false;
            const uint8_t *c = src + ip;
            const u32 b0 = c[0], lt = b0 & 3, sf = (b0 >> 2) & 3;
            D.lit_kind = lt;
            if (lt < 2) {
                D.lit_hdr = sf == 1 ? 2 : (sf == 3 ? 3 : 1);
                if (D.lit_hdr >= size) return false;
                const u32 v = z_le(c, (int)D.lit_hdr);
                D.lsize = D.lit_hdr == 1 ? v >> 3 : v >> 4;
                D.lit_csize = lt == 0 ? D.lsize : 1;
            } else {
                D.lit_hdr = sf < 2 ? 3 : sf + 2;
                if (D.lit_hdr >= size) return false;
                const u32 bits = sf < 2 ? 10 : (sf == 2 ? 14 : 18);
                const u64 v = (u64)z_le(c, 3) | ((u64)z_le(c + 3, (int)D.lit_hdr - 3) << 24);
                D.lsize = (u32)(v >> 4) & ((1u << bits) - 1);
                D.lit_csize = (u32)(v >> (4 + bits)) & ((1u << bits) - 1);
                D.four = sf != 0;
                if (lt == 2) def_huf = J.blk + k;
                D.def_huf = def_huf;
                if (def_huf == ~0u) return false;
            }
            if (D.lsize > gbz::ZS_BLOCK_MAX) return false;
            u32 at = D.lit_hdr + D.lit_csize;
            if (at >= size) return false;
            u32 ns = c[at++];
            if (ns >= 128) {
                const int more = ns < 255 ? 1 : 2;
                if (at + more > size) return false;
                ns = more == 1 ? ((ns - 128) << 8) + c[at] : z_le(c + at, 2) + 0x7F00;
                at += more;
            }
            D.nseq = ns;
            D.seq_at = at;
            if (ns) {
                if (at >= size) return false;
                const u32 modes = c[at];
                if (modes & 3) return false;
                for (int x = 0; x < 3; x++) {
                    if (((modes >> (6 - 2 * x)) & 3) != 3) def[x] = J.blk + k;
                    if (def[x] == ~0u) return false;
                    D.def_tab[x] = def[x];
                }
            } else if (at != size) {
                return false;
            }
            D.lit_off = lit;
            D.seq_off = seq;
            lit += lt == 0 ? 0 : D.lsize;
            seq += ns;
            // a literal and three bytes of a match are output bytes each
            if (lit > J.dst_len || (u64)seq * 3 > J.dst_len) return false;
        }
        B[k++] = D;
        ip += in_file;
        if (bh & 1) break;
    }
    if ((fhd >> 2) & 1) ip += 4;  // checksum
    *n_blocks = k;
    return ip == n;
}

__global__ void __launch_bounds__(128) k_pz_blocks(const __grid_constant__ ZArgs A) {
    const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= A.n) return;
    const InflateJob J = A.jobs[j];
    u32 k = 0;
    if (!pz_walk(A, j, J, &k)) {
        A.n_blk[j] = 0;
        A.odd[atomicAdd(&A.work->n_odd, 1u)] = j;
        return;
    }
    A.n_blk[j] = k;
    u32 nc = 0;
    for (u32 i = 0; i < k; i++) nc += A.blk[J.blk + i].type == 2;
    u32 at = nc ? atomicAdd(&A.work->n_list, nc) : 0;
    for (u32 i = 0; i < k; i++)
        if (A.blk[J.blk + i].type == 2) A.list[at++] = J.blk + i;
}

// One warp's tables.  The Huffman table is used up before the sequence
// tables are built.
constexpr int ZE_WARPS = 4;
constexpr int Z_LL = 0, Z_OF = 512, Z_ML = 768, Z_CELLS = 1280;
struct alignas(16) ZTables {  // the ring is written 16 bytes at a time
    union {
        uint16_t huf[1u << gbz::ZS_HUF_LOG];
        // sequence cells: next state's baseline (16 bits) | its bits (8) | its bits + the code's extra bits (8)
        u32 cell[Z_CELLS];
    };
    union {
        u32 wt[64];
        u32 ring[256];  // two 512-byte pieces of the sequences' bit stream
    };
    uint8_t sym[Z_CELLS];
    int q[32];      // per sequence of a batch: stream position before it, and its three states
    u32 state[32];
    int log[3], at, bad;
};

// A described table's bytes, -1 if malformed.
__device__ __forceinline__ int64_t pz_skip(u32 mode, int which, const uint8_t *p, int64_t n) {
    if (mode == 1) return n < 1 ? -1 : 1;
    if (mode != 2) return 0;
    int16_t norm[64];
    int ns, log;
    return gbz::zs_read_ncount(p, n, which == 1 ? gbz::ZS_OF_LOG : gbz::ZS_LL_LOG, which == 0 ? 36 : (which == 1 ? 32 : 53),
                               norm, &ns, &log);
}

// The three sequence tables of block b into T (one lane); T.at: offset of
// the bit stream in the block.
__device__ __noinline__ bool pz_tables(const ZArgs &A, const ZBlk &b, ZTables &T) {
    for (int x = 0; x < 3; x++) {
        const ZBlk &D = A.blk[b.def_tab[x]];
        const uint8_t *p = A.file + D.src + D.seq_at;
        const int64_t n = (int64_t)D.size - D.seq_at;
        const u32 modes = p[0];
        int64_t pos = 1;
        for (int y = 0; y < x; y++) {
            const int64_t u = pz_skip((modes >> (6 - 2 * y)) & 3, y, p + pos, n - pos);
            if (u < 0) return false;
            pos += u;
        }
        bool have = false;
        const int64_t u = gbz::zs_seq_table((int)(modes >> (6 - 2 * x)) & 3, x, p + pos, n - pos,
                                            T.cell + (x == 0 ? Z_LL : (x == 1 ? Z_OF : Z_ML)), nullptr, &T.log[x],
                                            x == 1 ? gbz::ZS_OF_LOG : gbz::ZS_LL_LOG, x == 0 ? 36 : (x == 1 ? 32 : 53),
                                            &have);
        if (u < 0) return false;
    }
    const uint8_t *p = A.file + b.src + b.seq_at;
    const int64_t n = (int64_t)b.size - b.seq_at;
    int64_t pos = 1;
    for (int y = 0; y < 3; y++) {
        const int64_t u = pz_skip(((u32)p[0] >> (6 - 2 * y)) & 3, y, p + pos, n - pos);
        if (u < 0) return false;
        pos += u;
    }
    T.at = (int)(b.seq_at + pos);
    return true;
}

// Bits [q, q + n) of the ring, n <= 31.
__device__ __forceinline__ u32 z_rd(const u32 *ring, int q, int n) {
    const int w = q >> 5;
    return __funnelshift_r(ring[w & 255], ring[(w + 1) & 255], q & 31) & ((1u << n) - 1);
}

__device__ __forceinline__ u32 z_less(u32 r) { return (r & Z_SYM) ? r + 1 : r - 1; }

// The literals of block b (Huffman, RLE) into the scratch, by one warp.
__device__ __forceinline__ bool pz_literals(const ZArgs &A, const ZBlk &b, uint8_t *out, ZTables &T, int lane) {
    const uint8_t *c = A.file + b.src + b.lit_hdr;
    if (b.lit_kind == 1) {
        const uint8_t v = c[0];
        for (u32 i = lane; i < b.lsize; i += 32) out[i] = v;
        return true;
    }
    if (lane == 0) {
        const ZBlk &D = A.blk[b.def_huf];
        int mb = 0;
        const int64_t used = gbz::zs_huf_table(A.file + D.src + D.lit_hdr, D.lit_csize, T.huf, T.wt, &mb);
        T.at = b.lit_kind == 2 ? (int)used : 0;
        T.log[0] = mb;
        T.bad = used < 0;
    }
    __syncwarp();
    if (T.bad) return false;
    const uint8_t *p = c + T.at;
    const int64_t cn = (int64_t)b.lit_csize - T.at;
    bool ok = true;
    if (!b.four) {
        if (lane == 0) ok = gbz::zs_huf_stream(p, cn, T.huf, T.log[0], out, b.lsize);
    } else {
        const int64_t seg = ((int64_t)b.lsize + 3) / 4;
        if (cn < 6 || 3 * seg > (int64_t)b.lsize) return false;
        const int64_t s1 = z_le(p, 2), s2 = z_le(p + 2, 2), s3 = z_le(p + 4, 2), s4 = cn - 6 - s1 - s2 - s3;
        if (s4 < 0) return false;
        if (lane < 4) {
            const int64_t at = 6 + (lane > 0 ? s1 : 0) + (lane > 1 ? s2 : 0) + (lane > 2 ? s3 : 0);
            const int64_t len = lane == 0 ? s1 : (lane == 1 ? s2 : (lane == 2 ? s3 : s4));
            ok = gbz::zs_huf_stream(p + at, len, T.huf, T.log[0], out + lane * seg,
                                    lane < 3 ? seg : (int64_t)b.lsize - 3 * seg);
        }
    }
    return __all_sync(FULL, ok);
}

// The sequences of block b into the scratch, by one warp: the first lane
// follows the three states through the bit stream, noting each sequence's
// position and states, 32 at a time; then every lane reads one sequence's
// extra bits.  The stream is kept in shared memory, the next 512 bytes
// already in registers.  What bounds it: the first lane's chain of one table
// load, the bit count's addition and the extraction of the next states per
// sequence.
__device__ __forceinline__ bool pz_sequences(const ZArgs &A, ZBlk &b, u64 base, ZTables &T, int lane) {
    if (lane == 0) T.bad = !pz_tables(A, b, T);
    __syncwarp();
    if (T.bad) return false;
#pragma unroll
    for (int x = 0; x < 3; x++) {
        const int at = x == 0 ? Z_LL : (x == 1 ? Z_OF : Z_ML);
        for (int i = lane; i < (1 << T.log[x]); i += 32) {
            const u32 c = T.cell[at + i], s = c & 0xffu, nb = (c >> 8) & 0xffu;
            u32 xb;
            int xn = (int)s;
            if (x == 0) gbz::zs_ll(s, &xb, &xn);
            if (x == 2) gbz::zs_ml(s, &xb, &xn);
            T.cell[at + i] = (c >> 16) | (nb << 16) | ((nb + (u32)xn) << 24);
            T.sym[at + i] = (uint8_t)s;
        }
    }
    const uint8_t *sb = A.file + b.src + T.at;
    const int size = (int)b.size - T.at;
    if (size <= 0) return false;
    const u32 last = sb[size - 1];
    if (last == 0) return false;
    // positions are bits from the 16-byte boundary at or below the stream's first byte
    const int d = (int)((uintptr_t)sb & 15);
    const uint8_t *al = sb - d;
    const int q_end = 8 * d;
    int q = q_end + (size - 1) * 8 + (31 - __clz(last));
    auto load = [&](int blk) {  // 16 bytes per lane of piece blk (pieces that hold no byte of the stream: zeros)
        const int at = blk * 512 + lane * 16;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (blk >= 0 && at < d + size) v = __ldg((const uint4 *)(al + at));
        return v;
    };
    int low = ((q - 1) >> 12) - 1;  // lowest piece in the ring
    ((uint4 *)T.ring)[((low + 1) & 1) * 32 + lane] = load(low + 1);
    ((uint4 *)T.ring)[(low & 1) * 32 + lane] = load(low);
    uint4 ahead = load(low - 1);
    __syncwarp();
    u32 sl = 0, so = 0, sm = 0;
    if (lane == 0) {
        q -= T.log[0];
        sl = z_rd(T.ring, q, T.log[0]);
        q -= T.log[1];
        so = z_rd(T.ring, q, T.log[1]);
        q -= T.log[2];
        sm = z_rd(T.ring, q, T.log[2]);
    }
    q = __shfl_sync(FULL, q, 0);
    u32 r0 = b.first ? 1 : Z_SYM, r1 = b.first ? 4 : Z_SYM | (1u << 29), r2 = b.first ? 8 : Z_SYM | (2u << 29);
    u64 lits = 0;
    bool bad = false;
    const u32 nseq = b.nseq;
    for (u32 k0 = 0; k0 < nseq; k0 += 32) {
        const int cnt = (int)min(32u, nseq - k0);
        // a batch reads at most 32 * 89 bits below q
        while (low > ((q - 1) >> 12) - 1) {
            low--;
            ((uint4 *)T.ring)[(low & 1) * 32 + lane] = ahead;
            ahead = load(low - 1);
        }
        __syncwarp();
        if (lane == 0) {
            const bool final = k0 + 32 >= nseq;
            for (int k = 0; k < cnt; k++) {
                // the 64 bits below q, loaded beside the cells
                const int w = (q - 64) >> 5;
                const u32 a0 = T.ring[w & 255], a1 = T.ring[(w + 1) & 255], a2 = T.ring[(w + 2) & 255];
                const u32 cl = T.cell[Z_LL + sl], co = T.cell[Z_OF + so], cm = T.cell[Z_ML + sm];
                T.q[k] = q;
                T.state[k] = sl | (sm << 9) | (so << 18);
                const u32 nl = (cl >> 16) & 0xffu, nm = (cm >> 16) & 0xffu, no = (co >> 16) & 0xffu;
                const int take = (int)((cl >> 24) + (co >> 24) + (cm >> 24));
                if (final && k + 1 == cnt) {  // the last sequence: no next states
                    q -= take - (int)(nl + nm + no);
                    break;
                }
                q -= take;
                u32 v = 0;
                if (take <= 64) {
                    const u32 sh = (u32)(q + take) & 31;
                    const u64 win = ((u64)__funnelshift_r(a1, a2, sh) << 32) | __funnelshift_r(a0, a1, sh);
                    if (take) v = (u32)(win >> (64 - take));
                } else {
                    const int ww = q >> 5;
                    v = __funnelshift_r(T.ring[ww & 255], T.ring[(ww + 1) & 255], q & 31);
                }
                so = (co & 0xffffu) + (v & ((1u << no) - 1));
                sm = (cm & 0xffffu) + ((v >> no) & ((1u << nm) - 1));
                sl = (cl & 0xffffu) + ((v >> (no + nm)) & ((1u << nl) - 1));
            }
        }
        __syncwarp();
        u32 ll = 0, ml = 0, off = 4;  // off: the offset value until resolved
        if (lane < cnt) {
            const u32 st = T.state[lane];
            u32 lb, mb;
            int xl, xm;
            const int xo = T.sym[Z_OF + (st >> 18)];
            gbz::zs_ll(T.sym[Z_LL + (st & 511)], &lb, &xl);
            gbz::zs_ml(T.sym[Z_ML + ((st >> 9) & 511)], &mb, &xm);
            int p = T.q[lane] - xo;
            off = (1u << xo) + z_rd(T.ring, p, xo);
            p -= xm;
            ml = mb + z_rd(T.ring, p, xm);
            p -= xl;
            ll = lb + z_rd(T.ring, p, xl);
            if (off > 3 && ((off - 3) & Z_SYM)) bad = true;
        }
        lits += __reduce_add_sync(FULL, ll);
        q = __shfl_sync(FULL, q, 0);
        if (!__any_sync(FULL, off <= 3)) {  // every offset is a new one
            off -= 3;
            const u32 n0 = __shfl_sync(FULL, off, cnt - 1), n1 = __shfl_sync(FULL, off, max(cnt - 2, 0)),
                      n2 = __shfl_sync(FULL, off, max(cnt - 3, 0));
            r2 = cnt > 2 ? n2 : (cnt > 1 ? r0 : r1);
            r1 = cnt > 1 ? n1 : r0;
            r0 = n0;
        } else {
            u32 mine = 0;
            for (int k = 0; k < cnt; k++) {
                const u32 v = __shfl_sync(FULL, off, k), zero = __shfl_sync(FULL, ll, k) == 0;
                u32 o;
                if (v > 3) {
                    o = v - 3;
                    r2 = r1;
                    r1 = r0;
                    r0 = o;
                } else {
                    const u32 idx = zero ? v : v - 1;  // 0..3
                    o = idx == 0 ? r0 : (idx == 1 ? r1 : (idx == 2 ? r2 : z_less(r0)));
                    if (idx >= 2) r2 = r1;
                    if (idx >= 1) {
                        r1 = r0;
                        r0 = o;
                    }
                }
                if (lane == k) mine = o;
            }
            off = mine;
        }
        if (lane < cnt) {
            A.seq_ll[base + k0 + lane] = ll;
            A.seq_ml[base + k0 + lane] = ml;
            A.seq_off[base + k0 + lane] = off;
        }
    }
    if (lane == 0) {
        b.used = (u32)min(lits, (u64)0xffffffffu);
        b.rep[0] = r0;
        b.rep[1] = r1;
        b.rep[2] = r2;
    }
    return !__any_sync(FULL, bad) && q == q_end && lits <= b.lsize;
}

__global__ void __launch_bounds__(ZE_WARPS * 32) k_pz_entropy(const __grid_constant__ ZArgs A) {
    static_assert(sizeof(ZTables) % 16 == 0 && offsetof(ZTables, ring) % 16 == 0, "ring alignment");
    __shared__ ZTables s_tab[ZE_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ZTables &T = s_tab[warp];
    const u32 n = A.work->n_list;
    for (;;) {
        u32 i = 0;
        if (lane == 0) i = atomicAdd(&A.work->claim_entropy, 1u);
        i = __shfl_sync(FULL, i, 0);
        if (i >= n) return;  // the whole warp
        ZBlk &b = A.blk[A.list[i]];
        const InflateJob &J = A.jobs[b.piece];
        bool ok = true;
        if (b.lit_kind != 0) ok = pz_literals(A, b, A.lits + J.aux + b.lit_off, T, lane);
        __syncwarp();
        if (ok && b.nseq) {
            ok = pz_sequences(A, b, J.aux / 3 + b.seq_off, T, lane);
        } else if (lane == 0 && !b.nseq) {  // the repeat offsets pass through
            b.used = 0;
            for (u32 x = 0; x < 3; x++) b.rep[x] = b.first ? (x == 0 ? 1 : 4 * x) : Z_SYM | (x << 29);
        }
        if (lane == 0) b.bad = !ok;
        __syncwarp();
    }
}

constexpr int ZB_SEQ = 2 * XT;  // sequences of a batch
struct ZByteShared {
    u32 map[X_MAP];
    u32 o[ZB_SEQ + 1], l[ZB_SEQ + 1], off[ZB_SEQ];  // per sequence: output place, literal place, offset
    u64 sums[XT / 32];
    u32 job;
};

__device__ __forceinline__ u32 z_offset(u32 v, u32 r0, u32 r1, u32 r2) {
    if (!(v & Z_SYM)) return v;
    const u32 k = (v >> 29) & 3, less = v & 0x1fffffffu, r = k == 0 ? r0 : (k == 1 ? r1 : r2);
    return r > less ? r - less : 0;
}

// One compressed block's bytes at dst + op.
__device__ __forceinline__ bool pz_block_bytes(const ZArgs &A, const InflateJob &J, const ZBlk &b, uint8_t *dst, u32 &op,
                                               u32 r0, u32 r1, u32 r2, ZByteShared &S) {
    const u32 t = threadIdx.x, cap = J.dst_len;
    if (b.bad) return false;
    const uint8_t *lit = b.lit_kind == 0 ? A.file + b.src + b.lit_hdr : A.lits + J.aux + b.lit_off;
    const u64 base = J.aux / 3 + b.seq_off;
    u32 lp = 0;
    for (u32 k0 = 0; k0 < b.nseq; k0 += ZB_SEQ) {
        const u32 cnt = min((u32)ZB_SEQ, b.nseq - k0);
        u32 ll[2] = {0, 0}, ml[2] = {0, 0}, off[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const u32 i = 2 * t + k;
            if (i < cnt) {
                ll[k] = A.seq_ll[base + k0 + i];
                ml[k] = A.seq_ml[base + k0 + i];
                off[k] = z_offset(A.seq_off[base + k0 + i], r0, r1, r2);
            }
        }
        // output places in the low half, literal places in the high half
        u64 total;
        u64 at = x_scan((u64)(ll[0] + ml[0] + ll[1] + ml[1]) | ((u64)(ll[0] + ll[1]) << 32), S.sums, &total);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const u32 i = 2 * t + k, o = (u32)at, l = (u32)(at >> 32);
            S.o[i] = o;
            S.l[i] = l;
            S.off[i] = off[k];
            if (i < cnt)
                bad |= (u64)lp + l + ll[k] > b.lsize || (u64)op + o + ll[k] + ml[k] > cap || off[k] == 0 ||
                       off[k] > op + o + ll[k];
            at += (u64)(ll[k] + ml[k]) | ((u64)ll[k] << 32);
        }
        if (t == 0) {
            S.o[ZB_SEQ] = (u32)total;
            S.l[ZB_SEQ] = (u32)(total >> 32);
        }
        if (__syncthreads_or(bad)) return false;
        const u32 all = (u32)total;
        for (u32 w = 0; w < all; w += XW) {
            const u32 n = min((u32)XW, all - w);
            if (t * XPER < n) {
                u32 bt = w + t * XPER;
                const u32 stop_all = min(bt + XPER, w + n);
                u32 i = 0, hi = ZB_SEQ;
                while (hi - i > 1) {
                    const u32 mid = (i + hi) >> 1;
                    if (S.o[mid] <= bt) i = mid;
                    else hi = mid;
                }
                for (;; i++) {
                    const u32 e0 = S.o[i], l0 = S.l[i], mat = e0 + (S.l[i + 1] - l0), end = min(S.o[i + 1], stop_all);
                    if (bt < mat) {
                        const u32 stop = min(mat, stop_all);
                        u32 s = X_LIT | (lp + l0 + (bt - e0));
                        for (; bt < stop; bt++) S.map[x_at(bt - w)] = s++;
                    }
                    if (bt < end) {
                        const u32 of = S.off[i], m = bt - mat, from = op + mat - of;
                        u32 r = m < of ? m : m % of;
                        for (; bt < end; bt++) {
                            S.map[x_at(bt - w)] = from + r;
                            r = r + 1 == of ? 0 : r + 1;
                        }
                    }
                    if (bt >= stop_all) break;
                }
            }
            __syncthreads();
            x_write(S.map, n, op + w, dst, lit);
            __syncthreads();
        }
        op += all;
        lp += (u32)(total >> 32);
    }
    const u32 rest = b.lsize - lp;  // lp <= lsize: checked above
    if (rest > cap - op) return false;
    x_copy(dst + op, lit + lp, rest);
    op += rest;
    return true;
}

__global__ void __launch_bounds__(XT, 3) k_pz_bytes(const __grid_constant__ ZArgs A) {
    extern __shared__ __align__(16) unsigned char x_smem[];
    ZByteShared &S = *(ZByteShared *)x_smem;
    for (;;) {
        if (threadIdx.x == 0) S.job = atomicAdd(&A.work->claim_bytes, 1u);
        __syncthreads();
        const u32 j = S.job;
        if (j >= A.n) return;
        const u32 nb = A.n_blk[j];
        const InflateJob J = A.jobs[j];
        uint8_t *dst = A.img + J.dst;
        bool ok = nb != 0;
        u32 op = 0, r0 = 1, r1 = 4, r2 = 8;
        for (u32 k = 0; ok && k < nb; k++) {
            const ZBlk &b = A.blk[J.blk + k];
            if (b.type == 2) {
                ok = pz_block_bytes(A, J, b, dst, op, r0, r1, r2, S);
                const u32 n0 = z_offset(b.rep[0], r0, r1, r2), n1 = z_offset(b.rep[1], r0, r1, r2),
                          n2 = z_offset(b.rep[2], r0, r1, r2);
                r0 = n0;
                r1 = n1;
                r2 = n2;
            } else if (b.size > J.dst_len - op) {
                ok = false;
            } else {
                if (b.type == 0) {
                    x_copy(dst + op, A.file + b.src, b.size);
                } else {
                    const uint8_t v = A.file[b.src];
                    for (u32 i = threadIdx.x; i < b.size; i += XT) dst[op + i] = v;
                }
                op += b.size;
            }
            __syncthreads();
        }
        ok = ok && op == J.dst_len;
        if (threadIdx.x == 0 && nb) {  // without blocks the piece is already on the list
            if (ok) x_level(J, dst, false, A.lvl);
            else A.odd[atomicAdd(&A.work->n_odd, 1u)] = j;
        }
        __syncthreads();
    }
}

// The pieces that the steps above left: one warp per piece, its first lane
// decoding with the warp's 13.3 KB of tables in `scratch`.  A frame that
// does not decode to exactly dst_len bytes sets ERR_CORRUPT.
__global__ void __launch_bounds__(128, 5) k_pz_serial(const __grid_constant__ ZArgs A, gbz::ZsScratch *scratch) {
    if ((threadIdx.x & 31) != 0) return;
    const u32 me = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = gridDim.x * (blockDim.x >> 5);
    gbz::ZsScratch &Z = scratch[me];
    const u32 n = A.work->n_odd;
    for (u32 i = me; i < n; i += warps) {
        const InflateJob J = A.jobs[A.odd[i]];
        uint8_t *dst = A.img + J.dst;
        const int64_t got = gbz::zstd_decompress(A.file + J.src, J.src_len, dst, J.dst_len, Z);
        const bool bad = got != (int64_t)J.dst_len;
        if (bad) atomicOr(&A.ctl->err, (u32)ERR_CORRUPT);
        x_level(J, dst, bad, A.lvl);
    }
}

}  // namespace gb
