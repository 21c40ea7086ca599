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
//
// 8M-row file of INT32 dictionary, INT16 and INT64 PLAIN columns (1M-row
// groups, 65,536-row pages, 113 MB of page bytes): SNAPPY 20.0 -> 1.16 ms,
// ZSTD 50.8 -> 3.10 ms (blocks 0.02, entropy 2.43, bytes 0.65 ms) against one
// warp per page.  What is left is the chain of the longest page: 50 pieces of
// 8 KB (SNAPPY), a block of 31,600 sequences at ~115 cycles each (ZSTD).
#pragma once

#include "gb_kernels.cuh"
#include "gb_zstd.h"

namespace gb {

constexpr int XT = 1024;     // threads of a block
constexpr int X_CTAS = 1;   // blocks of an SM: 64 registers a thread (two of 32 registers spill and took 1.4 times as long)
constexpr int XW = 16384;    // output bytes of a window
constexpr u32 X_HIST = 32768;  // latest output bytes kept in shared memory (most copies reach less far back)
constexpr u32 X_LIT = 0x80000000u;  // source: a literal (index in the low bits), else an output position
constexpr u32 X_LONG = 64;   // an element over this length is filled by a warp
constexpr int X_NLONG = XW / X_LONG + 2;  // at most so many of them touch a window

struct XLong {
    u32 at, len, base, period;  // output place (of the batch), bytes, first source, its period (copies)
};
struct alignas(16) XShared {
    u32 map[XW + 8];  // of a window's byte at output position p: entry p - (window's position rounded down to 4)
    uint8_t hist[X_HIST];
    XLong lng[X_NLONG];
    u32 n_long[2];  // this window's, the next one's
};

// One element's sources into the map of window [w, w + n) of a batch that
// starts at output position op: its bytes [at, at + len) come from base on,
// repeating after `period` bytes.
__device__ __forceinline__ void x_fill(XShared &X, u32 op, u32 w, u32 n, int par, u32 at, u32 len, u32 base, u32 period) {
    const u32 b0 = max(at, w), b1 = min(at + len, w + n);
    if (b0 >= b1) return;
    if (b1 - b0 > X_LONG) {
        X.lng[atomicAdd(&X.n_long[par], 1u)] = {at, len, base, period};
        return;
    }
    u32 r = b0 - at;
    if (r >= period) r %= period;
    u32 *m = X.map + (b0 - w + ((op + w) & 3)), *end = m + (b1 - b0);
    for (; m < end; m++) {
        *m = base + r;
        r = r + 1 == period ? 0 : r + 1;
    }
}

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

// The n bytes of window [w, w + n) of a batch that starts at output position
// op, once every element is in the map or on the long list: literals at lit
// (those with an index of lit_near + [0, near_n) in shared memory at near),
// earlier output in the ring from position `from` on (until the window itself
// takes its place), else in dst.  A source is an earlier position than the
// byte it feeds, so following it ends; entries are replaced by what they lead
// to, which shortens the chains of the bytes behind (any value another thread
// reads meanwhile leads to the same byte).  A thread makes four bytes at a
// time.  Ends with a barrier.
__device__ __forceinline__ void x_write(XShared &X, u32 w, u32 n, int par, u32 op, uint8_t *dst, const uint8_t *lit,
                                        const uint8_t *near, u32 lit_near, u32 near_n, u32 &from) {
    __syncthreads();
    const u32 nl = X.n_long[par], w0 = op + w, wa = w0 & ~3u;
    if (threadIdx.x == 0) X.n_long[par ^ 1] = 0;
    if (nl) {
        const XLong L0 = X.lng[0];
        if (nl == 1 && (L0.base & X_LIT) && L0.at <= w && L0.at + L0.len >= w + n) {  // one literal covers the window
            x_copy(dst + w0, lit + (L0.base & ~X_LIT) + (w - L0.at), n);
            from = w0 + n;  // not in the ring
            __syncthreads();
            return;
        }
        for (u32 i = threadIdx.x >> 5; i < nl; i += XT / 32) {
            const XLong L = X.lng[i];
            const u32 b0 = max(L.at, w), b1 = min(L.at + L.len, w + n);
            for (u32 b = b0 + (threadIdx.x & 31); b < b1; b += 32) {
                u32 r = b - L.at;
                if (r >= L.period) r %= L.period;
                X.map[w0 + (b - w) - wa] = L.base + r;
            }
        }
        __syncthreads();
    }
    const u32 ring = max(from + X_HIST, w0 + n) - X_HIST;
    const u32 quads = (w0 - wa + n + 3) >> 2;
    const bool words = ((uintptr_t)dst & 3) == 0;
    for (u32 q = threadIdx.x; q < quads; q += XT) {
        volatile u32 *map = X.map;
        const uint4 s4 = *(const uint4 *)(X.map + 4 * q);
        u32 s[4] = {s4.x, s4.y, s4.z, s4.w};
        const u32 p = wa + 4 * q;
        // bytes outside the window: any source that ends the search
        if (p < w0 || p + 4 > w0 + n) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (p + j < w0 || p + j >= w0 + n) s[j] = X_LIT | lit_near;
        }
        // literals count as negative: a source in the window is one at or above w0
        bool chased = false;
        while (max(max((int)s[0], (int)s[1]), max((int)s[2], (int)s[3])) >= (int)w0) {
            chased = true;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if ((int)s[j] >= (int)w0) s[j] = map[s[j] - wa];
        }
        if (chased) *(uint4 *)(X.map + 4 * q) = make_uint4(s[0], s[1], s[2], s[3]);
        u32 v[4];
        bool far = false;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const u32 i = s[j] & ~X_LIT, k = i - lit_near;
            const bool is_lit = (s[j] & X_LIT) != 0, ok = is_lit ? k < near_n : i >= ring;
            v[j] = ok ? *(is_lit ? near + k : X.hist + (i & (X_HIST - 1))) : 0;
            far |= !ok;
        }
        if (far) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const u32 i = s[j] & ~X_LIT;
                if (s[j] & X_LIT) {
                    if (i - lit_near >= near_n) v[j] = __ldg(lit + i);
                } else if (i < ring) {
                    v[j] = dst[i];
                }
            }
        }
        if (p >= w0 && p + 4 <= w0 + n) {
            const u32 x = v[0] | (v[1] << 8) | (v[2] << 16) | (v[3] << 24);
            *(u32 *)(X.hist + (p & (X_HIST - 1))) = x;
            if (words) {
                *(u32 *)(dst + p) = x;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) dst[p + j] = (uint8_t)v[j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (p + j >= w0 && p + j < w0 + n) {
                    dst[p + j] = (uint8_t)v[j];
                    X.hist[(p + j) & (X_HIST - 1)] = (uint8_t)v[j];
                }
        }
    }
    __syncthreads();
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
// takes SN_C compressed bytes at a time, in segments of 64 (an element with
// its length in the tag spans at most 62).  One lane per segment walks the
// chain that would begin at the segment's first byte; then it walks from
// where the segment before ends until it meets that chain, as two chains
// nearly always do within a few elements: from there on they are the same,
// and the segment's end does not depend on where it was entered.  One thread
// follows the segments' ends and walks again only where they did not meet or
// a long literal skips segments.
constexpr int SN_C = 8192;  // compressed bytes parsed at a time
constexpr int SN_SEG = SN_C / 64;
constexpr int SN_PER = SN_C / XT;   // positions of a thread
constexpr int SN_EL = SN_PER / 2;   // elements that can start there

constexpr int SN_J = SN_C + 2 * SN_SEG;  // entries of a jump table: 2 pad entries per segment
struct SnapShared {
    XShared x;  // its map holds the jump tables until the elements are known
    u32 words[SN_C / 4 + 4];           // the compressed bytes, as aligned words
    u64 mask[SN_SEG];                  // the starts
    u32 exit[SN_SEG];                  // where a segment's chain leaves it
    u32 sums[XT / 32];
    u32 skips[SN_SEG / 32];
    u32 changed, next, job, ip, bad;
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

// Barrier of the first SN_SEG threads.
__device__ __forceinline__ void sn_sync() {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(SN_SEG) : "memory");
}

// The first segment from s on whose chain does not end in the next one.
__device__ __forceinline__ u32 sn_skip(const u32 *skips, u32 s) {
    u32 g = skips[s >> 5] & (0xffffffffu << (s & 31));
    while (!g) {
        s = (s | 31) + 1;
        g = skips[s >> 5];
    }
    return (s & ~31u) + __ffs(g) - 1;
}

__device__ __forceinline__ u32 sn_at(u32 e) { return e + 2 * (e >> 6); }

// The starts of the staged piece into S.mask, by the first SN_SEG threads; S.next:
// where the last element ends (SN_C or above; 0xffff: beyond what a jump
// holds).  jump: per position, where an element there ends; jump4: four
// elements on, but no further than out of the segment.
__device__ __forceinline__ void sn_starts(SnapShared &S, const uint16_t *jump, const uint16_t *jump4) {
    const u32 t = threadIdx.x, end = (t + 1) * 64;
    u32 entry = t * 64, exit = entry;
    while (exit < end) exit = jump4[sn_at(exit)];
    S.exit[t] = exit;
    // enter each segment where the one before it ends, again for those whose entry changed
    for (int round = 0; round < SN_SEG; round++) {
        sn_sync();
        const u32 in = t ? S.exit[t - 1] : 0;
        const bool again = t && in != entry && (in >> 6) == t;
        if (t == 0) S.changed = 0;
        sn_sync();
        if (again) {
            entry = in;
            u32 e = in;
            while (e < end) e = jump4[sn_at(e)];
            if (e != exit) {
                S.changed = 1;
                S.exit[t] = exit = e;
            }
        }
        sn_sync();
        if (!S.changed) break;
    }
    u64 m = 0;
    for (u32 e = entry; e < end;) {
        const u32 next = jump4[sn_at(e)];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (e < end) {
                m |= 1ull << (e & 63);
                if (k < 3) e = jump[sn_at(e)];
            }
        }
        e = next;
    }
    S.mask[t] = m;
    // every segment was entered where the one before it ends: all is as it should be, unless one is skipped
    const unsigned g = __ballot_sync(FULL, t + 1 == SN_SEG || (exit >> 6) != t + 1);
    if ((t & 31) == 0) S.skips[t >> 5] = g;
    sn_sync();
    if (t == 0) {
        u32 q = sn_skip(S.skips, 0);  // segments up to q are right
        for (;;) {
            u32 x = S.exit[q];
            const u32 to = min(x >> 6, (u32)SN_SEG);
            for (u32 k = q + 1; k < to; k++) S.mask[k] = 0;
            if (x >= SN_C) {
                S.next = x;
                break;
            }
            u64 p = 0;
            while (x < (to + 1) * 64) {
                p |= 1ull << (x & 63);
                x = jump[sn_at(x)];
            }
            S.mask[to] = p;
            q = to;
            if (x == S.exit[to]) q = sn_skip(S.skips, to);  // the segments behind it stand
            else S.exit[to] = x;
        }
    }
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
    u32 ip = S.ip, op = 0, from = 0;
    int par = 0;
    if (S.bad) return false;
    static_assert(sizeof(S.x.map) >= 3 * SN_J * sizeof(uint16_t), "jump tables in the map");
    uint16_t *jump = (uint16_t *)S.x.map, *jump2 = jump + SN_J, *jump4 = jump2 + SN_J;
    if (t == 0) S.x.n_long[0] = 0;
    while (op < dlen) {
        if (ip >= slen) return false;
        const u32 a = (u32)((uintptr_t)(src + ip) & 3);
        const u32 *blk = (const u32 *)(src + ip - a);
        // words with a byte of [ip, slen), up to SN_C + 8 bytes from ip
        for (u32 k = t; k < SN_C / 4 + 3; k += XT) S.words[k] = 4 * (u64)k < (u64)(slen - ip) + a ? __ldg(blk + k) : 0u;
        __syncthreads();
        const uint8_t *c = (const uint8_t *)S.words + a;
        const u32 avail = min((u32)SN_C, slen - ip);
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            const u32 i = t + k * XT, tag = c[i], ty = tag & 3u;
            u32 cs = ty == 0 ? (tag >> 2) + 2 : 2 + ((0x310u >> (4 * (ty - 1))) & 15u);  // copies: 2, 3, 5 bytes
            if (tag >= 240 && ty == 0) cs = min(sn_decode(c + i).cs, 0x10000u);
            // past the page's end: to the next segment, where all chains meet
            jump[sn_at(i)] = (uint16_t)(i < avail ? min(i + cs, 0xffffu) : (i | 63) + 1);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            const u32 i = t + k * XT;
            u32 e = jump[sn_at(i)];
            if (e < (i | 63) + 1) e = jump[sn_at(e)];
            jump2[sn_at(i)] = (uint16_t)e;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SN_PER; k++) {
            const u32 i = t + k * XT;
            u32 e = jump2[sn_at(i)];
            if (e < (i | 63) + 1) e = jump2[sn_at(e)];
            jump4[sn_at(i)] = (uint16_t)e;
        }
        __syncthreads();
        if (t < SN_SEG) sn_starts(S, jump, jump4);
        __syncthreads();
        // the elements that start at this thread's positions.  Only the last
        // one of all can be longer than the compressed bytes it lies in:
        // lengths are clamped for the scan
        u32 bits = (u32)(S.mask[t / (64 / SN_PER)] >> (t * SN_PER & 63)) & ((1u << SN_PER) - 1);
        u32 len[SN_EL], val[SN_EL], sum = 0;
        bool mybad = false;
        u32 last = 0;  // compressed position after the last element here
#pragma unroll
        for (int k = 0; k < SN_EL; k++) {
            len[k] = 0;
            val[k] = 1;
            const u32 i = t * SN_PER + __ffs(bits) - 1;
            if (bits && i < avail) {
                const SnapElem e = sn_decode(c + i);
                val[k] = e.lit ? X_LIT | (ip + i + e.hdr) : e.off;
                len[k] = min(e.len, 1u << 30);
                last = i + e.cs;
                // a length of 2^30 or more, or an offset that looks like a literal: never valid in a page below 2 GB
                if (e.len == 0 || e.len >= (1u << 30) || (!e.lit && (e.off == 0 || (e.off & X_LIT)))) len[k] |= 1u << 30;
                sum += len[k] & ~(1u << 30);
                bits &= bits - 1;
            } else {
                bits = 0;
            }
        }
        u32 total, o = x_scan(sum, S.sums, &total);
        u32 at = o;
#pragma unroll
        for (int k = 0; k < SN_EL; k++) {
            const u32 l = len[k] & ~(1u << 30);
            const u64 pos = (u64)op + at;
            // elements after the last output byte are ignored
            if (len[k] && pos < dlen && ((len[k] >> 30) || pos + l > dlen || (!(val[k] & X_LIT) && val[k] > pos))) mybad = true;
            at += l;
        }
        if (last && (u64)op + at - 1 < dlen && sum && (u64)ip + last > slen) mybad = true;
        if (__syncthreads_or(mybad)) return false;
        total = min(total, dlen - op);
        for (u32 w = 0; w < total; w += XW) {
            const u32 n = min((u32)XW, total - w);
            at = o;
#pragma unroll
            for (int k = 0; k < SN_EL; k++) {
                if (len[k])
                    x_fill(S.x, op, w, n, par, at, len[k], (val[k] & X_LIT) ? val[k] : op + at - val[k],
                           (val[k] & X_LIT) ? 0xffffffffu : val[k]);
                at += len[k];
            }
            x_write(S.x, w, n, par, op, dst, src, c, ip, SN_C, from);
            par ^= 1;
        }
        op += total;
        if (avail < SN_C) {
            ip = slen;
        } else if (S.next >= 0xffff) {  // a literal that jumps do not reach over: it is the last element
            if (last > SN_C) S.ip = last;
            __syncthreads();
            ip += S.ip;
        } else {
            ip += S.next;
        }
        __syncthreads();
    }
    return true;
}

// Stored and SNAPPY pieces: a block claims pieces from a counter (zero at
// launch), longest first, until none is left.
__global__ void __launch_bounds__(XT, X_CTAS) k_pq_inflate(const uint8_t *__restrict__ file, const InflateJob *jobs,
                                                      uint32_t n, uint32_t *next, uint8_t *img, uint32_t *lvl, Ctl *ctl) {
    extern __shared__ __align__(16) unsigned char x_smem[];
    SnapShared &S = *(SnapShared *)x_smem;
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

// Small pieces, where there are many, one warp each (k_pq_inflate_small): no
// barriers, and 48 of them on an SM at once instead of one.  The warp decodes a round of elements at a time.  Lane L reads the 8
// compressed bytes at ip + L (one aligned word per lane, redistributed by
// shuffles) and decodes the element a tag there would be; the chain of real
// tags from ip (each start plus its element's compressed size) is walked with
// shuffles over the lanes' sizes, up to the first start at or past ip + 32.
// An exclusive scan of the starts' lengths places each element in the output.
// Each output byte of the round gets its source in a per-warp shared map: a
// compressed position (literal) or an earlier output position (copy; an
// overlapping copy repeats its first `offset` bytes).  A source inside the
// round is followed through the map to a byte written before the round or a
// literal byte, so that all bytes of a round are independent and the warp
// writes them with one load and one store each.  A literal longer than 64
// bytes (the last element of its round) is copied by the whole warp after
// the round.  Every length and offset is checked against the piece's bounds;
// a malformed block sets ERR_CORRUPT and stops.
#define SNW_MAP 1024   // output bytes of one round: at most 16 elements of at most 64 bytes
#define SNW_LONG 64    // literals longer than this are copied by the warp
#define SNW_LIT 0x80000000u

__device__ __forceinline__ void sn_warp_piece(const uint8_t *__restrict__ file, const InflateJob J, uint8_t *img, u32 *lvl,
                                              Ctl *ctl, u32 *map, const int lane) {
    const uint8_t *src = file + J.src;
    uint8_t *dst = img + J.dst;
    bool bad = false;
    if (J.mode == 0) {
        for (u32 i = lane; i < J.src_len; i += 32) dst[i] = src[i];
    } else {
        const u32 slen = J.src_len, dlen = J.dst_len;
        u32 ip = 0, op = 0;
        if (lane == 0) {  // the preamble: the uncompressed length
            u64 ulen = 0;
            int sh = 0;
            for (;;) {
                if (ip >= slen || sh > 28) {
                    bad = true;
                    break;
                }
                const uint8_t b = src[ip++];
                ulen |= (u64)(b & 0x7f) << sh;
                if (!(b & 0x80)) break;
                sh += 7;
            }
            if (ulen != dlen) bad = true;
        }
        bad = __shfl_sync(FULL, (int)bad, 0) != 0;
        ip = __shfl_sync(FULL, ip, 0);
        while (!bad && op < dlen) {
            if (ip >= slen) {
                bad = true;
                break;
            }
            // bytes [ip + lane, ip + lane + 8): lanes 0..10 load the aligned words over
            // [ip, ip + 40) and the warp redistributes them
            const uint8_t *blk = (const uint8_t *)((uintptr_t)(src + ip) & ~(uintptr_t)3);
            u32 word = 0;
            if (lane < 11) {
                const uint8_t *wp = blk + 4 * lane;
                if (blk >= src && blk + 44 <= src + slen) {
                    word = __ldg((const u32 *)wp);
                } else {
                    for (int k = 0; k < 4; k++)
                        if (wp + k >= src && wp + k < src + slen) word |= (u32)__ldg(wp + k) << (8 * k);
                }
            }
            const u32 sh0 = (u32)((uintptr_t)(src + ip) & 3) + (u32)lane;
            const u32 w0 = __shfl_sync(FULL, word, sh0 >> 2);
            const u32 w1 = __shfl_sync(FULL, word, (sh0 >> 2) + 1);
            const u32 w2 = __shfl_sync(FULL, word, (sh0 >> 2) + 2);
            const u32 lo = __funnelshift_r(w0, w1, 8 * (sh0 & 3)), hi = __funnelshift_r(w1, w2, 8 * (sh0 & 3));
            // the element a tag at ip + lane would be (selects, no branches)
            const u32 tag = lo & 0xffu, t = tag & 3u, l6 = tag >> 2;
            const u32 rest = (lo >> 8) | (hi << 24);  // bytes 1..4 after the tag
            const u32 nb = l6 >= 60 ? l6 - 59 : 0;     // a literal's length bytes
            const u32 lraw = nb ? rest & (0xffffffffu >> (32 - 8 * nb)) : l6;
            const u32 hdr = t == 0 ? 1 + nb : (t == 1 ? 2 : (t == 2 ? 3 : 5));
            const u32 len = t == 0 ? lraw + 1 : (t == 1 ? 4 + (l6 & 7u) : l6 + 1);  // 0 after a wrap
            const u32 off = t == 1 ? ((tag >> 5) << 8) | (rest & 0xffu) : (t == 2 ? rest & 0xffffu : rest);
            const u32 cs = t != 0 ? hdr : (lraw >= 0x7fff0000u ? 0x7fffffffu : hdr + lraw + 1);
            // the chain of starts from ip
            const u32 avail = min(32u, slen - ip);
            u32 pos = 0, mask = 0;
            while (pos < avail) {
                mask |= 1u << pos;
                pos += __shfl_sync(FULL, cs, pos);
            }
            const bool start = (mask >> lane) & 1u;
            // lengths clamped in the scan (16 starts of at most 2^26 cannot wrap); the one
            // element that may be longer, a long literal, is the round's last start
            u32 mylen = start ? min(len, 1u << 26) : 0, incl = mylen;
            for (int d = 1; d < 32; d <<= 1) {
                const u32 y = __shfl_up_sync(FULL, incl, d);
                if (lane >= d) incl += y;
            }
            const u32 excl = incl - mylen;  // round-relative output position
            u32 total = __shfl_sync(FULL, incl, 31);
            const u32 p = ip + (u32)lane;  // compressed position of this lane's tag
            const u64 o = (u64)op + excl;
            const bool live = start && o < dlen;  // elements after the last output byte are ignored
            const bool mybad = live && ((u64)p + cs > slen || len == 0 || o + len > dlen ||
                                        (t != 0 && (off == 0 || off > o)));
            if (__any_sync(FULL, mybad)) {
                bad = true;
                break;
            }
            // outputs past dlen (trailing elements) and the long literal are not mapped
            if (total > dlen - op) total = dlen - op;
            const u32 lmask = __ballot_sync(FULL, live && t == 0 && len > SNW_LONG);
            u32 mapped = total, lit_at = 0, lit_len = 0, lit_src = 0;
            if (lmask) {
                const int ll = __ffs(lmask) - 1;
                mapped = __shfl_sync(FULL, excl, ll);
                lit_len = __shfl_sync(FULL, len, ll);
                lit_src = __shfl_sync(FULL, p + hdr, ll);
                lit_at = op + mapped;
                total = mapped + lit_len;
            }
            if (mapped > SNW_MAP) {  // unreachable: 16 starts of at most 64 bytes
                bad = true;
                break;
            }
            if (start && excl < mapped) {
                // a literal's byte b comes from q + b; a copy's from o - off + (b mod off)
                const u32 base = t == 0 ? SNW_LIT | (p + hdr) : (u32)o - off;
                const u32 per = t == 0 ? 0xffffffffu : off;
                for (u32 b = 0, r = 0; b < len; b++) {
                    map[excl + b] = base + r;
                    r = r + 1 == per ? 0 : r + 1;
                }
            }
            __syncwarp();
            for (u32 k = lane; k < mapped; k += 32) {
                u32 s = map[k];
                while (!(s & SNW_LIT) && s >= op) s = map[s - op];
                dst[op + k] = (s & SNW_LIT) ? __ldg(src + (s & ~SNW_LIT)) : dst[s];
            }
            if (lit_len) {
                for (u32 b = lane; b < lit_len; b += 32) dst[lit_at + b] = __ldg(src + lit_src + b);
            }
            __syncwarp();
            op += total;
            ip += pos;
        }
    }
    if (bad && lane == 0) atomicOr(&ctl->err, (u32)ERR_CORRUPT);
    __syncwarp();
    if (lane == 0) x_level(J, dst, bad, lvl);
}

// Each warp claims pieces from a counter (zero at launch) until none is left.
__global__ void __launch_bounds__(256) k_pq_inflate_small(const uint8_t *__restrict__ file, const InflateJob *jobs,
                                                          uint32_t n, uint32_t *next, uint8_t *img, uint32_t *lvl,
                                                          Ctl *ctl) {
    __shared__ u32 s_map[8][SNW_MAP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (;;) {
        u32 j = 0;
        if (lane == 0) j = atomicAdd(next, 1u);
        j = __shfl_sync(FULL, j, 0);
        if (j >= n) return;  // the whole warp
        sn_warp_piece(file, jobs[j], img, lvl, ctl, s_map[warp], lane);
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
// descriptors, anything malformed) is marked and decoded from the start by the
// serial decoder (k_pz_serial), whose verdict counts.
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
    u32 n_list, claim_entropy, claim_bytes, n_odd, claim_odd;
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
    u32 *odd;       // per piece: 1, for the serial decoder
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
        A.odd[j] = 1;
        atomicAdd(&A.work->n_odd, 1u);
        return;
    }
    A.n_blk[j] = k;
    A.odd[j] = 0;
    u32 nc = 0;
    for (u32 i = 0; i < k; i++) nc += A.blk[J.blk + i].type == 2;
    u32 at = nc ? atomicAdd(&A.work->n_list, nc) : 0;
    for (u32 i = 0; i < k; i++)
        if (A.blk[J.blk + i].type == 2) A.list[at++] = J.blk + i;
}

// One warp's tables.  The Huffman table is used up before the sequence
// tables are built.

constexpr int Z_LL = 0, Z_OF = 512, Z_ML = 768, Z_CELLS = 1280;
struct alignas(16) ZTables {  // the ring is written 16 bytes at a time
    union {
        uint16_t huf[1u << gbz::ZS_HUF_LOG];
        // sequence cells: the next state's bits (5 bits) | the code's extra bits (6) | 0 | four times the next state's
        // baseline from bit 19 on.  The sum of three cells holds the sums of the bits in the same places.
        u32 cell[Z_CELLS];
    };
    union {
        u32 wt[64];
        u32 ring[256];  // two 512-byte pieces of the sequences' bit stream
    };
    u32 val[Z_CELLS];  // per cell: the code's baseline (24 bits) | its extra bits (8)
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

// The sequences of block b into the scratch, by one warp.  The three states
// are followed through the bit stream by all lanes alike (the loads are
// broadcasts and nothing diverges), lane k keeping the position and states of
// the k-th of 32 sequences; then every lane reads its sequence's extra bits.
// The stream is kept in shared memory, the next 512 bytes already in
// registers.  What bounds it: the chain from a sequence's cells over the sum
// of their bit counts and the extraction of the next states to the next
// cells; the 64 bits below the position are therefore loaded beside the
// cells.
__device__ __forceinline__ bool pz_sequences(const ZArgs &A, ZBlk &b, u64 base, ZTables &T, int lane) {
    if (lane == 0) T.bad = !pz_tables(A, b, T);
    __syncwarp();
    if (T.bad) return false;
#pragma unroll
    for (int x = 0; x < 3; x++) {
        const int at = x == 0 ? Z_LL : (x == 1 ? Z_OF : Z_ML);
        for (int i = lane; i < (1 << T.log[x]); i += 32) {
            const u32 c = T.cell[at + i], s = c & 0xffu, nb = (c >> 8) & 0xffu;
            u32 xb = 0;
            int xn = (int)s;
            if (x == 0) gbz::zs_ll(s, &xb, &xn);
            if (x == 2) gbz::zs_ml(s, &xb, &xn);
            T.cell[at + i] = nb | ((u32)xn << 5) | ((c >> 16) << 21);  // (base * 4) << 19
            T.val[at + i] = xb | ((u32)xn << 24);
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
    u32 sl, so, sm;
    q -= T.log[0];
    sl = z_rd(T.ring, q, T.log[0]);
    q -= T.log[1];
    so = z_rd(T.ring, q, T.log[1]);
    q -= T.log[2];
    sm = z_rd(T.ring, q, T.log[2]);
    sl *= 4;  // states are kept as byte offsets of their cells
    so *= 4;
    sm *= 4;
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
        int my_q = 0;
        u32 my_l = 0, my_o = 0, my_m = 0;
        auto step = [&](int k) {
            const u32 cl = *(const u32 *)((const char *)(T.cell + Z_LL) + sl);
            const u32 co = *(const u32 *)((const char *)(T.cell + Z_OF) + so);
            const u32 cm = *(const u32 *)((const char *)(T.cell + Z_ML) + sm);
            // the 96 bits below q (at most 63 + 26 are read)
            const int w = (q >> 5) - 3;
            const u32 a0 = T.ring[w & 255], a1 = T.ring[(w + 1) & 255], a2 = T.ring[(w + 2) & 255], a3 = T.ring[(w + 3) & 255];
            const u32 h0 = __funnelshift_r(a0, a1, (u32)q), h1 = __funnelshift_r(a1, a2, (u32)q), h2 = __funnelshift_r(a2, a3, (u32)q);
            if (k == lane) {
                my_q = q;
                my_l = sl;
                my_o = so;
                my_m = sm;
            }
            const u32 all = cl + co + cm, extra = (all >> 5) & 63;
            q -= (int)((all & 31) + extra);
            // the next states' bits, LL, ML, OF from the top: shifts take a cell's low 5 bits
            const u32 head = __funnelshift_l(extra < 32 ? h1 : h0, extra < 32 ? h2 : h1, extra);
            sl = (cl >> 19) + 4 * __funnelshift_l(head, 0u, cl);
            const u32 h_m = __funnelshift_l(0u, head, cl);
            sm = (cm >> 19) + 4 * __funnelshift_l(h_m, 0u, cm);
            so = (co >> 19) + 4 * __funnelshift_l(__funnelshift_l(0u, h_m, cm), 0u, co);
        };
        if (cnt == 32) {
#pragma unroll 8
            for (int k = 0; k < 32; k++) step(k);
        } else {
            for (int k = 0; k < cnt; k++) step(k);
        }
        my_l >>= 2;
        my_o >>= 2;
        my_m >>= 2;
        // after the last sequence no next states are read: their bits are not there
        if (k0 + 32 >= nseq) {
            const u32 n = (T.cell[Z_LL + my_l] + T.cell[Z_OF + my_o] + T.cell[Z_ML + my_m]) & 31;
            q += (int)__shfl_sync(FULL, n, cnt - 1);
        }
        u32 ll = 0, ml = 0, off = 4;  // off: the offset value until resolved
        if (lane < cnt) {
            const u32 vl = T.val[Z_LL + my_l], vm = T.val[Z_ML + my_m];
            const int xo = (int)(T.val[Z_OF + my_o] >> 24), xm = (int)(vm >> 24), xl = (int)(vl >> 24);
            int p = my_q - xo;
            off = (1u << xo) + z_rd(T.ring, p, xo);
            p -= xm;
            ml = (vm & 0xffffffu) + z_rd(T.ring, p, xm);
            p -= xl;
            ll = (vl & 0xffffffu) + z_rd(T.ring, p, xl);
            if (off > 3 && ((off - 3) & Z_SYM)) bad = true;
        }
        lits += __reduce_add_sync(FULL, ll);
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

__global__ void __launch_bounds__(32) k_pz_entropy(const __grid_constant__ ZArgs A) {
    static_assert(sizeof(ZTables) % 16 == 0 && offsetof(ZTables, ring) % 16 == 0, "ring alignment");
    __shared__ ZTables T;
    const int lane = threadIdx.x;
    const u32 n = A.work->n_list;
    for (;;) {
        u32 i = 0;
        if (lane == 0) i = atomicAdd(&A.work->claim_entropy, 1u);
        i = __shfl_sync(FULL, i, 0);
        if (i >= n) return;
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
    XShared x;
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
                                               u32 &from, int &par, u32 r0, u32 r1, u32 r2, ZByteShared &S) {
    const u32 t = threadIdx.x, cap = J.dst_len;
    if (b.bad) return false;
    const uint8_t *lit = b.lit_kind == 0 ? A.file + b.src + b.lit_hdr : A.lits + J.aux + b.lit_off;
    const u64 base = J.aux / 3 + b.seq_off + 2 * t;
    const u32 nseq = b.nseq, lsize = b.lsize;
    u32 lp = 0;
    u32 ll[2], ml[2], off[2];
    auto load = [&](u32 k0) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            ll[k] = ml[k] = off[k] = 0;
            if (k0 + 2 * t + k < nseq) {
                ll[k] = A.seq_ll[base + k0 + k];
                ml[k] = A.seq_ml[base + k0 + k];
                off[k] = z_offset(A.seq_off[base + k0 + k], r0, r1, r2);
            }
        }
    };
    for (u32 k0 = 0; k0 < nseq; k0 += ZB_SEQ) {
        load(k0);
        // output places in the low half, literal places in the high half
        u64 total;
        const u64 at = x_scan((u64)(ll[0] + ml[0] + ll[1] + ml[1]) | ((u64)(ll[0] + ll[1]) << 32), S.sums, &total);
        u32 o = (u32)at, l = lp + (u32)(at >> 32);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (k0 + 2 * t + k < nseq)
                bad |= (u64)l + ll[k] > lsize || (u64)op + o + ll[k] + ml[k] > cap || off[k] == 0 || off[k] > op + o + ll[k];
            o += ll[k] + ml[k];
            l += ll[k];
        }
        if (__syncthreads_or(bad)) return false;
        const u32 all = (u32)total;
        for (u32 w = 0; w < all; w += XW) {
            const u32 n = min((u32)XW, all - w);
            o = (u32)at;
            l = lp + (u32)(at >> 32);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                x_fill(S.x, op, w, n, par, o, ll[k], X_LIT | l, 0xffffffffu);
                o += ll[k];
                l += ll[k];
                x_fill(S.x, op, w, n, par, o, ml[k], op + o - off[k], off[k]);
                o += ml[k];
            }
            x_write(S.x, w, n, par, op, dst, lit, S.x.hist, lsize, 1, from);
            par ^= 1;
        }
        op += all;
        lp += (u32)(total >> 32);
    }
    const u32 rest = lsize - lp;  // lp <= lsize: checked above
    if (rest > cap - op) return false;
    if (rest) {
        x_copy(dst + op, lit + lp, rest);
        op += rest;
        from = op;  // not in the ring
    }
    return true;
}

__global__ void __launch_bounds__(XT, X_CTAS) k_pz_bytes(const __grid_constant__ ZArgs A) {
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
        u32 op = 0, from = 0, r0 = 1, r1 = 4, r2 = 8;
        int par = 0;
        if (threadIdx.x == 0) S.x.n_long[0] = 0;
        __syncthreads();
        for (u32 k = 0; ok && k < nb; k++) {
            const ZBlk &b = A.blk[J.blk + k];
            if (b.type == 2) {
                ok = pz_block_bytes(A, J, b, dst, op, from, par, r0, r1, r2, S);
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
                from = op;
            }
            __syncthreads();
        }
        ok = ok && op == J.dst_len;
        if (threadIdx.x == 0 && nb) {  // without blocks the piece is already marked
            if (ok) {
                x_level(J, dst, false, A.lvl);
            } else {
                A.odd[j] = 1;
                atomicAdd(&A.work->n_odd, 1u);
            }
        }
        __syncthreads();
    }
}

// The pieces that the steps above marked: one warp per piece, claimed longest
// first, its first lane decoding with the warp's 13.3 KB of tables in
// `scratch`.  Launch bounds of 5 blocks an SM hold a thread to 96 registers: 20
// warps an SM decode at once.  2M rows in pages of three columns and four frames,
// 368 pages of up to 128 KB: 12.3 ms; 14.9 with the file as a plain pointer of
// ZArgs (its loads waited for the page's stores) and the job kept in registers
// past the decode.  A frame that does not decode to exactly dst_len bytes sets
// ERR_CORRUPT.
__global__ void __launch_bounds__(128, 5) k_pz_serial(const uint8_t *__restrict__ file, const InflateJob *jobs, u32 n,
                                                      ZWork *work, const u32 *odd, uint8_t *img, uint32_t *lvl, Ctl *ctl,
                                                      gbz::ZsScratch *scratch) {
    if ((threadIdx.x & 31) != 0 || work->n_odd == 0) return;
    gbz::ZsScratch &Z = scratch[(blockIdx.x * blockDim.x + threadIdx.x) >> 5];
    for (;;) {
        const u32 i = atomicAdd(&work->claim_odd, 1u);
        if (i >= n) return;
        if (!odd[i]) continue;
        const InflateJob &J = jobs[i];
        const int64_t got = gbz::zstd_decompress(file + J.src, J.src_len, img + J.dst, J.dst_len, Z);
        const bool bad = got != (int64_t)J.dst_len;
        if (bad) atomicOr(&ctl->err, (u32)ERR_CORRUPT);
        x_level(J, img + J.dst, bad, lvl);
    }
}

}  // namespace gb
