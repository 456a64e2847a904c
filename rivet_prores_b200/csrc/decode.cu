// decode.cu -- the RDD 36 decoding process (§7) as sm_100a kernels.
//
//   k_locate   one CTA per picture: the big-endian u16 slice table, scanned
//              into slice offsets (src/decode.rs:202-221), each slice's
//              place in the picture (src/header.rs:308-320), and the first
//              slice that runs past picture_size.
//   k_entropy  persistent; one lane per slice component (Y', Cb, Cr, alpha):
//              the slice header (src/decode.rs:301-338), then the DC and
//              run/level/sign codes of the interleaved scan (:484-540) as a
//              list of (position, value) entries, or the alpha
//              run/difference codes (:570-595) straight into the alpha plane;
//              the lanes of a warp step together.
//   k_idct     one warp per 32 blocks, a lane each: the entries dequantised
//              into shared memory, the 8x8 IDCT in the crate's exact
//              single-precision order (src/dct.rs:36-66,
//              src/dsp/scalar.rs:8-12) and the sample conversion, stored as
//              woven 16-byte rows (src/decode.rs:395-438).
//   k_status   one CTA per picture: the first failing slice component.
//
// The f32 arithmetic uses __fmul_rn/__fadd_rn so that nothing is contracted
// into an FMA: the decoded samples are bit-identical to the crate's.

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "chain.h"
#include "codec_tables.h"
#include "device_types.h"
#include "pair_math.h"

namespace prores {

__device__ uint8_t d_scan[2][64];  // scanned index of each raster position, progressive and interlaced
__constant__ float c_idct_basis[64];  // T[x][u] (dct_basis)

namespace {


// floor(v) clamped to [0, max] (max an integer below 2^16), as an integer:
// clamping before the floor gives the same value as after it for integer
// bounds, and adding 2^23 rounded down leaves floor(v) in the low bits.
__device__ __forceinline__ uint32_t floor_clamped(float v, float max) {
    const float c = fminf(fmaxf(v, 0.0f), max);
    return __float_as_uint(__fadd_rd(c, 8388608.0f)) & 0xFFFFu;
}

// q exactly, for |q| < 2^22: q added to the significand of 1.5 2^23.
__device__ __forceinline__ float small_int_to_float(int32_t q) {
    return __fadd_rn(__int_as_float(0x4B400000 + q), -12582912.0f);
}

__device__ __forceinline__ uint64_t bswap64(uint64_t v) {
    uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
    return ((uint64_t)__byte_perm(lo, 0, 0x0123) << 32) | __byte_perm(hi, 0, 0x0123);
}

__device__ __forceinline__ uint32_t be16(const uint8_t *p) { return ((uint32_t)p[0] << 8) | p[1]; }

// MSB-first reader over [start, end) bits of the bitstream buffer: a pair of
// aligned 64-bit words funnel-shifted to the position; bits past `end` read
// as zero (the crate's BitReader::peek64, src/bits.rs:30-40). The word after
// the pair is fetched one word ahead, so moving on to the next word never
// waits for memory. The buffer has at least 24 bytes of padding after the
// last data word, so the words read never leave it.
struct Bits {
    const uint64_t *w;
    uint64_t pos, end, idx, w0, w1, w2;

    __device__ __forceinline__ uint64_t ld(uint64_t i) const { return bswap64(__ldg(w + i)); }
    __device__ __forceinline__ void init(const uint8_t *base, uint64_t byte_off, uint64_t len) {
        init_at(base, byte_off * 8, (byte_off + len) * 8);
    }
    // The same over bits [from, to).
    __device__ __forceinline__ void init_at(const uint8_t *base, uint64_t from, uint64_t to) {
        w = reinterpret_cast<const uint64_t *>(base);
        pos = from;
        end = to;
        idx = pos >> 6;
        w0 = ld(idx);
        w1 = ld(idx + 1);
        w2 = ld(idx + 2);
    }
    __device__ __forceinline__ uint64_t remaining() const { return end - pos; }
    __device__ __forceinline__ uint64_t peek() {
        uint64_t i = pos >> 6;
        if (i != idx) {
            if (i == idx + 1) {
                w0 = w1;
                w1 = w2;
                w2 = ld(i + 2);
            } else {
                w0 = ld(i);
                w1 = ld(i + 1);
                w2 = ld(i + 2);
            }
            idx = i;
        }
        uint32_t sh = (uint32_t)(pos & 63);
        uint64_t v = sh ? (w0 << sh) | (w1 >> (64 - sh)) : w0;
        uint64_t rem = end - pos;
        if (rem < 64) v &= rem ? (~0ull << (64 - rem)) : 0ull;
        return v;
    }
    // `n` (1..57) bits as a number (src/bits.rs:61-72).
    __device__ __forceinline__ int read(uint32_t n, uint64_t &v) {
        if ((uint64_t)n > remaining()) return DE_PAST_END;
        v = peek() >> (64 - n);
        pos += n;
        return DE_OK;
    }
};

// One symbol of codebook `cb` (src/vlc.rs:207-230), read bit by bit as the
// crate reads it, naming any failure exactly as the crate does.
__device__ __forceinline__ int read_sym(Bits &b, Codebook cb, uint32_t &sym) {
    uint64_t w = b.peek();
    uint64_t rem = b.remaining();
    uint32_t lz = clz64(w);
    if (lz > kMaxPrefix) return DE_PREFIX;
    if ((uint64_t)lz >= rem) return DE_PAST_END;
    b.pos += lz;
    rem -= lz;
    w = b.peek();
    if (!cb.eg && lz <= cb.q) {
        uint32_t need = 1u + cb.r;
        if (need > rem) return DE_PAST_END;
        uint64_t v = (w >> (64 - need)) & ((1ull << cb.r) - 1);
        b.pos += need;
        sym = (uint32_t)(((uint64_t)lz << cb.r) | v);
        return DE_OK;
    }
    uint32_t qe = cb.eg ? lz : lz - (cb.q + 1u);
    uint32_t ke = cb.eg ? cb.r : cb.e;
    uint64_t off = cb.eg ? 0ull : ((uint64_t)(cb.q + 1u) << cb.r);
    uint32_t need = qe + ke + 1u;
    if (need > rem) return DE_PAST_END;
    uint64_t v = w >> (64 - need);
    b.pos += need;
    uint64_t n = v - (1ull << ke) + off;
    if (n > kMaxSymbol) return DE_RANGE;
    sym = (uint32_t)n;
    return DE_OK;
}

// A component's coefficient list, in a region of 2 cap 32-bit words (cap =
// 64 n_blocks, the component's positions): entries from the front, each
// (scanned index << 21) | (magnitude << 5) | sign, in which a table entry's
// level and 32 times the index are in place. Magnitudes from kListBigMag up go to the back of the region as whole values, the k-th at
// 2 cap - 1 - k, and their entry holds kListBigMag + k. Half the bytes of
// (index, value) pairs of 32-bit words, for values of any size.
constexpr uint32_t kListBigMag = (1u << 16) - 2048u;
constexpr uint32_t kListBig = 1u << 31;  // in a list's count: it has values at the back of its region

struct CoefList {
    uint32_t *w;
    uint32_t cap, big, count;
    // The last four entries. They go out 16 bytes at a time: every lane has a
    // region of its own, so each lane's store takes the memory pipe a cycle,
    // and one store an entry held up the table reads queued behind it.
    uint4 last;
    __device__ __forceinline__ void push(bool ok, uint32_t e) {
        last.x = ok ? last.y : last.x;
        last.y = ok ? last.z : last.y;
        last.z = ok ? last.w : last.z;
        last.w = ok ? e : last.w;
        count += ok ? 1u : 0u;
        if (ok && (count & 3u) == 0) *reinterpret_cast<uint4 *>(w + count - 4u) = last;
    }
    __device__ __forceinline__ void finish() {
        const uint32_t n = count & 3u;
        if (n > 2u) w[count - 3u] = last.y;
        if (n > 1u) w[count - 2u] = last.z;
        if (n > 0u) w[count - 1u] = last.w;
    }
    __device__ __forceinline__ void put(uint32_t n, int32_t v) {
        uint32_t mag = v < 0 ? 0u - (uint32_t)v : (uint32_t)v;
        uint32_t sign = (uint32_t)(v < 0);
        if (mag >= kListBigMag) {
            w[2u * cap - 1u - big] = (uint32_t)v;
            mag = kListBigMag + big;
            sign = 0;
            big++;
        }
        push(true, (n << 21) | (mag << 5) | sign);
    }
    // If `ok`, the coefficient at n32 / 32 whose level is that of table entry
    // e2 and whose sign is the top bit of t.
    __device__ __forceinline__ void put_code(bool ok, uint32_t n32, uint32_t e2, uint32_t t) {
        push(ok, (n32 << 16) + ((e2 & 0xFE0u) | (t >> 31)));
    }
};

// A component's coefficients as one small integer (int8_t or int16_t) per
// scanned position in shared memory (zeroed beforehand: only the coded ones
// are written). A value the type cannot hold, other than its most negative
// one, is marked with that one (wide_mark<T>) and kept at the same position
// of a 32-bit array in global memory, which is otherwise never touched.
template <class T>
__device__ __forceinline__ constexpr int32_t wide_mark() {
    return sizeof(T) == 1 ? -128 : -32768;
}

template <class T>
struct SlotOut {
    T *slot;
    int32_t *wide;
    __device__ __forceinline__ void put(uint32_t n, int32_t v) {
        if (v > wide_mark<T>() && v <= -(wide_mark<T>() + 1)) {
            slot[n] = (T)v;
        } else {
            slot[n] = (T)wide_mark<T>();
            wide[n] = v;
        }
    }
    __device__ __forceinline__ void put_code(bool ok, uint32_t n32, uint32_t e2, uint32_t t) {
        const int32_t level = (int32_t)((e2 >> 5) & 127u);
        if (ok) slot[n32 >> 5] = (T)((int32_t)t < 0 ? -level : level);
    }
};

// The codeword of codebook `cb` at the top of `t` (32 bits, all data), as
// read_sym's general path reads it, when it is no longer than 32 bits and
// its symbol is in range; false otherwise (read_sym then reads it, and
// names any failure).
__device__ __forceinline__ bool window_code(uint32_t t, Codebook cb, uint32_t &sym, uint32_t &len) {
    const uint32_t lz = __clz(t);
    if (!cb.eg && lz <= cb.q) {
        len = lz + 1u + cb.r;
        sym = (lz << cb.r) | (cb.r ? (t << (lz + 1u)) >> (32u - cb.r) : 0u);
        return true;
    }
    const uint32_t qe = cb.eg ? lz : lz - (cb.q + 1u);
    const uint32_t ke = cb.eg ? cb.r : cb.e;
    const uint32_t need = qe + ke + 1u;
    if (lz + need > 32u) return false;
    len = lz + need;
    const uint64_t n = (uint64_t)((t << lz) >> (32u - need)) - (1ull << ke) +
                       (cb.eg ? 0ull : (uint64_t)(cb.q + 1u) << cb.r);
    if (n > kMaxSymbol) return false;
    sym = (uint32_t)n;
    return true;
}

// Readers of a component's bits for the lanes of a warp that run together:
// two 32-bit words, MSB first, a bit offset in the first, and the component's
// bits from there on. top() is the next 32 bits (those past the component's
// end are its neighbour's), advance() moves on by up to 32 bits, check() lets
// the reader fetch ahead; between two checks it moves on by 4 words at most.
__device__ __forceinline__ uint32_t be32(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

// Words straight from global memory, two of them on their way. A lane that
// moves on waits for what any lane loaded last: the fused decoder's reader,
// which has no shared memory to spare.
struct WordReader {
    const uint32_t *next;  // the word after the two on their way
    uint32_t w0, w1, raw1, raw2, pos;
    int32_t nleft;  // the bits left, negated
    __device__ __forceinline__ void init(const uint64_t *base, uint64_t from, uint64_t to) {
        next = reinterpret_cast<const uint32_t *>(base) + (from >> 5);
        w0 = be32(__ldg(next));
        w1 = be32(__ldg(next + 1));
        raw1 = __ldg(next + 2);
        raw2 = __ldg(next + 3);
        next += 4;
        pos = (uint32_t)from & 31u;
        nleft = -(int32_t)(to - from);
    }
    __device__ __forceinline__ uint32_t left() const { return (uint32_t)-nleft; }
    __device__ __forceinline__ uint32_t top() const { return __funnelshift_l(w1, w0, pos); }
    // The 32 bits from `off` (at most 32) bits on.
    __device__ __forceinline__ uint32_t top_at(uint32_t off) const {
        const uint32_t p = pos + off;
        return __funnelshift_l(p < 32u ? w1 : be32(raw1), p < 32u ? w0 : w1, p);
    }
    __device__ __forceinline__ void advance(uint32_t len) {
        pos += len;
        nleft += (int32_t)len;
        if (pos >= 32u) {
            pos -= 32u;
            w0 = w1;
            w1 = be32(raw1);
            raw1 = raw2;
            raw2 = __ldg(next++);
        }
    }
    __device__ __forceinline__ void check(uint32_t, bool) {}
};

// Words from a ring of 8 a lane in shared memory, filled 16 bytes at a time
// at the checks, each from a load made at a check before. A register that any
// lane has a load in flight to stalls the whole warp when it is next read, so
// the loads land where only a check reads them: with the words taken from
// registers as loaded (WordReader) a warp waited out a load nearly every code
// (11 of 16 stall cycles an instruction). Fetches reach at most 16 words past
// the read position.
struct RingReader {
    uint32_t *ring;    // this lane's word 0; word k is ring[32 (k & 7)]
    const uint4 *src;  // the block after q
    uint4 q;           // the ring's next block
    uint32_t w0, w1, w2, pos;
    int32_t nleft;
    uint32_t rd, wr;  // the number of w2, and of the next word the ring gets
    __device__ __forceinline__ void put(uint4 v) {
        uint32_t *at = ring + 32u * (wr & 7u);  // wr is a multiple of 4
        at[0] = be32(v.x);
        at[32] = be32(v.y);
        at[64] = be32(v.z);
        at[96] = be32(v.w);
        wr += 4;
    }
    __device__ __forceinline__ void init(const uint64_t *base, uint64_t from, uint64_t to) {
        src = reinterpret_cast<const uint4 *>(base) + (from >> 7);
        const uint4 a = __ldg(src), b = __ldg(src + 1);
        q = __ldg(src + 2);
        src += 3;
        wr = 0;
        put(a);
        put(b);
        rd = (((uint32_t)from >> 5) & 3u) + 2u;
        w0 = ring[32u * (rd - 2u)];
        w1 = ring[32u * (rd - 1u)];
        w2 = ring[32u * rd];
        pos = (uint32_t)from & 31u;
        nleft = -(int32_t)(to - from);
    }
    __device__ __forceinline__ uint32_t left() const { return (uint32_t)-nleft; }
    __device__ __forceinline__ uint32_t top() const { return __funnelshift_l(w1, w0, pos); }
    // The 32 bits from `off` (at most 32) bits on.
    __device__ __forceinline__ uint32_t top_at(uint32_t off) const {
        const uint32_t p = pos + off;
        return __funnelshift_l(p < 32u ? w1 : w2, p < 32u ? w0 : w1, p);
    }
    // No branch: a lane that stays within its word loads the same w2 again.
    __device__ __forceinline__ void advance(uint32_t len) {
        pos += len;
        nleft += (int32_t)len;
        const bool on = pos >= 32u;
        w0 = on ? w1 : w0;
        w1 = on ? w2 : w1;
        rd += on ? 1u : 0u;
        pos &= 31u;
        w2 = ring[32u * (rd & 7u)];
    }
    __device__ __forceinline__ void check(uint32_t mask, bool live) {
        do {
            // Words rd to wr - 1 are still to come; a block fits beside 4.
            if (live && wr - rd < 5u) {
                put(q);
                q = __ldg(src++);
            }
        } while (__any_sync(mask, live && wr - rd < 5u));
    }
};

// The DC part of scanned_coefficients() (src/decode.rs:486-498): the first
// DC by EG5, each next one as a difference by Table 9 on the previous
// difference, the sign flipped after a negative one. The lanes of `mask` run
// it together, four codes between checks. A code that is 32 bits or fewer and
// all data is read from top(): with z leading zeros, EGk is 2 z + k + 1 bits,
// z + k + 1 of them n + 2^k; Table 9's (1, 2, 3) for |difference| 2 is 3 or 4
// bits with z <= 1, from there on 2 z + 2 bits, z + 2 of them n itself. Any
// other code waits for the end of the four and goes by the general reader,
// which names any failure.
template <class Reader, class Out>
__device__ __forceinline__ int decode_dc(uint32_t mask, bool live, Reader &r, const Bits &b, uint32_t n_blocks, Out &out) {
    int err = DE_OK;
    uint32_t i = 0;
    int32_t prev_dc = 0, prev_diff = 3;
    const auto take = [&](uint32_t sym) {
        const int32_t n = symbol_to_signed(sym);
        if (i == 0) {
            prev_dc = n;
        } else {
            prev_diff = prev_diff < 0 ? -n : n;
            const int64_t s = (int64_t)prev_dc + prev_diff;
            if (s > INT32_MAX || s < INT32_MIN) err = DE_DC_OVERFLOW;
            prev_dc = (int32_t)s;
        }
        if (!err) out.put(i++, prev_dc);
        live = err == DE_OK;
    };
    while (__any_sync(mask, live && i < n_blocks)) {
        bool stuck = false;
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
            const uint32_t t = r.top(), z = __clz(t);
            const uint32_t a = i == 0 ? 5u : min((uint32_t)abs(prev_diff), 3u), e = a == 2u ? 1u : a;
            const bool rice = a == 2u && z <= 1u;
            const uint32_t len = rice ? z + 3u : 2u * z + e + 1u;
            const uint32_t sym = rice ? (z << 2) | ((t << (z + 1u)) >> 30)
                                      : ((t << z) >> ((31u - z - e) & 31u)) - (a == 2u ? 0u : 1u << e);
            if (live && i < n_blocks) {
                stuck = r.nleft > -32 || len > 32u;
                if (!stuck) {
                    r.advance(len);
                    take(sym);
                }
            }
        }
        r.check(mask, live);
        if (__any_sync(mask, stuck)) {
            if (stuck) {
                Bits g;
                g.init_at(reinterpret_cast<const uint8_t *>(b.w), b.end - r.left(), b.end);
                uint32_t sym = 0;
                err = read_sym(g, i == 0 ? kFirstDcBook : dc_book(prev_diff), sym);
                if (!err) {
                    r.init(b.w, g.pos, b.end);
                    take(sym);
                }
                live = err == DE_OK;
            }
            r.check(mask, live);
        }
    }
    return err;
}

// The AC part of scanned_coefficients() (src/decode.rs:499-540): every
// coefficient the codes give, in scanned-index order, handed to `out`; the
// positions not handed over are zero. The lanes of `mask` run it together, a
// component each (`live` false: none). A step reads one run, level and sign
// from the prefix tables without a branch; a lane whose code is not there, or
// runs past its data or its positions, stays where it is, and after four
// steps such lanes leave the others for one code. Bits past the end of the
// component read as zero, as the crate's reader has them, so the tables serve
// to the last code. What they do not hold goes by window_code and, for
// codewords over 32 bits and for naming every failure as the crate does, by
// read_sym. `r` is at the first AC code; `b` gives the bitstream and the end.
template <class Reader, class Out>
__device__ __forceinline__ int decode_ac(uint32_t mask, bool live, Reader &r, const Bits &b, uint32_t n_blocks,
                                         Out &out, const uint16_t *run_tab, const uint16_t *level_tab) {
    const char *run_bytes = reinterpret_cast<const char *>(run_tab);
    const char *level_bytes = reinterpret_cast<const char *>(level_tab);
    const uint32_t total32 = n_blocks * 64u * 32u;
    uint32_t n32 = n_blocks * 32u;  // 32 times the position
    // The rows of previous run 4 and previous level 1.
    uint32_t rrow = 2u << kBookRowShift, lrow = 1u << kBookRowShift;
    int err = DE_OK;
    bool ok = false, done = false;  // of a lane's last step
    if (!live) r.nleft = 0;         // done from the start
    const auto step = [&]() {
        // Zeros past the end: 32 - left bits when that is positive.
        const uint32_t past = (uint32_t)__viaddmax_s32(r.nleft, 32, 0);
        const uint32_t t = r.top() & __funnelshift_lc(0u, 0xFFFFFFFFu, past);
        const uint32_t e1 = *reinterpret_cast<const uint16_t *>(run_bytes + (rrow | ((t >> 20) & 0xFFEu)));
        const uint32_t t2 = __funnelshift_l(0u, t, e1);
        const uint32_t e2 = *reinterpret_cast<const uint16_t *>(level_bytes + (lrow | ((t2 >> 20) & 0xFFEu)));
        const uint32_t t3 = __funnelshift_l(0u, t2, e2);
        const uint32_t len = (e1 & 15u) + (e2 & 15u) + 1u;  // at most 23
        const uint32_t at32 = n32 + (e1 & 0xFE0u);
        // endOfData(): 31 or fewer bits remain, all zero (no run code is).
        done = past > 0 && t == 0;
        ok = ((e1 | e2) & kBookMiss) == 0 && r.nleft + (int32_t)len <= 0 && at32 < total32;
        out.put_code(ok, at32, e2, t3);
        n32 = ok ? at32 + 32u : n32;
        rrow = ok ? e1 & (7u << kBookRowShift) : rrow;
        lrow = ok ? e2 & (7u << kBookRowShift) : lrow;
        r.advance(ok ? len : 0u);
    };
    // One code by any means, at most 65 bits.
    const auto slow_step = [&]() {
        const uint32_t total = n_blocks * 64u;
        uint32_t run = 0, lvl = 0, l = 0, n = n32 >> 5;
        bool have_run = false, have_level = false, neg = false;
        if (r.nleft <= -32) {  // all of top() is data
            have_run = window_code(r.top(), run_book_of_row(rrow >> kBookRowShift), run, l);
            if (have_run) {
                n += run;
                if (n >= total) err = DE_RUN_PAST_END;
                r.advance(l);
                if (r.nleft <= -32) have_level = window_code(r.top(), level_book_of_row(lrow >> kBookRowShift), lvl, l);
                if (have_level) {
                    r.advance(l);
                    if (r.nleft == 0 && !err) err = DE_PAST_END;
                    neg = r.top() >> 31;
                    r.advance(1u);
                }
            }
        }
        if (!have_level && !err) {
            Bits g;
            g.init_at(reinterpret_cast<const uint8_t *>(b.w), b.end - r.left(), b.end);
            if (!have_run) {
                err = read_sym(g, run_book_of_row(rrow >> kBookRowShift), run);
                n += run;
                if (!err && n >= total) err = DE_RUN_PAST_END;
            }
            if (!err) err = read_sym(g, level_book_of_row(lrow >> kBookRowShift), lvl);
            if (!err && g.remaining() < 1) err = DE_PAST_END;
            if (!err) {
                neg = g.peek() >> 63;
                r.init(b.w, g.pos + 1, b.end);
            }
        }
        if (!err) {
            const int32_t level = (int32_t)lvl + 1;
            out.put(n, neg ? -level : level);
            n32 = (n + 1u) * 32u;
            rrow = run_book_row(run) << kBookRowShift;
            lrow = level_book_row(lvl) << kBookRowShift;
        } else {
            r.nleft = 0;
        }
    };
    for (;;) {
        step();
        step();
        step();
        step();
        r.check(mask, !done);
        const bool stuck = !ok && !done;
        if (__any_sync(mask, stuck)) {
            if (stuck) slow_step();
            r.check(mask, !done && err == DE_OK);
        } else if (!__any_sync(mask, !done)) {
            break;
        }
    }
    return err;
}

__device__ __forceinline__ uint16_t rescale(uint32_t a, uint64_t m, bool identity) {
    return identity ? (uint16_t)a : (uint16_t)(((uint64_t)a * m + (1ull << 39)) >> 40);
}

// Where a slice's alpha samples go, and how they are coded.
struct AlphaArea {
    uint16_t *row;         // the slice's first sample
    uint64_t pitch;        // samples from a row to the next of the picture
    uint32_t cols, ncols;  // coded samples a row (16 a macroblock), those inside the picture
    uint32_t rows;         // rows inside the picture
    uint32_t bits;
    uint64_t rescale_m;
    bool identity;
};

__device__ __forceinline__ AlphaArea alpha_area(const FrameDesc &fd, const PicDesc &pd, const SliceDesc &sd,
                                                uint16_t *alpha) {
    AlphaArea a;
    a.bits = fd.alpha_bits;
    a.cols = 16u * sd.mbs;
    a.rows = (uint32_t)sd.mb_y + 1u < pd.height_in_mb ? 16u : pd.height - 16u * (pd.height_in_mb - 1u);
    const uint32_t x0 = 16u * sd.mb_x;
    a.ncols = min(a.cols, fd.width - x0);
    a.row = (fd.out_alpha ? fd.out_alpha : alpha + fd.alpha_off) +
            (uint64_t)(pd.first_row + pd.row_step * (16u * sd.mb_y)) * fd.width + x0;
    a.pitch = (uint64_t)pd.row_step * fd.width;
    a.rescale_m = fd.rescale_m;
    a.identity = fd.rescale_identity != 0;
    return a;
}

// scanned_alpha() (src/decode.rs:570-595) and its placement (:365-389). The
// lanes of `mask` run it together, a slice each. A step reads a difference
// and its run when the last run is used up, and adds samples of the run to a
// group of 8, which goes out as one 16-byte store when it is full (a row is a
// whole number of groups): a lane in a long run and a lane with a code for
// every sample take the same steps. A code that runs past its data or the
// slice waits for the end of three steps and goes by the general reader,
// which names the failure.
template <class Reader>
__device__ __forceinline__ int decode_alpha(uint32_t mask, bool live, Reader &r, const Bits &b, AlphaArea a) {
    const uint32_t count = a.cols * 16u, needed = a.cols * a.rows;
    const int32_t value_mask = (int32_t)((1u << a.bits) - 1u);
    const uint32_t mag_bits = a.bits == 8 ? 3u : 6u;
    int32_t prev = -1;
    uint32_t n = 0, run_left = 0;  // samples up to the end of the run, those of it not placed
    uint32_t pair = 0;             // the run's sample, twice
    uint32_t fill = 0, col = 0, row = 0;
    uint4 group = make_uint4(0, 0, 0, 0);
    int err = DE_OK;
    bool done = !live, stuck = false;
    const auto start_run = [&](int32_t diff, uint32_t run) {
        prev = (int32_t)((uint32_t)prev + (uint32_t)diff) & value_mask;
        pair = 0x10001u * rescale((uint32_t)prev, a.rescale_m, a.identity);
        run_left = run;
        n += run;
    };
    const auto step = [&]() {
        const bool need = run_left == 0 && !done;
        const uint32_t past = (uint32_t)__viaddmax_s32(r.nleft, 32, 0);
        const uint32_t t = r.top() & __funnelshift_lc(0u, 0xFFFFFFFFu, past);
        // Tables 13 and 14: `1` and the difference in full, or `0`, magnitude
        // - 1 and a sign.
        const bool full = t >> 31;
        const int32_t mag = (int32_t)((t << 1) >> (32u - mag_bits)) + 1;
        const bool neg = (t << (1u + mag_bits)) >> 31;
        const int32_t diff = full ? (int32_t)((t << 1) >> (32u - a.bits)) : (neg ? -mag : mag);
        const uint32_t dlen = full ? 1u + a.bits : 2u + mag_bits;
        // Table 12: `1`; `0` and 4 bits of run - 1; or 5 zeros and 11 bits.
        const uint32_t u = r.top_at(dlen);
        const uint32_t r4 = (u << 1) >> 28;
        const uint32_t run = u >> 31 ? 1u : (r4 ? r4 + 1u : ((u << 5) >> 21) + 1u);
        const uint32_t rlen = u >> 31 ? 1u : (r4 ? 5u : 16u);
        const bool end = n >= count || (n >= needed && past > 0 && t == 0);
        const bool ok = need && !end && r.nleft + (int32_t)(dlen + rlen) <= 0 && n + run <= count;
        done = done || (need && end);
        stuck = need && !end && !ok;
        if (ok) start_run(diff, run);
        r.advance(ok ? dlen : 0u);
        r.advance(ok ? rlen : 0u);
        // The samples from `fill` on take the run's value; those past its
        // end are overwritten later.
        const uint32_t k = min(run_left, 8u - fill);
        const auto keep = [&](uint32_t at) {  // of the two samples from `at`, the bits of those before `fill`
            return ~__funnelshift_lc(0u, 0xFFFFFFFFu, (uint32_t)max(16 * ((int32_t)fill - (int32_t)at), 0));
        };
        const auto merge = [&](uint32_t w, uint32_t at) { return (w & keep(at)) | (pair & ~keep(at)); };
        group.x = merge(group.x, 0);
        group.y = merge(group.y, 2);
        group.z = merge(group.z, 4);
        group.w = merge(group.w, 6);
        fill += k;
        run_left -= k;
        if (fill == 8u) {
            fill = 0;
            if (row < a.rows && col < a.ncols) {
                uint16_t *dst = a.row + col;
                if (col + 8u <= a.ncols && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
                    *reinterpret_cast<uint4 *>(dst) = group;
                } else {
                    const uint32_t words[4] = {group.x, group.y, group.z, group.w};
#pragma unroll
                    for (uint32_t x = 0; x < 8; x++)
                        if (col + x < a.ncols) dst[x] = (uint16_t)(words[x / 2u] >> (16u * (x & 1u)));
                }
            }
            col += 8u;
            if (col == a.cols) {
                col = 0;
                row++;
                a.row += a.pitch;
            }
        }
    };
    // A code of the general reader.
    const auto slow_step = [&]() {
        Bits g;
        g.init_at(reinterpret_cast<const uint8_t *>(b.w), b.end - r.left(), b.end);
        uint64_t v = 0;
        int32_t diff = 0;
        uint32_t run = 1;
        err = g.read(1, v);
        if (!err && v == 1) {
            err = g.read(a.bits, v);
            diff = (int32_t)v;
        } else if (!err) {
            err = g.read(mag_bits, v);
            const int32_t mag = (int32_t)v + 1;
            if (!err) err = g.read(1, v);
            diff = v ? -mag : mag;
        }
        if (!err) err = g.read(1, v);
        if (!err && v == 0) {
            err = g.read(4, v);
            if (!err && v == 0) err = g.read(11, v);
            run = (uint32_t)v + 1u;
        }
        if (!err && n + run > count) err = DE_ALPHA_RUN;
        if (!err) {
            start_run(diff, run);
            r.init(b.w, g.pos, b.end);
        } else {
            done = true;
        }
    };
    for (;;) {
        step();
        step();
        step();
        r.check(mask, !done);
        if (__any_sync(mask, stuck)) {
            if (stuck) slow_step();
            stuck = false;
            r.check(mask, !done);
        } else if (!__any_sync(mask, !done)) {
            break;
        }
    }
    return err;
}

// One component by one lane of any warp (the fused decoder).
template <class Out>
__device__ int decode_component(Bits &b, uint32_t n_blocks, Out &out, const uint16_t *run_tab,
                                const uint16_t *level_tab) {
    const uint32_t mask = __activemask();
    WordReader r;
    r.init(b.w, b.pos, b.end);
    const int err = decode_dc(mask, true, r, b, n_blocks, out);
    const int ac_err = decode_ac(mask, err == DE_OK, r, b, n_blocks, out, run_tab, level_tab);
    return err ? err : ac_err;
}

__device__ int decode_alpha_alone(Bits &b, const AlphaArea &a) {
    WordReader r;
    r.init(b.w, b.pos, b.end);
    return decode_alpha(__activemask(), true, r, b, a);
}

// The slice header (src/decode.rs:301-338) and where component `comp` (0
// Y', 1 Cb, 2 Cr, 3 alpha) lies in the slice. A header failure comes back
// (the Y' item reports it; the other components then report nothing).
__device__ int2 component_range(const uint8_t *sb, uint32_t size, bool has_alpha, uint32_t comp, uint32_t &start,
                                uint32_t &len) {
    const uint32_t min_header = has_alpha ? 8u : 6u;
    uint32_t hs = 0, ys = 0, cbs = 0, crs = 0;
    if (size < min_header) return make_int2(DE_SLICE_SHORT, 0);
    hs = sb[0] >> 3;
    const uint32_t qi = sb[1];
    if (hs < min_header || hs > size) return make_int2(DE_SLICE_HDR_SIZE, (int)hs);
    if (qi < 1 || qi > 224) return make_int2(DE_QINDEX, (int)qi);
    ys = be16(sb + 2);
    cbs = be16(sb + 4);
    const uint32_t body = size - hs;
    if (has_alpha) {
        crs = be16(sb + 6);
    } else {
        if (ys + cbs > body) return make_int2(DE_COMP_SIZES, 0);
        crs = body - ys - cbs;
    }
    if (ys + cbs + crs > body) return make_int2(DE_COMP_SIZES, 0);
    start = hs;
    if (comp == 0) {
        len = ys;
    } else if (comp == 1) {
        start += ys;
        len = cbs;
    } else if (comp == 2) {
        start += ys + cbs;
        len = crs;
    } else {
        start += ys + cbs + crs;
        len = size - start;
    }
    return make_int2(DE_OK, 0);
}

// One work item a lane: component `comp` (0 Y', 1 Cb, 2 Cr, 3 alpha) of slice
// `s`, or none (`valid` false). All lanes of the warp come here together.
__device__ __forceinline__ void decode_items(const DecodeLaunch &d, bool valid, uint32_t comp, uint32_t s,
                                             const uint16_t *run_tab, const uint16_t *level_tab, uint32_t *ring) {
    Bits b{};
    CoefList list{};
    uint32_t n_blocks = 0;
    bool live = false, live_alpha = false;  // a colour component, an alpha component to decode
    AlphaArea area{};
    int2 status = make_int2(DE_OK, 0);
    if (valid) {
        const SliceDesc sd = d.slices[s];
        const PicDesc &pd = d.pics[sd.pic];
        // A picture that failed before decoding is never read.
        valid = d.pic_status[sd.pic].locate_slice < 0;
        const FrameDesc &fd = d.frames[pd.frame];
        const bool has_alpha = fd.alpha_bits != 0;
        if (valid && (comp < 3 || has_alpha)) {
            uint32_t start = 0, len = 0;
            const int2 hdr_err = component_range(d.bits + sd.off, sd.size, has_alpha, comp, start, len);
            if (hdr_err.x != DE_OK) {
                if (comp == 0) status = hdr_err;
            } else {
                b.init(d.bits, sd.off + start, len);
                if (comp == 3) {
                    area = alpha_area(fd, pd, sd, d.alpha);
                    live_alpha = true;
                } else {
                    const uint32_t cpm = fd.chroma == 2 ? 2u : 4u;
                    n_blocks = (comp == 0 ? 4u : cpm) * sd.mbs;
                    const uint64_t base = sd.coef + (comp == 0 ? 0ull : 64ull * sd.mbs * (4u + (comp - 1u) * cpm));
                    list.w = reinterpret_cast<uint32_t *>(d.coef + base);
                    list.cap = 64u * n_blocks;
                    live = true;
                }
            }
        }
    }
    __syncwarp();
    RingReader r{};
    r.ring = ring;
    if (live || live_alpha) r.init(b.w, b.pos, b.end);
    r.check(0xffffffffu, live || live_alpha);
    if (__any_sync(0xffffffffu, live_alpha)) {
        const int err = decode_alpha(0xffffffffu, live_alpha, r, b, area);
        if (live_alpha) status.x = err;
    }
    if (__any_sync(0xffffffffu, live)) {
        const int dc_err = decode_dc(0xffffffffu, live, r, b, n_blocks, list);
        const int ac_err = decode_ac(0xffffffffu, live && dc_err == DE_OK, r, b, n_blocks, list, run_tab, level_tab);
        if (live) {
            status.x = dc_err ? dc_err : ac_err;
            list.finish();
        }
    }
    if (valid) {
        // Every run writes every count of the slices it decodes (a failing
        // component's too), so k_idct never reads a stale one.
        if (comp < 3) d.coef_count[3ull * s + comp] = list.count | (list.big ? kListBig : 0u);
        d.slot_status[4ull * s + comp] = status;
    }
}

// ------------------------------------------------------------------ kernels

constexpr int kLocateThreads = 1024;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__global__ void __launch_bounds__(kLocateThreads) k_locate(DecodeLaunch d) {
    chain_start();
    chain_wait();
    __shared__ uint32_t warp_sums[kLocateThreads / 32];
    __shared__ uint64_t carry;
    __shared__ int first_bad;
    const PicDesc p = d.pics[blockIdx.x];
    const FrameDesc &fd = d.frames[p.frame];
    const uint32_t cpm = fd.chroma == 2 ? 2u : 4u;
    const uint32_t coef_per_mb = 64u * (4u + 2u * cpm);
    const uint32_t S = 1u << p.log2_slice_mbs;
    const uint32_t full = p.width_in_mb >> p.log2_slice_mbs;
    const uint32_t rem_mbs = p.width_in_mb & (S - 1u);
    const uint8_t *table = d.bits + p.off + p.header_size;
    const uint64_t data_start = p.off + p.header_size + 2ull * p.n_slices;
    const uint64_t limit = p.off + p.picture_size;
    if (threadIdx.x == 0) {
        carry = 0;
        first_bad = INT32_MAX;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t chunk = 0; chunk < p.n_slices; chunk += kLocateThreads) {
        const uint32_t k = chunk + threadIdx.x;
        const uint32_t size = k < p.n_slices ? be16(table + 2ull * k) : 0u;
        uint32_t incl = warp_incl_scan(size);
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            uint32_t ws = warp_sums[lane];
            warp_sums[lane] = warp_incl_scan(ws);
        }
        __syncthreads();
        const uint64_t excl = carry + (warp ? warp_sums[warp - 1] : 0u) + incl - size;
        if (k < p.n_slices) {
            const uint64_t off = data_start + excl;
            if (off + size > limit) atomicMin(&first_bad, (int)k);
            const uint32_t row = k / p.slices_per_row, j = k - row * p.slices_per_row;
            uint32_t mb_x, mbs;
            if (j < full) {
                mb_x = j * S;
                mbs = S;
            } else {
                // The slices after the full ones halve down the binary digits
                // of what is left (src/header.rs:308-320).
                uint32_t idx = j - full;
                mb_x = full * S;
                mbs = 1;
                for (int bit = (int)p.log2_slice_mbs - 1; bit >= 0; bit--) {
                    if (!(rem_mbs & (1u << bit))) continue;
                    if (idx == 0) {
                        mbs = 1u << bit;
                        break;
                    }
                    mb_x += 1u << bit;
                    idx--;
                }
            }
            SliceDesc sd;
            sd.off = off;
            sd.size = size;
            sd.pic = blockIdx.x;
            sd.mb_x = (uint16_t)mb_x;
            sd.mb_y = (uint16_t)row;
            sd.mbs = mbs;
            sd.coef = p.coef_base + ((uint64_t)row * p.width_in_mb + mb_x) * coef_per_mb;
            d.slices[p.slice_base + k] = sd;
            // The slice's items for k_idct: its parts, or a group's once (the
            // fused decode alone has none).
            const IdctShape shape = idct_shape(fd.chroma, p.log2_slice_mbs);
            if (!d.idct_items) {
            } else if (shape.slices > 1u) {
                if (k % shape.slices == 0)
                    d.idct_items[p.idct_base + k / shape.slices] =
                        make_uint4(p.slice_base + k, min(shape.slices, p.n_slices - k) << 8, blockIdx.x, p.frame);
            } else {
                for (uint32_t part = 0; part < shape.parts; part++)
                    d.idct_items[p.idct_base + k * shape.parts + part] =
                        make_uint4(p.slice_base + k, (1u << 8) | part, blockIdx.x, p.frame);
            }
        }
        __syncthreads();
        if (threadIdx.x == kLocateThreads - 1) carry += (warp ? warp_sums[warp - 1] : 0u) + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        PicStatus st;
        st.locate_slice = first_bad == INT32_MAX ? -1 : first_bad;
        st.slot = -1;
        st.code = 0;
        st.aux = 0;
        d.pic_status[blockIdx.x] = st;
    }
}

constexpr int kEntropyMaxThreads = 512;

// Persistent: each warp takes 32 x entropy_per_lane slice components per
// grab of the work counter, a lane each in turn, component-major, until the
// list runs out. The alpha components come first: where a frame has alpha,
// its codes take a lane several times as long as a colour component, and
// started last they would leave the launch waiting on them.
//
// Bound by the length of a component's chain of codes (small batches: a step
// waits for two table reads one after the other) and by integer issue (8 UHD
// frames: 60 % of the slots, 68 % of the ALU pipe, 29 of 32 lanes at work).
// 32 UHD 4:2:2 frames take 680 us, one 175, 8 UHD 4:4:4 frames with 16-bit
// alpha 1030; with a branch for every case, loads and single-entry stores
// among the steps, 1810, 535 and 2770. 83 registers, given out as 88, leave
// two CTAs of 8 warps an SM; held to 64, for four, the spills cost 14 %.
__global__ void __launch_bounds__(kEntropyMaxThreads) k_entropy(DecodeLaunch d) {
    chain_start();
    extern __shared__ __align__(16) unsigned char smem[];
    uint16_t *run_tab = reinterpret_cast<uint16_t *>(smem), *level_tab = run_tab + kBookTableWords;
    // Each warp's ring: word k of lane l at [32 k + l].
    uint32_t *ring = reinterpret_cast<uint32_t *>(level_tab + kBookTableWords) + 8u * (threadIdx.x & ~31u) + (threadIdx.x & 31u);
    for (uint32_t i = threadIdx.x; i < kBookTableWords / 2; i += blockDim.x) {
        reinterpret_cast<uint32_t *>(run_tab)[i] = reinterpret_cast<const uint32_t *>(d.tables.run_books)[i];
        reinterpret_cast<uint32_t *>(level_tab)[i] = reinterpret_cast<const uint32_t *>(d.tables.level_books)[i];
    }
    chain_wait();
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t items = 4u * d.n_slices;
    const uint32_t per_lane = d.entropy_per_lane > 0 ? d.entropy_per_lane : 1u;
    const uint32_t grab = 32u * per_lane;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(d.work_counter, grab);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= items) break;
        for (uint32_t k = 0; k < per_lane; k++) {
            const uint32_t item = base + 32u * k + lane;
            const uint32_t kind = item / d.n_slices, s = item - kind * d.n_slices;
            decode_items(d, item < items, kind == 0 ? 3u : kind - 1u, s, run_tab, level_tab, ring);
        }
    }
}

// Placement of block b of macroblock m (src/decode.rs:395-413).
__device__ __forceinline__ void block_xy(uint32_t comp, uint32_t chroma, uint32_t mb_x, uint32_t mb_y, uint32_t m,
                                         uint32_t b, uint32_t &bx, uint32_t &by) {
    const uint32_t x = mb_x + m, y0 = 16u * mb_y;
    if (comp == 0) {
        bx = 16u * x + 8u * (b & 1u);
        by = y0 + 8u * (b >> 1);
    } else if (chroma == 2) {
        bx = 8u * x;
        by = y0 + 8u * b;
    } else {
        bx = 16u * x + 8u * (b >> 1);
        by = y0 + 8u * (b & 1u);
    }
}

// k_idct: a warp takes up to 32 blocks (IdctShape), a lane each for the
// transform. The warp dequantises the components' lists into its own shared
// memory, every lane runs its block's rows and then its columns from there
// with the paired sums of pair_math.h (13 instructions a sample for both
// passes, from 24 with a product for every term), and stores whole 16-byte
// rows from registers: neighbouring lanes hold neighbouring blocks, so a
// store covers 256 contiguous bytes and nothing is staged. No barrier wider
// than a warp; the next list words are on their way while the last are
// placed. Bound by issue (66 % of the slots, 37 instructions a sample at 36 %
// non-zeros) and by the 24 warps an SM that the blocks' 8.7 kB leave room for
// (20, at 102 registers: 11 % slower; 16: 25 %), in CTAs of 2, whose place is
// free sooner than one of 4 (813 us). 32 UHD 4:2:2 frames take 801 us, where a
// CTA per slice with index arithmetic for every row and column task and all 64
// products took 1990; a mixed batch 424 for 1585.
constexpr int kIdctWarps = 2;
// A block's floats in shared memory: 64 and 4 more, so that eight lanes'
// 16-byte reads of the same place in neighbouring blocks meet no bank twice.
constexpr uint32_t kBlockStride = 68;
struct IdctWarp {
    float f[32 * kBlockStride];
    // By scanned index, luma then chroma: the weight, which as a float has
    // its low 16 bits clear, with the raster position's byte offset in them.
    uint32_t weight[2][64];
};

// floor(a), floor(b) as integers clamped to [0, 2^16), a in the low half (an
// infinity clamps, a NaN gives 0, as a maximum with 0 would).
__device__ __forceinline__ uint32_t floor_pair(float a, float b) {
    uint32_t r;
    asm("{\n\t.reg .s32 i, j;\n\tcvt.rmi.s32.f32 i, %1;\n\tcvt.rmi.s32.f32 j, %2;\n\t"
        "cvt.pack.sat.u16.s32 %0, j, i;\n\t}"
        : "=r"(r)
        : "f"(a), "f"(b));
    return r;
}

// The column pass of four columns t (in shared memory: t[8 v] is row v's
// four), rows in order, zero rows (clear in `rows`) skipped, and the
// conversion floor(v scale + bias) clamped. Stored columns are in the order
// the row pass leaves them: 0, 1, 3, 2 (kForward) or 7, 6, 4, 5; words kFirst
// and kFirst + 1 of out[y] get row y's samples in picture order.
template <int kFirst, bool kForward>
__device__ __forceinline__ void idct_columns(const float *t, uint32_t rows, float oscale, uint64_t bias2, uint32_t max2,
                                             uint32_t (&out)[8][4]) {
    Pairs8 c[4];
    const auto term = [&](auto v) {
        constexpr int u = decltype(v)::value;
        if (u > 0 && !((rows >> u) & 1u)) return;
        const float4 r = *reinterpret_cast<const float4 *>(t + 8 * u);
        pairs_term<u, u == 0>(c[0], r.x, c_idct_basis);
        pairs_term<u, u == 0>(c[1], r.y, c_idct_basis);
        pairs_term<u, u == 0>(c[2], r.z, c_idct_basis);
        pairs_term<u, u == 0>(c[3], r.w, c_idct_basis);
    };
    term(std::integral_constant<int, 0>{});
    term(std::integral_constant<int, 1>{});
    term(std::integral_constant<int, 2>{});
    term(std::integral_constant<int, 3>{});
    term(std::integral_constant<int, 4>{});
    term(std::integral_constant<int, 5>{});
    term(std::integral_constant<int, 6>{});
    term(std::integral_constant<int, 7>{});
    // Two rows, ya and yb, of the pair m of every column.
    const auto put = [&](uint64_t Pairs8::*m, int ya, int yb) {
        float lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float a, b;
            pair_split(c[k].*m, a, b);
            pair_split(pair_add(pair_of(__fmul_rn(a, oscale), __fmul_rn(b, oscale)), bias2), lo[k], hi[k]);
        }
        if (kForward) {
            out[ya][kFirst] = __vminu2(floor_pair(lo[0], lo[1]), max2);
            out[ya][kFirst + 1] = __vminu2(floor_pair(lo[3], lo[2]), max2);
            out[yb][kFirst] = __vminu2(floor_pair(hi[0], hi[1]), max2);
            out[yb][kFirst + 1] = __vminu2(floor_pair(hi[3], hi[2]), max2);
        } else {
            out[ya][kFirst] = __vminu2(floor_pair(lo[2], lo[3]), max2);
            out[ya][kFirst + 1] = __vminu2(floor_pair(lo[1], lo[0]), max2);
            out[yb][kFirst] = __vminu2(floor_pair(hi[2], hi[3]), max2);
            out[yb][kFirst + 1] = __vminu2(floor_pair(hi[1], hi[0]), max2);
        }
    };
    put(&Pairs8::o01, 0, 1);
    put(&Pairs8::o32, 3, 2);
    put(&Pairs8::o45, 4, 5);
    put(&Pairs8::o76, 7, 6);
}

__global__ void __launch_bounds__(32 * kIdctWarps, 12) k_idct(DecodeLaunch d) {
    chain_start();
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    IdctWarp &w = reinterpret_cast<IdctWarp *>(smem)[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t index = blockIdx.x * kIdctWarps + (threadIdx.x >> 5);
    if (index >= d.n_idct_items) return;
    // The item names its picture and frame, so every descriptor is fetched at
    // once, and the first list words once those are there.
    const uint4 item = d.idct_items[index];
    const uint32_t first = item.x, n_slices = item.y >> 8, part = item.y & 255u;
    const PicDesc &pd = d.pics[item.z];
    const FrameDesc &fd = d.frames[item.w];
    if (d.pic_status[item.z].locate_slice >= 0) return;
    const uint32_t cpm = fd.chroma == 2 ? 2u : 4u;
    const IdctShape shape = idct_shape(fd.chroma, pd.log2_slice_mbs);
    // The components [c0, c1) of the item's slices.
    uint32_t c0, c1;
    idct_components(shape, cpm, part, c0, c1);
    const uint32_t n_lists = n_slices * (c1 - c0);

    // Lane l < n_lists looks after list l: slice l / (c1 - c0)'s component.
    const uint32_t per = c1 - c0;
    uint32_t list_coef = 0, list_n = 0, list_nb = 1, list_at = 0;  // region / 64, entries, blocks, first lane
    uint32_t list_xy = 0;                                          // the slice's place in macroblocks
    float list_q8 = 0.0f;                                          // qScale / 8
    if (lane < n_lists) {
        const uint32_t j = per == 1u ? lane : (per == 2u ? lane >> 1 : lane / 3u), c = c0 + lane - j * per;
        const SliceDesc sd = d.slices[first + j];
        list_n = d.coef_count[3ull * (first + j) + c];
        const uint32_t qi = sd.size >= 2 ? d.bits[sd.off + 1] : 1u;
        list_q8 = (float)qscale(min(max(qi, 1u), 224u)) * 0.125f;
        list_nb = (c == 0 ? 4u : cpm) * sd.mbs;
        const uint32_t start = c == 0 ? 0u : sd.mbs * (4u + (c - 1u) * cpm);
        list_coef = (uint32_t)(sd.coef >> 6) + start;
        list_at = j * shape.blocks + start - (c0 == 0 ? 0u : sd.mbs * (4u + (c0 - 1u) * cpm));
        list_xy = sd.mb_x | ((uint32_t)sd.mb_y << 16);
    }
    // This lane's block: its list and component, and its place there.
    uint32_t my_list = 32, my_comp = 0, my_blk = 0;

    // A list's state for the whole warp, and four of its entries from `i` on
    // (this lane's: i + 4 lane).
    struct List {
        const uint32_t *words;
        uint32_t n, nb, at, shift, comp;
        bool big;
        float q8;
    };
    const auto open = [&](uint32_t l, uint32_t comp) {
        List r;
        r.words = reinterpret_cast<const uint32_t *>(d.coef + ((uint64_t)__shfl_sync(0xffffffffu, list_coef, l) << 6));
        r.nb = __shfl_sync(0xffffffffu, list_nb, l);
        r.n = __shfl_sync(0xffffffffu, list_n, l);
        r.big = (r.n & kListBig) != 0;
        r.n = min(r.n & ~kListBig, 64u * r.nb);
        r.at = __shfl_sync(0xffffffffu, list_at, l);
        r.q8 = __shfl_sync(0xffffffffu, list_q8, l);
        r.shift = 31u - __clz(r.nb);
        r.comp = comp;
        if (lane - r.at < r.nb) {
            my_list = l;
            my_comp = comp;
            my_blk = lane - r.at;
        }
        return r;
    };
    const auto fetch = [&](const List &l, uint32_t i) {
        i += 4u * lane;
        return i < l.n ? *reinterpret_cast<const uint4 *>(l.words + i) : make_uint4(0, 0, 0, 0);
    };
    List list = open(0, c0);
    uint4 e = fetch(list, 0);

    // Zeros, and the picture's weights in scanned order.
#pragma unroll
    for (uint32_t i = 0; i < kBlockStride / 4u; i++)
        reinterpret_cast<float4 *>(w.f)[32u * i + lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
        const uint32_t r = (i & 1u) * 32u + lane;
        const float weight = (float)d.weights[fd.weights * 128u + 32u * i + lane];
        w.weight[i >> 1][d_scan[pd.interlaced_scan][r]] = __float_as_uint(weight) | (4u * r);
    }
    __syncwarp();

    // The coefficient lists, dequantised (F = QF W qScale / 8,
    // src/decode.rs:356; W qScale / 8 is exact) into the blocks. Positions
    // are below the component's end: k_entropy stops at a run that passes it.
    for (uint32_t l = 0; l < n_lists; l++) {
        List next = list;
        uint4 ahead = make_uint4(0, 0, 0, 0);
        if (l + 1u < n_lists) {
            next = open(l + 1u, list.comp + 1u == c1 ? c0 : list.comp + 1u);
            ahead = fetch(next, 0);
        }
        const uint32_t *table = w.weight[list.comp > 0 ? 1 : 0];
        char *blocks = reinterpret_cast<char *>(w.f + list.at * kBlockStride);
        const auto put = [&](uint32_t x, float v) {
            const uint32_t pos = x >> 21;
            const uint32_t t = table[pos >> list.shift];
            const float scale = __fmul_rn(__uint_as_float(t & 0xFFFF0000u), list.q8);
            *reinterpret_cast<float *>(blocks + (pos & (list.nb - 1u)) * (4u * kBlockStride) + (t & 0xFFFFu)) =
                __fmul_rn(v, scale);
        };
        const auto small = [](uint32_t x) {
            return __uint_as_float(__float_as_uint(__uint2float_rn((x >> 5) & 0xFFFFu)) | (x << 31));
        };
        const auto place = [&](uint32_t x) { put(x, small(x)); };
        uint32_t i = 0;
        if (!list.big) {
            for (; i + 128u <= list.n; i += 128u) {
                const uint4 x = e;
                e = fetch(list, i + 128u);
                place(x.x);
                place(x.y);
                place(x.z);
                place(x.w);
            }
            i += 4u * lane;
            if (i < list.n) place(e.x);
            if (i + 1u < list.n) place(e.y);
            if (i + 2u < list.n) place(e.z);
            if (i + 3u < list.n) place(e.w);
        } else {
            for (i = lane; i < list.n; i += 32u) {
                const uint32_t x = list.words[i], mag = (x >> 5) & 0xFFFFu;
                put(x, mag < kListBigMag ? small(x)
                                         : __int2float_rn((int32_t)list.words[128u * list.nb - 1u - (mag - kListBigMag)]));
            }
        }
        list = next;
        e = ahead;
    }
    __syncwarp();

    // Row pass: tmp[v][x] = sum_u F[v][u] T[x][u], u in order (src/dct.rs:
    // 38-53), each lane its block's rows over their coefficients, in the
    // order 0, 1, 3, 2, 7, 6, 4, 5 the sums come in. A row that is zero in
    // all 32 blocks stays zero.
    float *blk = w.f + lane * kBlockStride;
    uint32_t rows = 1u;
#pragma unroll 1
    for (uint32_t v = 0; v < 8; v++) {
        const float4 a = *reinterpret_cast<const float4 *>(blk + 8u * v);
        const float4 b = *reinterpret_cast<const float4 *>(blk + 8u * v + 4u);
        const uint32_t any = __float_as_uint(a.x) | __float_as_uint(a.y) | __float_as_uint(a.z) | __float_as_uint(a.w) |
                             __float_as_uint(b.x) | __float_as_uint(b.y) | __float_as_uint(b.z) | __float_as_uint(b.w);
        if (!__any_sync(0xffffffffu, any != 0)) continue;
        rows |= 1u << v;
        Pairs8 o;
        pairs_term<0, true>(o, a.x, c_idct_basis);
        pairs_term<1, false>(o, a.y, c_idct_basis);
        pairs_term<2, false>(o, a.z, c_idct_basis);
        pairs_term<3, false>(o, a.w, c_idct_basis);
        pairs_term<4, false>(o, b.x, c_idct_basis);
        pairs_term<5, false>(o, b.y, c_idct_basis);
        pairs_term<6, false>(o, b.z, c_idct_basis);
        pairs_term<7, false>(o, b.w, c_idct_basis);
        *reinterpret_cast<ulonglong2 *>(blk + 8u * v) = make_ulonglong2(o.o01, o.o32);
        *reinterpret_cast<ulonglong2 *>(blk + 8u * v + 4u) = make_ulonglong2(o.o76, o.o45);
    }

    // Column pass and conversion, half a block's columns at a time.
    uint32_t px[8][4];
    {
        const uint64_t bias2 = pair_of(fd.out_bias, fd.out_bias);
        const uint32_t max1 = (1u << fd.bit_depth) - 1u, max2 = max1 | (max1 << 16);
        idct_columns<0, true>(blk, rows, fd.out_scale, bias2, max2, px);
        idct_columns<2, false>(blk + 4, rows, fd.out_scale, bias2, max2, px);
    }

    // A 16-byte row of the block at a time: neighbouring lanes' blocks are
    // neighbours in the picture.
    const uint32_t xy = __shfl_sync(0xffffffffu, list_xy, my_list);
    if (my_list == 32u) return;
    const uint32_t mb_shift = my_comp == 0 || cpm == 4u ? 2u : 1u;
    uint32_t bx, by;
    block_xy(my_comp, fd.chroma, xy & 0xFFFFu, xy >> 16, my_blk >> mb_shift, my_blk & ((1u << mb_shift) - 1u), bx, by);
    const uint32_t pw = fd.plane_w[my_comp];
    if (bx >= pw || by >= pd.height) return;
    uint16_t *plane = fd.out_planes ? fd.out_planes + (fd.plane_off[my_comp] - fd.plane_off[0])
                                    : d.planes + fd.plane_off[my_comp];
    uint16_t *dst = plane + (uint64_t)(pd.first_row + pd.row_step * by) * pw + bx;
    const uint64_t pitch = (uint64_t)pd.row_step * pw;
    const uint32_t cols = min(8u, pw - bx), n_rows = min(8u, pd.height - by);
#pragma unroll
    for (uint32_t y = 0; y < 8; y++, dst += pitch) {
        if (y >= n_rows) break;
        if (cols == 8u && ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0)) {
            *reinterpret_cast<uint4 *>(dst) = make_uint4(px[y][0], px[y][1], px[y][2], px[y][3]);
        } else {
#pragma unroll
            for (uint32_t x = 0; x < 8; x++)
                if (x < cols) dst[x] = (uint16_t)(px[y][x / 2u] >> (16u * (x & 1u)));
        }
    }
}

// ------------------------------------------------------------ fused decode
//
// k_decode: the whole per-slice chain in one kernel (src/decode.rs:292-391).
// A CTA takes a group of consecutive slices of the flat list at a time
// (grabbed from a work counter) and
//   1. zeroes the group's coefficient slots in shared memory (one int16 per
//      scanned position of every component) and sets the slices up: where
//      their positions and blocks start, their dequantisation factors;
//   2. decodes every component of the group, one thread each (Y' of every
//      slice, then Cb, Cr, alpha), straight into the slots; alpha goes to
//      its plane as it is decoded;
//   3. transforms every block of the group, one thread each, in registers:
//      dequantise, the 8x8 IDCT in the crate's single-precision order,
//      conversion, and 16-byte row stores into the woven planes.
// No coefficient leaves the chip; the bitstream is read once and the planes
// written once.

constexpr int kDecodeThreads = 128;
constexpr uint32_t kMaxGroup = 32;  // slices a CTA decodes at once (4 items each <= 128 threads)

// Figures 4 and 5, folded into immediates in the unrolled transform:
// scan_at<IL>(8 v + u) is the scanned index of row v, column u.
struct ScanPair {
    uint8_t v[2][64];
};
__device__ constexpr ScanPair scan_pair() {
    ScanPair s{};
    for (int i = 0; i < 64; i++) {
        s.v[0][i] = kProgressiveScan[i];
        s.v[1][i] = kInterlacedScan[i];
    }
    return s;
}
template <int IL>
__device__ __forceinline__ constexpr uint32_t scan_at(int i) {
    constexpr ScanPair s = scan_pair();
    return s.v[IL][i];
}

// A slice of a CTA's group.
struct GroupSlice {
    uint32_t pos;         // its first position in the group's slots
    uint32_t blk;         // its first block in the group's list of blocks
    uint32_t nb_y, nb_c;  // blocks of Y' and of each chroma component
    uint32_t live;        // decoded at all (its picture's slices were located)
};



// One block: dequantise (F = QF scale, src/dsp/scalar.rs:8-12), the IDCT's
// row pass tmp[v][x] = sum_u F[v][u] T[x][u] and column pass
// f[y][x] = sum_v T[y][v] tmp[v][x], each sum in the crate's order
// (src/dct.rs:36-66), then floor(f s + b) clamped, stored row by row. Every
// term is computed: a zero term adds nothing to a non-zero sum and only
// flips the sign of a zero one, which the conversion cannot see, so the
// crate's skipped zero rows and its leading 0 + come out the same.
template <int IL, class T>
__device__ __forceinline__ void idct_block(const T *cs, const int32_t *wide, uint32_t nb, uint32_t blk,
                                           const float *sc, float oscale, float obias, float omax, uint16_t *row0,
                                           uint64_t row_pitch, uint32_t cols, uint32_t rows) {
    float t[64];
#pragma unroll
    for (int v = 0; v < 8; v++) {
        float f[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint32_t n = scan_at<IL>(8 * v + u) * nb + blk;
            const int32_t q = cs[n];
            const float fq = q == wide_mark<T>() ? __int2float_rn(wide[n]) : small_int_to_float(q);
            f[u] = __fmul_rn(fq, sc[8 * v + u]);
        }
#pragma unroll
        for (int x = 0; x < 8; x++) {
            float acc = __fmul_rn(f[0], c_idct_basis[8 * x]);
#pragma unroll
            for (int u = 1; u < 8; u++) acc = __fadd_rn(acc, __fmul_rn(f[u], c_idct_basis[8 * x + u]));
            t[8 * v + x] = acc;
        }
    }
#pragma unroll
    for (int y = 0; y < 8; y++) {
        uint32_t px[8];
#pragma unroll
        for (int x = 0; x < 8; x++) {
            float acc = __fmul_rn(c_idct_basis[8 * y], t[x]);
#pragma unroll
            for (int v = 1; v < 8; v++) acc = __fadd_rn(acc, __fmul_rn(c_idct_basis[8 * y + v], t[8 * v + x]));
            px[x] = floor_clamped(__fadd_rn(__fmul_rn(acc, oscale), obias), omax);
        }
        if ((uint32_t)y >= rows) continue;
        uint16_t *dst = row0 + (uint64_t)y * row_pitch;
        if (cols == 8u && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
            uint4 w;
            w.x = __byte_perm(px[0], px[1], 0x5410);
            w.y = __byte_perm(px[2], px[3], 0x5410);
            w.z = __byte_perm(px[4], px[5], 0x5410);
            w.w = __byte_perm(px[6], px[7], 0x5410);
            __stcs(reinterpret_cast<uint4 *>(dst), w);
        } else {
#pragma unroll
            for (int x = 0; x < 8; x++)
                if ((uint32_t)x < cols) dst[x] = (uint16_t)px[x];
        }
    }
}

template <class T>
__global__ void __launch_bounds__(kDecodeThreads) k_decode(DecodeLaunch d) {
    chain_start();
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    uint16_t *run_tab = reinterpret_cast<uint16_t *>(smem);
    uint16_t *level_tab = run_tab + kBookTableWords;
    GroupSlice *gs = reinterpret_cast<GroupSlice *>(level_tab + kBookTableWords);  // kMaxGroup
    float *scale = reinterpret_cast<float *>(gs + kMaxGroup);                    // [group][luma, chroma][64]
    T *slots = reinterpret_cast<T *>(scale + 128u * d.group);                   // group_positions
    __shared__ uint32_t s_group, s_blocks;

    for (uint32_t i = threadIdx.x; i < kBookTableWords / 2; i += kDecodeThreads) {
        reinterpret_cast<uint32_t *>(run_tab)[i] = reinterpret_cast<const uint32_t *>(d.tables.run_books)[i];
        reinterpret_cast<uint32_t *>(level_tab)[i] = reinterpret_cast<const uint32_t *>(d.tables.level_books)[i];
    }
    const uint32_t n_groups = (d.n_slices + d.group - 1u) / d.group;
    int32_t *wide_all = reinterpret_cast<int32_t *>(d.coef);
    for (;;) {
        __syncthreads();  // the last group's blocks are all transformed (and the tables are in)
        if (threadIdx.x == 0) s_group = atomicAdd(d.work_counter, 1u);
        __syncthreads();
        const uint32_t g = s_group;
        if (g >= n_groups) break;
        const uint32_t first = g * d.group;
        const uint32_t count = min(d.group, d.n_slices - first);

        // 1. Zeroed slots; the slices' places in the group.
        for (uint32_t i = threadIdx.x; i < d.group_positions * sizeof(T) / 16u; i += kDecodeThreads)
            reinterpret_cast<int4 *>(slots)[i] = make_int4(0, 0, 0, 0);
        if (threadIdx.x < 32) {
            const uint32_t k = threadIdx.x;
            GroupSlice e{};
            uint32_t n_pos = 0, n_blk = 0;
            if (k < count) {
                const SliceDesc sd = d.slices[first + k];
                const uint32_t cpm = d.frames[d.pics[sd.pic].frame].chroma == 2 ? 2u : 4u;
                e.nb_y = 4u * sd.mbs;
                e.nb_c = cpm * sd.mbs;
                e.live = d.pic_status[sd.pic].locate_slice < 0;
                n_pos = 64u * (e.nb_y + 2u * e.nb_c);
                n_blk = e.live ? e.nb_y + 2u * e.nb_c : 0u;
            }
            const uint32_t ip = warp_incl_scan(n_pos), ib = warp_incl_scan(n_blk);
            e.pos = ip - n_pos;
            e.blk = ib - n_blk;
            if (k < count) gs[k] = e;
            if (k == 31) s_blocks = ib;
        }
        // F = QF W qScale / 8, one factor per raster position (src/decode.rs:356).
        for (uint32_t i = threadIdx.x; i < 128u * count; i += kDecodeThreads) {
            const uint32_t k = i >> 7, which = (i >> 6) & 1u, r = i & 63u;
            const SliceDesc sd = d.slices[first + k];
            const FrameDesc &fd = d.frames[d.pics[sd.pic].frame];
            uint32_t qi = sd.size >= 2 ? d.bits[sd.off + 1] : 1u;
            qi = qi < 1u ? 1u : (qi > 224u ? 224u : qi);
            scale[i] = (float)((uint32_t)d.weights[fd.weights * 128u + which * 64u + r] * qscale(qi)) / 8.0f;
        }
        __syncthreads();

        // 2. Entropy decoding. Thread i takes item kind i / count of slice
        // i % count: kind 0 its Y', kind 1 its Cb and then its Cr for 4:2:2
        // (together about as long as Y') or its Cb for 4:4:4, kind 2 the
        // Cr of a 4:4:4 slice, kind 3 its alpha; so the threads of a warp
        // mostly decode codes of about equal length.
        for (uint32_t i = threadIdx.x; i < 4u * count; i += kDecodeThreads) {
            const uint32_t kind = i / count, k = i - kind * count;
            const GroupSlice e = gs[k];
            if (!e.live) continue;  // never read: the picture failed before decoding
            const uint32_t s = first + k;
            const SliceDesc sd = d.slices[s];
            const PicDesc &pd = d.pics[sd.pic];
            const FrameDesc &fd = d.frames[pd.frame];
            const bool pair = fd.chroma == 2;  // 4:2:2: Cb and Cr on one thread
            uint32_t c = kind, last = kind;
            if (kind == 1 && pair) last = 2;
            if (kind == 2 && pair) continue;
            for (; c <= last; c++) {
                const bool has_alpha = fd.alpha_bits != 0;
                int2 *status = d.slot_status + 4ull * s + c;
                if (c == 3 && !has_alpha) {
                    *status = make_int2(DE_OK, 0);
                    continue;
                }
                uint32_t start = 0, len = 0;
                const int2 he = component_range(d.bits + sd.off, sd.size, has_alpha, c, start, len);
                if (he.x != DE_OK) {
                    *status = c == 0 ? he : make_int2(DE_OK, 0);
                    continue;
                }
                Bits b;
                b.init(d.bits, sd.off + start, len);
                int err;
                if (c == 3) {
                    err = decode_alpha_alone(b, alpha_area(fd, pd, sd, d.alpha));
                } else {
                    const uint32_t nb = c == 0 ? e.nb_y : e.nb_c;
                    const uint32_t off = c == 0 ? 0u : 64u * (e.nb_y + (c - 1u) * e.nb_c);
                    SlotOut<T> out{slots + e.pos + off, wide_all + sd.coef + off};
                    err = decode_component(b, nb, out, run_tab, level_tab);
                }
                *status = make_int2(err, 0);
            }
        }
        __syncthreads();

        // 3. Every block: transform, convert, store.
        const uint32_t n_blocks = s_blocks;
        for (uint32_t bi = threadIdx.x; bi < n_blocks; bi += kDecodeThreads) {
            uint32_t k = 0;
            while (k + 1u < count && gs[k + 1u].blk <= bi) k++;
            const GroupSlice e = gs[k];
            const SliceDesc sd = d.slices[first + k];
            const PicDesc &pd = d.pics[sd.pic];
            const FrameDesc &fd = d.frames[pd.frame];
            uint32_t local = bi - e.blk, c = 0, nb = e.nb_y, off = 0;
            if (local >= e.nb_y) {
                local -= e.nb_y;
                c = local < e.nb_c ? 1u : 2u;
                local -= (c - 1u) * e.nb_c;
                nb = e.nb_c;
                off = 64u * (e.nb_y + (c - 1u) * e.nb_c);
            }
            const uint32_t per_mb = c == 0 ? 4u : (fd.chroma == 2 ? 2u : 4u);
            const uint32_t m = local / per_mb, bb = local - m * per_mb;
            uint32_t bx, by;
            block_xy(c, fd.chroma, sd.mb_x, sd.mb_y, m, bb, bx, by);
            const uint32_t pw = fd.plane_w[c];
            if (bx >= pw || by >= pd.height) continue;  // wholly outside the picture
            uint16_t *plane =
                fd.out_planes ? fd.out_planes + (fd.plane_off[c] - fd.plane_off[0]) : d.planes + fd.plane_off[c];
            uint16_t *row0 = plane + (uint64_t)(pd.first_row + pd.row_step * by) * pw + bx;
            const uint64_t pitch = (uint64_t)pd.row_step * pw;
            const float *sc = scale + (2u * k + (c > 0 ? 1u : 0u)) * 64u;
            const T *cs = slots + e.pos + off;
            const int32_t *wide = wide_all + sd.coef + off;
            const uint32_t cols = min(8u, pw - bx), rows = min(8u, pd.height - by);
            if (pd.interlaced_scan)
                idct_block<1>(cs, wide, nb, local, sc, fd.out_scale, fd.out_bias, fd.out_max, row0, pitch, cols, rows);
            else
                idct_block<0>(cs, wide, nb, local, sc, fd.out_scale, fd.out_bias, fd.out_max, row0, pitch, cols, rows);
        }
    }
}

constexpr int kStatusThreads = 256;

__global__ void __launch_bounds__(kStatusThreads) k_status(DecodeLaunch d) {
    chain_start();
    chain_wait();
    __shared__ int best;
    const PicDesc p = d.pics[blockIdx.x];
    if (threadIdx.x == 0) best = INT32_MAX;
    __syncthreads();
    if (d.pic_status[blockIdx.x].locate_slice < 0) {
        const uint64_t first = 4ull * p.slice_base, n = 4ull * p.n_slices;
        for (uint64_t i = threadIdx.x; i < n; i += kStatusThreads) {
            if (d.slot_status[first + i].x != DE_OK) {
                atomicMin(&best, (int)i);
                break;  // later slots of this thread are further on
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && best != INT32_MAX) {
        const int2 st = d.slot_status[4ull * p.slice_base + best];
        d.pic_status[blockIdx.x].slot = best;
        d.pic_status[blockIdx.x].code = st.x;
        d.pic_status[blockIdx.x].aux = st.y;
    }
}

}  // namespace

cudaError_t upload_scans() {
    uint8_t s[2][64];
    for (int i = 0; i < 64; i++) {
        s[0][i] = kProgressiveScan[i];
        s[1][i] = kInterlacedScan[i];
    }
    return cudaMemcpyToSymbol(d_scan, s, sizeof s);
}

cudaError_t launch_locate(const DecodeLaunch &d, cudaStream_t s) {
    if (d.n_pics == 0) return cudaSuccess;
    return launch_chained(k_locate, d.n_pics, kLocateThreads, 0, s, d);
}

// The prefix tables, and 8 words a lane for the rings: 56 KB for 8 warps, of
// which an SM would hold four (its registers hold two).
static size_t entropy_smem_bytes(int warps_per_block) { return 2 * 2 * kBookTableWords + 1024u * warps_per_block; }

cudaError_t launch_entropy(const DecodeLaunch &d, const EntropyShape &shape, cudaStream_t s) {
    if (d.n_slices == 0) return cudaSuccess;
    return launch_chained(k_entropy, shape.grid, 32 * shape.warps_per_block, entropy_smem_bytes(shape.warps_per_block),
                          s, d);
}

static size_t idct_smem_bytes() { return kIdctWarps * sizeof(IdctWarp); }

cudaError_t launch_idct(const DecodeLaunch &d, cudaStream_t s) {
    if (d.n_idct_items == 0) return cudaSuccess;
    return launch_chained(k_idct, (d.n_idct_items + kIdctWarps - 1) / kIdctWarps, 32 * kIdctWarps, idct_smem_bytes(),
                          s, d);
}

cudaError_t launch_status(const DecodeLaunch &d, cudaStream_t s) {
    if (d.n_pics == 0) return cudaSuccess;
    return launch_chained(k_status, d.n_pics, kStatusThreads, 0, s, d);
}

size_t decode_smem_bytes(uint32_t group, uint32_t group_positions, uint32_t slot_bytes) {
    return 2 * 2 * kBookTableWords + sizeof(GroupSlice) * kMaxGroup + 512u * group + slot_bytes * group_positions;
}

// The most shared memory a CTA of k_decode may take (a group of 8-macroblock
// 4:4:4 slices fills about a hundred kilobytes).
constexpr size_t kDecodeSmemMax = 200u << 10;

int decode_grid(int device, uint32_t group, uint32_t group_positions, uint32_t slot_bytes) {
    int sms = 0, fit = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const size_t smem = decode_smem_bytes(group, group_positions, slot_bytes);
    if (slot_bytes == 1)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_decode<int8_t>, kDecodeThreads, smem);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_decode<int16_t>, kDecodeThreads, smem);
    return sms * (fit > 0 ? fit : 1);
}

cudaError_t launch_decode(const DecodeLaunch &d, int grid, cudaStream_t s) {
    if (d.n_slices == 0) return cudaSuccess;
    const size_t smem = decode_smem_bytes(d.group, d.group_positions, d.slot_bytes);
    if (d.group < 1 || d.group > kMaxGroup || d.group_positions % 16u != 0 || smem > kDecodeSmemMax ||
        (d.slot_bytes != 1 && d.slot_bytes != 2))
        return cudaErrorInvalidValue;
    const uint32_t groups = (d.n_slices + d.group - 1u) / d.group;
    const int g = grid > 0 && (uint32_t)grid < groups ? grid : (int)groups;
    return d.slot_bytes == 1 ? launch_chained(k_decode<int8_t>, g, kDecodeThreads, smem, s, d)
                             : launch_chained(k_decode<int16_t>, g, kDecodeThreads, smem, s, d);
}

cudaError_t configure_decode_kernels() {
    cudaError_t e = cudaFuncSetAttribute(k_idct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)idct_smem_bytes());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_entropy, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)entropy_smem_bytes(kEntropyMaxThreads / 32));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_decode<int16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDecodeSmemMax);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_decode<int8_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDecodeSmemMax);
    if (e != cudaSuccess) return e;
    float basis[64];
    dct_basis(basis);
    if ((e = cudaMemcpyToSymbol(c_idct_basis, basis, sizeof basis)) != cudaSuccess) return e;
    return upload_scans();
}

int entropy_grid(int device, int warps_per_block, int blocks_per_sm) {
    int sms = 0, fit = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_entropy, 32 * warps_per_block,
                                                  entropy_smem_bytes(warps_per_block));
    if (fit < 1) fit = 1;
    const int per_sm = blocks_per_sm > 0 && blocks_per_sm < fit ? blocks_per_sm : fit;
    return sms * per_sm;
}

}  // namespace prores
