// encode.cu -- the encoder (the crate's src/encode.rs) as sm_100a kernels.
//
//   k_fdct        one warp per 32 blocks: edge-replicated 8x8 gathers, p = s
//                 512/2^b - 256 and the FDCT in the crate's exact
//                 single-precision order (src/encode.rs:488-555,
//                 src/dct.rs:70-93), written in the slice's scanned order once
//                 per frame.
//   k_alpha_size  one warp per slice: the lossless alpha codes' size
//                 (src/encode.rs:838-868, :457-470); it does not depend on
//                 the quantiser.
//   k_rc_init / k_cost / k_rc_step
//                 the rate control's probe sequence replayed exactly: 224,
//                 then mid = lo + (hi - lo) / 2 while lo < hi
//                 (src/encode.rs:685-713). k_cost sizes every slice of every
//                 picture still searching at that picture's probe, one warp
//                 per slice component (quantise + exact bit count,
//                 src/dsp/scalar.rs:19-39, src/encode.rs:398-409); k_rc_step
//                 sums a picture's slices and moves its interval.
//   k_cost_window the next kWindow finer quantisers below the uniform one.
//   k_deep_select / k_cost_deep
//                 the quantisers below those, for the slices likely to need
//                 them.
//   k_share_prep / k_shareout / k_share_final
//                 the sequential share-out of the slack
//                 (src/encode.rs:769-793), a warp per picture; its block's
//                 other warps cost any deeper quantiser it needs.
//   k_layout / k_frame
//                 slice offsets (an exclusive scan per picture), picture and
//                 frame sizes, the frame and picture headers.
//   k_pack        one warp per slice component: its codes bit-packed into
//                 shared memory and from there into the frame
//                 (src/encode.rs:413-437, :797-829); k_pack_headers the slice
//                 headers and table entries, k_pack_alpha the alpha codes.
//
// Output bits are OR-ed into a zeroed buffer as big-endian 32-bit words, so
// writers that share a word never need to be ordered.

#include <cuda_runtime.h>

#include <cstdint>

#include "chain.h"
#include "codec_tables.h"
#include "encode_types.h"
#include "pair_math.h"

namespace prores {

__constant__ uint8_t c_enc_scan[2][64];
__constant__ float c_fdct_basis[64];  // T[x][u], the same values as the decoder's

namespace {

constexpr float kAcRounding = 0.42f;  // src/encode.rs:204

__device__ __forceinline__ uint32_t bswap32(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

// ORs `value` into the bit field [bitpos, bitpos + len) (MSB first; the
// value's leading zeros are the field's) of a big-endian bit buffer.
__device__ __forceinline__ void put_field(uint32_t *out, uint64_t bitpos, uint64_t value, uint32_t len) {
    const uint32_t nb = bit_len64(value);
    if (nb == 0) return;
    const uint64_t start = bitpos + len - nb;
    uint32_t *w = out + (start >> 5);
    const uint32_t o = (uint32_t)(start & 31);
    const uint32_t first = 32 - o;
    if (nb <= first) {
        atomicOr(w, bswap32((uint32_t)(value << (first - nb))));
        return;
    }
    const uint32_t rest = nb - first;
    atomicOr(w, bswap32((uint32_t)(value >> rest)));
    if (rest <= 32) {
        atomicOr(w + 1, bswap32((uint32_t)(value << (32 - rest))));
    } else {
        atomicOr(w + 1, bswap32((uint32_t)(value >> (rest - 32))));
        atomicOr(w + 2, bswap32((uint32_t)(value << (64 - rest))));
    }
}

// floor(|x| + r) as an integer: |x| + r is positive, so truncation is the
// floor (and both saturate alike from 2^31 up).
__device__ __forceinline__ int32_t magnitude(float x, float r) { return __float2int_rz(__fadd_rn(fabsf(x), r)); }

__device__ __forceinline__ int32_t quantise1(float f, float inv, float r) {
    // x = F inv; QF = sign(x) floor(|x| + r) (src/dsp/scalar.rs:19-39).
    const float x = __fmul_rn(f, inv);
    const int32_t q = magnitude(x, r);
    return x < 0.0f ? -q : q;
}

// ---------------------------------------------------------------- fdct

constexpr int kFdctWarps = 3;
constexpr int kMaxSliceCoefs = 64 * 12 * 8;

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

// An 8-point forward transform: o[j] is outputs 2 j and 2 j + 1, each the sum
// of in[x] T[x][u] with x in order, summed as a pair; the products stay
// scalar (see pair_math.h), and the first is not added to 0 (which changes
// only the sign of a zero, and no quantised value).
__device__ __forceinline__ void fdct8(const float (&in)[8], uint64_t (&o)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
        for (int x = 0; x < 8; x++) {
            const uint64_t term =
                pair_of(__fmul_rn(in[x], c_fdct_basis[8 * x + 2 * j]), __fmul_rn(in[x], c_fdct_basis[8 * x + 2 * j + 1]));
            o[j] = x == 0 ? term : pair_add(o[j], term);
        }
    }
}

// Up to 32 blocks a warp, a lane each (IdctShape: a component of 32 blocks,
// several of fewer, or several slices). A lane loads its block's 8 rows,
// transforms them (rows, then columns, in the crate's order) in its own column
// of shared memory, [position][lane], so nothing is exchanged and no bank is
// met twice. Then the warp writes the components out in scanned order, 16
// bytes a lane, with the largest |F| of every 32 coefficients (8 lanes).
// Bound by issue (74 % of the slots, 49 instructions a sample, of which the
// sums' terms are 23): 30 UHD 4:2:2 frames take 852 us, 1463 with a warp per
// component (half the lanes idle in 4:2:2 chroma, more in narrow slices) and a
// reduction for every position's maximum; a mixed batch 515 for 1796. Rows are
// loaded two ahead (12 % slower without). 27 warps fill an SM's shared memory,
// in blocks of 3, since a block's place is free only when its last warp is
// done (24 warps, in blocks of 4: 915 us; of 2: 878; of 1: 892).
struct FdctWarp {
    float t[64][32];
    uint8_t raster[64];  // of each scanned position
};

__global__ void __launch_bounds__(32 * kFdctWarps, 9) k_fdct(EncodeLaunch e) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    FdctWarp &w = reinterpret_cast<FdctWarp *>(smem)[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t index = blockIdx.x * kFdctWarps + (threadIdx.x >> 5);
    if (index >= e.n_fdct_items) return;  // the whole warp
    // The item's picture: the last whose items start at or before it, of 32
    // places at a time, so a round more for every 32 times the pictures. (From
    // end to end, 32 at a time, 131,072 frames of 16x16 took 31.9 ms, now 0.8.)
    uint32_t pic = 0, step = 1;
    while (32u * step < e.n_pics) step *= 32u;
    for (; step > 0; step >>= 5) {
        const uint32_t i = pic + step * lane;
        const uint32_t m = __ballot_sync(0xffffffffu, i < e.n_pics && e.pics[i].fdct_base <= index);
        pic += step * (31u - __clz(m));
    }
    const EncPicDesc &pd = e.pics[pic];
    const EncFrameDesc &fd = e.frames[pd.frame];
    const uint32_t cpm = fd.chroma == 2 ? 2u : 4u;
    const IdctShape shape = idct_shape(fd.chroma, pd.log2_slice_mbs);
    const uint32_t local = index - pd.fdct_base;
    const uint32_t first = shape.slices > 1u ? local * shape.slices : local / shape.parts;
    const uint32_t part = shape.slices > 1u ? 0u : local - first * shape.parts;
    const uint32_t n_slices = min(shape.slices, pd.n_slices - first);
    uint32_t c0, c1;
    idct_components(shape, cpm, part, c0, c1);
    w.raster[c_enc_scan[pd.interlaced_scan][lane]] = (uint8_t)lane;
    w.raster[c_enc_scan[pd.interlaced_scan][lane + 32u]] = (uint8_t)(lane + 32u);

    // This lane's block.
    const uint32_t j = lane / shape.blocks;
    if (j < n_slices) {
        const EncSliceDesc sd = e.slices[pd.slice_base + first + j];
        const uint32_t nb_y = c0 == 0 ? 4u * sd.mbs : 0u, nb_c = cpm * sd.mbs;
        uint32_t b = lane - j * shape.blocks, c = 0;
        if (b >= nb_y) {
            b -= nb_y;
            c = max(c0, 1u);
            if (b >= nb_c) {
                b -= nb_c;
                c++;
            }
            if (b >= nb_c) c = 3u;  // past the item's blocks
        }
        if (c < c1) {
            const uint32_t per_shift = c == 0 || cpm == 4u ? 2u : 1u;
            uint32_t bx, by;
            block_xy(c, fd.chroma, sd.mb_x, sd.mb_y, b >> per_shift, b & ((1u << per_shift) - 1u), bx, by);
            const uint32_t pw = fd.plane_w[c];
            const uint16_t *plane = e.in + fd.in_off[c] + (uint64_t)pd.first_row * pw;
            const float scale = fd.in_scale;
            const bool wide = bx + 8u <= pw;
            // Row y's eight samples; the last picture row and column repeat.
            const auto load = [&](uint32_t y) {
                const uint16_t *line = plane + (uint64_t)(pd.row_step * min(by + y, pd.height - 1u)) * pw;
                if (wide && (reinterpret_cast<uintptr_t>(line + bx) & 15u) == 0)
                    return __ldg(reinterpret_cast<const uint4 *>(line + bx));
                uint32_t v[8];
#pragma unroll
                for (uint32_t x = 0; x < 8; x++) v[x] = __ldg(line + min(bx + x, pw - 1u));  // bx may be past the plane
                return make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
            };
            uint4 row = load(0), next = load(1);
            // p = s 512 / 2^b - 256: the product is exact, so one rounding
            // is the crate's two.
#pragma unroll 1
            for (uint32_t y = 0; y < 8; y++) {
                const uint4 after = load(min(y + 2u, 7u));  // two rows ahead
                const uint32_t words[4] = {row.x, row.y, row.z, row.w};
                float p[8];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    p[2 * i] = __fmaf_rn((float)(words[i] & 0xFFFFu), scale, -256.0f);
                    p[2 * i + 1] = __fmaf_rn((float)(words[i] >> 16), scale, -256.0f);
                }
                row = next;
                next = after;
                uint64_t o[4];
                fdct8(p, o);
#pragma unroll
                for (int k = 0; k < 4; k++) pair_split(o[k], w.t[8 * y + 2 * k][lane], w.t[8 * y + 2 * k + 1][lane]);
            }
            // Columns: F[v][u] = sum_y T[y][v] tmp[y][u], y in order from 0.
#pragma unroll 1
            for (uint32_t u = 0; u < 8; u++) {
                float col[8];
#pragma unroll
                for (int y = 0; y < 8; y++) col[y] = w.t[8 * y + u][lane];
                uint64_t o[4];
                fdct8(col, o);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    pair_split(o[k], w.t[16 * k + u][lane], w.t[16 * k + 8 + u][lane]);
            }
        }
    }
    __syncwarp();

    // The components, one after another.
    for (uint32_t k = 0; k < n_slices; k++) {
        const EncSliceDesc sd = e.slices[pd.slice_base + first + k];
        uint32_t at = k * shape.blocks;
        for (uint32_t c = c0; c < c1; c++) {
            const uint32_t nb = (c == 0 ? 4u : cpm) * sd.mbs;
            const uint64_t coef = sd.coef + (c == 0 ? 0u : 64u * sd.mbs * (4u + (c - 1u) * cpm));
            float *out = e.coef + coef, *cmax = e.coef_max + (coef >> 5);
            if (nb >= 4u) {
                const uint32_t shift = 29u - __clz(nb);  // four blocks of a position a lane
#pragma unroll 4
                for (uint32_t i = lane; i < 16u * nb; i += 32u) {
                    const uint32_t r = w.raster[i >> shift], b = 4u * (i & ((1u << shift) - 1u));
                    const float4 v = *reinterpret_cast<const float4 *>(&w.t[r][at + b]);
                    reinterpret_cast<float4 *>(out)[i] = v;
                    float m = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
                    if ((lane & 7u) == 0) cmax[i >> 3] = m;
                }
            } else {
#pragma unroll
                for (uint32_t i = lane; i < 64u; i += 32u) {  // both blocks of a position
                    const float2 v = *reinterpret_cast<const float2 *>(&w.t[w.raster[i]][at]);
                    reinterpret_cast<float2 *>(out)[i] = v;
                    float m = fmaxf(fabsf(v.x), fabsf(v.y));
#pragma unroll
                    for (int o = 1; o < 16; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                    if ((lane & 15u) == 0) cmax[i >> 4] = m;
                }
            }
            at += nb;
        }
    }
}

// ---------------------------------------------------------------- alpha

constexpr int kAlphaWarps = 4;
constexpr int kMaxAlphaValues = 16 * 16 * 8;

struct AlphaScratch {
    uint16_t start[kMaxAlphaValues + 1];
    uint16_t value[kMaxAlphaValues];
};

__device__ __forceinline__ uint32_t alpha_diff_len(int32_t diff, uint32_t bits) {
    const uint32_t a = diff < 0 ? 0u - (uint32_t)diff : (uint32_t)diff;
    const uint32_t mag = bits == 8 ? 3u : 6u, max = bits == 8 ? 8u : 64u;
    return (a >= 1u && a <= max) ? 2u + mag : 1u + bits;
}
__device__ __forceinline__ uint32_t alpha_run_len(uint32_t run) { return run == 1u ? 1u : (run <= 16u ? 5u : 16u); }

// The slice's alpha values (16 rows of 16 mbs, edges repeated, converted to
// the coded bits) into runs; returns the run count. A run cannot pass 2048
// values: a slice has at most 2048.
__device__ uint32_t alpha_runs(const EncodeLaunch &e, const EncSliceDesc &sd, const EncPicDesc &pd,
                               const EncFrameDesc &fd, AlphaScratch &sc) {
    const int lane = threadIdx.x & 31;
    const uint32_t cols = 16u * sd.mbs, count = 16u * cols;
    const uint32_t width = fd.width, x0 = 16u * sd.mb_x;
    const uint16_t max_in = (uint16_t)(0xFFFFu >> (16u - fd.bit_depth));
    const uint16_t *plane = e.alpha_in + fd.alpha_in_off;
    const uint32_t cshift = (uint32_t)__ffs(cols) - 1u;  // cols is 16 times a power of two
    uint32_t n_runs = 0;
    uint32_t prev = 0;
    // 256 values (count is a multiple) a round: their eight loads are all
    // issued before the first is used.
    for (uint32_t base = 0; base < count; base += 256) {
        uint32_t vals[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t i = base + 32u * k + lane;
            const uint32_t r = i >> cshift, n = i & (cols - 1u);
            const uint32_t row = pd.first_row + pd.row_step * min(16u * sd.mb_y + r, pd.height - 1u);
            vals[k] = __ldg(plane + (uint64_t)row * width + min(x0 + n, width - 1u));
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t i = base + 32u * k + lane;
            uint32_t a = vals[k] < max_in ? vals[k] : max_in;
            const uint32_t v = fd.rescale_identity ? a : (uint32_t)(((uint64_t)a * fd.rescale_m + (1ull << 39)) >> 40);
            const uint32_t before = __shfl_up_sync(0xffffffffu, v, 1);
            const uint32_t left = lane == 0 ? prev : before;
            const bool is_start = i == 0 || v != left;
            const uint32_t mask = __ballot_sync(0xffffffffu, is_start);
            if (is_start) {
                const uint32_t idx = n_runs + __popc(mask & ((1u << lane) - 1u));
                sc.start[idx] = (uint16_t)i;
                sc.value[idx] = (uint16_t)v;
            }
            n_runs += __popc(mask);
            prev = __shfl_sync(0xffffffffu, v, 31);
        }
    }
    if (lane == 0) sc.start[n_runs] = (uint16_t)count;
    __syncwarp();
    return n_runs;
}

__device__ __forceinline__ uint32_t alpha_run_bits(const AlphaScratch &sc, uint32_t j, uint32_t bits, uint32_t &dlen) {
    const int32_t prev = j ? (int32_t)sc.value[j - 1] : -1;
    dlen = alpha_diff_len((int32_t)sc.value[j] - prev, bits);
    return dlen + alpha_run_len((uint32_t)sc.start[j + 1] - sc.start[j]);
}

__global__ void __launch_bounds__(32 * kAlphaWarps) k_alpha_size(EncodeLaunch e) {
    chain_wait();
    __shared__ AlphaScratch scratch[kAlphaWarps];
    const uint32_t s = blockIdx.x * kAlphaWarps + (threadIdx.x >> 5);
    if (s >= e.n_slices) return;
    const int lane = threadIdx.x & 31;
    const EncSliceDesc sd = e.slices[s];
    const EncPicDesc &pd = e.pics[sd.pic];
    const EncFrameDesc &fd = e.frames[pd.frame];
    if (fd.alpha_bits == 0) {
        if (lane == 0) e.alpha_bytes[s] = 0;
        return;
    }
    AlphaScratch &sc = scratch[threadIdx.x >> 5];
    const uint32_t n_runs = alpha_runs(e, sd, pd, fd, sc);
    uint32_t bits = 0;
    for (uint32_t j = lane; j < n_runs; j += 32) {
        uint32_t dlen;
        bits += alpha_run_bits(sc, j, fd.alpha_bits, dlen);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bits += __shfl_xor_sync(0xffffffffu, bits, o);
    if (lane == 0) e.alpha_bytes[s] = (bits + 7u) / 8u;
}

// ---------------------------------------------------------------- quantisers

// A lower bound on the |F| that quantise to a non-zero AC level at inverse
// weight inv. A level is non-zero when fl(fl(|F| inv) + 0.42f) >= 1, which
// needs the exact sum fl(|F| inv) + 0.42f to reach 1 - 2^-25 (the midpoint
// below 1), and so |F| inv >= (1 - 2^-25 - 0.42f)(1 - 2^-24). The bound takes
// a margin of 2^-22 and is rounded down, so every non-zero lies at or above
// it; the kernels re-quantise each candidate exactly.
__device__ __forceinline__ float nonzero_bound(float inv) {
    constexpr double y0 = 1.0 - 1.0 / (1 << 25) - (double)kAcRounding;
    return __double2float_rd(__ddiv_rn(y0 * (1.0 - 1.0 / (1 << 22)), (double)inv));
}

// A CTA per set and quantization_index, one after another in the grid's x
// (y and z end at 65535): inv[scan[k]] = 8 / (W[k] qScale), laid out as beside
// kQuantStride, in single precision for luma and chroma
// (src/encode.rs:303-329), the non-zero bound of each, and the least bound
// over each chunk of 32 scanned coefficients. On the host the 225 quantisers
// of a set took about half a millisecond of every call.
__global__ void __launch_bounds__(128) k_quant(float *quant, const uint8_t *keys) {
    __shared__ float bound[128];
    const uint32_t set = blockIdx.x / 225u, qi = blockIdx.x - 225u * set;
    const uint32_t i = threadIdx.x, k = i & 63u, g = i >> 6;
    const uint8_t *key = keys + kQuantKey * set;
    float *t = quant + (uint64_t)blockIdx.x * kQuantStride;
    const uint32_t at = 64u * g + c_enc_scan[key[128]][k];
    const float inv = __fdiv_rn(8.0f, (float)((uint32_t)key[i] * qscale(qi < 1u ? 1u : qi)));
    t[at] = inv;
    bound[at] = nonzero_bound(inv);
    t[128u + at] = bound[at];
    __syncthreads();
    // Chunk j of a component of n blocks is positions 32 j / n to 32 (j + 1) / n - 1.
    if (k < 60u) {
        const uint32_t shift = 31u - __clz((k + 4u) >> 1), n = 1u << shift, j = k - (2u * n - 4u);
        float m = bound[64u * g + 32u * j / n];
        for (uint32_t p = 32u * j / n + 1u; p < 32u * (j + 1u) / n; p++) m = fminf(m, bound[64u * g + p]);
        t[256u + 60u * g + k] = m;
    }
}

// ---------------------------------------------------------------- costing

// One component's view of a quantiser table (layout beside kQuantStride):
// inverse weights and non-zero bounds by scanned position, and the bound of
// each 32-coefficient chunk of a component of its block count.
struct CompQuant {
    const float *inv, *bound, *chunk;
};

__device__ __forceinline__ CompQuant comp_quant(const float *qb, uint32_t comp, uint32_t n_blocks) {
    const uint32_t g = comp > 0 ? 1u : 0u;
    CompQuant c;
    c.inv = qb + 64u * g;
    c.bound = qb + 128u + 64u * g;
    c.chunk = n_blocks >= 32u ? c.bound : qb + 256u + 60u * g + (2u * n_blocks - 4u);
    return c;
}

// Code lengths by context for the warps that count bits: of run symbols
// below 63, and of level symbols below 127 with the sign bit added. The last
// column stands for every symbol past those (kLongCode: no two lengths of
// the rest add up to it).
constexpr uint32_t kRunLens = 64, kLevelLens = 128, kLongCode = 128;
struct CountTables {
    // Both indices are context x kRow + symbol; a row is 33 words, so that
    // neighbouring contexts lie in different banks.
    static constexpr uint32_t kRow = 132;
    uint8_t run[16][kRow];
    uint8_t level[9][kRow];
    uint8_t pad[12];  // a whole number of 16-byte words
    // Copies the device's table (built once, by configure_encode_kernels).
    __device__ __forceinline__ void fill();
};
__device__ uint4 d_count_tables[sizeof(CountTables) / sizeof(uint4)];

__device__ __forceinline__ void CountTables::fill() {
    for (uint32_t i = threadIdx.x; i < sizeof(CountTables) / sizeof(uint4); i += blockDim.x)
        reinterpret_cast<uint4 *>(this)[i] = d_count_tables[i];
}

void build_count_tables(CountTables &t) {
    t = CountTables{};
    for (uint32_t c = 0; c < 16; c++)
        for (uint32_t n = 0; n < kRunLens; n++)
            t.run[c][n] = (uint8_t)(n + 1u < kRunLens ? cb_len32(run_book(c), n) : kLongCode);
    for (uint32_t c = 0; c < 9; c++)
        for (uint32_t n = 0; n < kLevelLens; n++)
            t.level[c][n] = (uint8_t)(n + 1u < kLevelLens ? cb_len32(level_book(c), n) + 1u : kLongCode);
}

// A warp's non-zeros on their way from the quantiser to the code tables, in
// scanned order: (position << 16) + level symbol, both below 2^15 (a
// component with larger levels, which only samples far above their depth's
// range can make, is counted by warp_wide_bits). The two entries before the
// first hold the state a component starts with (previous run 4, previous
// level 1), then the last two counted.
constexpr uint32_t kGroupRuns = 4;  // runs of 128 coefficients quantised before codes are counted
constexpr uint32_t kNonzeroBuf = 2 + 63 + 128 * kGroupRuns + 3;
constexpr uint32_t kWeightsAt = kNonzeroBuf, kIdsAt = kNonzeroBuf + 64;
// Words of shared memory a warp's count takes: its list, then the inverse
// weights and chunk numbers it works with.
constexpr uint32_t kCountWords = kIdsAt + 8;
// Components with more than this many live chunks of every 8 are read whole,
// the others by the list of their live chunks (30 UHD frames, the probe at
// quantiser index 56: 372 us at 3, 382 at 2, 415 at 5; 16 4:4:4 12-bit fields
// 76, 78 and 82).
constexpr uint32_t kLiveOf8 = 3;
static_assert(64u * kLiveOf8 / 8u <= 4u * (kCountWords - kIdsAt), "the list holds a 32-block component's live chunks");
// |F| from here on may make a level symbol of 2^15: 8 / (W qScale) is at most 4.
constexpr float kWideCoef = 8191.0f;

// The bits of a run and level (with its sign) past the tables: `n` its entry
// less the position before it, `k` the same of the non-zero before it.
__device__ __noinline__ uint32_t long_code_bits(uint32_t e0, uint32_t e1, uint32_t e2) {
    const uint32_t run = (e0 >> 16) - (e1 >> 16) - 1u;
    const uint32_t prev_run = ((e1 >> 16) - (e2 >> 16) - 1u) & 0xFFFFu;
    return cb_len32(run_book(prev_run), run) + cb_len32(level_book(e1 & 0xFFFFu), e0 & 0xFFFFu) + 1u;
}

// Sums the bits of two neighbouring non-zeros a lane, the entries c = (c.x,
// c.y) after the two before them, b; `n` of them are there (below 1: none).
// Each one's run is coded by the run before it, its level by the level before
// it, with a sign. All contexts are in the four entries. Run and level go
// through every step as the two halves of a word: an entry less the position
// before it and 1, clamped to the tables' last columns or to the contexts'
// last rows, is one instruction.
constexpr uint32_t kCodeCols = ((kRunLens - 1u) << 16) | (kLevelLens - 1u), kCodeRows = (15u << 16) | 8u;
struct CountSink {
    static constexpr bool kSign = false;
    const CountTables &t;
    uint32_t bits;
    __device__ __forceinline__ void pairs(uint2 b, uint2 c, int32_t n) {
        const uint32_t nbx = ~b.x & 0xFFFF0000u, nby = ~b.y & 0xFFFF0000u, ncx = ~c.x & 0xFFFF0000u;
        const uint32_t i0 = __viaddmin_s16x2(b.y, nbx, kCodeRows) * CountTables::kRow + __viaddmin_s16x2(c.x, nby, kCodeCols);
        const uint32_t i1 = __viaddmin_s16x2(c.x, nby, kCodeRows) * CountTables::kRow + __viaddmin_s16x2(c.y, ncx, kCodeCols);
        const uint8_t *run = &t.run[0][0], *level = &t.level[0][0];
        uint32_t l0 = (uint32_t)run[i0 >> 16] + level[i0 & 0xFFFFu];
        uint32_t l1 = (uint32_t)run[i1 >> 16] + level[i1 & 0xFFFFu];
        if ((l0 | l1) >= kLongCode) {
            if (l0 >= kLongCode) l0 = long_code_bits(c.x, b.y, b.x);
            if (l1 >= kLongCode && n > 1) l1 = long_code_bits(c.y, c.x, b.y);
        }
        bits += (n > 0 ? l0 : 0u) + (n > 1 ? l1 : 0u);
    }
};

// kShared: f and cmax point into shared memory; else into global memory, where
// a kernel of the chain wrote them.
template <bool kShared>
__device__ __forceinline__ float coef_load(const float *f, uint32_t i) {
    if constexpr (kShared)
        return f[i];
    else
        return chain_load(f + i);
}

// Length of the code of a DC difference's symbol n by a = min(|previous
// difference|, 3) (Table 9), and with a = 5 of the first DC's (EG5). EGk is
// 2 floor(log2(n + 2^k)) - k + 1 bits, and a is k but for a = 2, whose
// codebook (1, 2, 3) has (n >> 2) + 3 bits below 8 and from there on, as
// 2^3 is also where its Rice part ends, 2 floor(log2(n)).
__device__ __forceinline__ uint32_t dc_len(uint32_t a, uint32_t n) {
    const uint32_t add = a == 2u ? 0u : 1u << a, sub = a == 2u ? 2u : a + 1u;
    const uint32_t len = 2u * bit_len32(n + add) - sub;
    return a == 2u && n < 8u ? (n >> 2) + 3u : len;
}

// What a component's count starts from, loaded ahead: each lane's two chunk
// maxima and its DC.
struct CompHead {
    float max_lo, max_hi, dc;
};

template <bool kShared>
__device__ __forceinline__ CompHead comp_head(const float *f, const float *cmax, uint32_t n_blocks) {
    const uint32_t lane = threadIdx.x & 31u, chunks = 2u * n_blocks;
    CompHead h{0.0f, 0.0f, 0.0f};
    if (lane < chunks) h.max_lo = coef_load<kShared>(cmax, lane);
    if (lane + 32u < chunks) h.max_hi = coef_load<kShared>(cmax, lane + 32u);
    if (lane < n_blocks) h.dc = coef_load<kShared>(f, lane);
    return h;
}

// A warp's list of non-zeros: filled 32 or 512 coefficients at a time, handed
// to `sink` 64 non-zeros at a time, two neighbouring ones a lane (see
// CountSink and PackSink: both get them with the whole warp together). With
// kSign an entry's bit 15 is the coefficient's sign.
template <class Sink>
struct NonzeroList {
    static constexpr bool kSign = Sink::kSign;
    Sink &sink;
    uint32_t *buf;
    uint32_t first, end;  // shared addresses of buf + 2 and past the last entry
    __device__ __forceinline__ NonzeroList(Sink &s, uint32_t *b, uint32_t n_blocks) : sink(s) {
        buf = b;
        first = end = (uint32_t)__cvta_generic_to_shared(b + 2);
        if ((threadIdx.x & 31u) == 0) {
            b[0] = (n_blocks - 6u) << 16;
            b[1] = ((n_blocks - 1u) << 16) | 1u;
        }
    }
    // A lane's coefficient of a chunk; tag = (position << 16) - 0x4B000001.
    // The store is a predicated instruction: as a branch it took about as
    // many instructions again as all the rest.
    __device__ __forceinline__ void add(float v, float inv, uint32_t tag, uint32_t below) {
        // y = |F inv| + 0.42 (src/dsp/scalar.rs:19-39); adding 2^23 rounded
        // down leaves floor(y) in the low bits.
        const float y = __fadd_rn(fabsf(__fmul_rn(v, inv)), kAcRounding);
        const uint32_t b = __ballot_sync(0xffffffffu, y >= 1.0f);
        const uint32_t at = end + 4u * __popc(b & below);
        uint32_t entry = __float_as_uint(__fadd_rd(y, 8388608.0f)) + tag;
        if (kSign) entry += (__float_as_uint(v) >> 16) & 0x8000u;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %2, 0f3F800000;\n\t@p st.shared.u32 [%0], %1;\n\t}"
                     :
                     : "r"(at), "r"(entry), "f"(y)
                     : "memory");
        end += 4u * __popc(b);
    }
    // Four coefficients a lane of each of kRuns runs of 128 positions: y the
    // quantised magnitudes before their floor (with kSign, signed), `counts` the lane's non-zeros
    // by run (a byte each), `tag` of the lane's first position.
    template <uint32_t kRuns>
    __device__ __forceinline__ void add_runs(const float (&y)[4 * kRuns], uint32_t counts, uint32_t tag) {
        // Sums over the lanes up to this one; at most 128 a byte.
        uint32_t sums = counts;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
            asm volatile("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\tshfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n\t"
                         "@p add.u32 %0, %0, t;\n\t}"
                         : "+r"(sums)
                         : "r"(o));
        const uint32_t totals = __shfl_sync(0xffffffffu, sums, 31);
        const uint32_t before = sums - counts;
#pragma unroll
        for (uint32_t r = 0; r < kRuns; r++) {
            uint32_t at = end + 4u * ((before >> (8 * r)) & 255u);
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                // Adding 2^23 rounded down leaves floor(y) in the low bits.
                const float m = fabsf(y[4 * r + k]);
                uint32_t entry = __float_as_uint(__fadd_rd(m, 8388608.0f)) + tag + ((128u * r + k) << 16);
                if (kSign) entry += (__float_as_uint(y[4 * r + k]) >> 16) & 0x8000u;
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %2, 0f3F800000;\n\t@p st.shared.u32 [%0], %1;\n\t"
                             "@p add.u32 %0, %0, 4;\n\t}"
                             : "+r"(at)
                             : "r"(entry), "f"(m)
                             : "memory");
            }
            end += 4u * ((totals >> (8 * r)) & 255u);
        }
    }
    // Hands the whole groups of 64 over; what is left, and the two entries
    // before it, go to the front.
    __device__ __forceinline__ void drain() {
        const uint32_t lane = threadIdx.x & 31u;
        __syncwarp();
        const uint32_t full = ((end - first) >> 2) & ~63u;
        if (full) {
            const uint2 *q = reinterpret_cast<const uint2 *>(buf) + lane;
#pragma unroll 1
            for (const uint2 *stop = q + full / 2u; q < stop; q += 32) sink.pairs(q[0], q[1], 2);
            const uint2 keep = q[0];
            const uint32_t last = buf[full + 64u];
            __syncwarp();
            reinterpret_cast<uint2 *>(buf)[lane] = keep;
            if (lane == 0) buf[64] = last;
            __syncwarp();
            end -= 4u * full;
        }
    }
    __device__ __forceinline__ void finish() {
        const uint32_t lane = threadIdx.x & 31u;
        const uint2 *q = reinterpret_cast<const uint2 *>(buf) + lane;
        const int32_t n = (int32_t)((end - first) >> 2) - (int32_t)(2u * lane);
        // Where there is no entry, any valid one, not used.
        uint2 b = q[0], c = q[1];
        if (n < 1) b = make_uint2(0u, 5u << 16), c.x = 6u << 16;
        if (n < 2) c.y = (c.x & 0xFFFF0000u) + (1u << 16);
        if (end != first) sink.pairs(b, c, n);
    }
};

template <bool kShared>
__device__ __forceinline__ float4 coef_load4(const float *f) {
    if constexpr (kShared)
        return *reinterpret_cast<const float4 *>(f);
    else
        return chain_load4(f);
}

// The AC non-zeros of a component of 2^kLog blocks, every coefficient in turn. A lane takes four neighbouring positions of each run
// of 128, four runs at a time; how many non-zeros the lanes below hold in
// each run comes from one scan of four byte counts.
template <int kLog, bool kShared, class Sink>
__device__ __forceinline__ void warp_dense(const float *f, const float *inv, Sink &sink, uint32_t *buf) {
    constexpr uint32_t kBlocks = 1u << kLog, kRuns = kBlocks / 2u;
    constexpr uint32_t kGroup = kRuns < kGroupRuns ? kRuns : kGroupRuns;
    constexpr bool kSplit = kBlocks == 2u;  // a lane's four positions are of two scan positions
    const uint32_t lane = threadIdx.x & 31u;
    // The 64 inverse weights, where every run finds its own at a constant
    // distance: run r's positions of this lane start at 128 r + 4 lane, their
    // weight's place is (128 r >> kLog) + (4 lane >> kLog).
    float *w = reinterpret_cast<float *>(buf + kWeightsAt);
    w[lane] = __ldg(inv + lane);
    w[lane + 32u] = __ldg(inv + lane + 32u);
    __syncwarp();
    w += (4u * lane) >> kLog;
    NonzeroList<Sink> list(sink, buf, kBlocks);
    f += 4u * lane;
#pragma unroll 1
    for (uint32_t g = 0; g < kRuns; g += kGroup) {
        float y[4 * kGroup];
#pragma unroll
        for (uint32_t r = 0; r < kGroup; r++) {
            const float4 v = coef_load4<kShared>(f + 128u * r);
            y[4 * r] = v.x;
            y[4 * r + 1] = v.y;
            y[4 * r + 2] = v.z;
            y[4 * r + 3] = v.w;
        }
        if (g == 0 && 4u * lane < kBlocks) {  // the DCs
            y[0] = y[1] = 0.0f;
            if (!kSplit) y[2] = y[3] = 0.0f;
        }
        uint32_t counts = 0;
#pragma unroll
        for (uint32_t r = 0; r < kGroup; r++) {
            const float wa = w[(128u * r) >> kLog], wb = kSplit ? w[((128u * r) >> kLog) + 1u] : wa;
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                // |F inv| + 0.42 (src/dsp/scalar.rs:19-39), a non-zero from 1 up.
                const float m = __fadd_rn(fabsf(__fmul_rn(y[4 * r + k], k < 2 ? wa : wb)), kAcRounding);
                y[4 * r + k] = Sink::kSign ? copysignf(m, y[4 * r + k]) : m;
                if (m >= 1.0f) counts += 1u << (8 * r);
            }
        }
        list.template add_runs<kGroup>(y, counts, ((128u * g + 4u * lane) << 16) - 0x4B000001u);
        list.drain();
        f += 128u * kGroup;
        w += (128u * kGroup) >> kLog;
    }
    list.finish();
}

// The same for a component with few chunks that may hold a non-zero, whose
// numbers are the first `n` bytes of `ids`: 8 of them in flight at a time.
template <bool kShared, class Sink>
__device__ __forceinline__ void warp_sparse(const float *f, const float *inv, uint32_t n_blocks, const uint2 *ids,
                                            uint32_t n, Sink &sink, uint32_t *buf) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t shift = 31u - __clz(n_blocks);
    NonzeroList<Sink> list(sink, buf, n_blocks);
#pragma unroll 1
    for (uint32_t k = 0; k < n; k += 8) {
        const uint2 id = ids[k >> 3];
        float v[8], iv[8];
        uint32_t p[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            p[i] = 32u * (((i < 4 ? id.x : id.y) >> (8 * (i & 3))) & 255u) + lane;
            v[i] = iv[i] = 0.0f;
            if (k + i < n) {
                v[i] = coef_load<kShared>(f, p[i]);
                iv[i] = __ldg(inv + (p[i] >> shift));
            }
        }
        if (p[0] < n_blocks) v[0] = 0.0f;  // the DCs
#pragma unroll
        for (uint32_t i = 0; i < 8; i++)
            if (k + i < n) list.add(v[i], iv[i], (p[i] << 16) - 0x4B000001u, below);
        list.drain();
    }
    list.finish();
}

// Every AC non-zero of a component to `sink`: all chunks in turn, or where
// few are live (the bits of live_hi:live_lo) those by their list.
template <bool kShared, class Sink>
__device__ __forceinline__ void warp_nonzeros(const float *f, const float *inv, uint32_t n_blocks, uint32_t live_lo,
                                              uint32_t live_hi, Sink &sink, uint32_t *buf) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t n_live = __popc(live_lo) + __popc(live_hi);
    if (kLiveOf8 * 2u * n_blocks < 8u * n_live) {
        switch (n_blocks) {
        case 32: warp_dense<5, kShared>(f, inv, sink, buf); break;
        case 16: warp_dense<4, kShared>(f, inv, sink, buf); break;
        case 8: warp_dense<3, kShared>(f, inv, sink, buf); break;
        case 4: warp_dense<2, kShared>(f, inv, sink, buf); break;
        default: warp_dense<1, kShared>(f, inv, sink, buf); break;
        }
    } else if (n_live) {
        // The live chunks' numbers, in order (at most 24).
        uint8_t *ids = reinterpret_cast<uint8_t *>(buf + kIdsAt);
        if ((live_lo >> lane) & 1u) ids[__popc(live_lo & below)] = (uint8_t)lane;
        if ((live_hi >> lane) & 1u) ids[__popc(live_lo) + __popc(live_hi & below)] = (uint8_t)(lane + 32u);
        __syncwarp();
        warp_sparse<kShared>(f, inv, n_blocks, reinterpret_cast<const uint2 *>(ids), n_live, sink, buf);
    }
}

// The chunks of a component that may hold a non-zero at `cq`'s quantiser.
__device__ __forceinline__ void live_chunks(const CompHead &h, uint32_t n_blocks, const CompQuant &cq, uint32_t &lo,
                                            uint32_t &hi) {
    const uint32_t lane = threadIdx.x & 31u;
    lo = __ballot_sync(0xffffffffu, lane < 2u * n_blocks && h.max_lo >= __ldg(cq.chunk + lane));
    hi = 0;
    if (n_blocks == 32u) hi = __ballot_sync(0xffffffffu, h.max_hi >= __ldg(cq.chunk + lane + 32u));
}

// A lane's DC (lanes below n_blocks) as its code's symbol and its codebook by
// `a` (see dc_len): EG5 of the first, then Table 9 by |previous difference|,
// the sign flipped after a negative one.
__device__ __forceinline__ uint32_t dc_symbol(float dc, float inv0, uint32_t &a) {
    const uint32_t lane = threadIdx.x & 31u;
    const int32_t q = quantise1(dc, inv0, 0.5f);
    const int32_t left = __shfl_up_sync(0xffffffffu, q, 1);
    const int32_t diff = (int32_t)((uint32_t)q - (uint32_t)left);
    const int32_t before = __shfl_up_sync(0xffffffffu, diff, 1);
    const int32_t prev_diff = lane == 0 ? 5 : (lane == 1 ? 3 : before);
    const int32_t value = lane == 0 ? q : (prev_diff < 0 ? -diff : diff);
    a = min((uint32_t)abs(prev_diff), lane == 0 ? 5u : 3u);
    // 0, -1, 1, -2, 2, ... -> 0, 1, 2, 3, 4, ...
    return ((uint32_t)value << 1) ^ (uint32_t)(value >> 31);
}

// The AC codes of a component with levels of any size (its largest |F| reaches
// kWideCoef), the whole warp, 32 positions at a time: a lane with a non-zero
// finds the one before it in the lanes' vote, and that one's run and level,
// its contexts, by shuffles (one lane walking alone held its whole warp: 4
// 1080p frames of samples past their depth's range took 1430 us, now 274).
// emit(coded, run, level, negative, previous run,
// previous level), every lane each time.
template <bool kShared, class Emit>
__device__ __forceinline__ void warp_wide_codes(const float *f, const float *inv, uint32_t n_blocks, Emit emit) {
    const uint32_t lane = threadIdx.x & 31u, shift = 31u - __clz(n_blocks);
    uint32_t last_run = 4, last_level = 1, next = n_blocks;  // of the last code, and the position after it
    for (uint32_t p0 = n_blocks; p0 < 64u * n_blocks; p0 += 32u) {
        const uint32_t p = p0 + lane;
        float x = 0.0f;
        if (p < 64u * n_blocks) x = __fmul_rn(coef_load<kShared>(f, p), __ldg(inv + (p >> shift)));
        const int32_t m = magnitude(x, kAcRounding);
        const uint32_t coded = __ballot_sync(0xffffffffu, m >= 1);
        if (!coded) continue;
        const uint32_t before = coded & ((1u << lane) - 1u), from = 31u - __clz(before);
        const uint32_t run = p - (before ? p0 + from + 1u : next), level = (uint32_t)m - 1u;
        const uint32_t run_before = __shfl_sync(0xffffffffu, run, from), level_before = __shfl_sync(0xffffffffu, level, from);
        emit(m >= 1, run, level, x < 0.0f, before ? run_before : last_run, before ? level_before : last_level);
        const uint32_t top = 31u - __clz(coded);
        last_run = __shfl_sync(0xffffffffu, run, top);
        last_level = __shfl_sync(0xffffffffu, level, top);
        next = p0 + top + 1u;
    }
}

template <bool kShared>
__device__ __noinline__ uint32_t warp_wide_bits(const float *f, const float *inv, uint32_t n_blocks) {
    uint32_t bits = 0;
    warp_wide_codes<kShared>(f, inv, n_blocks, [&](bool coded, uint32_t run, uint32_t level, bool, uint32_t prev_run,
                                                   uint32_t prev_level) {
        if (coded) bits += cb_len32(run_book(prev_run), run) + cb_len32(level_book(prev_level), level) + 1u;
    });
    return bits;
}

// Bits of one quantised component (src/encode.rs:398-409), the whole warp.
// Two stages, 512 coefficients at a time: the warp quantises them (16 a lane,
// their loads all in flight at once) and appends the non-zeros to a list in
// order; then each lane takes two neighbouring non-zeros of a full 64 and
// looks their code lengths up. So zeros cost no per-code work, and no code
// waits for the one before it. Where most chunks quantise to zero only the
// others are read. Every lane gets the sum.
//
// Bound by issue (79 % of the slots; 29 thread instructions a coefficient at
// 36 % non-zeros, DRAM at 4.8 TB/s): 30 UHD 4:2:2 frames take 430 us a probe
// near the answer, where a lane per component walking its codes in order, each
// look-up waiting for the last, took 800; 30 1080p frames 123 us for 700.
template <bool kShared = false>
__device__ __forceinline__ uint32_t warp_component_bits(const float *f, const CompHead &h, uint32_t n_blocks, const CompQuant &cq,
                                        const CountTables &t, uint32_t *buf) {
    uint32_t live_lo, live_hi, a;
    live_chunks(h, n_blocks, cq, live_lo, live_hi);
    const uint32_t symbol = dc_symbol(h.dc, __ldg(cq.inv), a), len = dc_len(a, symbol);
    CountSink sink{t, (threadIdx.x & 31u) < n_blocks ? len : 0u};
    __syncwarp();  // the last component's entries are read
    if (__any_sync(0xffffffffu, fmaxf(h.max_lo, h.max_hi) >= kWideCoef))
        sink.bits += warp_wide_bits<kShared>(f, cq.inv, n_blocks);
    else
        warp_nonzeros<kShared>(f, cq.inv, n_blocks, live_lo, live_hi, sink, buf);
    return __reduce_add_sync(0xffffffffu, sink.bits);
}

// The quantiser table of quantization_index qi (layout beside kQuantStride).
__device__ __forceinline__ const float *quant_base(const EncodeLaunch &e, const EncPicDesc &pd, uint32_t qi) {
    return e.quant + ((uint64_t)pd.quant * 225u + qi) * kQuantStride;
}

__device__ __forceinline__ void comp_layout(const EncFrameDesc &fd, uint32_t mbs, uint32_t comp, uint32_t &n_blocks,
                                            uint32_t &offset) {
    const uint32_t cpm = fd.chroma == 2 ? 2u : 4u;
    n_blocks = (comp == 0 ? 4u : cpm) * mbs;
    offset = comp == 0 ? 0u : 64u * mbs * (4u + (comp - 1u) * cpm);
}

// Bytes of one slice component at quantiser qi, the whole warp.
__device__ __forceinline__ uint32_t warp_component_bytes(const EncodeLaunch &e, const EncSliceDesc &sd,
                                                         const EncPicDesc &pd, const EncFrameDesc &fd, uint32_t comp,
                                                         uint32_t qi, const CountTables &t, uint32_t *buf) {
    uint32_t nb, off;
    comp_layout(fd, sd.mbs, comp, nb, off);
    const CompQuant q = comp_quant(quant_base(e, pd, qi), comp, nb);
    const float *f = e.coef + sd.coef + off;
    const uint32_t bits =
        warp_component_bits(f, comp_head<false>(f, e.coef_max + ((sd.coef + off) >> 5), nb), nb, q, t, buf);
    return (bits + 7u) / 8u;
}

constexpr int kCostThreads = 256;
constexpr int kCostBlocks = 4;      // CTAs an SM (5, at 48 registers: 7 % slower)
constexpr uint32_t kCostTake = 4;   // items a warp of k_cost takes at once, at most (2: 3 % slower; 19, as 4 rounds a warp: 7 %)
// Above this many items a warp its next ones are taken before it costs those
// it has: the counter's answer, about 1 us, is then waited for beside them. A
// warp that holds items it has not begun leaves others idle at the end, so
// with fewer they are taken when it is done (one UHD frame, 3 items a warp:
// 27 -> 25 us a probe; 30 1080p frames, 19 a warp, are better off ahead).
constexpr uint32_t kGrabAhead = 8;

// A warp per slice component, (component, slice) component-major. Its first
// items go by its place, so that a batch with an item a warp has each warp at
// work (all from the counter, 16-20 us a probe of one 1080p frame, now 13-15).
// From then on a warp takes `take` neighbouring items (at most 32) from the
// probe's counter at a time: its lanes look the items' places up side by side,
// so the chain of descriptor loads is waited for once, and the items are
// costed in turn.
__global__ void __launch_bounds__(kCostThreads, kCostBlocks) k_cost(EncodeLaunch e, int step, uint32_t take) {
    chain_start();
    __shared__ __align__(16) CountTables t;
    __shared__ __align__(8) uint32_t buf[kCostThreads / 32][kCountWords];
    t.fill();
    chain_wait();
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t items = 3u * e.n_slices;
    const uint32_t warps = gridDim.x * (kCostThreads / 32);
    const bool ahead = items > kGrabAhead * warps;
    uint32_t grab = (blockIdx.x * (kCostThreads / 32) + (threadIdx.x >> 5)) * take;
    for (;;) {
        const uint32_t base = __shfl_sync(0xffffffffu, grab, 0);
        if (base >= items) break;
        if (ahead && lane == 0) grab = warps * take + atomicAdd(e.cost_taken + step, take);
        // This lane's item: its first coefficient (a multiple of 64), its
        // quantiser table and component group, its block count (0: none).
        const uint32_t item = base + lane;
        uint32_t my_coef = 0, my_quant = 0, my_blocks = 0, my_bytes = 0, out = 0;
        if (lane < take && item < items) {
            const uint32_t comp = item < e.n_slices ? 0u : (item < 2u * e.n_slices ? 1u : 2u);
            const uint32_t s = item - comp * e.n_slices;
            const EncSliceDesc sd = e.slices[s];
            const uint32_t qi = (uint32_t)e.state[sd.pic].probe_qi, set = e.state[sd.pic].quant;
            out = 3u * s + comp;
            const uint32_t off = comp == 0 ? 0u : 64u * sd.mbs * (4u + (comp - 1u) * sd.cpm);
            my_coef = (uint32_t)((sd.coef + off) >> 6);
            my_quant = ((set * 225u + qi) << 1) | (comp > 0 ? 1u : 0u);
            if (qi != 0) my_blocks = (comp == 0 ? 4u : sd.cpm) * sd.mbs;
        }
        const uint32_t costed = __ballot_sync(0xffffffffu, my_blocks != 0);
        // With no picture left to cost (each is down to one quantiser, or the
        // coarsest did not fit its target) the other items are not looked at:
        // 4 UHD frames 10 us for such a probe, 39 with them. Asked only by a warp
        // whose items are all settled, so it costs the other probes nothing.
        if (!costed && step > 0 && e.searching[step] == 0) break;
        // The next item's maxima and DCs are on their way while one is costed.
        CompHead next_head{};
        uint32_t next_blocks = 0;
        const float *next_f = e.coef;
        const auto look = [&](uint32_t j) {
            const uint64_t coef = (uint64_t)__shfl_sync(0xffffffffu, my_coef, j) << 6;
            next_blocks = __shfl_sync(0xffffffffu, my_blocks, j);
            next_f = e.coef + coef;
            next_head = comp_head<false>(next_f, e.coef_max + (coef >> 5), next_blocks);
        };
        if (costed) look((uint32_t)__ffs(costed) - 1u);
        for (uint32_t left = costed; left;) {
            const uint32_t j = (uint32_t)__ffs(left) - 1u;
            left &= left - 1u;
            const CompHead h = next_head;
            const uint32_t nb = next_blocks;
            const float *f = next_f;
            if (left) look((uint32_t)__ffs(left) - 1u);
            const uint32_t quant = __shfl_sync(0xffffffffu, my_quant, j);
            const CompQuant q = comp_quant(e.quant + (uint64_t)(quant >> 1) * kQuantStride, quant & 1u, nb);
            const uint32_t bits = warp_component_bits(f, h, nb, q, t, buf[threadIdx.x >> 5]);
            if (lane == j) my_bytes = (bits + 7u) / 8u;
        }
        if (my_blocks) e.probe_comp[(uint64_t)step * 3u * e.n_slices + out] = my_bytes;
        if (!ahead && lane == 0) grab = warps * take + atomicAdd(e.cost_taken + step, take);
    }
}

// A slice's size from its component bytes, and whether every 16-bit size
// field holds it (src/encode.rs:671-681).
__device__ __forceinline__ uint64_t slice_total(uint32_t hdr, const uint32_t c[3], uint32_t alpha, bool &fits) {
    const uint64_t t = (uint64_t)hdr + c[0] + c[1] + c[2] + alpha;
    fits = t <= 65535u && c[0] <= 65535u && c[1] <= 65535u && c[2] <= 65535u;
    return t;
}

// Macroblocks from slice (mb_x, mb_y) to the end of the picture: the
// share-out's remaining_mbs (src/encode.rs:737-741, :771).
__device__ __forceinline__ uint64_t mbs_from(const EncPicDesc &pd, const EncSliceDesc &sd) {
    return (uint64_t)pd.width_in_mb * pd.height_in_mb - ((uint64_t)sd.mb_y * pd.width_in_mb + sd.mb_x);
}

// The probe step that costed quantiser qi for this picture, or -1. The crate
// reuses only the probe at uniform - 1 (src/encode.rs:743-749) and costs
// the later window levels afresh; a size is a function of the slice and
// the quantiser alone, so reusing any probe at a window's quantiser gives
// the same sizes and changes no choice.
__device__ __forceinline__ int probe_step_for(const EncPicState &st, int32_t qi) {
#pragma unroll
    for (int k = 0; k < kProbeSteps; k++)
        if (qi >= 1 && st.step_qi[k] == (uint32_t)qi) return k;
    return -1;
}

// Component sizes at window level j (quantiser uniform - 1 - j) of slice s:
// from a probe at that quantiser when there is one, else the window.
__device__ __forceinline__ const uint32_t *level_comp(const EncodeLaunch &e, const EncPicState &st, uint32_t j,
                                                      uint32_t s) {
    const int step = probe_step_for(st, st.uniform - 1 - (int32_t)j);
    if (step >= 0) return e.probe_comp + ((uint64_t)step * e.n_slices + s) * 3u;
    return e.win_comp + ((uint64_t)j * e.n_slices + s) * 3u;
}

// The slices whose window level is costed, as a list: level 0 takes every
// slice of a picture that has finer quantisers to share out; a later level
// the slices (at no level that a probe sized already)
// whose size at the level before fits and is within the most their share
// can come to (the crate's prefetch rule, src/encode.rs:741-767). The list
// order is the atomics' and steers nothing but speed.
__global__ void __launch_bounds__(kCostThreads) k_window_select(EncodeLaunch e, int level) {
    chain_start();
    chain_wait();
    const uint32_t s = blockIdx.x * kCostThreads + threadIdx.x;
    const int lane = threadIdx.x & 31;
    bool take = false;
    if (s < e.n_slices) {
        const EncSliceDesc sd = e.slices[s];
        const EncPicState st = e.state[sd.pic];
        const int32_t qi = st.uniform - 1 - level;
        if (st.fits_at_all && st.uniform > 1 && qi >= 1 && probe_step_for(st, qi) < 0) {
            take = true;
            if (level > 0) {
                const EncPicDesc &pd = e.pics[sd.pic];
                const uint32_t *prev = level_comp(e, st, (uint32_t)level - 1u, s);
                take = prev[0] != kNotCosted;
                if (take) {
                    const uint32_t alpha = e.alpha_bytes[s];
                    const uint32_t pc[3] = {prev[0], prev[1], prev[2]};
                    bool fits, f2;
                    const uint64_t n = slice_total(pd.header_bytes, pc, alpha, fits);
                    const uint32_t *u = e.probe_comp + ((uint64_t)st.hi_probe * e.n_slices + s) * 3u;
                    const uint32_t uc[3] = {u[0], u[1], u[2]};
                    const uint64_t used = slice_total(pd.header_bytes, uc, alpha, f2);
                    const uint64_t slack = st.budget - st.hi_total;
                    const uint64_t most = used + slack * sd.mbs / mbs_from(pd, sd);
                    take = fits && n <= most;
                }
                if (!take) e.win_comp[((uint64_t)level * e.n_slices + s) * 3u] = kNotCosted;
            }
        }
    }
    const uint32_t m = __ballot_sync(0xffffffffu, take);
    if (m) {
        const int leader = __ffs(m) - 1;
        uint32_t at = 0;
        if (lane == leader) at = atomicAdd(e.win_count + level, (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (take) e.win_list[at + __popc(m & ((1u << lane) - 1u))] = s;
    }
}

// Costs the listed slices at window level `level` (quantiser uniform - 1 -
// level), a warp per (slice, component).
__global__ void __launch_bounds__(kCostThreads, kCostBlocks) k_cost_window(EncodeLaunch e, int level) {
    chain_start();
    chain_wait();
    __shared__ __align__(16) CountTables t;
    __shared__ __align__(8) uint32_t buf[kCostThreads / 32][kCountWords];
    const uint32_t items = 3u * e.win_count[level], stride = gridDim.x * (kCostThreads / 32);
    if (blockIdx.x * (kCostThreads / 32) >= items) return;  // the whole block
    t.fill();
    __syncthreads();
    for (uint32_t item = blockIdx.x * (kCostThreads / 32) + (threadIdx.x >> 5); item < items; item += stride) {
        const uint32_t comp = item % 3u, s = e.win_list[item / 3u];
        const EncSliceDesc sd = e.slices[s];
        const uint32_t qi = (uint32_t)(e.state[sd.pic].uniform - 1 - level);
        const EncPicDesc &pd = e.pics[sd.pic];
        const uint32_t bytes =
            warp_component_bytes(e, sd, pd, e.frames[pd.frame], comp, qi, t, buf[threadIdx.x >> 5]);
        if ((threadIdx.x & 31) == 0) e.win_comp[((uint64_t)level * e.n_slices + s) * 3u + comp] = bytes;
    }
}

// The levels past the window, costed ahead of the share-out, every slice at
// once: a slice whose last window level fits and is
// within its likely allowance goes on to the next finer quantiser, and so
// on while the size it just found fits and stays within that allowance,
// for up to kDeepLevels levels. A slice's ladder depends on nothing but its
// own sizes and its picture's slack, so the slices need not wait for one
// another; the share-out then reads these sizes instead of costing them one
// slice after another (which it still does for a level past the ladder).
//
// The likely allowance is the slice's share of the picture's slack in
// proportion to its macroblocks, plus a quarter, plus one step (its size
// change a finer quantiser, as estimated below), and never above the most
// its share can come to (the crate's prefetch rule: the whole slack from
// the slice on, if no slice before it took any). For a slice whose step is
// under a quarter of its share it is that most, and so it is, for at most
// kTailLevels levels, for a picture's last kTailSlices slices. The
// share-out's allowance for a slice is what the slices before it left,
// which stays near the proportional share but for the last slices of a
// picture; the most is far above it there (the last slice's is the whole
// slack), and a ladder to the most for every slice costed several
// quantisers of every slice of a picture's tail for nothing. What the
// ladder leaves out only moves work to the share-out, never changes a
// size.
constexpr uint32_t kTailSlices = 16;  // a picture's tail: slices within this many slices' macroblocks of its end
constexpr uint32_t kTailLevels = 4;

// The slices with a ladder, listed (in the atomics' order, which steers
// nothing but speed).
__global__ void __launch_bounds__(kCostThreads) k_deep_select(EncodeLaunch e) {
    chain_start();
    chain_wait();
    const uint32_t s = blockIdx.x * kCostThreads + threadIdx.x;
    DeepItem item{};
    if (s < e.n_slices) {
        const EncSliceDesc sd = e.slices[s];
        const EncPicState st = e.state[sd.pic];
        e.deep_count[s] = 0;
        if (st.fits_at_all && st.uniform - kWindow > 1) {
            const EncPicDesc &pd = e.pics[sd.pic];
            const uint32_t hb = pd.header_bytes, alpha = e.alpha_bytes[s];
            const uint32_t *u = e.probe_comp + ((uint64_t)st.hi_probe * e.n_slices + s) * 3u;
            const uint32_t uc[3] = {u[0], u[1], u[2]};
            bool f0;
            const uint64_t used = slice_total(hb, uc, alpha, f0);
            const uint64_t slack = st.budget - st.hi_total;
            const uint64_t most = used + slack * sd.mbs / mbs_from(pd, sd);
            const uint64_t share = slack * sd.mbs / ((uint64_t)pd.width_in_mb * pd.height_in_mb);
            const uint32_t *c = level_comp(e, st, kWindow - 1, s);
            bool fits = false;
            uint64_t n = ~0ull;
            if (c[0] != kNotCosted) {
                const uint32_t cc[3] = {c[0], c[1], c[2]};
                n = slice_total(hb, cc, alpha, fits);
            }
            // The slice's step: its size change a finer quantiser, the larger
            // of the first step and the mean of the window's next three (the
            // first can be far larger than the rest: above quantiser index
            // 128 a step of the index is 4 of qScale, below it 1).
            const uint32_t *c1 = level_comp(e, st, 0, s);
            uint64_t step = 0, n1 = 0;
            if (c1[0] != kNotCosted) {
                const uint32_t cc[3] = {c1[0], c1[1], c1[2]};
                bool f1;
                n1 = slice_total(hb, cc, alpha, f1);
                step = n1 > used ? n1 - used : 0u;
                if (c[0] != kNotCosted) step = min(step, n > n1 ? (n - n1) / (uint64_t)(kWindow - 1) : 0u);
            }
            // A slice whose step is small beside its share (a coarse
            // quantiser, where a step often changes no size) walks many
            // levels wherever its allowance lands: its ladder goes to the
            // most. So do the last slices of a picture, where what the slices
            // before left gathers, for at most kTailLevels levels.
            const bool coarse = 4u * step <= share;
            const bool tail = mbs_from(pd, sd) <= (uint64_t)kTailSlices * sd.mbs;
            const uint64_t likely = coarse || tail ? most : min(most, used + share + share / 4u + step);
            const uint32_t levels = coarse ? (uint32_t)kDeepLevels : (tail ? kTailLevels : (uint32_t)kDeepLevels);
            uint32_t peak = 0;
#pragma unroll
            for (int j = 0; j < kWindow; j++) {
                const uint32_t *cj = level_comp(e, st, (uint32_t)j, s);
                const uint32_t cc[3] = {cj[0], cj[1], cj[2]};
                bool fj;
                const uint64_t nj = cj[0] == kNotCosted ? 0u : slice_total(hb, cc, alpha, fj);
                peak = max(peak, cj[0] == kNotCosted || !fj ? ~0u : (uint32_t)nj);
            }
            if (fits && n <= likely)
                item = DeepItem{likely, s, min(levels, (uint32_t)(st.uniform - 1 - kWindow)), hb + alpha, peak};
        }
    }
    const uint32_t m = __ballot_sync(0xffffffffu, item.levels != 0);
    if (m) {
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t at = 0;
        if (lane == (uint32_t)__ffs(m) - 1u) at = atomicAdd(e.deep_listed, (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1);
        if (item.levels) e.deep_list[at + __popc(m & ((1u << lane) - 1u))] = item;
    }
}

// Blocks take the listed slices, with a warp for each component and each of
// the next kDeepTries levels. Bound by the longest ladders, whose levels
// follow one another: a warp a slice, component after component and level
// after level, took one UHD frame 44 us, 30 of them 128 and 32 frames of mixed
// sizes 394; this takes 13, 25 and 76 with both its kernels. In smaller teams,
// four times 3 warps a block for a level at a time: 29, 33 and 181; twice 6
// warps: 18, 21 and 107; the same with a list of each block's own 32 slices
// instead of the one of all: 77, 126 and 378 (neighbours' ladders are long
// together).
constexpr uint32_t kDeepTries = 4;
constexpr uint32_t kDeepThreads = 32 * 3 * kDeepTries;
constexpr int kDeepBlocks = 2;

__global__ void __launch_bounds__(kDeepThreads, kDeepBlocks) k_cost_deep(EncodeLaunch e) {
    chain_start();
    __shared__ __align__(16) CountTables t;
    __shared__ __align__(8) uint32_t buf[kDeepThreads / 32][kCountWords];
    __shared__ uint32_t now, sizes[2][kDeepTries][3];
    t.fill();
    chain_wait();
    __syncthreads();
    const uint32_t listed = e.deep_listed[0];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t comp = warp % 3u, ahead = warp / 3u;
    for (;;) {
        if (threadIdx.x == 0) now = atomicAdd(e.deep_listed + 1, 1u);
        __syncthreads();
        if (now >= listed) return;
        const DeepItem item = e.deep_list[now];
        const EncSliceDesc sd = e.slices[item.s];
        const EncPicDesc &pd = e.pics[sd.pic];
        const EncFrameDesc &fd = e.frames[pd.frame];
        // Level j is quantiser finest - j, which item.levels keeps above 0.
        const uint32_t finest = (uint32_t)(e.state[sd.pic].uniform - 1 - kWindow);
        uint32_t j = 0, peak = item.peak;
        bool more = true;
        for (uint32_t turn = 0; more; turn ^= 1u) {
            if (j + ahead < item.levels) {
                const uint32_t bytes = warp_component_bytes(e, sd, pd, fd, comp, finest - j - ahead, t, buf[warp]);
                if (lane == 0) sizes[turn][ahead][comp] = bytes;
            }
            __syncthreads();
            for (uint32_t a = 0; more && a < kDeepTries; a++) {
                const uint32_t c3[3] = {sizes[turn][a][0], sizes[turn][a][1], sizes[turn][a][2]};
                bool fits;
                const uint64_t n = slice_total(item.hba, c3, 0, fits);
                peak = max(peak, fits ? (uint32_t)n : ~0u);
                if (threadIdx.x == 0)
                    e.deep[(uint64_t)item.s * kDeepLevels + j] =
                        make_uint2(min(c3[0], 65535u) | (min(c3[1], 65535u) << 16),
                                   min(c3[2], 65535u) | ((peak <= 65535u ? peak : 0u) << 16));
                j++;
                more = fits && n <= item.likely && j < item.levels;
            }
        }
        if (threadIdx.x == 0) e.deep_count[item.s] = j;
    }
}

// Threads a picture of k_rc_init and k_rc_step, at most and at least (rc_threads).
constexpr int kRcThreads = 1024, kRcThreadsMin = 64;

__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v, uint64_t *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    uint64_t t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
    return t;
}

__global__ void __launch_bounds__(kRcThreads) k_rc_init(EncodeLaunch e) {
    chain_start();
    chain_wait();
    __shared__ uint64_t sh[kRcThreads / 32];
    const EncPicDesc pd = e.pics[blockIdx.x];
    uint64_t a = 0;
    if (e.any_alpha)
        for (uint32_t k = threadIdx.x; k < pd.n_slices; k += blockDim.x) a += e.alpha_bytes[pd.slice_base + k];
    const uint64_t alpha = block_sum_u64(a, sh);
    if (threadIdx.x == 0) {
        // Alpha is lossless and comes on top of the rate; the picture
        // header and the slice table come out of it (src/encode.rs:686-689).
        const uint64_t overhead = 8u + 2ull * pd.n_slices;
        const uint64_t b = pd.budget_in + alpha;
        EncPicState st{};
        st.budget = b > overhead ? b - overhead : 0;
        st.lo = 1;
        st.hi = 224;
        st.probe_qi = 224;
        st.hi_probe = 0;
        st.fits_at_all = 0;
        st.uniform = 224;
        st.quant = pd.quant;
        e.state[blockIdx.x] = st;
        if (blockIdx.x == 0) {
            for (int j = 0; j < kWindow; j++) e.win_count[j] = 0;
            for (int j = 0; j < kProbeSteps; j++) e.cost_taken[j] = e.searching[j] = 0;
            e.deep_listed[0] = e.deep_listed[1] = 0;
        }
    }
}

__global__ void __launch_bounds__(kRcThreads) k_rc_step(EncodeLaunch e, int step) {
    chain_start();
    chain_wait();
    __shared__ uint64_t sh[kRcThreads / 32];
    __shared__ int all_fit;
    const EncPicDesc pd = e.pics[blockIdx.x];
    const EncPicState st0 = e.state[blockIdx.x];
    if (st0.probe_qi == 0) return;
    if (threadIdx.x == 0) all_fit = 1;
    __syncthreads();
    uint64_t sum = 0;
    bool fit = true;
#pragma unroll 4
    for (uint32_t k = threadIdx.x; k < pd.n_slices; k += blockDim.x) {
        const uint32_t s = pd.slice_base + k;
        const uint32_t *c = e.probe_comp + ((uint64_t)step * e.n_slices + s) * 3u;
        const uint32_t cc[3] = {c[0], c[1], c[2]};
        bool f;
        sum += slice_total(pd.header_bytes, cc, e.any_alpha ? e.alpha_bytes[s] : 0u, f);
        fit = fit && f;
    }
    if (!fit) all_fit = 0;
    const uint64_t total = block_sum_u64(sum, sh);
    if (threadIdx.x == 0) {
        EncPicState st = st0;
        st.step_qi[step] = (uint8_t)st.probe_qi;
        const bool ok = all_fit && total <= st.budget;
        if (step == 0) {
            // totals(224): if even the coarsest quantiser does not fit, it is
            // used throughout (src/encode.rs:701-713).
            st.fits_at_all = ok;
            st.hi_probe = 0;
            st.hi_total = total;
            if (!ok) {
                st.probe_qi = 0;
                st.uniform = 224;
            }
        } else if (ok) {
            st.hi = st.probe_qi;
            st.hi_probe = step;
            st.hi_total = total;
        } else {
            st.lo = st.probe_qi + 1;
        }
        if (st.fits_at_all) {
            if (st.lo < st.hi) {
                st.probe_qi = st.lo + (st.hi - st.lo) / 2;
            } else {
                st.probe_qi = 0;
                st.uniform = st.hi;
            }
        }
        e.state[blockIdx.x] = st;
        if (st.probe_qi != 0 && step + 1 < kProbeSteps) atomicAdd(e.searching + step + 1, 1u);
    }
}

// The share-out (src/encode.rs:769-793). With D = remaining_budget -
// remaining_base, slice i steps from the uniform quantiser to the next finer
// one while that size n fits and n <= base + floor(D mbs / remaining_mbs),
// i.e. while n <= base or D >= ceil((n - base) remaining_mbs / mbs); D then
// falls by what the slice took over its base. Three kernels:
//   k_share_prep   every slice in parallel: its base and, for each window
//                  level, the threshold on D and the size over the base;
//   k_shareout     one warp per picture, the only serial part: D against
//                  the thresholds (the window's, then each slice's deep
//                  ladder from k_cost_deep), 32 slices at a time, their
//                  thresholds copied ahead; where a slice gets past all of
//                  them, the block's other warps cost the next quantisers;
//   k_share_final  every slice in parallel: its quantiser and sizes.
constexpr uint32_t kDeepFlag = 0x80000000u;  // share_steps: sizes are in final_comp already

__global__ void k_share_prep(EncodeLaunch e) {
    chain_start();
    chain_wait();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= e.n_slices) return;
    const EncSliceDesc sd = e.slices[s];
    const EncPicState st = e.state[sd.pic];
    SharePrep pr{};
    if (st.uniform > 1 && st.fits_at_all) {
        const EncPicDesc &pd = e.pics[sd.pic];
        const uint32_t hb = pd.header_bytes, alpha = e.alpha_bytes[s];
        const uint32_t *u = e.probe_comp + ((uint64_t)st.hi_probe * e.n_slices + s) * 3u;
        const uint32_t uc[3] = {u[0], u[1], u[2]};
        bool f;
        const uint64_t base = slice_total(hb, uc, alpha, f);
        const uint64_t rem = mbs_from(pd, sd);
        const uint32_t shift = 31u - __clz(sd.mbs);
        pr.base = (uint32_t)base;
        pr.hba = hb + alpha;
        pr.rem = (uint32_t)rem;
        pr.shift = (uint8_t)shift;
        uint64_t run = 0;
        uint32_t levels = 0;  // the walk's levels before it stops whatever D is
        bool stopped = false;
#pragma unroll
        for (int j = 0; j < kWindow; j++) {
            const bool more = st.uniform - j > 1;
            const uint32_t *c = more ? level_comp(e, st, (uint32_t)j, s) : nullptr;
            const bool known = more && c[0] != kNotCosted;
            if (!stopped && more && !known) pr.uncosted_at_end = 1;
            stopped = stopped || !known;
            pr.thr[j] = ~0ull;
            if (stopped) continue;
            const uint32_t cc[3] = {c[0], c[1], c[2]};
            bool fits;
            const uint64_t n = slice_total(hb, cc, alpha, fits);
            const uint64_t thr = !fits ? ~0ull : n <= base ? 0ull : ((((n - base) * rem) + sd.mbs - 1) >> shift);
            run = run > thr ? run : thr;
            pr.thr[j] = run;
            pr.delta[j] = (int32_t)((int64_t)n - (int64_t)base);
            levels++;
        }
        if (!stopped) {
            pr.deep_count = (uint8_t)min(e.deep_count[s], (uint32_t)(st.uniform - 1 - kWindow));
            levels += pr.deep_count;
            pr.uncosted_at_end = st.uniform - (int32_t)levels > 1;
        }
        pr.levels = (uint8_t)levels;
    }
    e.share_prep[s] = pr;
}

// The size at a level past the window, from a slice's deep ladder (a level that
// fits).
__device__ __forceinline__ uint32_t deep_size(const SharePrep &p, uint2 v) {
    return p.hba + (v.x & 0xFFFFu) + (v.x >> 16) + (v.y & 0xFFFFu);
}

// The deep levels (level j at deep[32 j]) that D lets the slice take, all of
// the window's taken. A level's threshold on D grows with its size, so the
// running maximum of the thresholds is at most D where the ladder's peak is
// within the allowance that D gives: a binary search of the peaks, which only
// grow, from the levels taken at the last D (`last`) on. (A table of 64-bit
// thresholds for each chunk of 32 slices took 6,500 cycles to build where the
// ladders are long: 96 frames of mixed sizes 3.43 -> 2.66 ms without it.)
__device__ __forceinline__ uint32_t deep_steps(const SharePrep &p, const uint2 *deep, uint32_t last, uint64_t D) {
    const uint64_t allowed = p.base + (D << p.shift) / p.rem;
    const uint32_t limit = (uint32_t)min(allowed, (uint64_t)65535u);
    const auto taken = [&](uint32_t j) { return (deep[32u * j].y >> 16) - 1u < limit; };
    uint32_t lo = 0, hi = p.deep_count;
    if (last > 0 && !taken(last - 1u))
        hi = last - 1u;
    else if (last < hi && !taken(last))
        lo = hi = last;
    else
        lo = last;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (taken(mid))
            lo = mid + 1u;
        else
            hi = mid;
    }
    return lo;
}

// Quantisers costed at a time for a slice that needs one nobody costed, and
// the warps that do, one per component and quantiser (32 frames of mixed
// sizes: 686, 603 and 551 us with 1, 2 and 4; the others have none).
constexpr int kShareTries = 4;
constexpr int kShareHelpers = 3 * kShareTries;
constexpr int kShareThreads = 32 * (1 + kShareHelpers);

// What k_shareout's first warp asks the others for, and their answer.
struct ShareJob {
    uint64_t D;
    uint32_t slice;  // ~0: no more
    uint32_t steps;  // taken so far; with kDeepFlag once sizes are in final_comp
    int32_t delta;   // the size over the base after them
    uint32_t base;
};

struct ShareShared {
    CountTables t;
    // The slice being costed, copied in once (its coefficients, then its
    // chunk maxima): the warps walk it for every quantiser they try.
    __align__(16) float stage[kMaxSliceCoefs + kMaxSliceCoefs / 32];
    __align__(8) uint32_t buf[kShareHelpers][kCountWords];
    uint32_t sizes[2][kShareTries][3];
    ShareJob job;
    // Per lane, of the 32 slices being settled and of the next ones: their
    // thresholds (16-byte words, of two chunks ahead) and their ladders (of one
    // ahead).
    uint4 prep[3][sizeof(SharePrep) / sizeof(uint4)][32];
    uint2 ladder[2][kDeepLevels][32];
};

__device__ __forceinline__ void copy8_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Barriers of k_shareout: a job is posted / its answer is (all threads); the
// helpers among themselves.
__device__ __forceinline__ void share_barrier(int id, int threads) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int kJobPosted = 1, kJobDone = 2, kHelpersOnly = 3;

// A helper warp: costs one component of the slice at one of the kShareTries
// next finer quantisers, until the slice no longer fits its allowance (fixed
// during the slice's walk).
__device__ void share_help(const EncodeLaunch &e, const EncPicDesc &pd, int32_t uniform, ShareShared &sh) {
    const uint32_t h = (threadIdx.x >> 5) - 1u, lane = threadIdx.x & 31u;
    const uint32_t c = h % 3u, ahead = h / 3u, tid = threadIdx.x - 32u;
    const EncFrameDesc &fd = e.frames[pd.frame];
    for (;;) {
        share_barrier(kJobPosted, kShareThreads);
        const ShareJob job = sh.job;
        if (job.slice == ~0u) return;
        const uint32_t s = job.slice;
        const EncSliceDesc sd = e.slices[s];
        const uint32_t alpha = e.alpha_bytes[s];
        const uint32_t cpm = fd.chroma == 2 ? 2u : 4u;
        const uint32_t total = 64u * (4u + 2u * cpm) * sd.mbs;
        float *const smax = sh.stage + kMaxSliceCoefs;
        for (uint32_t i = tid; i < total / 4u; i += 32u * kShareHelpers)
            copy16_async(sh.stage + 4u * i, e.coef + sd.coef + 4u * i);
        const float *msrc = e.coef_max + (sd.coef >> 5);
        for (uint32_t i = tid; i < total / 32u; i += 32u * kShareHelpers) smax[i] = msrc[i];
        const uint64_t allowed = job.base + job.D * sd.mbs / mbs_from(pd, sd);
        copies_wait();
        share_barrier(kHelpersOnly, 32 * kShareHelpers);
        uint32_t nb, off;
        comp_layout(fd, sd.mbs, c, nb, off);
        const float *f = sh.stage + off;
        const CompHead head = comp_head<true>(f, smax + (off >> 5), nb);
        uint32_t steps = job.steps, c3[3] = {0, 0, 0};
        int32_t delta = job.delta, qi = uniform - (int32_t)job.steps;
        bool any = false, more = qi > 1;
        for (uint32_t turn = 0; more; turn ^= 1u) {
            const int32_t mine = qi - 1 - (int32_t)ahead;
            if (mine >= 1) {
                const CompQuant q = comp_quant(quant_base(e, pd, (uint32_t)mine), c, nb);
                const uint32_t bits = warp_component_bits<true>(f, head, nb, q, sh.t, sh.buf[h]);
                if (lane == 0) sh.sizes[turn][ahead][c] = (bits + 7u) / 8u;
            }
            share_barrier(kHelpersOnly, 32 * kShareHelpers);
            for (int a = 0; more && a < kShareTries; a++) {
                const uint32_t n3[3] = {sh.sizes[turn][a][0], sh.sizes[turn][a][1], sh.sizes[turn][a][2]};
                bool fits;
                const uint64_t n = slice_total(pd.header_bytes, n3, alpha, fits);
                if (!(fits && n <= allowed)) {
                    more = false;
                    break;
                }
                qi -= 1;
                steps++;
                delta = (int32_t)n - (int32_t)job.base;
                c3[0] = n3[0];
                c3[1] = n3[1];
                c3[2] = n3[2];
                any = true;
                more = qi > 1;
            }
        }
        if (tid == 0) {
            if (any) {
                e.final_comp[3ull * s] = c3[0];
                e.final_comp[3ull * s + 1] = c3[1];
                e.final_comp[3ull * s + 2] = c3[2];
                steps |= kDeepFlag;
            }
            sh.job.steps = steps;
            sh.job.delta = delta;
        }
        share_barrier(kJobDone, kShareThreads);
    }
}

// The settling warp: 32 slices at a time.
__device__ void share_settle(const EncodeLaunch &e, const EncPicDesc &pd, uint64_t D, ShareShared &sh) {
    const int lane = threadIdx.x & 31;
    constexpr uint32_t kPrepWords = sizeof(SharePrep) / sizeof(uint4);
    // What the next chunks need is copied to shared memory while one is
    // settled, a lane's slice by the lane, which alone reads it.
    const auto fetch_prep = [&](uint32_t k0, uint32_t slot) {
        if (k0 + lane >= pd.n_slices) return;
        const uint4 *src = reinterpret_cast<const uint4 *>(e.share_prep + pd.slice_base + k0 + lane);
#pragma unroll
        for (uint32_t w = 0; w < kPrepWords; w++) copy16_async(&sh.prep[slot][w][lane], src + w);
    };
    const auto load_prep = [&](uint32_t slot) {
        union {
            SharePrep p;
            uint4 w[kPrepWords];
        } u;
#pragma unroll
        for (uint32_t w = 0; w < kPrepWords; w++) u.w[w] = sh.prep[slot][w][lane];
        return u.p;
    };
    const auto fetch_ladder = [&](uint32_t k0, uint32_t slot, uint32_t half) {
        if (k0 + lane >= pd.n_slices) return;
        const uint32_t count = load_prep(slot).deep_count;
        const uint2 *src = e.deep + (uint64_t)(pd.slice_base + k0 + lane) * kDeepLevels;
#pragma unroll 4
        for (uint32_t j = 0; j < count; j++) copy8_async(&sh.ladder[half][j][lane], src + j);
    };
    fetch_prep(0, 0);
    copies_wait();
    fetch_prep(32, 1);
    fetch_ladder(0, 0, 0);
    uint32_t slot = 0, half = 0;
    for (uint32_t k0 = 0; k0 < pd.n_slices; k0 += 32) {
        const uint32_t k = k0 + lane;
        const bool live = k < pd.n_slices;
        copies_wait();
        const uint32_t slot1 = slot == 2u ? 0u : slot + 1u, slot2 = slot1 == 2u ? 0u : slot1 + 1u;
        fetch_prep(k0 + 64, slot2);
        fetch_ladder(k0 + 32, slot1, half ^ 1u);
        // Past the picture's end: no level, at any D.
        SharePrep mine{};
        if (live) {
            mine = load_prep(slot);
        } else {
#pragma unroll
            for (int j = 0; j < kWindow; j++) mine.thr[j] = ~0ull;
        }
        const uint2 *my_deep = &sh.ladder[half][0][lane];
        uint32_t last_deep = 0;  // deep levels taken at the last D
        uint32_t my_steps = 0;
        uint32_t done = 0;  // lanes below are settled
        while (done < 32u) {
            // The walk is sequential: a slice's slack D is what the slices
            // before it left. Each lane guesses its D and takes its steps
            // there; the guesses are redone from the exclusive sum of the
            // steps' size changes until no lane's steps change. A lane's D
            // depends only on the lanes before it, so after t rounds the
            // first t lanes are exact and the fixed point reached (at most 33
            // rounds) is the sequential walk's. The first lane that needs a
            // level nobody costed, and those after it, wait for the helpers
            // to cost it.
            uint64_t myD = D;
            uint32_t ks = 0, guessed = 0;           // the steps at myD, and those it came from
            int32_t mine_dl = 0, before = 0;        // a size that fits is below 2^16
            uint32_t upto_deep = 0;                 // the lanes up to the first deep one; 0: none is
            for (int round = 0; round < 34; round++) {
                ks = 0;
                mine_dl = 0;
                if ((uint32_t)lane >= done) {
#pragma unroll
                    for (int j = 0; j < kWindow; j++) {
                        const bool taken = mine.thr[j] <= myD;
                        ks += taken;
                        mine_dl = taken ? mine.delta[j] : mine_dl;
                    }
                }
                const bool past = ks == (uint32_t)kWindow && mine.deep_count > 0;
                if (__any_sync(0xffffffffu, past)) {
                    if (past) last_deep = deep_steps(mine, my_deep, last_deep, myD);
                    if (past && last_deep) {
                        ks += last_deep;
                        mine_dl = (int32_t)(deep_size(mine, my_deep[32u * (last_deep - 1u)]) - mine.base);
                    }
                }
                const uint32_t deep_mask =
                    __ballot_sync(0xffffffffu, (uint32_t)lane >= done && mine.uncosted_at_end && ks == mine.levels);
                const uint32_t moved = __ballot_sync(0xffffffffu, ks != guessed);
                upto_deep = deep_mask ? deep_mask ^ (deep_mask - 1u) : 0u;
                if (!(moved & (upto_deep ? upto_deep : ~0u))) break;
                guessed = ks;
                // Inclusive sum over the lanes.
                int32_t incl = mine_dl;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                before = incl - mine_dl;
                myD = (uint64_t)((int64_t)D - before);
            }
            const uint32_t f = upto_deep ? 31u - (uint32_t)__clz(upto_deep) : 32u;
            // Lanes done .. f - 1 are settled at myD with ks steps.
            if ((uint32_t)lane >= done && (uint32_t)lane < f) my_steps = ks;
            if (f == 32u) {
                // Every lane settled: D after the chunk.
                D = (uint64_t)((int64_t)D - __shfl_sync(0xffffffffu, before + mine_dl, 31));
                break;
            }
            // The deep lane, at its exact D.
            D = (uint64_t)((int64_t)D - __shfl_sync(0xffffffffu, before, f));
            if (lane == (int)f) sh.job = ShareJob{D, pd.slice_base + k, ks, mine_dl, mine.base};
            share_barrier(kJobPosted, kShareThreads);
            share_barrier(kJobDone, kShareThreads);
            if (lane == (int)f) my_steps = sh.job.steps;
            D = (uint64_t)((int64_t)D - sh.job.delta);
            done = f + 1;
        }
        if (live) e.share_steps[pd.slice_base + k] = my_steps;
        slot = slot1;
        half ^= 1u;
    }
    if (lane == 0) sh.job.slice = ~0u;
    share_barrier(kJobPosted, kShareThreads);
}

// A block per picture: a warp that settles its slices, and helpers. Bound by
// the settling warp's chain: about 1170 cycles a chunk of 32 UHD slices, of
// them 700 in its two rounds (thresholds against D, the votes, a scan), 200 to
// start the next chunks' copies. One UHD frame 122 -> 73 us, 30 of them 152 ->
// 85, and 32 frames of mixed sizes, whose slices often get past their ladders,
// 1243 -> 503. Before, each round ended with a scan, also to find that nothing
// had moved; each chunk built tables of its lanes' thresholds first (10,000 cycles
// where the ladders are long); and the one warp copied a slice past its ladder
// in and costed it alone (24,000 cycles a slice, 7,000 now).
__global__ void __launch_bounds__(kShareThreads) k_shareout(EncodeLaunch e) {
    chain_start();
    extern __shared__ __align__(16) uint8_t share_smem[];
    ShareShared &sh = *reinterpret_cast<ShareShared *>(share_smem);
    sh.t.fill();
    chain_wait();
    __syncthreads();
    const EncPicDesc pd = e.pics[blockIdx.x];
    const EncPicState st = e.state[blockIdx.x];
    if (!(st.uniform > 1 && st.fits_at_all)) {
        for (uint32_t k = threadIdx.x; k < pd.n_slices; k += kShareThreads) e.share_steps[pd.slice_base + k] = 0;
        return;
    }
    if (threadIdx.x < 32u)
        share_settle(e, pd, st.budget - st.hi_total, sh);
    else
        share_help(e, pd, st.uniform, sh);
}

__global__ void k_share_final(EncodeLaunch e) {
    chain_start();
    chain_wait();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= e.n_slices) return;
    const EncSliceDesc sd = e.slices[s];
    const EncPicState st = e.state[sd.pic];
    const uint32_t steps = e.share_steps[s];
    const uint32_t n = steps & ~kDeepFlag;
    e.final_qi[s] = (uint32_t)st.uniform - n;
    if (steps & kDeepFlag) return;  // written by the walk
    if (n > (uint32_t)kWindow) {
        // From the slice's deep ladder (a level the slice fits at, so no
        // size there is saturated).
        const uint2 v = e.deep[(uint64_t)s * kDeepLevels + (n - 1u - kWindow)];
        e.final_comp[3ull * s] = v.x & 0xFFFFu;
        e.final_comp[3ull * s + 1] = v.x >> 16;
        e.final_comp[3ull * s + 2] = v.y & 0xFFFFu;
        return;
    }
    const uint32_t *c = n == 0 ? e.probe_comp + ((uint64_t)st.hi_probe * e.n_slices + s) * 3u
                               : level_comp(e, st, n - 1u, s);
    e.final_comp[3ull * s] = c[0];
    e.final_comp[3ull * s + 1] = c[1];
    e.final_comp[3ull * s + 2] = c[2];
}

// ---------------------------------------------------------------- layout

constexpr int kLayoutThreads = 1024;

__device__ __forceinline__ uint64_t warp_incl_scan64(uint64_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Slice offsets within the picture (after its header and table) and the
// picture's size (src/encode.rs:820-829).
__global__ void __launch_bounds__(kLayoutThreads) k_layout(EncodeLaunch e) {
    chain_start();
    chain_wait();
    __shared__ uint64_t warp_sums[kLayoutThreads / 32];
    __shared__ uint64_t carry;
    const EncPicDesc pd = e.pics[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 8u + 2ull * pd.n_slices;
    if (threadIdx.x == 0 && blockIdx.x == 0) *e.pack_taken = 0;
    __syncthreads();
    for (uint32_t chunk = 0; chunk < pd.n_slices; chunk += kLayoutThreads) {
        const uint32_t k = chunk + threadIdx.x;
        uint64_t size = 0;
        if (k < pd.n_slices) {
            const uint32_t s = pd.slice_base + k;
            const uint32_t cc[3] = {e.final_comp[3ull * s], e.final_comp[3ull * s + 1], e.final_comp[3ull * s + 2]};
            bool f;
            size = slice_total(pd.header_bytes, cc, e.alpha_bytes[s], f);
        }
        const uint64_t incl = warp_incl_scan64(size);
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 0) warp_sums[lane] = warp_incl_scan64(warp_sums[lane]);
        __syncthreads();
        const uint64_t excl = carry + (warp ? warp_sums[warp - 1] : 0u) + incl - size;
        if (k < pd.n_slices) e.slice_off[pd.slice_base + k] = excl;
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_sums[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) e.state[blockIdx.x].pic_size = carry;
}

// Picture places and sizes, the frame header and frame_size, the picture
// headers (src/header.rs:174-199, :292-304). One thread per frame.
__global__ void k_frame(EncodeLaunch e) {
    chain_start();
    chain_wait();
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= e.n_frames) return;
    const EncFrameDesc fd = e.frames[f];
    uint64_t pos = fd.header_len;
    for (uint32_t i = 0; i < fd.n_pics; i++) {
        e.state[fd.first_pic + i].pic_off = pos;
        pos += e.state[fd.first_pic + i].pic_size;
    }
    e.frame_size[f] = pos;
    const bool over = pos > fd.out_cap;
    e.frame_status[f] = over ? 1u : 0u;
    if (over) return;
    const uint64_t base = fd.out_base * 8u;
    const uint8_t *h = e.headers + (uint64_t)kHeaderSlot * fd.header_slot;
    put_field(e.out, base, (uint32_t)pos, 32);  // frame_size
    for (uint32_t b = 4; b < fd.header_len; b++) put_field(e.out, base + 8ull * b, h[b], 8);
    for (uint32_t i = 0; i < fd.n_pics; i++) {
        const EncPicDesc &pd = e.pics[fd.first_pic + i];
        const EncPicState &st = e.state[fd.first_pic + i];
        const uint64_t at = base + 8ull * st.pic_off;
        put_field(e.out, at, 8u << 3, 8);
        put_field(e.out, at + 8, (uint32_t)st.pic_size, 32);
        put_field(e.out, at + 40, pd.n_slices <= 65535u ? pd.n_slices : 0u, 16);
        put_field(e.out, at + 56, (pd.log2_slice_mbs & 3u) << 4, 8);
    }
}

// ---------------------------------------------------------------- packing

// The writer's tables by context: a code's length << 24 | its significant
// bits, of run symbols below 63 and of level symbols below 127 with room for
// the sign bit; 0 in the last column, for every symbol past those. Both are
// indexed by context x kRow + symbol; neighbouring contexts start in
// different banks.
struct PackTables {
    static constexpr uint32_t kRow = kLevelLens + 1;
    uint32_t run[16][kRow];  // kRunLens used
    uint32_t level[9][kRow];
    uint32_t pad[3];  // a whole number of 16-byte words
    __device__ __forceinline__ void fill();
};
__device__ uint4 d_pack_tables[sizeof(PackTables) / sizeof(uint4)];

__device__ __forceinline__ void PackTables::fill() {
    for (uint32_t i = threadIdx.x; i < sizeof(PackTables) / sizeof(uint4); i += blockDim.x)
        reinterpret_cast<uint4 *>(this)[i] = d_pack_tables[i];
}

void build_pack_tables(PackTables &t) {
    t = PackTables{};
    for (uint32_t c = 0; c < 16; c++)
        for (uint32_t n = 0; n + 1 < kRunLens; n++)
            t.run[c][n] = (cb_len32(run_book(c), n) << 24) | (uint32_t)cb_bits(run_book(c), n);
    for (uint32_t c = 0; c < 9; c++)
        for (uint32_t n = 0; n + 1 < kLevelLens; n++)
            t.level[c][n] = ((cb_len32(level_book(c), n) + 1u) << 24) | ((uint32_t)cb_bits(level_book(c), n) << 1);
}

// A warp's output bits: fields, a lane each, are placed by a scan of their
// lengths and OR-ed into words in shared memory, which go out 32 at a time,
// the first and the last (which neighbours share) by an atomic OR. A batch of
// fields is at most kBatchBits bits.
constexpr uint32_t kBatchBits = 64 * 56;
constexpr uint32_t kPackWords = 32 + kBatchBits / 32 + 4;
struct WarpBits {
    uint32_t *buf;    // kPackWords words, zero past `bits`
    uint32_t base;    // its shared address
    uint32_t *out;    // where word 0 goes
    uint32_t bits;    // held, from bit 0 of word 0 on
    bool shared;      // word 0 is shared with what comes before
    // Once a warp; finish() leaves the buffer zero again.
    __device__ __forceinline__ void clear(uint32_t *b) {
        buf = b;
        base = (uint32_t)__cvta_generic_to_shared(b);
        for (uint32_t i = threadIdx.x & 31u; i < kPackWords; i += 32u) buf[i] = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void start(uint32_t *o, uint64_t bitpos) {
        out = o + (bitpos >> 5);
        bits = (uint32_t)bitpos & 31u;
        shared = true;
    }
    // Room for the lane's `len` bits, in lane order; returns its place.
    __device__ __forceinline__ uint32_t place(uint32_t len) {
        uint32_t sum = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
            asm volatile("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\tshfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n\t"
                         "@p add.u32 %0, %0, t;\n\t}"
                         : "+r"(sum)
                         : "r"(o));
        const uint32_t at = bits + sum - len;
        bits += __shfl_sync(0xffffffffu, sum, 31);
        return at;
    }
    // If `n` > 0, ORs `v` into word `w` of the buffer.
    __device__ __forceinline__ void or_word(uint32_t w, uint32_t v, int32_t n) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %2, 0;\n\t@p red.shared.or.b32 [%0], %1;\n\t}"
                     :
                     : "r"(base + 4u * w), "r"(v), "r"(n)
                     : "memory");
    }
    // ORs a field of `len` bits (at most 32; 0: none) in at bit `at`.
    __device__ __forceinline__ void put32(uint32_t at, uint32_t value, uint32_t len) {
        const uint32_t v = __funnelshift_lc(0u, value, 32u - len), o = at & 31u, w = at >> 5;
        or_word(w, v >> o, (int32_t)len);
        or_word(w + 1u, __funnelshift_r(0u, v, o), (int32_t)(o + len) - 32);
    }
    // The same of up to 64 bits.
    __device__ __forceinline__ void put(uint32_t at, uint64_t value, uint32_t len) {
        const uint64_t v = len ? value << (64u - len) : 0ull;
        const uint32_t hi = (uint32_t)(v >> 32), lo = (uint32_t)v, o = at & 31u, w = at >> 5;
        or_word(w, hi >> o, (int32_t)len);
        or_word(w + 1u, __funnelshift_r(lo, hi, o), (int32_t)(o + len) - 32);
        or_word(w + 2u, __funnelshift_r(0u, lo, o), (int32_t)(o + len) - 64);
    }
    // The whole words out, once there are 32.
    __device__ __forceinline__ void drain() {
        __syncwarp();
        if (bits >= 32u * 32u) flush(bits >> 5);
    }
    __device__ __forceinline__ void flush(uint32_t words) {
        const uint32_t lane = threadIdx.x & 31u;
        const uint32_t part = buf[words];
        __syncwarp();
        for (uint32_t i = lane; i < words; i += 32u) {
            const uint32_t v = bswap32(buf[i]);
            buf[i] = 0;
            if (i == 0 && shared)
                atomicOr(out, v);
            else
                out[i] = v;
        }
        __syncwarp();
        if (lane == 0) {
            buf[words] = 0;
            buf[0] = part;
        }
        __syncwarp();
        out += words;
        bits &= 31u;
        shared = shared && words == 0;
    }
    // Zero bits to the next byte boundary, then everything out.
    __device__ __forceinline__ void finish() {
        __syncwarp();
        if (bits >= 32u) flush(bits >> 5);
        if ((threadIdx.x & 31u) == 0 && bits) {
            atomicOr(out, bswap32(buf[0]));
            buf[0] = 0;
        }
        __syncwarp();
    }
};

// Writes the codes of two neighbouring non-zeros a lane (see CountSink).
struct PackSink {
    static constexpr bool kSign = true;
    const PackTables &t;
    WarpBits &w;
    // The code of entry e after the entries p and pp, at any length.
    __device__ __noinline__ static uint64_t long_code(uint32_t e, uint32_t p, uint32_t pp, uint32_t &len) {
        const uint32_t run = (e >> 16) - (p >> 16) - 1u, prev_run = ((p >> 16) - (pp >> 16) - 1u) & 0xFFFFu;
        const uint32_t level = e & 0x7FFFu, sign = (e >> 15) & 1u;
        const Codebook rb = run_book(prev_run), lb = level_book(p & 0x7FFFu);
        const uint32_t ll = cb_len32(lb, level);
        len = cb_len32(rb, run) + ll + 1u;
        return (((cb_bits(rb, run) << ll) | cb_bits(lb, level)) << 1) | sign;
    }
    __device__ __forceinline__ void pairs(uint2 b, uint2 c, int32_t n) {
        constexpr uint32_t kNoSign = 0xFFFF7FFFu;
        const uint32_t sign0 = (c.x >> 15) & 1u, sign1 = (c.y >> 15) & 1u;
        const uint32_t nbx = ~b.x & 0xFFFF0000u, nby = ~b.y & 0xFFFF0000u, ncx = ~c.x & 0xFFFF0000u;
        const uint32_t by = b.y & kNoSign, cx = c.x & kNoSign, cy = c.y & kNoSign;
        const uint32_t i0 = __viaddmin_s16x2(by, nbx, kCodeRows) * PackTables::kRow + __viaddmin_s16x2(cx, nby, kCodeCols);
        const uint32_t i1 = __viaddmin_s16x2(cx, nby, kCodeRows) * PackTables::kRow + __viaddmin_s16x2(cy, ncx, kCodeCols);
        const uint32_t *run = &t.run[0][0], *level = &t.level[0][0];
        const uint32_t r0 = run[i0 >> 16], l0 = level[i0 & 0xFFFFu];
        const uint32_t r1 = run[i1 >> 16], l1 = level[i1 & 0xFFFFu];
        uint32_t len0 = (r0 >> 24) + (l0 >> 24), len1 = (r1 >> 24) + (l1 >> 24);
        const bool long0 = n > 0 && (r0 == 0 || l0 == 0), long1 = n > 1 && (r1 == 0 || l1 == 0);
        len0 = n > 0 ? len0 : 0u;
        len1 = n > 1 ? len1 : 0u;
        // Codes of the tables: at most 28 bits, and mostly two in 32.
        const uint32_t v0 = (((r0 & 0xFFFFFFu) << (l0 >> 24)) | (l0 & 0xFFFFFFu)) + sign0;
        const uint32_t v1 = n > 1 ? (((r1 & 0xFFFFFFu) << (l1 >> 24)) | (l1 & 0xFFFFFFu)) + sign1 : 0u;
        if (!__any_sync(0xffffffffu, len0 + len1 > 32u || long0 || long1)) {
            w.put32(w.place(len0 + len1), (v0 << len1) | v1, len0 + len1);
        } else {
            uint64_t w0 = v0, w1 = v1;
            if (long0) w0 = long_code(c.x, b.y, b.x, len0);
            if (long1) w1 = long_code(c.y, c.x, b.y, len1);
            const uint32_t at = w.place(len0 + len1);
            w.put(at, w0, len0);
            w.put(at + len0, w1, len1);
        }
        w.drain();
    }
};

// The AC codes of a component with levels of any size. A level's code and sign
// are at most 64 bits, |F| of 16-bit samples staying below 2^21.
__device__ __noinline__ WarpBits warp_wide_write(WarpBits w, const float *f, const float *inv, uint32_t n_blocks) {
    warp_wide_codes<false>(f, inv, n_blocks, [&](bool coded, uint32_t run, uint32_t level, bool neg, uint32_t prev_run,
                                                 uint32_t prev_level) {
        const Codebook rb = run_book(prev_run), lb = level_book(prev_level);
        const uint32_t rlen = coded ? cb_len32(rb, run) : 0u, llen = coded ? cb_len32(lb, level) + 1u : 0u;
        const uint32_t at = w.place(rlen + llen);
        w.put(at, coded ? cb_bits(rb, run) : 0u, rlen);
        w.put(at + rlen, coded ? (cb_bits(lb, level) << 1) | (uint64_t)neg : 0u, llen);
        w.drain();
    });
    return w;
}

// Each slice component's codes (src/encode.rs:413-437), a warp each, taken as
// by k_cost: the non-zeros are gathered as for counting, and their codes
// placed 64 at a time.
//
// Bound by issue (72 % of the slots, 51 warp instructions for 32 coefficients
// at 36 % non-zeros). A lane per component, writing bit by bit into words it
// OR-ed to memory, took 1390 us for 30 UHD frames, 636 for 30 1080p and 474
// for one UHD frame (a lane's walk from end to end): 968, 265 and 50, and from a
// counter instead of the grid's stride 865, 245 and 50. Alpha, whose codes were
// OR-ed into memory one by one, goes through the same words: 8 UHD 4:4:4 frames
// with it 1595 -> 779.
__global__ void __launch_bounds__(kCostThreads, kCostBlocks) k_pack(EncodeLaunch e, uint32_t take) {
    chain_start();
    __shared__ __align__(16) PackTables t;
    __shared__ __align__(8) uint32_t buf[kCostThreads / 32][kCountWords];
    __shared__ uint32_t words[kCostThreads / 32][kPackWords];
    t.fill();
    chain_wait();
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t items = 3u * e.n_slices;
    WarpBits w;
    w.clear(words[warp]);
    const uint32_t warps = gridDim.x * (kCostThreads / 32);
    const bool ahead = items > kGrabAhead * warps;
    uint32_t grab = (blockIdx.x * (kCostThreads / 32) + (threadIdx.x >> 5)) * take;
    for (;;) {
        const uint32_t base = __shfl_sync(0xffffffffu, grab, 0);
        if (base >= items) break;
        if (ahead && lane == 0) grab = warps * take + atomicAdd(e.pack_taken, take);
        // This lane's item, as in k_cost, and the bit its codes start at.
        const uint32_t item = base + lane;
        uint32_t my_coef = 0, my_quant = 0, my_blocks = 0;
        uint64_t my_at = 0;
        if (lane < take && item < items) {
            const uint32_t comp = item < e.n_slices ? 0u : (item < 2u * e.n_slices ? 1u : 2u);
            const uint32_t s = item - comp * e.n_slices;
            const EncSliceDesc sd = e.slices[s];
            uint64_t at = e.slice_off[s];
            for (uint32_t c = 0; c < comp; c++) at += e.final_comp[3ull * s + c];
            const EncPicDesc &pd = e.pics[sd.pic];
            at += e.state[sd.pic].pic_off + pd.header_bytes + e.frames[pd.frame].out_base;
            const uint32_t off = comp == 0 ? 0u : 64u * sd.mbs * (4u + (comp - 1u) * sd.cpm);
            my_coef = (uint32_t)((sd.coef + off) >> 6);
            my_quant = ((pd.quant * 225u + e.final_qi[s]) << 1) | (comp > 0 ? 1u : 0u);
            if (e.frame_status[pd.frame] == 0) my_blocks = (comp == 0 ? 4u : sd.cpm) * sd.mbs;
            my_at = 8ull * at;
        }
        CompHead next_head{};
        uint32_t next_blocks = 0;
        uint64_t next_coef = 0;
        const auto look = [&](uint32_t j) {
            next_coef = (uint64_t)__shfl_sync(0xffffffffu, my_coef, j) << 6;
            next_blocks = __shfl_sync(0xffffffffu, my_blocks, j);
            next_head = comp_head<false>(e.coef + next_coef, e.coef_max + (next_coef >> 5), next_blocks);
        };
        uint32_t left = __ballot_sync(0xffffffffu, my_blocks != 0);
        if (left) look((uint32_t)__ffs(left) - 1u);
        while (left) {
            const uint32_t j = (uint32_t)__ffs(left) - 1u;
            left &= left - 1u;
            const CompHead h = next_head;
            const uint32_t nb = next_blocks;
            const uint64_t coef = next_coef;
            if (left) look((uint32_t)__ffs(left) - 1u);
            const uint32_t quant = __shfl_sync(0xffffffffu, my_quant, j);
            const uint64_t at = __shfl_sync(0xffffffffu, my_at, j);
            const CompQuant cq = comp_quant(e.quant + (uint64_t)(quant >> 1) * kQuantStride, quant & 1u, nb);
            const float *f = e.coef + coef;
            w.start(e.out, at);
            uint32_t live_lo, live_hi, a;
            live_chunks(h, nb, cq, live_lo, live_hi);
            const uint32_t symbol = dc_symbol(h.dc, __ldg(cq.inv), a);
            const uint32_t len = lane < nb ? dc_len(a, symbol) : 0u;
            // The code's significant bits: n + 2^k of EGk; the codebook for a
            // difference of 2 has (n & 3) + 4 below 8, from there on n itself.
            const uint32_t code = a == 2u ? (symbol < 8u ? (symbol & 3u) + 4u : symbol) : symbol + (1u << a);
            w.put(w.place(len), code, len);
            w.drain();
            if (__any_sync(0xffffffffu, fmaxf(h.max_lo, h.max_hi) >= kWideCoef)) {
                w = warp_wide_write(w, f, cq.inv, nb);
            } else {
                PackSink sink{t, w};
                warp_nonzeros<false>(f, cq.inv, nb, live_lo, live_hi, sink, buf[warp]);
            }
            w.finish();
        }
        if (!ahead && lane == 0) grab = warps * take + atomicAdd(e.pack_taken, take);
    }
}

// A slice's alpha codes, the whole warp, a run and its difference a lane.
__device__ void alpha_write(const EncodeLaunch &e, const EncSliceDesc &sd, const EncPicDesc &pd,
                            const EncFrameDesc &fd, AlphaScratch &sc, uint32_t *words, uint64_t bitpos) {
    const int lane = threadIdx.x & 31;
    const uint32_t n_runs = alpha_runs(e, sd, pd, fd, sc);
    const uint32_t bits = fd.alpha_bits;
    const uint32_t max = bits == 8 ? 8u : 64u;
    WarpBits w;
    w.clear(words);
    w.start(e.out, bitpos);
    for (uint32_t base = 0; base < n_runs; base += 32) {
        const uint32_t j = base + lane;
        uint32_t dlen = 0, len = 0;
        if (j < n_runs) len = alpha_run_bits(sc, j, bits, dlen);
        uint64_t field = 0;
        if (j < n_runs) {
            const int32_t prev = j ? (int32_t)sc.value[j - 1] : -1;
            const int32_t diff = (int32_t)sc.value[j] - prev;
            const uint32_t a = diff < 0 ? 0u - (uint32_t)diff : (uint32_t)diff;
            // Tables 13/14: `0`, |d| - 1, sign; or `1` and d mod 2^bits.
            if (a >= 1u && a <= max)
                field = ((a - 1u) << 1) | (uint32_t)(diff < 0);
            else
                field = (1u << bits) | ((uint32_t)diff & ((1u << bits) - 1u));
            // Table 12: `1`; `0` and 4 bits of run - 1; or 5 zeros and 11 bits.
            const uint32_t run = (uint32_t)sc.start[j + 1] - sc.start[j];
            field = (field << (len - dlen)) | (run == 1u ? 1u : run - 1u);
        }
        w.put(w.place(len), field, len);
        w.drain();
    }
    w.finish();
}

// Slice headers and table entries, one thread per slice; alpha codes, one
// warp per slice.
__global__ void k_pack_headers(EncodeLaunch e) {
    chain_start();
    chain_wait();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= e.n_slices) return;
    const EncSliceDesc sd = e.slices[s];
    const EncPicDesc &pd = e.pics[sd.pic];
    if (e.frame_status[pd.frame]) return;
    const EncFrameDesc &fd = e.frames[pd.frame];
    const EncPicState &st = e.state[sd.pic];
    const uint32_t comp[3] = {e.final_comp[3ull * s], e.final_comp[3ull * s + 1], e.final_comp[3ull * s + 2]};
    const uint32_t hb = pd.header_bytes;
    const uint64_t slice_bit = 8ull * (fd.out_base + st.pic_off + e.slice_off[s]);
    bool f;
    const uint64_t total = slice_total(hb, comp, e.alpha_bytes[s], f);
    // slice_header_size << 3, quantization_index, the component sizes (the
    // Cr size only with alpha); the slice table's entry.
    put_field(e.out, slice_bit, hb << 3, 8);
    put_field(e.out, slice_bit + 8, e.final_qi[s], 8);
    put_field(e.out, slice_bit + 16, comp[0] & 0xFFFFu, 16);
    put_field(e.out, slice_bit + 32, comp[1] & 0xFFFFu, 16);
    if (hb == 8) put_field(e.out, slice_bit + 48, comp[2] & 0xFFFFu, 16);
    const uint64_t table_bit = 8ull * (fd.out_base + st.pic_off + 8u + 2ull * (s - pd.slice_base));
    put_field(e.out, table_bit, (uint32_t)(total & 0xFFFFu), 16);
}

__global__ void __launch_bounds__(32 * kAlphaWarps) k_pack_alpha(EncodeLaunch e) {
    chain_start();
    chain_wait();
    __shared__ AlphaScratch scratch[kAlphaWarps];
    __shared__ uint32_t words[kAlphaWarps][kPackWords];
    const uint32_t s = blockIdx.x * kAlphaWarps + (threadIdx.x >> 5);
    if (s >= e.n_slices) return;
    const EncSliceDesc sd = e.slices[s];
    const EncPicDesc &pd = e.pics[sd.pic];
    const EncFrameDesc &fd = e.frames[pd.frame];
    if (!fd.alpha_bits || e.frame_status[pd.frame]) return;
    const EncPicState &st = e.state[sd.pic];
    const uint32_t *c = e.final_comp + 3ull * s;
    const uint64_t at = 8ull * (fd.out_base + st.pic_off + e.slice_off[s] + pd.header_bytes + c[0] + c[1] + c[2]);
    alpha_write(e, sd, pd, fd, scratch[threadIdx.x >> 5], words[threadIdx.x >> 5], at);
}

}  // namespace

cudaError_t launch_quant(float *quant, const uint8_t *keys, uint32_t sets, cudaStream_t s) {
    k_quant<<<225u * sets, 128, 0, s>>>(quant, keys);
    return cudaGetLastError();
}

cudaError_t launch_fdct(const EncodeLaunch &e, cudaStream_t s) {
    if (!e.n_slices) return cudaSuccess;
    return launch_chained(k_fdct, (e.n_fdct_items + kFdctWarps - 1) / kFdctWarps, 32 * kFdctWarps,
                          kFdctWarps * sizeof(FdctWarp), s, e);
}

cudaError_t launch_alpha_size(const EncodeLaunch &e, cudaStream_t s) {
    if (!e.n_slices) return cudaSuccess;
    if (!e.any_alpha) return cudaSuccess;  // alpha_bytes is zeroed beforehand
    return launch_chained(k_alpha_size, (e.n_slices + kAlphaWarps - 1) / kAlphaWarps, 32 * kAlphaWarps, 0, s, e);
}

// A picture's threads in the bisection step: as many as leave every picture's
// block a place (2048 threads an SM), since more go through its slices sooner
// (9 steps of 30 UHD frames 162 us with 256, 107 with 1024) and blocks that wait
// for a place cost all of them a round (4,096 frames of 16x16 72 us a step with
// 1024 threads each, 10 with 64; 131,072 of them 2230 and 141).
static uint32_t rc_threads(const EncodeLaunch &e) {
    uint32_t threads = kRcThreads;
    while (threads > kRcThreadsMin && (uint64_t)threads * e.n_pics > 2048ull * (uint32_t)e.sm_count) threads /= 2;
    return threads;
}

cudaError_t launch_rc_init(const EncodeLaunch &e, cudaStream_t s) {
    if (!e.n_pics) return cudaSuccess;
    return launch_chained(k_rc_init, e.n_pics, rc_threads(e), 0, s, e);
}

// CTAs of a kernel that walks `items` warp items at a stride: all that are
// resident, or what the items need.
static uint32_t cost_grid(const EncodeLaunch &e, uint32_t items) {
    return std::min<uint32_t>((items + kCostThreads / 32 - 1) / (kCostThreads / 32), (uint32_t)(kCostBlocks * e.sm_count));
}

// Items a warp takes at once: enough to share the look-ups, few enough that
// the last ones do not hold the launch up (a component takes a warp about 6 us
// when all warps are busy).
static uint32_t cost_take(const EncodeLaunch &e, uint32_t items) {
    const uint32_t warps = (uint32_t)(kCostBlocks * e.sm_count) * (kCostThreads / 32);
    return std::max(1u, std::min(kCostTake, items / (8u * warps)));
}

cudaError_t launch_cost(const EncodeLaunch &e, int step, cudaStream_t s) {
    if (!e.n_slices) return cudaSuccess;
    const uint32_t items = 3u * e.n_slices;
    return launch_chained(k_cost, cost_grid(e, items), kCostThreads, 0, s, e, step, cost_take(e, items));
}

cudaError_t launch_rc_step(const EncodeLaunch &e, int step, cudaStream_t s) {
    if (!e.n_pics) return cudaSuccess;
    return launch_chained(k_rc_step, e.n_pics, rc_threads(e), 0, s, e, step);
}

cudaError_t launch_cost_window(const EncodeLaunch &e, int level, cudaStream_t s) {
    if (!e.n_slices) return cudaSuccess;
    const uint32_t items = 3u * e.n_slices;
    cudaError_t err =
        launch_chained(k_window_select, (e.n_slices + kCostThreads - 1) / kCostThreads, kCostThreads, 0, s, e, level);
    if (err != cudaSuccess) return err;
    // Blocks past the list's end return.
    return launch_chained(k_cost_window, cost_grid(e, items), kCostThreads, 0, s, e, level);
}

cudaError_t launch_cost_deep(const EncodeLaunch &e, cudaStream_t s) {
    if (!e.n_slices) return cudaSuccess;
    cudaError_t err = launch_chained(k_deep_select, (e.n_slices + kCostThreads - 1) / kCostThreads, kCostThreads, 0, s, e);
    if (err != cudaSuccess) return err;
    return launch_chained(k_cost_deep, (uint32_t)(kDeepBlocks * e.sm_count), kDeepThreads, 0, s, e);
}

cudaError_t launch_shareout(const EncodeLaunch &e, cudaStream_t s) {
    if (!e.n_pics) return cudaSuccess;
    cudaError_t err = launch_chained(k_share_prep, (e.n_slices + 255) / 256, 256, 0, s, e);
    if (err != cudaSuccess) return err;
    err = launch_chained(k_shareout, e.n_pics, kShareThreads, sizeof(ShareShared), s, e);
    if (err != cudaSuccess) return err;
    return launch_chained(k_share_final, (e.n_slices + 255) / 256, 256, 0, s, e);
}

cudaError_t launch_layout(const EncodeLaunch &e, cudaStream_t s) {
    cudaError_t err = e.n_pics ? launch_chained(k_layout, e.n_pics, kLayoutThreads, 0, s, e) : cudaSuccess;
    if (err != cudaSuccess || !e.n_frames) return err;
    return launch_chained(k_frame, (e.n_frames + 127) / 128, 128, 0, s, e);
}

cudaError_t launch_pack(const EncodeLaunch &e, cudaStream_t s) {
    if (!e.n_slices) return cudaSuccess;
    const uint32_t items = 3u * e.n_slices;
    cudaError_t err = launch_chained(k_pack, cost_grid(e, items), kCostThreads, 0, s, e, cost_take(e, items));
    if (err != cudaSuccess) return err;
    err = launch_chained(k_pack_headers, (e.n_slices + 255) / 256, 256, 0, s, e);
    if (err != cudaSuccess || !e.any_alpha) return err;
    return launch_chained(k_pack_alpha, (e.n_slices + kAlphaWarps - 1) / kAlphaWarps, 32 * kAlphaWarps, 0, s, e);
}

cudaError_t configure_encode_kernels() {
    static_assert(sizeof(FdctWarp) % 16 == 0, "the warps' areas are 16-byte aligned");
    cudaError_t err0 = cudaFuncSetAttribute(k_shareout, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)sizeof(ShareShared));
    if (err0 != cudaSuccess) return err0;
    CountTables tables;
    build_count_tables(tables);
    if ((err0 = cudaMemcpyToSymbol(d_count_tables, &tables, sizeof tables)) != cudaSuccess) return err0;
    PackTables codes;
    build_pack_tables(codes);
    if ((err0 = cudaMemcpyToSymbol(d_pack_tables, &codes, sizeof codes)) != cudaSuccess) return err0;
    float basis[64];
    dct_basis(basis);
    cudaError_t err = cudaMemcpyToSymbol(c_fdct_basis, basis, sizeof basis);
    if (err != cudaSuccess) return err;
    uint8_t sc[2][64];
    for (int i = 0; i < 64; i++) {
        sc[0][i] = kProgressiveScan[i];
        sc[1][i] = kInterlacedScan[i];
    }
    return cudaMemcpyToSymbol(c_enc_scan, sc, sizeof sc);
}

}  // namespace prores
