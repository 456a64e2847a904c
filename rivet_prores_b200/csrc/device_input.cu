// Frames that arrive as a MOV (or a run of MOV samples) and frames that
// already lie in device memory.
//
// The crate finds whole frames in a file without parsing the container
// (tests/sample.rs:20-38, examples/prores_bench.rs:103-121): at each byte
// position i from 4, the four bytes "icpf" with a big-endian frame_size of
// at least 28 at i - 4 that ends inside the data are a frame, and the scan
// resumes where that frame ends; anything else moves on by one byte.
// prores_scan_frames restates that walk on the host. On the device a kernel
// finds every "icpf" at once (all candidates, whatever frame they fall in),
// and the host resolves them in position order with the same rule, which
// gives the same frames: a candidate inside an accepted frame is exactly one
// the sequential walk never reaches.
//
// prores_decode_device then decodes such frames where they lie: the host
// fetches only the header bytes it plans with (the frame header, then each
// picture header), the bitstreams are copied device to device into the
// workspace's padded buffer, and the kernels write the planes straight into
// the caller's device buffers.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "engine.h"

#define PR_CUDA(expr, what)                     \
    do {                                        \
        Status st_ = cuda_status((expr), what); \
        if (st_) return st_;                    \
    } while (0)

namespace prores {
namespace {

constexpr int kScanThreads = 256;
constexpr uint32_t kScanSpan = 16;  // positions a thread checks

__device__ __forceinline__ uint8_t byte_at(const uint8_t *data, uint64_t i) { return __ldg(data + i); }

// Every position i (4 <= i, i + 4 <= len) where "icpf" starts, with the
// big-endian word before it, appended in no particular order.
__global__ void __launch_bounds__(kScanThreads) k_scan_icpf(const uint8_t *data, uint64_t len, uint64_t *pos,
                                                            uint32_t *size, unsigned int *count, uint32_t cap) {
    const uint64_t t = (uint64_t)blockIdx.x * kScanThreads + threadIdx.x;
    const uint64_t lo = max((uint64_t)4, t * kScanSpan);
    const uint64_t hi = min(t * kScanSpan + kScanSpan, len >= 3 ? len - 3 : 0);  // i + 4 <= len
    for (uint64_t i = lo; i < hi; i++) {
        if (byte_at(data, i) != 'i' || byte_at(data, i + 1) != 'c' || byte_at(data, i + 2) != 'p' ||
            byte_at(data, i + 3) != 'f')
            continue;
        const uint32_t sz = ((uint32_t)byte_at(data, i - 4) << 24) | ((uint32_t)byte_at(data, i - 3) << 16) |
                            ((uint32_t)byte_at(data, i - 2) << 8) | (uint32_t)byte_at(data, i - 1);
        const unsigned int k = atomicAdd(count, 1u);
        if (k < cap) {
            pos[k] = i;
            size[k] = sz;
        }
    }
}

// The crate's acceptance rule for the "icpf" at i with frame_size `size`.
bool accepted(uint64_t i, uint64_t size, uint64_t len) { return size >= 28 && i - 4 + size <= len; }

size_t resolve(std::vector<std::pair<uint64_t, uint32_t>> &cand, uint64_t len, prores_span *out, size_t cap) {
    std::sort(cand.begin(), cand.end());
    size_t n = 0;
    uint64_t next = 4;  // the sequential walk's position
    for (const auto &c : cand) {
        if (c.first < next || !accepted(c.first, c.second, len)) continue;
        if (n < cap) out[n] = prores_span{(size_t)(c.first - 4), (size_t)c.second};
        n++;
        next = c.first - 4 + c.second;
    }
    return n;
}

int fail_status(const Status &s) {
    set_last_error(s);
    return s.code;
}

Status check_spans(const prores_span *frames, int n, size_t data_len) {
    for (int i = 0; i < n; i++)
        if (frames[i].offset > data_len || frames[i].len > data_len - frames[i].offset)
            return make_status(PRORES_CONFIG, strf("frame %d lies outside the %zu bytes given", i, data_len));
    return Status();
}

// The header bytes planning reads of a frame: the frame header, then the
// header of each picture, side by side (zero where the frame is shorter).
struct HeadSlot {
    uint8_t head[kFrameHeadBytes];
    uint8_t pic[2][kPictureHeaderSize];
};
constexpr int kHeadBatch = 64;  // frames a launch, their spans passed as its argument
struct HeadSpans {
    prores_span span[kHeadBatch];
};

// A warp per frame gathers its slot, walking to the picture headers as
// plan_decode does: the first after the frame header, the second after the
// first picture. `out` is page-locked host memory, which the warps write
// themselves: one launch and one wait for what took a copy a frame in each
// of three rounds (32 frames: about 100 us a round, probing and decoding).
__global__ void __launch_bounds__(32 * 4) k_gather_heads(const uint8_t *data, HeadSpans spans, int n, HeadSlot *out) {
    const int i = (int)(blockIdx.x * 4 + (threadIdx.x >> 5));
    const uint32_t lane = threadIdx.x & 31u;
    if (i >= n) return;
    const uint8_t *frame = data + spans.span[i].offset;
    const uint64_t len = spans.span[i].len;
    const auto at = [&](uint64_t pos) -> uint32_t { return pos < len ? byte_at(frame, pos) : 0u; };
    for (uint32_t k = lane; k < kFrameHeadBytes; k += 32u) out[i].head[k] = (uint8_t)at(k);
    uint64_t pos = 8u + ((at(8) << 8) | at(9));
    for (int p = 0; p < 2; p++) {
        if (lane < kPictureHeaderSize) out[i].pic[p][lane] = (uint8_t)at(pos + lane);
        pos += ((uint64_t)at(pos + 1) << 24) | (at(pos + 2) << 16) | (at(pos + 3) << 8) | at(pos + 4);
    }
}

// The header bytes of every frame of a call, fetched from device memory.
struct DeviceHeads {
    std::vector<HeadSlot> slots;
    std::vector<size_t> lens;

    Status fetch(Workspace &ws, const uint8_t *d_data, const prores_span *frames, int n, cudaStream_t s) {
        slots.resize(n);
        lens.resize(n);
        if (!n) return Status();
        PR_CUDA(ws.host_small.reserve(sizeof(HeadSlot) * n), "cudaMallocHost");
        HeadSlot *host = static_cast<HeadSlot *>(ws.host_small.p);
        for (int first = 0; first < n; first += kHeadBatch) {
            const int count = std::min(kHeadBatch, n - first);
            HeadSpans spans{};
            std::copy(frames + first, frames + first + count, spans.span);
            k_gather_heads<<<(count + 3) / 4, 32 * 4, 0, s>>>(d_data, spans, count, host + first);
            PR_CUDA(cudaGetLastError(), "k_gather_heads");
        }
        Status w = wait_stream(s, ws.wait_ms, "header fetch");
        if (w) return w;
        std::copy(host, host + n, slots.begin());
        for (int i = 0; i < n; i++) lens[i] = frames[i].len;
        return Status();
    }

    const uint8_t *head(int i) const { return slots[i].head; }

    // Bytes [pos, pos + len) of frame i, if a slot holds them.
    const uint8_t *bytes(int i, size_t pos, size_t len) const {
        const HeadSlot &slot = slots[i];
        if (pos > lens[i] || len > lens[i] - pos) return nullptr;
        if (pos == 0 && len <= sizeof slot.head) return slot.head;
        size_t at = 8 + (((size_t)slot.head[8] << 8) | slot.head[9]);
        for (const uint8_t *p : {slot.pic[0], slot.pic[1]}) {
            if (pos == at && len <= kPictureHeaderSize) return p;
            at += ((size_t)p[1] << 24) | ((size_t)p[2] << 16) | ((size_t)p[3] << 8) | p[4];
        }
        return len == 0 ? slot.head : nullptr;
    }
};

}  // namespace
}  // namespace prores

using namespace prores;

extern "C" {

size_t prores_scan_frames(const uint8_t *data, size_t len, prores_span *frames, size_t cap) {
    size_t n = 0;
    size_t i = 4;
    while (data && i + 4 <= len) {
        if (memcmp(data + i, "icpf", 4) == 0) {
            const uint64_t size = ((uint64_t)data[i - 4] << 24) | ((uint64_t)data[i - 3] << 16) |
                                  ((uint64_t)data[i - 2] << 8) | (uint64_t)data[i - 1];
            if (accepted(i, size, len)) {
                if (n < cap) frames[n] = prores_span{i - 4, (size_t)size};
                n++;
                i += size - 4;
                continue;
            }
        }
        i++;
    }
    return n;
}

int prores_scan_frames_device(prores_ctx *ctx, const uint8_t *d_data, size_t len, prores_span *frames, size_t cap,
                              size_t *count, void *stream) {
    if (!ctx || (!d_data && len) || !count) return fail_status(make_status(PRORES_CONFIG, "no context or data"));
    cudaSetDevice(ctx->impl.device);
    auto ws = ctx->impl.acquire();
    if (!ws) return fail_status(make_status(PRORES_DEVICE, "no stream"));
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ws->stream;
    Status st;
    uint32_t room = 1u << 16;
    std::vector<std::pair<uint64_t, uint32_t>> cand;
    for (int attempt = 0; attempt < 2 && !st; attempt++) {
        // Candidate positions, their words, and the counter.
        st = cuda_status(ws->slices.reserve((size_t)room * 12 + 64), "cudaMalloc");
        if (st) break;
        uint64_t *pos = ws->slices.as<uint64_t>();
        uint32_t *size = reinterpret_cast<uint32_t *>(pos + room);
        unsigned int *counter = reinterpret_cast<unsigned int *>(size + room);
        st = cuda_status(cudaMemsetAsync(counter, 0, sizeof(unsigned int), s), "memset");
        const uint64_t threads = len / kScanSpan + 1;
        const uint64_t blocks = (threads + kScanThreads - 1) / kScanThreads;
        if (!st && len >= 8) {
            k_scan_icpf<<<(unsigned int)blocks, kScanThreads, 0, s>>>(d_data, len, pos, size, counter, room);
            st = cuda_status(cudaGetLastError(), "k_scan_icpf");
        }
        if (!st) st = cuda_status(ws->host_small.reserve((size_t)room * 12 + 64), "cudaMallocHost");
        if (st) break;
        uint8_t *host = static_cast<uint8_t *>(ws->host_small.p);
        unsigned int found = 0;
        st = cuda_status(cudaMemcpyAsync(host, counter, sizeof found, cudaMemcpyDeviceToHost, s), "scan");
        if (!st) st = wait_stream(s, ws->wait_ms, "scan");
        if (st) break;
        memcpy(&found, host, sizeof found);
        if (found > room) {  // more candidates than room: once more with room for all
            room = found;
            continue;
        }
        if (found) {
            st = cuda_status(cudaMemcpyAsync(host, pos, 8ull * found, cudaMemcpyDeviceToHost, s), "scan");
            if (!st)
                st = cuda_status(cudaMemcpyAsync(host + 8ull * found, size, 4ull * found, cudaMemcpyDeviceToHost, s),
                                 "scan");
            if (!st) st = wait_stream(s, ws->wait_ms, "scan");
            if (st) break;
            cand.resize(found);
            for (unsigned int k = 0; k < found; k++) {
                memcpy(&cand[k].first, host + 8ull * k, 8);
                memcpy(&cand[k].second, host + 8ull * found + 4ull * k, 4);
            }
        }
        *count = resolve(cand, len, frames, cap);
        break;
    }
    ctx->impl.release_or_retire(std::move(ws));
    return st ? fail_status(st) : PRORES_OK;
}

int prores_probe_device(prores_ctx *ctx, const uint8_t *d_data, size_t data_len, const prores_span *frames, int n,
                        uint32_t out_bit_depth, prores_frame *info, int *status) {
    if (!ctx || n < 0 || (n && (!frames || !info || !status)))
        return fail_status(make_status(PRORES_CONFIG, "no context or frames"));
    Status st = check_spans(frames, n, data_len);
    if (st) return fail_status(st);
    cudaSetDevice(ctx->impl.device);
    auto ws = ctx->impl.acquire();
    if (!ws) return fail_status(make_status(PRORES_DEVICE, "no stream"));
    DeviceHeads heads;
    st = heads.fetch(*ws, d_data, frames, n, ws->stream);
    ctx->impl.release_or_retire(std::move(ws));
    if (st) return fail_status(st);
    std::vector<Status> errs(n);
    for (int i = 0; i < n; i++) {
        errs[i] = probe_frame(heads.head(i), frames[i].len, out_bit_depth, &info[i]);  // reads the frame header only
        status[i] = errs[i].code;
    }
    set_batch_errors(errs);
    return PRORES_OK;
}

int prores_decode_device(prores_ctx *ctx, const uint8_t *d_data, size_t data_len, const prores_span *frames, int n,
                         uint32_t out_bit_depth, prores_frame *out, int *status, void *stream) {
    if (!ctx || n < 0 || (n && (!frames || !out || !status)))
        return fail_status(make_status(PRORES_CONFIG, "no context or frames"));
    Status st = check_spans(frames, n, data_len);
    if (st) return fail_status(st);
    cudaSetDevice(ctx->impl.device);
    auto ws = ctx->impl.acquire();
    if (!ws) return fail_status(make_status(PRORES_DEVICE, "no stream"));
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ws->stream;
    DeviceHeads heads;
    st = heads.fetch(*ws, d_data, frames, n, s);
    DecodePlan plan;
    std::vector<prores_buf> bufs(n);
    for (int i = 0; i < n; i++) bufs[i] = prores_buf{d_data + frames[i].offset, frames[i].len};
    const FrameBytes read = [&](int i, size_t pos, size_t len) { return heads.bytes(i, pos, len); };
    if (!st) st = plan_decode(bufs.data(), n, out_bit_depth, plan, &read);
    // The planes go straight into the caller's device buffers.
    for (int i = 0; i < n && !st; i++) {
        const DecodeFrame &f = plan.frames[i];
        if (f.err || f.desc < 0) continue;
        prores_frame &o = out[i];
        if (!o.data || o.data_len < f.samples || (f.alpha_samples && (!o.alpha || o.alpha_len < f.alpha_samples)))
            st = make_status(PRORES_CONFIG, "an output buffer is smaller than its frame");
        FrameDesc &fd = plan.fdesc[f.desc];
        fd.out_planes = o.data;
        fd.out_alpha = f.alpha_samples ? o.alpha : nullptr;
    }
    plan.planes_total = 0;  // nothing lands in the workspace's plane buffers
    plan.alpha_total = 0;
    if (!st) st = upload_decode(ctx->impl, *ws, plan, s);
    if (!st) st = upload_decode_bits(*ws, plan, bufs.data(), s);
    if (!st) st = enqueue_decode(ctx->impl, *ws, plan, s, nullptr);
    Status first;
    if (!st) st = fetch_decode(*ws, plan, s, out, status, &first, true);
    if (st) {
        ctx->impl.release_or_retire(std::move(ws));
        return fail_status(st);
    }
    ctx->impl.release(std::move(ws));
    if (first) set_last_error(first);
    return PRORES_OK;
}

}  // extern "C"
