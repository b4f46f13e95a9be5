// ss_stage.cu -- staged copies (see ss_stage.h).
#include "ss_stage.h"

#include "ss_engine.h"
#include "ss_shares.h"

#include <algorithm>
#include <cstring>
#include <thread>

namespace ssb {

namespace {

// Measured with 16 host cores: creating the 3-player turn's session (211 MB of
// leaf values up) 30 ms plain, 27 / 20 / 16.5 / 14.9 / 15.6 with 1 / 2 / 4 / 8
// / 12 threads; its leaf values (126 MB down) 34 ms plain, 24.8 / 17.0 / 12.6 /
// 11.2 / 10.9.  Pieces of 512 KiB or 4 MiB: 17 ms instead of 14.9 up.
constexpr size_t kPiece = size_t(1) << 20;
constexpr int kMaxThreads = 8;
// below this the plain call is as fast as starting threads
constexpr size_t kStageMin = size_t(4) << 20;

enum class Way { up, down };

// One thread's share [0, bytes) through its two pieces of page-locked memory.
cudaError_t move_share(Way way, int device, char *dst, const char *src, size_t bytes, char *buf, cudaStream_t s) {
    cudaError_t e = cudaSetDevice(device);
    cudaEvent_t done[2] = {nullptr, nullptr};
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
    const size_t n = (bytes + kPiece - 1) / kPiece;
    auto size = [&](size_t k) { return std::min(kPiece, bytes - k * kPiece); };
    auto fetch = [&](size_t k) {
        cudaError_t r = cudaMemcpyAsync(buf + (k & 1) * kPiece, src + k * kPiece, size(k), cudaMemcpyDeviceToHost, s);
        return r == cudaSuccess ? cudaEventRecord(done[k & 1], s) : r;
    };
    if (way == Way::down)
        for (size_t k = 0; k < std::min<size_t>(2, n) && e == cudaSuccess; ++k) e = fetch(k);
    for (size_t k = 0; k < n && e == cudaSuccess; ++k) {
        char *b = buf + (k & 1) * kPiece;
        if (way == Way::up) {
            if (k >= 2) e = cudaEventSynchronize(done[k & 1]);
            if (e != cudaSuccess) break;
            std::memcpy(b, src + k * kPiece, size(k));
            e = cudaMemcpyAsync(dst + k * kPiece, b, size(k), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaEventRecord(done[k & 1], s);
        } else {
            e = cudaEventSynchronize(done[k & 1]);
            if (e != cudaSuccess) break;
            std::memcpy(dst + k * kPiece, b, size(k));
            if (k + 2 < n) e = fetch(k + 2);
        }
    }
    // the pieces go back to the pool on return: wait for whatever still uses
    // them, after an error too
    for (int i = 0; i < 2; ++i)
        if (done[i]) {
            const cudaError_t w = cudaEventSynchronize(done[i]);
            if (e == cudaSuccess) e = w;
            cudaEventDestroy(done[i]);
        }
    return e;
}

cudaError_t staged(Way way, void *dst, const void *src, size_t bytes, cudaStream_t s) {
    const int cores = static_cast<int>(std::thread::hardware_concurrency());
    const int nt = std::max(1, std::min({kMaxThreads, cores > 0 ? cores : 1, static_cast<int>(bytes / kStageMin)}));
    char *buf = bytes < kStageMin ? nullptr : static_cast<char *>(host_block_take(2 * kPiece * nt));
    if (!buf) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes,
                                              way == Way::up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, s);
        return e == cudaSuccess && way == Way::down ? cudaStreamSynchronize(s) : e;
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) {
        const size_t share = (bytes / nt + kPiece - 1) / kPiece * kPiece;   // whole pieces; the last takes the rest
        cudaError_t got[kMaxThreads] = {};
        run_shares<kMaxThreads>(nt, [&](int i) {
            const size_t at = std::min(bytes, share * i), end = i + 1 == nt ? bytes : std::min(bytes, share * (i + 1));
            if (at < end)
                got[i] = move_share(way, device, static_cast<char *>(dst) + at, static_cast<const char *>(src) + at,
                                    end - at, buf + 2 * kPiece * i, s);
        });
        for (cudaError_t g : got)
            if (e == cudaSuccess) e = g;
    }
    host_block_give(buf);
    return e;
}

}  // namespace

cudaError_t stage_upload(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    return staged(Way::up, dst, src, bytes, s);
}

cudaError_t stage_download(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    return staged(Way::down, dst, src, bytes, s);
}

}  // namespace ssb
