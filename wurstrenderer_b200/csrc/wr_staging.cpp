#include "wr_staging.h"

#include <algorithm>
#include <cstring>

namespace wr {

std::shared_ptr<Staging> Staging::shared() {
    static std::mutex m;
    static std::weak_ptr<Staging> last;
    std::lock_guard<std::mutex> lock(m);
    std::shared_ptr<Staging> s = last.lock();
    if (!s) {
        s.reset(new Staging());
        last = s;
    }
    return s;
}

Staging::~Staging() {
    {
        std::lock_guard<std::mutex> lock(m_);
        stop_ = true;
    }
    start_.notify_all();
    for (std::thread &t : threads_) t.join();
    if (pinned_) cudaFreeHost(pinned_);
}

// makes the buffers and threads once; false while the large copies so far, `bytes` more with this one, are
// not worth them, and when they cannot be had
bool Staging::prepare(size_t bytes) {
    if (pinned_) return true;
    copied_ += bytes;
    if (copied_ <= kPrepareAfter) return false;
    void *p = nullptr;
    if (cudaHostAlloc(&p, 2 * kThreads * kPiece, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();   // out of pinned memory: the driver copies
        return false;
    }
    pinned_ = static_cast<char *>(p);
    // as many threads as half the cores take, so that a small machine keeps some for its own work
    const int others = std::min<int>(kThreads, std::max(2u, std::thread::hardware_concurrency() / 2)) - 1;
    try {
        for (int k = 1; k <= others; ++k) threads_.emplace_back([this, k] { work(k); });
    } catch (...) {
        // fewer threads than wanted share the work
    }
    return true;
}

void Staging::work(int k) {
    int seen = 0;
    std::unique_lock<std::mutex> lock(m_);
    while (true) {
        start_.wait(lock, [&] { return stop_ || turn_ != seen; });
        if (stop_) return;
        seen = turn_;
        if (k >= wanted_) continue;
        lock.unlock();
        task_(k);
        lock.lock();
        if (--running_ == 0) done_.notify_one();
    }
}

// pieces k, k + parts, ... of the copy, through this share's two pinned buffers
cudaError_t Staging::share(int k, int parts, bool up, char *host, char *dev, size_t bytes, cudaStream_t st, int device) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    char *buf[2] = {pinned_ + size_t(2 * k) * kPiece, pinned_ + size_t(2 * k + 1) * kPiece};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (cudaEvent_t &v : ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    const size_t pieces = (bytes + kPiece - 1) / kPiece;
    struct Flight { size_t piece; bool live; } flight[2] = {{0, false}, {0, false}};
    auto size_of = [&](size_t i) { return std::min(kPiece, bytes - i * kPiece); };
    // waits for a buffer's piece and, on the way to the host, copies it out
    auto finish = [&](int b) {
        if (!flight[b].live) return;
        flight[b].live = false;
        const cudaError_t w = cudaEventSynchronize(ev[b]);
        if (e == cudaSuccess) e = w;
        if (!up && w == cudaSuccess) memcpy(host + flight[b].piece * kPiece, buf[b], size_of(flight[b].piece));
    };
    int b = 0;
    for (size_t i = size_t(k); i < pieces && e == cudaSuccess; i += size_t(parts), b ^= 1) {
        finish(b);
        if (e != cudaSuccess) break;
        if (up) {
            memcpy(buf[b], host + i * kPiece, size_of(i));
            e = cudaMemcpyAsync(dev + i * kPiece, buf[b], size_of(i), cudaMemcpyHostToDevice, st);
        } else {
            e = cudaMemcpyAsync(buf[b], dev + i * kPiece, size_of(i), cudaMemcpyDeviceToHost, st);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
        if (e == cudaSuccess) flight[b] = {i, true};
    }
    finish(b);       // the older piece first
    finish(b ^ 1);
    // after an error a piece without an event may still be on the bus: its buffer is free with the stream
    if (e != cudaSuccess) cudaStreamSynchronize(st);
    for (cudaEvent_t v : ev)
        if (v) cudaEventDestroy(v);
    return e;
}

cudaError_t Staging::copy(bool up, char *host, char *dev, size_t bytes, cudaStream_t st) {
    const cudaMemcpyKind kind = up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    void *to = up ? dev : host;
    const void *from = up ? host : dev;
    bool direct = bytes < kDirectBytes;
    if (!direct) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
            cudaGetLastError();
            direct = true;
        } else {
            direct = a.type != cudaMemoryTypeUnregistered;   // pinned or managed
        }
    }
    std::unique_lock<std::mutex> lock(use_, std::defer_lock);
    if (direct || !lock.try_lock() || !prepare(bytes)) return cudaMemcpyAsync(to, from, bytes, kind, st);
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const size_t pieces = (bytes + kPiece - 1) / kPiece;
    const int parts = int(std::min<size_t>(threads_.size() + 1, pieces));
    std::vector<cudaError_t> result(size_t(parts), cudaSuccess);
    {
        std::lock_guard<std::mutex> l(m_);
        task_ = [&](int k) { result[size_t(k)] = share(k, parts, up, host, dev, bytes, st, device); };
        wanted_ = parts;
        running_ = parts - 1;
        ++turn_;
    }
    start_.notify_all();
    result[0] = share(0, parts, up, host, dev, bytes, st, device);
    {
        std::unique_lock<std::mutex> l(m_);
        done_.wait(l, [&] { return running_ == 0; });
        task_ = nullptr;
    }
    for (cudaError_t r : result)
        if (e == cudaSuccess) e = r;
    return e;
}

cudaError_t Staging::to_host(void *host, const void *dev, size_t bytes, cudaStream_t st) {
    return copy(false, static_cast<char *>(host), static_cast<char *>(const_cast<void *>(dev)), bytes, st);
}

cudaError_t Staging::to_device(void *dev, const void *host, size_t bytes, cudaStream_t st) {
    return copy(true, static_cast<char *>(const_cast<void *>(host)), static_cast<char *>(dev), bytes, st);
}

}  // namespace wr
