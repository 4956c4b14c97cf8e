// Large copies between device memory and the caller's pageable memory.
//
// The driver moves pageable memory through a staging buffer of its own on the calling thread: the
// film of a 1024x512 render (12.6 MB) took 1.0 ms that way, the images of 24 jobs (61 MB) 14 ms,
// most of it first touches of a fresh array's pages. Here a few threads share a copy: each stages
// its pieces through pinned memory, one piece on the bus while another is copied in host memory
// (0.5 and 4 ms; a million rays' queries 13.3 -> 6.4 ms, 200,003 guide points 2.3 -> 1.2).
// Pinned memory and copies below kDirectBytes go straight to the driver, and so do the first
// kPrepareAfter bytes of large copies: the buffers and threads take 15 ms to make, which a program that
// loads a scene, renders a frame and ends would pay for nothing (400x300 from a fresh scene: 4.6 ms by
// the driver, 18 with them), and staging saves 0.05 to 0.4 ms a MB.
#pragma once

#include <condition_variable>
#include <cstddef>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

namespace wr {

class Staging {
public:
    // the process's staging buffers and threads (16 MB and up to 7 threads, made when enough has been
    // copied), shared by the scenes that hold the pointer and given back with the last of them
    static std::shared_ptr<Staging> shared();
    ~Staging();

    // Both copy after the work already in `st` and before what it is given next; the host array is
    // complete, or free again, once the caller has waited for `st`.
    cudaError_t to_host(void *host, const void *dev, size_t bytes, cudaStream_t st);
    cudaError_t to_device(void *dev, const void *host, size_t bytes, cudaStream_t st);

private:
    static constexpr int kThreads = 8;                   // the calling thread and up to seven others
    static constexpr size_t kPiece = size_t(1) << 20;    // staged at a time; two per thread
    static constexpr size_t kDirectBytes = size_t(2) << 20;
    static constexpr size_t kPrepareAfter = size_t(64) << 20;

    cudaError_t copy(bool up, char *host, char *dev, size_t bytes, cudaStream_t st);
    cudaError_t share(int k, int parts, bool up, char *host, char *dev, size_t bytes, cudaStream_t st, int device);
    bool prepare(size_t bytes);
    void work(int k);

    std::mutex use_;                     // one copy at a time; another thread's goes to the driver
    size_t copied_ = 0;                  // bytes of large copies before the buffers were made
    char *pinned_ = nullptr;
    std::vector<std::thread> threads_;
    std::mutex m_;
    std::condition_variable start_, done_;
    std::function<void(int)> task_;      // what the threads do in this turn
    int turn_ = 0, wanted_ = 0, running_ = 0;
    bool stop_ = false;
};

}  // namespace wr
