// Copies between pageable host memory and the device.
//
// cudaMemcpyAsync stages pageable memory through the driver's pinned buffer with one host
// thread: 17 GB/s, while the link moves 33 (in) to 56 (out).  HostCopier cuts the copies
// into chunks that the caller and two helpers move through pinned buffers of their own, each
// filling (draining) one buffer while the other is in flight.  copy() keeps the driver's
// contract for pageable memory: towards the device it returns once the source may be reused,
// towards the host once the data is there.
// Measured, whole calls (driver's staging -> this): 512x512 Gauss transform, 9.4 MB in and
// 4.2 out, 1.11 -> 0.74 ms; 1024x1024 3.57 -> 1.98; 48 served images, 56 MB each way,
// 9.4 -> 5.6.  Three helpers and more gain nothing and vary more (0.74-1.0 at 512x512).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

namespace pgpu {

struct HostPiece {
    char* dst;
    const char* src;
    size_t bytes;
};

class HostCopier {
public:
    // two threads besides the caller's, which sleep between copies; pinned memory: 2 MB each
    static constexpr int kHelpers = 2;
    explicit HostCopier(int device);
    ~HostCopier();
    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;
    // The pieces in any order on st.  One call at a time (a second caller waits).
    cudaError_t copy(const std::vector<HostPiece>& pieces, cudaMemcpyKind kind, cudaStream_t st);
    // The host side of a copy that copy() takes: ordinary pageable memory.  Pinned, managed
    // and device memory go to cudaMemcpyAsync, which moves them without a host thread.
    static bool pageable(const void* host);
    // enough cores for the helpers: alone, one thread is no faster than the driver's
    static bool available();

private:
    // A copy is cut into about twelve chunks of 512 KB to 1 MB: each costs the stream some
    // 10 us however small it is (48 served images: 64 KB 13 ms, 256 KB 7.6, 512 KB 5.8, 1 MB
    // 5.6), while few large ones leave a helper idle (256x256: 512 KB 0.354 ms, 1 MB 0.390).
    static constexpr size_t kMinChunk = 512 << 10, kMaxChunk = 1024 << 10;
    // a range of device memory and where the host's side of it begins; it may run over
    // several pieces that follow each other on the device
    struct Chunk {
        char* dev;
        size_t bytes, piece, offset;
    };
    struct Lane {
        char* pin[2] = {};
        cudaEvent_t ev[2] = {};
        int k = 0;
    };
    int device_;
    std::mutex call_;                 // held by copy()
    std::mutex mu_;                   // guards the members below
    std::condition_variable start_, done_;
    Lane lanes_[1 + kHelpers];        // [0]: the caller's
    std::vector<std::thread> threads_;
    bool stop_ = false;
    long long seq_ = 0;               // the current copy
    int wanted_ = 0, busy_ = 0;       // helpers it still takes, helpers at work on it
    std::vector<Chunk> chunks_;
    const HostPiece* pieces_ = nullptr;
    cudaMemcpyKind kind_ = cudaMemcpyHostToDevice;
    cudaStream_t st_ = nullptr;
    std::atomic<size_t> next_{0};
    std::atomic<int> err_{0};

    cudaError_t open(Lane& l);
    void helper(int lane);
    void work(Lane& l);
    void host_side(const Chunk& c, char* pin) const;
};

}  // namespace pgpu
