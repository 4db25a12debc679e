#include "host_copy.h"

#include <algorithm>
#include <cstring>

namespace pgpu {

HostCopier::HostCopier(int device) : device_(device) {
    threads_.reserve(kHelpers);
    for (int i = 1; i <= kHelpers; ++i) {
        try {
            threads_.emplace_back([this, i] { helper(i); });
        } catch (...) {   // no more threads to be had: those that run share the work
            break;
        }
    }
}

HostCopier::~HostCopier() {
    {
        std::lock_guard<std::mutex> lk(mu_);
        stop_ = true;
    }
    start_.notify_all();
    for (std::thread& t : threads_) t.join();
    for (Lane& l : lanes_)
        for (int s = 0; s < 2; ++s) {
            if (l.ev[s]) {
                cudaEventSynchronize(l.ev[s]);
                cudaEventDestroy(l.ev[s]);
            }
            if (l.pin[s]) cudaFreeHost(l.pin[s]);
        }
}

bool HostCopier::pageable(const void* host) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

bool HostCopier::available() { return std::thread::hardware_concurrency() >= 4; }

// a lane's buffers and events, made on the first copy that takes it
cudaError_t HostCopier::open(Lane& l) {
    for (int s = 0; s < 2; ++s) {
        cudaError_t e;
        if (!l.pin[s] && (e = cudaHostAlloc((void**)&l.pin[s], kMaxChunk, cudaHostAllocPortable))) {
            l.pin[s] = nullptr;
            return e;
        }
        if (!l.ev[s] && (e = cudaEventCreateWithFlags(&l.ev[s], cudaEventDisableTiming))) {
            l.ev[s] = nullptr;
            return e;
        }
    }
    return cudaSuccess;
}

void HostCopier::helper(int lane) {
    cudaSetDevice(device_);
    long long seen = 0;
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
        start_.wait(lk, [&] { return stop_ || (seq_ != seen && wanted_ > 0); });
        if (stop_) return;
        seen = seq_;
        --wanted_;
        ++busy_;
        lk.unlock();
        if (open(lanes_[lane]) == cudaSuccess) work(lanes_[lane]);
        else cudaGetLastError();   // no buffers: the others do it
        lk.lock();
        if (--busy_ == 0) done_.notify_all();
    }
}

// between a chunk's pinned buffer and the host memory of its pieces
void HostCopier::host_side(const Chunk& c, char* pin) const {
    size_t k = c.piece, o = c.offset;
    for (size_t left = c.bytes; left; ++k, o = 0) {
        const HostPiece& p = pieces_[k];
        const size_t n = std::min(left, p.bytes - o);
        if (kind_ == cudaMemcpyHostToDevice) memcpy(pin, p.src + o, n);
        else memcpy(p.dst + o, pin, n);
        pin += n;
        left -= n;
    }
}

// Takes chunks until none is left.  A chunk that was taken is finished before the return:
// queued on the stream (in), or in place (out).
void HostCopier::work(Lane& l) {
    cudaError_t e = cudaSuccess;
    int pending = -1;            // buffer whose chunk is on its way out
    Chunk out{};
    while (!e) {
        const size_t i = next_.fetch_add(1);
        const bool more = i < chunks_.size() && !err_.load();
        const int s = l.k;
        if (more) {
            const Chunk& c = chunks_[i];
            l.k ^= 1;
            // the buffer's last copy is over, also one on another stream (an event never
            // recorded is complete)
            if ((e = cudaEventSynchronize(l.ev[s]))) break;
            if (kind_ == cudaMemcpyHostToDevice) {
                host_side(c, l.pin[s]);
                if ((e = cudaMemcpyAsync(c.dev, l.pin[s], c.bytes, kind_, st_))) break;
            } else if ((e = cudaMemcpyAsync(l.pin[s], c.dev, c.bytes, kind_, st_))) {
                break;
            }
            if ((e = cudaEventRecord(l.ev[s], st_))) break;
        }
        if (kind_ == cudaMemcpyDeviceToHost) {
            if (pending >= 0) {
                if ((e = cudaEventSynchronize(l.ev[pending]))) break;
                host_side(out, l.pin[pending]);
                pending = -1;
            }
            if (more) {
                pending = s;
                out = chunks_[i];
            }
        }
        if (!more) break;
    }
    if (e) {
        int none = 0;
        err_.compare_exchange_strong(none, (int)e);
    }
}

cudaError_t HostCopier::copy(const std::vector<HostPiece>& pieces, cudaMemcpyKind kind, cudaStream_t st) {
    std::lock_guard<std::mutex> one(call_);
    if (open(lanes_[0]) != cudaSuccess) {   // no pinned memory: the driver's staging
        cudaGetLastError();
        for (const HostPiece& p : pieces)
            if (cudaError_t e = cudaMemcpyAsync(p.dst, p.src, p.bytes, kind, st)) return e;
        return cudaSuccess;
    }
    size_t total = 0;
    for (const HostPiece& p : pieces) total += p.bytes;
    const size_t chunk = std::min(std::max(total / 12 & ~(size_t)4095, kMinChunk), kMaxChunk);
    chunks_.clear();
    for (size_t k = 0; k < pieces.size(); ++k) {
        const HostPiece& p = pieces[k];
        char* dev = kind == cudaMemcpyHostToDevice ? p.dst : const_cast<char*>(p.src);
        for (size_t o = 0; o < p.bytes;) {
            Chunk* c = chunks_.empty() ? nullptr : &chunks_.back();
            if (!c || c->bytes == chunk || c->dev + c->bytes != dev + o) {
                chunks_.push_back({dev + o, 0, k, o});
                c = &chunks_.back();
            }
            const size_t n = std::min(chunk - c->bytes, p.bytes - o);
            c->bytes += n;
            o += n;
        }
    }
    pieces_ = pieces.data();
    if (chunks_.empty()) return cudaSuccess;
    kind_ = kind;
    st_ = st;
    next_ = 0;
    err_ = 0;
    {
        std::lock_guard<std::mutex> lk(mu_);
        ++seq_;
        wanted_ = (int)std::min(threads_.size(), chunks_.size() - 1);
    }
    start_.notify_all();
    work(lanes_[0]);
    {
        std::unique_lock<std::mutex> lk(mu_);
        wanted_ = 0;   // a helper still asleep has nothing left to take
        done_.wait(lk, [&] { return busy_ == 0; });
    }
    return (cudaError_t)err_.load();
}

}  // namespace pgpu
