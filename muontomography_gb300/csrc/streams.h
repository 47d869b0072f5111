// The streams and events of a handle or a call, and the side streams' work between a
// fork and its join.  Host code: the CUDA runtime's stream and event calls alone.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

namespace muto {

// Side streams the class kernels of a voxel pass are spread over (they touch
// disjoint voxels), with the events that fork them from the launching stream
// and join them back; inside stream capture they become parallel branches.
struct ClassFan {
    static constexpr int kSide = 3;
    cudaStream_t side[kSide] = {};
    cudaEvent_t fork = nullptr, join[kSide] = {};
    int n = 0;  // side streams in use (0: every class on the launching stream)
};

// Work on the first n side streams, from the fork on.  What is left before the join (an
// exception) waits for it: nothing that the launches made use is freed under them.
struct Forked {
    const ClassFan& fan;
    int n;
    bool joined = false;
    Forked(const ClassFan& f, int count) : fan(f), n(count) {}
    ~Forked() {
        if (joined) return;
        for (int q = 0; q < n; ++q) (void)cudaStreamSynchronize(fan.side[q]);
    }
    Forked(const Forked&) = delete;
    Forked& operator=(const Forked&) = delete;
};

// The streams and events of one handle (or call), from a small pool per device: creating
// and destroying them takes longer than a small scan's iterations.  A set goes
// back to the pool idle, all its streams waited for (a query first: 1 us, a wait on
// an idle stream 3); the pool keeps at most kKept sets a device, and none whose work
// failed.
struct HandleStreams {
    static constexpr int kOverlap = 5;
    int device = 0;
    cudaStream_t stream = nullptr;
    ClassFan fan{};
    cudaEvent_t ov_ev[kOverlap] = {};

    cudaError_t create(int dev) {
        device = dev;
        cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&fan.fork, cudaEventDisableTiming);
        for (int k = 0; e == cudaSuccess && k < ClassFan::kSide; ++k) {
            e = cudaStreamCreateWithFlags(&fan.side[k], cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&fan.join[k], cudaEventDisableTiming);
            fan.n = k + 1;
        }
        for (int k = 0; e == cudaSuccess && k < kOverlap; ++k) e = cudaEventCreateWithFlags(&ov_ev[k], cudaEventDisableTiming);
        return e;
    }
    void destroy() {
        for (int k = 0; k < ClassFan::kSide; ++k) {
            if (fan.side[k]) cudaStreamDestroy(fan.side[k]);
            if (fan.join[k]) cudaEventDestroy(fan.join[k]);
        }
        if (fan.fork) cudaEventDestroy(fan.fork);
        for (cudaEvent_t e : ov_ev)
            if (e) cudaEventDestroy(e);
        if (stream) cudaStreamDestroy(stream);
        *this = HandleStreams{};
    }
    static constexpr size_t kKept = 8;
    // (never destroyed: a handle of a program's own static object may outlive them)
    static std::mutex& mutex() {
        static std::mutex* m = new std::mutex;
        return *m;
    }
    static std::map<int, std::vector<HandleStreams>>& kept() {
        static auto* k = new std::map<int, std::vector<HandleStreams>>;
        return *k;
    }
    // the device's streams for a new handle
    static cudaError_t take(int dev, HandleStreams* out) {
        {
            std::lock_guard<std::mutex> lock(mutex());
            auto& k = kept()[dev];
            if (!k.empty()) {
                *out = k.back();
                k.pop_back();
                return cudaSuccess;
            }
        }
        HandleStreams h;
        const cudaError_t e = h.create(dev);
        if (e == cudaSuccess) *out = h;
        else h.destroy();
        return e;
    }
    static bool wait_for(cudaStream_t s) {
        const cudaError_t e = cudaStreamQuery(s);
        return (e == cudaErrorNotReady ? cudaStreamSynchronize(s) : e) == cudaSuccess;
    }
    // back to the pool, its work done (forked: the side streams may have been used)
    void give(bool forked = true) {
        if (!stream) return;
        bool idle = cudaStreamSynchronize(stream) == cudaSuccess;
        for (int k = 0; forked && k < fan.n; ++k) idle = wait_for(fan.side[k]) && idle;
        if (idle) {
            std::lock_guard<std::mutex> lock(mutex());
            auto& k = kept()[device];
            if (k.size() < kKept) {
                k.push_back(*this);
                *this = HandleStreams{};
                return;
            }
        }
        destroy();
    }
};

}  // namespace muto
