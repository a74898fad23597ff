// Work queued beside a caller's stream: side streams that start after what the
// caller's stream holds and that it waits for afterwards, whatever happens in
// between.  A plan run queues its buckets one after the other; when a later
// launch fails, the earlier buckets are already running and write Y, NODES and
// status, and the caller, told of the error, synchronises its own stream and
// frees them.  So the join is this object's destructor, not the last statement
// of the successful path.
#pragma once
#include <cuda_runtime_api.h>

namespace mgpu {

class StreamFork {
public:
    static constexpr int kMaxSides = 64;

private:
    struct Side {
        cudaStream_t st, look;
        cudaEvent_t done, look_done;
    };
    cudaStream_t caller_;
    cudaEvent_t start_;
    Side sides_[kMaxSides];  // with work, not joined yet; no allocation, so nothing here throws
    int n_ = 0;

    // `caller_` waits for `st`; the host does where that cannot be queued
    cudaError_t after(cudaStream_t st, cudaEvent_t done)
    {
        cudaError_t e = cudaEventRecord(done, st);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(caller_, done, 0);
        if (e != cudaSuccess) {
            cudaStreamSynchronize(st);
            cudaGetLastError();  // returned here, or behind an error reported already: not to the next launch check
        }
        return e;
    }

public:
    // `start` is recorded by begin(); neither it nor a side's events may be in
    // use by another thread until the object is gone
    StreamFork(cudaStream_t caller, cudaEvent_t start) : caller_(caller), start_(start) {}
    StreamFork(const StreamFork &) = delete;
    StreamFork &operator=(const StreamFork &) = delete;
    ~StreamFork()
    {
        for (int i = 0; i < n_; ++i) {
            const Side &s = sides_[i];
            // an error can leave the look-ahead stream's work unjoined with its main stream
            if (s.look) after(s.look, s.look_done);
            after(s.st, s.done);
        }
    }

    cudaError_t begin() { return cudaEventRecord(start_, caller_); }

    // From here on `st` (and a look-ahead stream that the work on it forks and
    // joins) belongs to the fork.
    cudaError_t to(cudaStream_t st, cudaEvent_t done, cudaStream_t look = nullptr, cudaEvent_t look_done = nullptr)
    {
        if (n_ == kMaxSides) return cudaErrorInvalidValue;
        const cudaError_t e = cudaStreamWaitEvent(st, start_, 0);
        if (e == cudaSuccess) sides_[n_++] = Side{st, look, done, look_done};
        return e;
    }

    // The successful path's join: the first error, every side joined all the same.
    cudaError_t join()
    {
        cudaError_t first = cudaSuccess;
        for (int i = 0; i < n_; ++i) {
            const cudaError_t e = after(sides_[i].st, sides_[i].done);
            if (first == cudaSuccess) first = e;
        }
        n_ = 0;
        return first;
    }
};

}  // namespace mgpu
