// Host side of large transfers: pageable caller memory goes through pinned buffers, copied by a few
// threads while the previous piece is on the bus.
//
// Measured on a 16-thread host: a 25 MB upload from pageable memory takes the driver 1.19 ms
// (21 GB/s); one thread copies 18 GB/s, four copy 60 GB/s, and the bus takes 47 GB/s from pinned
// memory. Below a few hundred KB a single copy into a pinned buffer (51 GB/s out of the cache) and
// one DMA beat the driver's path too (21 us against 27 us at 300 KB).
#pragma once
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

// Three helper threads, started on first use and kept until the process ends. One job at a time;
// a caller that finds them busy copies alone, so any number of threads may copy at once.
class CopyPool {
public:
    static CopyPool &get() {
        static CopyPool *p = new CopyPool();        // never destroyed: the helpers may outlive static teardown
        return *p;
    }
    void copy(void *dst, const void *src, size_t bytes) {
        if (bytes < MIN_SPLIT || !owner_.try_lock()) { std::memcpy(dst, src, bytes); return; }
        {
            std::lock_guard<std::mutex> l(m_);
            if (!started_) {
                for (int i = 0; i < HELPERS; i++) std::thread([this, i] { work(i); }).detach();
                started_ = true;
            }
            dst_ = static_cast<char *>(dst); src_ = static_cast<const char *>(src); bytes_ = bytes;
            left_ = HELPERS;
            job_++;
        }
        cv_.notify_all();
        part(HELPERS);
        std::unique_lock<std::mutex> l(m_);
        done_.wait(l, [this] { return left_ == 0; });
        l.unlock();
        owner_.unlock();
    }

private:
    static constexpr int HELPERS = 3;
    static constexpr size_t MIN_SPLIT = 1 << 19;
    void part(int i) {
        const size_t step = (bytes_ / (HELPERS + 1) + 63) & ~(size_t)63, a = step * i;
        if (a < bytes_) std::memcpy(dst_ + a, src_ + a, i == HELPERS || bytes_ - a < step ? bytes_ - a : step);
    }
    void work(int i) {
        unsigned long seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> l(m_);
                cv_.wait(l, [&] { return job_ != seen; });
                seen = job_;
            }
            part(i);
            std::lock_guard<std::mutex> l(m_);
            if (--left_ == 0) done_.notify_one();
        }
    }
    std::mutex owner_, m_;
    std::condition_variable cv_, done_;
    bool started_ = false;
    unsigned long job_ = 0;
    int left_ = 0;
    char *dst_ = nullptr;
    const char *src_ = nullptr;
    size_t bytes_ = 0;
};

// Pinned pieces of one device's uploads, each with the event of the last copy out of it.
struct UploadRing {
    static constexpr int N = 4;
    static constexpr size_t PIECE = 2u << 20;
    char *buf[N];
    cudaEvent_t ev[N];
    bool busy[N];
    int next;
};
static void upload_ring_free(UploadRing *r) {
    for (int i = 0; i < UploadRing::N; i++) {
        if (r->ev[i]) cudaEventDestroy(r->ev[i]);
        if (r->buf[i]) cudaFreeHost(r->buf[i]);
    }
    std::memset(r, 0, sizeof(*r));
}
// src (any host memory) -> dst (device) on `stream`. The source has been read when the call returns.
static cudaError_t upload_staged(UploadRing *r, void *dst, const void *src, size_t bytes, cudaStream_t stream) {
    if (bytes <= (64u << 10)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);   // the driver's inline path
    for (size_t off = 0; off < bytes; off += UploadRing::PIECE) {
        const size_t n = bytes - off < UploadRing::PIECE ? bytes - off : UploadRing::PIECE;
        const int i = r->next;
        r->next = (i + 1) % UploadRing::N;
        cudaError_t e;
        if (!r->buf[i] && ((e = cudaMallocHost(reinterpret_cast<void **>(&r->buf[i]), UploadRing::PIECE)) != cudaSuccess ||
                           (e = cudaEventCreateWithFlags(&r->ev[i], cudaEventDisableTiming)) != cudaSuccess)) return e;
        if (r->busy[i] && (e = cudaEventSynchronize(r->ev[i])) != cudaSuccess) return e;
        CopyPool::get().copy(r->buf[i], static_cast<const char *>(src) + off, n);
        if ((e = cudaMemcpyAsync(static_cast<char *>(dst) + off, r->buf[i], n, cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
            (e = cudaEventRecord(r->ev[i], stream)) != cudaSuccess) return e;
        r->busy[i] = true;
    }
    return cudaSuccess;
}

// src (device) -> dst (any host memory), after all work the stream waits for; done when the call returns. Pieces
// of 1 MB leave the device while earlier ones are copied out of the pinned buffers (the driver's pageable
// path moves 4 MB in 244 us, the bus in 84).
static cudaError_t download_staged(UploadRing *r, void *dst, const void *src, size_t bytes, cudaStream_t stream) {
    constexpr size_t STEP = 1u << 20;
    cudaError_t e;
    size_t out = 0;                             // pieces out: copied to dst
    const size_t np = (bytes + STEP - 1) / STEP;
    const int first = r->next;
    for (size_t in = 0; out < np;) {
        if (in < np && in - out < UploadRing::N) {
            const int i = (first + (int)(in % UploadRing::N)) % UploadRing::N;
            if (!r->buf[i] && ((e = cudaMallocHost(reinterpret_cast<void **>(&r->buf[i]), UploadRing::PIECE)) != cudaSuccess ||
                               (e = cudaEventCreateWithFlags(&r->ev[i], cudaEventDisableTiming)) != cudaSuccess)) return e;
            if (r->busy[i] && (e = cudaEventSynchronize(r->ev[i])) != cudaSuccess) return e;      // an upload's copy out of it
            const size_t n = bytes - in * STEP < STEP ? bytes - in * STEP : STEP;
            if ((e = cudaMemcpyAsync(r->buf[i], static_cast<const char *>(src) + in * STEP, n, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                (e = cudaEventRecord(r->ev[i], stream)) != cudaSuccess) return e;
            r->busy[i] = false;
            in++;
            continue;
        }
        const int i = (first + (int)(out % UploadRing::N)) % UploadRing::N;
        if ((e = cudaEventSynchronize(r->ev[i])) != cudaSuccess) return e;
        const size_t n = bytes - out * STEP < STEP ? bytes - out * STEP : STEP;
        CopyPool::get().copy(static_cast<char *>(dst) + out * STEP, r->buf[i], n);
        out++;
    }
    return cudaSuccess;
}

// Rows of a blocking call, between the caller's memory and a pinned buffer of the same size, in up to 16 pieces so
// that the bus works on one while the next is copied. Pieces of 256 KB and more: a copy command costs the host 4 us. (Waking
// the pool for a part of a megabyte costs more than it saves: a call with 1.5 MB each way took 100 us longer.)
struct IoPieces {
    static constexpr int N = 16;
    cudaEvent_t ev[N];
    static size_t piece(size_t bytes) {
        const size_t p = ((bytes + N - 1) / N + 4095) & ~(size_t)4095;
        return p < (256u << 10) ? 256u << 10 : p;
    }
    static void copy(void *dst, const void *src, size_t n) {
        if (n >= (1u << 20)) CopyPool::get().copy(dst, src, n);
        else std::memcpy(dst, src, n);
    }
    // src -> pinned -> dst; src has been read when the call returns
    static cudaError_t in(void *dst, void *pinned, const void *src, size_t bytes, cudaStream_t stream) {
        const size_t p = piece(bytes);
        for (size_t off = 0; off < bytes; off += p) {
            const size_t n = bytes - off < p ? bytes - off : p;
            copy(static_cast<char *>(pinned) + off, static_cast<const char *>(src) + off, n);
            const cudaError_t e = cudaMemcpyAsync(static_cast<char *>(dst) + off, static_cast<char *>(pinned) + off, n, cudaMemcpyHostToDevice, stream);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    // first half of src -> pinned -> dst: the copies off the device
    cudaError_t out_start(void *pinned, const void *src, size_t bytes, cudaStream_t stream) {
        const size_t p = piece(bytes);
        int i = 0;
        for (size_t off = 0; off < bytes; off += p, i++) {
            const size_t n = bytes - off < p ? bytes - off : p;
            cudaError_t e;
            if (!ev[i] && (e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming)) != cudaSuccess) return e;
            if ((e = cudaMemcpyAsync(static_cast<char *>(pinned) + off, static_cast<const char *>(src) + off, n, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                (e = cudaEventRecord(ev[i], stream)) != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    // second half, piece by piece; ready() is asked once the first piece is there (the kernels are done then)
    template <class Ready>
    bool out_finish(void *dst, const void *pinned, size_t bytes, Ready ready) {
        const size_t p = piece(bytes);
        int i = 0;
        for (size_t off = 0; off < bytes; off += p, i++) {
            if (cudaEventSynchronize(ev[i]) != cudaSuccess || (i == 0 && !ready())) return false;
            copy(static_cast<char *>(dst) + off, static_cast<const char *>(pinned) + off, bytes - off < p ? bytes - off : p);
        }
        return true;
    }
    void free() {
        for (int i = 0; i < N; i++)
            if (ev[i]) { cudaEventDestroy(ev[i]); ev[i] = nullptr; }
    }
};
