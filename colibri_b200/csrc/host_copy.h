// Host side of large transfers: pageable caller memory goes through pinned buffers, copied by a few
// threads while the previous piece is on the bus.
//
// Measured on a 16-thread host: a 25 MB upload from pageable memory takes the driver 1.19 ms
// (21 GB/s); one thread copies 18 GB/s, four copy 60 GB/s, and the bus takes 47 GB/s from pinned
// memory. Below a few hundred KB a single copy into a pinned buffer (51 GB/s out of the cache) and
// one DMA beat the driver's path too (21 us against 27 us at 300 KB).
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

// Helper threads, started on first use and kept until the process ends. One job at a time;
// a caller that finds them busy copies alone, so any number of threads may copy at once.
// A job is cut into pieces of 64 KB that the caller and whoever is awake take one after the other, so a copy never
// waits for a sleeping helper (waking one takes about 50 us, as long as 1 MB takes to copy). Helpers look for
// the next job for 200 us before they sleep: a call's result usually follows its input within that time. So a program
// that copies 256 KB or more at shorter intervals keeps them awake, on cores its own threads may want:
// COLI_CUDA_COPY_THREADS=0 turns them off, 1 to 3 sets their number (read once). Without it there are three, or a quarter of the
// host's hardware threads if that is less. One that the system does not grant is done without.
// Measured, three helpers / none: a group of 1.5 MB each way back to back 320 / 408 us, in calls 5 ms apart (helpers asleep) 405 to
// 434 / 416; uploads of 25 MB (one expert) 1150 / 2010, apart 1170 / 2170.
class CopyPool {
public:
    static CopyPool &get() {
        static CopyPool *p = new CopyPool();        // never destroyed: the helpers may outlive static teardown
        return *p;
    }
    void copy(void *dst, const void *src, size_t bytes) {
        if (bytes < MIN_SPLIT || bytes > MAX_JOB || limit_ == 0 || !owner_.try_lock()) {
            if (bytes > MAX_JOB)
                for (size_t off = 0; off < bytes; off += MAX_JOB)
                    copy(static_cast<char *>(dst) + off, static_cast<const char *>(src) + off, bytes - off < MAX_JOB ? bytes - off : MAX_JOB);
            else std::memcpy(dst, src, bytes);
            return;
        }
        const uint64_t n = (bytes + PIECE - 1) / PIECE;
        dst_.store(static_cast<char *>(dst), std::memory_order_relaxed);
        src_.store(static_cast<const char *>(src), std::memory_order_relaxed);
        bytes_.store(bytes, std::memory_order_relaxed);
        done_.store(0, std::memory_order_relaxed);
        const uint64_t job = (++epoch_ << 32) | (n << 16);
        ticket_.store(job, std::memory_order_seq_cst);
        if (!started_) {
            started_ = true;
            try {                               // (no exception may leave through the C entry points above)
                for (int i = 0; i < limit_; i++) std::thread([this] { work(); }).detach();
            } catch (const std::system_error &) {
            }
        }
        if (asleep_.load(std::memory_order_seq_cst)) {
            { std::lock_guard<std::mutex> l(m_); }
            cv_.notify_all();
        }
        take();
        while (done_.load(std::memory_order_acquire) < n) pause();       // pieces that helpers are in the middle of
        owner_.unlock();
    }

private:
    static constexpr int HELPERS = 3;
    static int helper_limit() {
        const char *e = std::getenv("COLI_CUDA_COPY_THREADS");
        const unsigned quarter = std::thread::hardware_concurrency() / 4;
        const int n = e && *e ? std::atoi(e) : (int)quarter;
        return n < 0 ? 0 : n > HELPERS ? HELPERS : n;
    }
    static constexpr size_t MIN_SPLIT = 1 << 18, PIECE = 1 << 16, MAX_JOB = (size_t)1 << 30;
    static void pause() {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }
    // Copies pieces of the current job until none is left. ticket_: job number | pieces << 16 | next piece; the
    // job's fields change only while its ticket has no piece left, so a piece won from a ticket belongs to what was read.
    void take() {
        uint64_t t = ticket_.load(std::memory_order_acquire);
        for (;;) {
            const uint64_t n = (t >> 16) & 0xFFFF, i = t & 0xFFFF;
            if (i >= n) return;
            char *dst = dst_.load(std::memory_order_relaxed);
            const char *src = src_.load(std::memory_order_relaxed);
            const size_t bytes = bytes_.load(std::memory_order_relaxed);
            if (!ticket_.compare_exchange_weak(t, t + 1, std::memory_order_acq_rel, std::memory_order_acquire)) continue;
            const size_t a = i * PIECE;
            std::memcpy(dst + a, src + a, bytes - a < PIECE ? bytes - a : PIECE);
            done_.fetch_add(1, std::memory_order_release);
            t = ticket_.load(std::memory_order_acquire);
        }
    }
    bool open() const {
        const uint64_t t = ticket_.load(std::memory_order_seq_cst);
        return (t & 0xFFFF) < ((t >> 16) & 0xFFFF);
    }
    void work() {
        for (;;) {
            take();
            const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(200);
            while (!open() && std::chrono::steady_clock::now() < until)
                for (int i = 0; i < 16; i++) pause();
            if (open()) continue;
            std::unique_lock<std::mutex> l(m_);
            asleep_.fetch_add(1, std::memory_order_seq_cst);
            cv_.wait(l, [this] { return open(); });
            asleep_.fetch_sub(1, std::memory_order_seq_cst);
        }
    }
    const int limit_ = helper_limit();
    std::mutex owner_, m_;
    std::condition_variable cv_;
    bool started_ = false;
    uint64_t epoch_ = 0;
    std::atomic<uint64_t> ticket_{0}, done_{0};
    std::atomic<size_t> bytes_{0};
    std::atomic<char *> dst_{nullptr};
    std::atomic<const char *> src_{nullptr};
    std::atomic<int> asleep_{0};
};

// Pinned pieces of one device's transfers, each with the event of the last copy out of it or into it. A transfer holds the
// ring from its first piece to its last: a thread that brings experts in and one that runs the model may share a device.
struct UploadRing {
    static constexpr int N = 4;
    static constexpr size_t PIECE = 2u << 20;
    char *buf[N] = {};
    cudaEvent_t ev[N] = {};
    bool busy[N] = {};
    int next = 0;
    std::mutex mu;
};
static void upload_ring_free(UploadRing *r) {
    for (int i = 0; i < UploadRing::N; i++) {
        if (r->ev[i]) cudaEventDestroy(r->ev[i]);
        if (r->buf[i]) cudaFreeHost(r->buf[i]);
        r->ev[i] = nullptr; r->buf[i] = nullptr; r->busy[i] = false;
    }
    r->next = 0;
}
// Buffer i of the ring, pinned on first use. Where the system has no pinned memory left the transfer goes without it, by
// the driver's own staging: slower, not refused.
static bool upload_ring_slot(UploadRing *r, int i) {
    if (r->buf[i]) return true;
    if (!r->ev[i] && cudaEventCreateWithFlags(&r->ev[i], cudaEventDisableTiming) != cudaSuccess) { r->ev[i] = nullptr; (void)cudaGetLastError(); return false; }
    void *p = nullptr;
    if (cudaMallocHost(&p, UploadRing::PIECE) != cudaSuccess) { (void)cudaGetLastError(); return false; }
    r->buf[i] = static_cast<char *>(p);
    return true;
}
// src (any host memory) -> dst (device) on `stream`. The source has been read when the call returns, small ones and
// pinned ones included: cudaMemcpyAsync straight from a pinned source would return before the copy has run.
static cudaError_t upload_staged(UploadRing *r, void *dst, const void *src, size_t bytes, cudaStream_t stream) {
    std::lock_guard<std::mutex> hold(r->mu);
    for (size_t off = 0; off < bytes; off += UploadRing::PIECE) {
        const size_t n = bytes - off < UploadRing::PIECE ? bytes - off : UploadRing::PIECE;
        const int i = r->next;
        r->next = (i + 1) % UploadRing::N;
        cudaError_t e;
        if (!upload_ring_slot(r, i)) {
            e = cudaMemcpyAsync(static_cast<char *>(dst) + off, static_cast<const char *>(src) + off, bytes - off, cudaMemcpyHostToDevice, stream);
            return e != cudaSuccess ? e : cudaStreamSynchronize(stream);
        }
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
// path moves 4 MB in 244 us, the bus in 84). ready() is asked once, when the first piece is there (the kernels before
// it are done then); if it says no, dst is left alone and nothing more is copied off the device.
template <class Ready>
static cudaError_t download_staged(UploadRing *r, void *dst, const void *src, size_t bytes, cudaStream_t stream, Ready ready) {
    constexpr size_t STEP = 1u << 20;
    std::lock_guard<std::mutex> hold(r->mu);
    cudaError_t e;
    size_t out = 0;                             // pieces out: copied to dst
    const size_t np = (bytes + STEP - 1) / STEP;
    const int first = r->next;
    for (size_t i = 0; i < np && i < (size_t)UploadRing::N; i++)
        if (!upload_ring_slot(r, (first + (int)i) % UploadRing::N)) {
            char few[16];                       // (a blocking copy: the kernels before it are done when it returns)
            if ((e = cudaMemcpyAsync(few, src, bytes < sizeof(few) ? bytes : sizeof(few), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                (e = cudaStreamSynchronize(stream)) != cudaSuccess || !ready()) return e;
            if ((e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream)) != cudaSuccess) return e;
            return cudaStreamSynchronize(stream);
        }
    for (size_t in = 0; out < np;) {
        if (in < np && in - out < UploadRing::N) {
            const int i = (first + (int)(in % UploadRing::N)) % UploadRing::N;
            if (r->busy[i] && (e = cudaEventSynchronize(r->ev[i])) != cudaSuccess) return e;      // the copy before, out of it or into it
            const size_t n = bytes - in * STEP < STEP ? bytes - in * STEP : STEP;
            if ((e = cudaMemcpyAsync(r->buf[i], static_cast<const char *>(src) + in * STEP, n, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                (e = cudaEventRecord(r->ev[i], stream)) != cudaSuccess) return e;
            r->busy[i] = true;                  // until its event has been waited for, here or by the buffer's next user
            in++;
            continue;
        }
        const int i = (first + (int)(out % UploadRing::N)) % UploadRing::N;
        if ((e = cudaEventSynchronize(r->ev[i])) != cudaSuccess) return e;
        r->busy[i] = false;
        if (out == 0 && !ready()) return cudaSuccess;
        const size_t n = bytes - out * STEP < STEP ? bytes - out * STEP : STEP;
        CopyPool::get().copy(static_cast<char *>(dst) + out * STEP, r->buf[i], n);
        out++;
    }
    return cudaSuccess;
}

// Rows of a blocking call, between the caller's memory and a pinned buffer of the same size, in up to 16 pieces so
// that the bus works on one while the next is copied. Pieces of 512 KB and more: a copy command costs the host 4 us,
// and four threads copy such a piece in about as long as the bus takes for it.
struct IoPieces {
    static constexpr int N = 16;
    cudaEvent_t ev[N];
    static size_t piece(size_t bytes) {
        const size_t p = ((bytes + N - 1) / N + 4095) & ~(size_t)4095;
        return p < (512u << 10) ? 512u << 10 : p;
    }
    // src -> pinned -> dst; src has been read when the call returns
    static cudaError_t in(void *dst, void *pinned, const void *src, size_t bytes, cudaStream_t stream) {
        const size_t p = piece(bytes);
        for (size_t off = 0; off < bytes; off += p) {
            const size_t n = bytes - off < p ? bytes - off : p;
            CopyPool::get().copy(static_cast<char *>(pinned) + off, static_cast<const char *>(src) + off, n);
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
            CopyPool::get().copy(static_cast<char *>(dst) + off, static_cast<const char *>(pinned) + off, bytes - off < p ? bytes - off : p);
        }
        return true;
    }
    void free() {
        for (int i = 0; i < N; i++)
            if (ev[i]) { cudaEventDestroy(ev[i]); ev[i] = nullptr; }
    }
};
