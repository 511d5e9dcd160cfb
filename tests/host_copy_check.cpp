// Host transfers (csrc/host_copy.h) against a small stand-in for the CUDA runtime that moves data as late as the
// real one may: a copy from or to pinned memory happens when its stream or event is waited for, a pageable source is read
// before the call returns. Prints "ok" and returns 0, or says what failed. Usage: host_copy_check CHECK
#include <dlfcn.h>
#include <dirent.h>
#include <errno.h>
#include <pthread.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
typedef struct Stream *cudaStream_t;
typedef struct Event *cudaEvent_t;
enum { cudaEventDisableTiming = 2 };

struct Stream { std::deque<std::function<void()>> ops; uint64_t pushed = 0, done = 0; };
struct Event { Stream *s = nullptr; uint64_t at = 0; };
static std::map<char *, size_t> g_pinned;             // page-locked host ranges
static int g_pin_budget = 1 << 30;                    // allocations of pinned memory that still succeed

static std::recursive_mutex g_rt;                    // the runtime may be entered by several threads
#define RT std::lock_guard<std::recursive_mutex> rt(g_rt)
static bool pinned(const void *p) {
    RT;
    auto it = g_pinned.upper_bound((char *)p);
    return it != g_pinned.begin() && (--it, (char *)p < it->first + it->second);
}
static void drain(Stream *s, uint64_t to) {
    RT;
    while (s->done < to) { s->ops.front()(); s->ops.pop_front(); s->done++; }
}
static cudaError_t cudaMallocHost(void **p, size_t n) {
    RT;
    if (g_pin_budget-- <= 0) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    g_pinned[(char *)*p] = n;
    return cudaSuccess;
}
static cudaError_t cudaGetLastError() { return cudaSuccess; }
static cudaError_t cudaFreeHost(void *p) { RT; g_pinned.erase((char *)p); std::free(p); return cudaSuccess; }
static cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = new Event(); return cudaSuccess; }
static cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
static cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { RT; e->s = s; e->at = s->pushed; return cudaSuccess; }
static cudaError_t cudaEventSynchronize(cudaEvent_t e) { RT; if (e->s) drain(e->s, e->at); return cudaSuccess; }
static cudaError_t cudaStreamSynchronize(cudaStream_t s) { drain(s, s->pushed); return cudaSuccess; }
static cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    RT;
    if (kind == cudaMemcpyHostToDevice && !pinned(src)) {
        auto copy = std::make_shared<std::vector<char>>((const char *)src, (const char *)src + n);
        s->ops.push_back([=] { std::memcpy(dst, copy->data(), n); });
    } else {
        s->ops.push_back([=] { std::memcpy(dst, src, n); });
    }
    s->pushed++;
    if (kind == cudaMemcpyDeviceToHost && !pinned(dst)) drain(s, s->pushed);
    return cudaSuccess;
}

#include "../colibri_b200/csrc/host_copy.h"

static std::atomic<int> g_threads_left{1 << 30};      // threads that may still be created
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    if (g_threads_left.fetch_sub(1) <= 0) return EAGAIN;
    static auto real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
    return real(t, a, f, arg);
}
static int threads() {                                 // of this process
    int n = 0;
    DIR *d = opendir("/proc/self/task");
    while (dirent *e = readdir(d)) n += e->d_name[0] != '.';
    closedir(d);
    return n;
}

#define REQUIRE(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

static std::vector<char> pattern(size_t n, unsigned seed) {
    std::vector<char> v(n);
    for (size_t i = 0; i < n; i++) { seed = seed * 1664525u + 1013904223u; v[i] = (char)(seed >> 24); }
    return v;
}
static const size_t SIZES[] = {1, 4, 4096, 65536, 65537, 300000, (2u << 20), (2u << 20) + 5, (11u << 20) + 12};

// The source of an upload, pinned or not, belongs to the caller again when the call returns.
static int upload_sources() {
    UploadRing ring;
    Stream s;
    for (size_t n : SIZES)
        for (int pin = 0; pin < 2; pin++) {
            const std::vector<char> want = pattern(n, (unsigned)n);
            std::vector<char> dev(n, 0);
            char *src;
            if (pin) REQUIRE(cudaMallocHost((void **)&src, n) == cudaSuccess); else src = (char *)std::malloc(n);
            std::memcpy(src, want.data(), n);
            REQUIRE(upload_staged(&ring, dev.data(), src, n, &s) == cudaSuccess);
            std::memset(src, 0x5A, n);                       // the caller reuses its buffer
            cudaStreamSynchronize(&s);
            REQUIRE(dev == want);
            if (pin) cudaFreeHost(src); else std::free(src);
        }
    upload_ring_free(&ring);
    return 0;
}

// Downloads arrive whole; one whose kernels failed leaves the destination alone, and what it had under way into the
// ring's buffers does not reach the transfer after it.
static int downloads() {
    UploadRing ring;
    Stream s;
    for (size_t n : SIZES)
        for (int fine = 0; fine < 2; fine++) {
            std::vector<char> dev = pattern(n, (unsigned)n + 1), dst(n, 0x11);
            const std::vector<char> untouched = dst, want = pattern(n, (unsigned)n + 2);
            REQUIRE(download_staged(&ring, dst.data(), dev.data(), n, &s, [&] { return fine != 0; }) == cudaSuccess);
            REQUIRE(dst == (fine ? dev : untouched));
            std::vector<char> up(n, 0);
            REQUIRE(upload_staged(&ring, up.data(), want.data(), n, &s) == cudaSuccess);
            cudaStreamSynchronize(&s);
            REQUIRE(up == want);
        }
    upload_ring_free(&ring);
    return 0;
}

// With no or too little pinned memory transfers take another way and are as whole.
static int no_pinned_memory() {
    for (int budget = 0; budget < UploadRing::N; budget++) {
        UploadRing ring;
        Stream s;
        g_pin_budget = budget;
        for (size_t n : SIZES) {
            const std::vector<char> want = pattern(n, (unsigned)n + budget);
            std::vector<char> dev(n, 0), back(n, 0x11), src = want;
            const std::vector<char> untouched = back;
            REQUIRE(upload_staged(&ring, dev.data(), src.data(), n, &s) == cudaSuccess);
            src.assign(n, 0x5A);
            REQUIRE(download_staged(&ring, back.data(), dev.data(), n, &s, [] { return false; }) == cudaSuccess);
            REQUIRE(back == untouched);
            REQUIRE(download_staged(&ring, back.data(), dev.data(), n, &s, [] { return true; }) == cudaSuccess);
            REQUIRE(dev == want && back == want);
        }
        upload_ring_free(&ring);
    }
    return 0;
}

// Rows of a blocking call: pieces of 512 KB, sixteen at most, whole both ways; a call whose kernels failed writes nothing.
static int row_pieces() {
    const size_t half = 512u << 10;
    const struct { size_t bytes; uint64_t pieces; } cases[] = {{1, 1}, {half, 1}, {half + 1, 2}, {16 * half, 16}, {16 * half + 4, 16},
                                                               {(40u << 20) + 12, 16}};
    for (const auto &c : cases) {
        IoPieces io = {};
        Stream s;
        const std::vector<char> want = pattern(c.bytes, (unsigned)c.bytes);
        std::vector<char> src = want, dev(c.bytes, 0), dst(c.bytes, 0x11);
        const std::vector<char> untouched = dst;
        void *pin;
        REQUIRE(cudaMallocHost(&pin, c.bytes) == cudaSuccess);
        REQUIRE(IoPieces::in(dev.data(), pin, src.data(), c.bytes, &s) == cudaSuccess && s.pushed == c.pieces);
        src.assign(c.bytes, 0x5A);
        REQUIRE(io.out_start(pin, dev.data(), c.bytes, &s) == cudaSuccess && s.pushed == 2 * c.pieces);
        REQUIRE(!io.out_finish(dst.data(), pin, c.bytes, [] { return false; }) && dst == untouched);
        REQUIRE(io.out_finish(dst.data(), pin, c.bytes, [] { return true; }) && dst == want && dev == want);
        io.free();
        cudaFreeHost(pin);
    }
    return 0;
}

// One ring, several threads with streams of their own: nobody's pieces reach another's transfer.
static int ring_of_several_threads() {
    UploadRing ring;
    std::atomic<int> bad{0};
    std::vector<Stream> streams(4);                   // (the ring's events remember them)
    std::vector<std::thread> users;
    for (int c = 0; c < 4; c++)
        users.emplace_back([&ring, &bad, &streams, c] {
            Stream &s = streams[c];
            for (int rep = 0; rep < 40; rep++) {
                const size_t n = SIZES[(rep + c) % 9];
                const std::vector<char> want = pattern(n, (unsigned)(n + 17 * c + rep));
                std::vector<char> dev(n, 0), back(n, 0), src = want;
                if (upload_staged(&ring, dev.data(), src.data(), n, &s) != cudaSuccess) bad++;
                src.assign(n, 0x5A);
                if (download_staged(&ring, back.data(), dev.data(), n, &s, [] { return true; }) != cudaSuccess) bad++;
                cudaStreamSynchronize(&s);
                if (dev != want || back != want) bad++;
            }
        });
    for (auto &t : users) t.join();
    upload_ring_free(&ring);
    REQUIRE(bad == 0);
    return 0;
}

static const size_t COPY_SIZES[] = {1, 65536, (1u << 18) - 1, 1u << 18, (1u << 18) + 1, (1u << 20) + 77, (9u << 20) + 3};

// Copies are whole with as many helpers as asked for (argument), as the system grants, or none.
static int helpers(int granted, int expected) {
    g_threads_left = granted;
    for (int rep = 0; rep < 3; rep++)
        for (size_t n : COPY_SIZES) {
            const std::vector<char> src = pattern(n, (unsigned)(n + rep));
            std::vector<char> dst(n, 0);
            CopyPool::get().copy(dst.data(), src.data(), n);
            REQUIRE(dst == src);
        }
    REQUIRE(threads() == 1 + expected);
    return 0;
}

// Several threads copy at once, each job whole and in its own buffer.
static int many_callers() {
    std::atomic<int> bad{0};
    std::vector<std::thread> callers;
    for (int c = 0; c < 6; c++)
        callers.emplace_back([c, &bad] {
            for (int rep = 0; rep < 60; rep++)
                for (size_t n : COPY_SIZES) {
                    if (n > (2u << 20) && rep % 10) continue;
                    const std::vector<char> src = pattern(n, (unsigned)(n * 31 + c * 7 + rep));
                    std::vector<char> dst(n, 0);
                    CopyPool::get().copy(dst.data(), src.data(), n);
                    if (dst != src) bad++;
                    if (rep % 16 == 15) usleep(400);          // long enough for the helpers to fall asleep
                }
        });
    for (auto &t : callers) t.join();
    REQUIRE(bad == 0);
    return 0;
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    int rc = 2;
    if (what == "upload_sources") rc = upload_sources();
    if (what == "downloads") rc = downloads();
    if (what == "ring_of_several_threads") rc = ring_of_several_threads();
    if (what == "row_pieces") rc = row_pieces();
    if (what == "no_pinned_memory") rc = no_pinned_memory();
    if (what == "helpers" && argc > 3) rc = helpers(std::atoi(argv[2]), std::atoi(argv[3]));
    if (what == "many_callers") rc = many_callers();
    if (rc == 2) std::printf("unknown check %s\n", what.c_str());
    if (rc == 0) std::puts("ok");
    return rc;
}
