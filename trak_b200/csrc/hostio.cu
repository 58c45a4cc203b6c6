// Pageable host memory <-> device memory: the numpy memmaps and host accumulators TRAKer keeps its features and
// scores in (trak/savers.py:363-442, trak/traker.py:632-667).
//
// A copy from or to pageable memory goes through a pinned buffer in any case; the driver's own does that with one
// host thread (measured: 11 GB/s host to device, one core's memory copy is 8 GB/s), while PCIe takes 55 GB/s.  Here
// a transfer is cut into chunks that alternate between the slots of a small pinned ring.  The host side of the chunks
// (a copy, or the fp32 accumulation `dst += chunk`) is done by several threads in pieces they take one after the
// other; the calling thread starts the PCIe copies and hands out slots, and takes pieces in between, so host and PCIe
// work run side by side with no meeting point per chunk (with one, waking and joining the threads took a third of
// the time at 4 MB a chunk, half at 2 MB).  Where a transfer stalls, as the first chunk does behind the stream's earlier
// work, the threads sleep.  Measured on 16 cores: 627 MB of features go up at 44 GB/s, 100 MB of
// scores come down at 37.
//
// The rings (16 MB per device and direction, made on first use: larger ones crowd the L3) and the threads outlive a
// call and serve every stream: a ring is locked for the length of a transfer, and each slot carries the event of the
// copy that last used it.  tb_host_staging_release gives the pinned memory back.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include <dlfcn.h>
#include <immintrin.h>
#include <sys/types.h>
#include <unistd.h>

#include "host_util.h"

namespace tb {

// ---- host threads ------------------------------------------------------------------------------
// Threads that help with one job at a time.  A job's body is run by every thread that comes while the job is open; it
// has to be able to finish with no helper at all (another caller has them, or this is a forked child).
//
// Where the process has an OpenMP runtime (torch's), the helpers are its team: after any parallel region its threads
// keep spinning for milliseconds, and threads of our own beside them would get half of the cores (a score block added
// to a host accumulator that had just been cleared: 27 GB/s with our own, 40 with the team).  Else a few of our own.
// Either way as many as the user asks for: the team's size, or OMP_NUM_THREADS (tb_host_threads tells).
struct OpenMp {
    void (*parallel)(void (*)(void*), void*, unsigned, unsigned) = nullptr;
    int (*max_threads)() = nullptr;
    int (*thread_num)() = nullptr;
    int (*in_parallel)() = nullptr;

    OpenMp() {
        // what the process's own code would be linked to, under whatever file name, else a libgomp that some module
        // has loaded for itself; never loads one
        void* lib = dlsym(RTLD_DEFAULT, "GOMP_parallel") ? RTLD_DEFAULT : dlopen("libgomp.so.1", RTLD_LAZY | RTLD_NOLOAD);
        max_threads = reinterpret_cast<int (*)()>(dlsym(lib, "omp_get_max_threads"));
        thread_num = reinterpret_cast<int (*)()>(dlsym(lib, "omp_get_thread_num"));
        in_parallel = reinterpret_cast<int (*)()>(dlsym(lib, "omp_in_parallel"));
        if (max_threads && thread_num && in_parallel)
            parallel = reinterpret_cast<void (*)(void (*)(void*), void*, unsigned, unsigned)>(dlsym(lib, "GOMP_parallel"));
    }
    static const OpenMp& get() {
        static const OpenMp omp;
        return omp;
    }
    // the calling thread's team; inside a parallel region the team is at work already
    int threads() const { return in_parallel() ? 1 : max_threads(); }

    struct Region {
        const OpenMp* omp;
        const std::function<void()>*body, *caller;
    };
    void run(const std::function<void()>& body, const std::function<void()>& caller) const {
        Region r{this, &body, &caller};
        // as many threads as everyone else asks for: a team of another size would be torn down and built again
        parallel([](void* p) {
            const Region& g = *static_cast<Region*>(p);
            if (g.omp->thread_num() == 0)
                (*g.caller)();
            else
                (*g.body)();
        }, &r, 0, 0);
    }
};

class HostThreads {
  public:
    static HostThreads& get() {
        static std::mutex mu;
        static HostThreads* pool = nullptr;  // never destroyed: its threads sleep until the process ends
        std::lock_guard<std::mutex> lk(mu);
        if (!pool || pool->pid_ != getpid()) pool = new HostThreads();  // a forked child has none of the threads
        return *pool;
    }

    // Threads that share a job, the calling one included: OMP_NUM_THREADS where it is a number, else most of the cores.
    static int wanted() {
        if (const char* env = getenv("OMP_NUM_THREADS")) {
            const long n = strtol(env, nullptr, 10);
            if (n > 0) return (int)std::min<long>(n, 256);
        }
        return std::max(1, std::min(MAX_HELPERS + 1, (int)std::thread::hardware_concurrency() - 1));
    }

    // `body` on the helpers while `caller` runs here; returns when both have ended.
    void help(const std::function<void()>& body, const std::function<void()>& caller) {
        std::unique_lock<std::mutex> busy(busy_, std::try_to_lock);
        if (!busy.owns_lock()) {
            caller();
            return;
        }
        auto job = std::make_shared<Job>(body);
        {
            std::lock_guard<std::mutex> lk(mu_);
            job_ = job;
            ++generation_;
        }
        wake_.notify_all();
        caller();
        job->closed.store(true);
        while (job->active.load() > 0) _mm_pause();
    }

  private:
    struct Job {
        explicit Job(const std::function<void()>& b) : body(b) {}
        const std::function<void()>& body;  // valid while the job is open or a helper is active
        std::atomic<bool> closed{false};
        std::atomic<int> active{0};
    };

    HostThreads() : pid_(getpid()) {
        for (int i = 1; i < wanted(); ++i) {
            try {
                std::thread([this] { loop(); }).detach();
            } catch (const std::system_error&) {  // no more threads to be had: those that are there do the work
                break;
            }
        }
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            std::shared_ptr<Job> job;
            {
                std::unique_lock<std::mutex> lk(mu_);
                wake_.wait(lk, [&] { return generation_ != seen; });
                seen = generation_;
                job = job_;
            }
            job->active.fetch_add(1);
            if (!job->closed.load()) job->body();
            job->active.fetch_sub(1);
        }
    }

    static constexpr int MAX_HELPERS = 11;
    const pid_t pid_;
    std::mutex busy_, mu_;
    std::condition_variable wake_;
    std::shared_ptr<Job> job_;
    uint64_t generation_ = 0;
};

// Threads that share the host side of a transfer started by this thread.
static int host_threads() { return OpenMp::get().parallel ? OpenMp::get().threads() : HostThreads::wanted(); }

// Waits a moment: pauses at first, sleeps once it has taken longer than a transfer that gets on ever stalls (a chunk
// crosses PCIe in 40 us; with sleeps from 20 us on, 2 MB came down in 300 us instead of 120).
struct Patience {
    int spins = 0;
    std::chrono::steady_clock::time_point since;

    void wait() {
        _mm_pause();
        if (++spins % 64) return;
        const auto now = std::chrono::steady_clock::now();
        if (spins == 64)
            since = now;
        else if (now - since > std::chrono::microseconds(400))
            std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
};

// ---- pinned rings ------------------------------------------------------------------------------
constexpr size_t CHUNK_BYTES = 2u << 20;
constexpr int SLOTS = 8;
constexpr size_t PIECE_BYTES = 128u << 10;  // what a thread takes at a time
constexpr int HOSTIO_MAX_DEV = 64;

struct Ring {
    std::mutex mu;
    uint8_t* buf = nullptr;
    cudaEvent_t ev[SLOTS] = {};
    bool in_flight[SLOTS] = {};

    int make() {  // with mu held and the device current
        if (buf) return TB_OK;
        void* p = nullptr;
        TB_CUDA(cudaHostAlloc(&p, CHUNK_BYTES * SLOTS, cudaHostAllocDefault));
        for (int i = 0; i < SLOTS; ++i) {
            const cudaError_t e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
            if (e != cudaSuccess) {
                for (int j = 0; j < i; ++j) cudaEventDestroy(ev[j]);
                cudaFreeHost(p);
                TB_CUDA(e);
            }
        }
        buf = static_cast<uint8_t*>(p);
        return TB_OK;
    }
    int settle(int slot) {  // the device is done with what was last put in this slot
        if (in_flight[slot]) TB_CUDA(cudaEventSynchronize(ev[slot]));
        in_flight[slot] = false;
        return TB_OK;
    }
    int release() {
        if (!buf) return TB_OK;
        for (int i = 0; i < SLOTS; ++i) {
            const int rc = settle(i);
            if (rc != TB_OK) return rc;
            TB_CUDA(cudaEventDestroy(ev[i]));
        }
        TB_CUDA(cudaFreeHost(buf));
        buf = nullptr;
        return TB_OK;
    }
};
static Ring g_up[HOSTIO_MAX_DEV], g_down[HOSTIO_MAX_DEV];

// One transfer in pieces.  Chunk c lives in slot c % SLOTS; its pieces may be worked on once `opened` > c (going up:
// the slot is free; going down: the chunk has arrived), and left[c] counts those not done yet.
struct Transfer {
    Ring& ring;
    const size_t bytes, chunk;
    const int chunks, pieces_per_chunk, pieces;
    const std::function<void(size_t, uint8_t*, size_t)> op;  // (offset, pinned address, length)
    std::atomic<int> next{0}, opened{0};
    std::atomic<bool> stop{false};
    std::vector<std::atomic<int>> left;

    Transfer(Ring& r, size_t n, std::function<void(size_t, uint8_t*, size_t)> f)
        : ring(r), bytes(n), chunk(chunk_of(n)), chunks((int)((n + chunk - 1) / chunk)),
          pieces_per_chunk((int)((chunk + PIECE_BYTES - 1) / PIECE_BYTES)), pieces(chunks * pieces_per_chunk),
          op(std::move(f)), left(chunks) {
        for (auto& l : left) l.store(pieces_per_chunk, std::memory_order_relaxed);
    }
    // about an eighth of the transfer, so that the stages of a short one overlap too
    static size_t chunk_of(size_t n) {
        return std::min(CHUNK_BYTES, std::max<size_t>(256u << 10, align_up((n + SLOTS - 1) / SLOTS, 4096)));
    }
    size_t offset(int c) const { return (size_t)c * chunk; }
    size_t length(int c) const { return std::min(chunk, bytes - offset(c)); }
    uint8_t* slot(int c) const { return ring.buf + (size_t)(c % SLOTS) * CHUNK_BYTES; }

    void piece(int p) {
        const int c = p / pieces_per_chunk;
        const size_t lo = (size_t)(p % pieces_per_chunk) * PIECE_BYTES, hi = std::min(lo + PIECE_BYTES, length(c));
        if (hi > lo) op(offset(c) + lo, slot(c) + lo, hi - lo);
        left[c].fetch_sub(1, std::memory_order_release);
    }
    void helper() {
        for (int p; (p = next.fetch_add(1, std::memory_order_relaxed)) < pieces;) {
            for (Patience idle; opened.load(std::memory_order_acquire) <= p / pieces_per_chunk; idle.wait())
                if (stop.load(std::memory_order_relaxed)) return;
            piece(p);
        }
    }
    // The calling thread's side: `advance` starts copies and opens chunks as far as it can without waiting, sets
    // `done` when nothing is left; in between this thread takes pieces of open chunks itself.
    int drive(const std::function<int(bool*)>& advance) {
        int rc = TB_OK;
        const std::function<void()> body = [this] { helper(); }, caller = [&] {
            int held = -1;  // a piece taken whose chunk was not open yet
            Patience idle;
            for (bool done = false; !done;) {
                const int before = opened.load(std::memory_order_relaxed);
                rc = advance(&done);
                if (rc != TB_OK) break;
                const int open = opened.load(std::memory_order_relaxed), coming = next.load(std::memory_order_relaxed);
                if (held < 0 && coming < pieces && coming / pieces_per_chunk < open) {
                    held = next.fetch_add(1, std::memory_order_relaxed);
                    if (held >= pieces) held = -1;
                }
                if (held >= 0 && held / pieces_per_chunk < open) {
                    piece(held);
                    held = -1;
                    idle = Patience();
                } else if (open != before) {
                    idle = Patience();
                } else if (!done) {
                    idle.wait();
                }
            }
            stop.store(true, std::memory_order_relaxed);
        };
        if (host_threads() < 2)
            caller();
        else if (OpenMp::get().parallel)
            OpenMp::get().run(body, caller);
        else
            HostThreads::get().help(body, caller);
        return rc;
    }
    bool worked(int c) const { return left[c].load(std::memory_order_acquire) == 0; }
};

// Whether the device is done with a slot; never waits.
static int slot_idle(Ring& ring, int slot, bool* idle) {
    *idle = true;
    if (!ring.in_flight[slot]) return TB_OK;
    const cudaError_t e = cudaEventQuery(ring.ev[slot]);
    if (e == cudaErrorNotReady) {
        *idle = false;
        return TB_OK;
    }
    TB_CUDA(e);
    ring.in_flight[slot] = false;
    return TB_OK;
}

// What one thread can do, the driver's own copy does better: up 10 to 20 GB/s against 7 to 15 through the ring, down 15
// to 21 against 9 to 15 (2 to 400 MB).  Memory that turns out to be pinned is waited for like any other.
static int copy_alone(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t stream) {
    TB_CUDA(cudaMemcpyAsync(dst, src, bytes, kind, stream));
    TB_CUDA(cudaStreamSynchronize(stream));
    return TB_OK;
}

}  // namespace tb

extern "C" {

int tb_host_to_device(int device, void* stream_, void* dst, const void* src, size_t bytes) {
    using namespace tb;
    if (bytes == 0) return TB_OK;
    if (!dst || !src || device < 0 || device >= HOSTIO_MAX_DEV) return TB_ERR_BAD_ARG;
    int rc = select_device(device, nullptr);
    if (rc != TB_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (host_threads() < 2) return copy_alone(dst, src, bytes, cudaMemcpyHostToDevice, stream);
    Ring& ring = g_up[device];
    std::lock_guard<std::mutex> lk(ring.mu);
    rc = ring.make();
    if (rc != TB_OK) return rc;
    const uint8_t* s = static_cast<const uint8_t*>(src);
    uint8_t* d = static_cast<uint8_t*>(dst);
    Transfer t(ring, bytes, [s](size_t at, uint8_t* pin, size_t n) { memcpy(pin, s + at, n); });
    int sent = 0, opened = 0;
    return t.drive([&](bool* done) {
        for (; sent < t.chunks && t.worked(sent); ++sent) {
            const int slot = sent % SLOTS;
            TB_CUDA(cudaMemcpyAsync(d + t.offset(sent), t.slot(sent), t.length(sent), cudaMemcpyHostToDevice, stream));
            TB_CUDA(cudaEventRecord(ring.ev[slot], stream));
            ring.in_flight[slot] = true;
        }
        // a slot is handed out again when its last chunk has been sent and the device has read it
        while (opened < t.chunks && opened < sent + SLOTS) {
            bool idle;
            const int r = slot_idle(ring, opened % SLOTS, &idle);
            if (r != TB_OK) return r;
            if (!idle) break;
            t.opened.store(++opened, std::memory_order_release);
        }
        *done = sent == t.chunks;
        return (int)TB_OK;
    });
}

int tb_device_to_host(int device, void* stream_, void* dst, const void* src, size_t bytes, int add_f32) {
    using namespace tb;
    if (bytes == 0) return TB_OK;
    if (!dst || !src || device < 0 || device >= HOSTIO_MAX_DEV || (add_f32 && (bytes % 4 || ((uintptr_t)dst & 3u))))
        return TB_ERR_BAD_ARG;
    int rc = select_device(device, nullptr);
    if (rc != TB_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (host_threads() < 2 && !add_f32) return copy_alone(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
    Ring& ring = g_down[device];
    std::lock_guard<std::mutex> lk(ring.mu);
    rc = ring.make();
    if (rc != TB_OK) return rc;
    const uint8_t* s = static_cast<const uint8_t*>(src);
    uint8_t* d = static_cast<uint8_t*>(dst);
    Transfer t(ring, bytes, [d, add_f32](size_t at, uint8_t* pin, size_t n) {
        if (!add_f32) {
            memcpy(d + at, pin, n);
            return;
        }
        const float* x = reinterpret_cast<const float*>(pin);
        float* y = reinterpret_cast<float*>(d + at);
        for (size_t j = 0; j < n / 4; ++j) y[j] += x[j];
    });
    int asked = 0, opened = 0, finished = 0;
    return t.drive([&](bool* done) {
        while (finished < opened && t.worked(finished)) ++finished;
        for (; asked < t.chunks && asked < finished + SLOTS; ++asked) {
            const int slot = asked % SLOTS;
            TB_CUDA(cudaMemcpyAsync(t.slot(asked), s + t.offset(asked), t.length(asked), cudaMemcpyDeviceToHost, stream));
            TB_CUDA(cudaEventRecord(ring.ev[slot], stream));
            ring.in_flight[slot] = true;
        }
        while (opened < asked) {
            bool idle;
            const int r = slot_idle(ring, opened % SLOTS, &idle);
            if (r != TB_OK) return r;
            if (!idle) break;
            t.opened.store(++opened, std::memory_order_release);
        }
        *done = finished == t.chunks;
        return (int)TB_OK;
    });
}

int tb_host_threads(int* openmp) {
    if (openmp) *openmp = tb::OpenMp::get().parallel ? 1 : 0;
    return tb::host_threads();
}

int tb_host_staging_release(void) {
    using namespace tb;
    int prev = 0;
    const bool restore = cudaGetDevice(&prev) == cudaSuccess;
    int rc = TB_OK;
    for (int dev = 0; dev < HOSTIO_MAX_DEV; ++dev)
        for (Ring* ring : {&g_up[dev], &g_down[dev]}) {
            std::lock_guard<std::mutex> lk(ring->mu);
            if (!ring->buf) continue;
            if (cudaSetDevice(dev) != cudaSuccess) continue;
            const int r = ring->release();
            if (r != TB_OK) rc = r;
        }
    if (restore) cudaSetDevice(prev);
    return rc;
}

}  // extern "C"
