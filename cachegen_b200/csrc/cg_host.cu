// Host side of the byte strings: memory that is not pinned to and from the GPU, through pinned staging memory,
// with the copies between the two kinds of host memory spread over a few threads and overlapped with the transfer.
//
// One thread copies 13 GB/s here and the bus takes 54, so a 30 MB chunk that was copied and then sent took
// both times after each other.  Eight threads copy 60 to 70 GB/s with stores that bypass the cache (16 threads
// 64, measured).  Each transfer takes about 4 us more than its bytes: 30 MB in pieces of half a megabyte 808 us, of
// 2 MB 632, of 8 MB 589, in one 577.  So the bytes are copied in small pieces but travel in transfers that grow from
// the first pieces on (to the GPU, where the copies come first) or shrink towards the last ones (from it): 30 MB
// to the GPU in 660 us, against 703 when every piece was sent as soon as it was copied.
#include <string.h>
#include <sys/mman.h>
#include <time.h>
#include <unistd.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "cg_common.cuh"
#include "cg_hostcopy.h"

namespace {

constexpr int64_t kPiece = 128 << 10;   // of a copy between host memories
constexpr int64_t kFirstSend = 256 << 10, kLastFetch = 512 << 10;  // the smallest transfer to the GPU, from it
constexpr int64_t kMostBytes = 8 << 20;                            // of a transfer that waits for its bytes to gather
constexpr int64_t kHugeFrom = 8 << 20;  // results from this size on ask for 2 MB pages
constexpr int kMaxThreads = 8;          // helpers at most: half the cores, up to this
constexpr int kSpinMicros = 60;         // a helper that has run out of work looks for more for this long
constexpr int kIdleSeconds = 5;         // ... sleeps for this long, and then ends

struct Piece {
    uint8_t *dst;
    const uint8_t *src;  // nullptr: the pages at dst are to be touched
    int64_t bytes;
    std::atomic<bool> done{false};
};

// One call's copies.  Pieces below `ready` may be taken, each by one thread.
struct Job {
    explicit Job(int n) : pieces(n) {}
    std::vector<Piece> pieces;
    std::atomic<int> ready{0}, next{0}, helpers{0};
    // what one thread does beside the copies: wanted (1), being done (2), done (3)
    std::atomic<int> beside{0};
    void (*run_beside)(void *) = nullptr;
    void *beside_of = nullptr;
    std::atomic<bool> stop{false};  // the job's pieces will not all be copied
    // does it if nobody else has begun to
    void take_beside() {
        int wanted = 1;
        if (!beside.compare_exchange_strong(wanted, 2, std::memory_order_acq_rel)) return;
        run_beside(beside_of);
        beside.store(3, std::memory_order_release);
    }
    // takes one piece and copies it; false if there is none to take now
    bool work() {
        int i = next.load(std::memory_order_relaxed);
        do {
            if (i >= ready.load(std::memory_order_acquire)) return false;
        } while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
        Piece &p = pieces[i];
        if (p.src) cg::copy_piece(p.dst, p.src, p.bytes);
        else for (int64_t k = 0; k < p.bytes; k += 4096) cg::touch_page(p.dst + k);  // may already hold data
        p.done.store(true, std::memory_order_release);
        return true;
    }
    bool taken() const { return next.load(std::memory_order_relaxed) >= static_cast<int>(pieces.size()); }
};

// Helper threads, shared by all callers; started when there is work, ended after a time without.
class Helpers {
  public:
    void add(Job *j) {
        std::lock_guard<std::mutex> lock(mu_);
        jobs_.push_back(j);
        const int cores = static_cast<int>(std::thread::hardware_concurrency());
        const int most = cores / 2 < kMaxThreads ? cores / 2 : kMaxThreads;
        const int want = static_cast<int>(j->pieces.size()) - 1 < most ? static_cast<int>(j->pieces.size()) - 1 : most;
        while (threads_ < want) {
            try {
                std::thread(&Helpers::run, this).detach();
            } catch (const std::exception &) {
                break;  // the caller copies by itself
            }
            ++threads_;
        }
        generation_.fetch_add(1, std::memory_order_release);
        wake_.notify_all();
    }
    // returns when no helper is inside the job any more
    void remove(Job *j) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            for (size_t i = 0; i < jobs_.size(); ++i)
                if (jobs_[i] == j) jobs_.erase(jobs_.begin() + static_cast<long>(i));
        }
        while (j->helpers.load(std::memory_order_acquire)) std::this_thread::yield();
    }

  private:
    void run() {
        using clock = std::chrono::steady_clock;
        auto idle_since = clock::now();
        for (;;) {
            Job *j = nullptr;
            uint64_t seen;
            {
                std::unique_lock<std::mutex> lock(mu_);
                seen = generation_.load(std::memory_order_acquire);
                for (Job *q : jobs_)
                    if (!q->taken() || q->beside.load(std::memory_order_acquire) == 1) {
                        j = q;
                        j->helpers.fetch_add(1, std::memory_order_acquire);
                        break;
                    }
            }
            if (j) {
                j->take_beside();
                while (!j->taken())
                    if (!j->work()) cg::spin_pause();
                j->helpers.fetch_sub(1, std::memory_order_release);
                idle_since = clock::now();
                continue;
            }
            if (clock::now() - idle_since < std::chrono::microseconds(kSpinMicros)) {
                while (generation_.load(std::memory_order_acquire) == seen &&
                       clock::now() - idle_since < std::chrono::microseconds(kSpinMicros))
                    cg::spin_pause();
                continue;
            }
            std::unique_lock<std::mutex> lock(mu_);
            if (generation_.load(std::memory_order_acquire) != seen) {
                idle_since = clock::now();
                continue;
            }
            if (wake_.wait_for(lock, std::chrono::seconds(kIdleSeconds)) == std::cv_status::timeout && jobs_.empty()) {
                --threads_;
                return;
            }
            idle_since = clock::now();
        }
    }
    std::mutex mu_;
    std::condition_variable wake_;
    std::vector<Job *> jobs_;
    std::atomic<uint64_t> generation_{0};
    int threads_ = 0;
};

// Never destroyed: helpers may still sleep in it when the process ends.  A forked child starts its own.
Helpers &helpers() {
    static std::mutex mu;
    static Helpers *pool = nullptr;
    static pid_t owner = 0;
    std::lock_guard<std::mutex> lock(mu);
    if (!pool || owner != getpid()) {
        pool = new Helpers;
        owner = getpid();
    }
    return *pool;
}

// A third of what is still to go, within bounds: no long transfer is left when everything else is done.
int64_t part_of(int64_t left, int64_t least, int64_t most) {
    const int64_t third = left / 3 / kPiece * kPiece;
    return third < least ? least : third > most ? most : third;
}

int64_t round_up(int64_t n) { return (n + 255) / 256 * 256; }

int check_segments(const cg_host_segment *segs, int n, const void *staging, int64_t staging_bytes, int64_t *pieces) {
    if (!segs || !staging) return CG_E_NULL;
    if (n <= 0) return CG_E_SHAPE;
    int64_t need = 0;
    *pieces = 0;
    for (int i = 0; i < n; ++i) {
        if (segs[i].bytes < 0) return CG_E_SHAPE;
        if (segs[i].bytes && (!segs[i].host || !segs[i].device)) return CG_E_NULL;
        need += round_up(segs[i].bytes);
        *pieces += (segs[i].bytes + kPiece - 1) / kPiece;
    }
    if (need > staging_bytes) return CG_E_CAPACITY;
    return *pieces > 0x7FFFFFFF ? CG_E_SHAPE : CG_OK;
}

}  // namespace

using namespace cg;

namespace {
// A part of a transfer to the GPU: it can go once the job's first `upto` pieces have been copied.
struct Part {
    uint8_t *to;
    const uint8_t *from;
    int64_t bytes;
    int upto;
};

// Sends the parts, in order, as the job's pieces are copied; the caller copies with the helpers.
cudaError_t send_parts(Job &job, const std::vector<Part> &parts, cudaStream_t st) {
    const int n = static_cast<int>(parts.size());
    int sent = 0, end = 0, copied_pieces = 0;
    int64_t left = 0, copied = 0, most = kFirstSend;  // bytes not sent yet; of those, the ones up to `end`
    for (const Part &p : parts) left += p.bytes;
    while (sent < n && !job.stop.load(std::memory_order_acquire)) {
        while (copied_pieces < static_cast<int>(job.pieces.size()) && job.pieces[copied_pieces].done.load(std::memory_order_acquire)) ++copied_pieces;
        for (; end < n && parts[end].upto <= copied_pieces; ++end) copied += parts[end].bytes;
        // all that has been copied in a row of the same tensor goes as one transfer
        const bool enough = end == n || copied >= part_of(left, kFirstSend, most);
        if (enough) {
            most = most < kMostBytes ? 2 * most : most;
            left -= copied;
            copied = 0;
        }
        while (enough && sent < end) {
            int64_t bytes = parts[sent].bytes;
            int e = sent + 1;
            while (e < end && parts[e].to == parts[sent].to + bytes && parts[e].from == parts[sent].from + bytes) bytes += parts[e++].bytes;
            const cudaError_t err = cudaMemcpyAsync(parts[sent].to, parts[sent].from, static_cast<size_t>(bytes), cudaMemcpyHostToDevice, st);
            if (err != cudaSuccess) return err;
            sent = e;
        }
        if (sent < n && !job.work()) cg::spin_pause();
    }
    return cudaSuccess;
}

// A byte string on its way into staging memory (cg_host_stage).
struct Stage {
    Stage(const void *h, int64_t n, void *s, int64_t size)
        : host(static_cast<const uint8_t *>(h)), staging(static_cast<uint8_t *>(s)), bytes(n), spare(round_up(n)), room(size), job(static_cast<int>((n + kPiece - 1) / kPiece)) {
        for (size_t k = 0; k < job.pieces.size(); ++k) {
            const int64_t a = static_cast<int64_t>(k) * kPiece;
            job.pieces[k].dst = staging + a;
            job.pieces[k].src = host + a;
            job.pieces[k].bytes = n - a < kPiece ? n - a : kPiece;
        }
        job.ready.store(static_cast<int>(job.pieces.size()), std::memory_order_release);
    }
    const uint8_t *host;
    uint8_t *staging;
    int64_t bytes, spare, room;  // of the byte string; where the staging memory is free; its size
    Job job;
    // cg_host_stage_ahead: the whole string goes to `ahead` on `stream`
    uint8_t *ahead = nullptr;
    cudaStream_t stream = nullptr;
    int device = 0;
    std::vector<Part> parts;
    cudaError_t error = cudaSuccess;
    static void send_ahead(void *self) {
        Stage &s = *static_cast<Stage *>(self);
        s.error = cudaSetDevice(s.device);
        if (s.error == cudaSuccess) s.error = send_parts(s.job, s.parts, s.stream);
    }
};

// Pieces of a byte string on the GPU to tensors of their own, whatever byte they start at: sixteen bytes a thread and pass, put
// together from the five words they lie in.  Bound by memory: the 30 MB of a Llama-7B chunk's blob in about 15 us.
constexpr int kSpreadSegments = 32, kSpreadThreads = 256;
struct SpreadList {
    uint8_t *dst[kSpreadSegments];
    const uint8_t *src[kSpreadSegments];
    int64_t bytes[kSpreadSegments];
};
__global__ void __launch_bounds__(kSpreadThreads) spread_kernel(const __grid_constant__ SpreadList list) {
    uint8_t *const dst = list.dst[blockIdx.y];
    const uint8_t *const src = list.src[blockIdx.y];
    const int64_t n = list.bytes[blockIdx.y], step = static_cast<int64_t>(gridDim.x) * kSpreadThreads * 16;
    const bool aligned = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
    const uint32_t shift = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src) & 3) * 8u;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(src) & ~static_cast<uintptr_t>(3));
    for (int64_t i = (static_cast<int64_t>(blockIdx.x) * kSpreadThreads + threadIdx.x) * 16; i < n; i += step) {
        if (aligned && i + 16 <= n) {
            uint32_t w[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) w[k] = k < 4 || shift ? __ldg(words + i / 4 + k) : 0u;
            *reinterpret_cast<uint4 *>(dst + i) = make_uint4(__funnelshift_r(w[0], w[1], shift), __funnelshift_r(w[1], w[2], shift),
                                                             __funnelshift_r(w[2], w[3], shift), __funnelshift_r(w[3], w[4], shift));
        } else {
            for (int64_t k = i; k < i + 16 && k < n; ++k) dst[k] = src[k];
        }
    }
}
}  // namespace

// No C++ exception may leave an entry: the callers are C.  What can throw is host memory that is not there, before the helpers know
// of a job, so nothing is in use when a job goes away.
extern "C" int cg_host_upload(const cg_host_segment *segs, int nsegs, void *staging, int64_t staging_bytes, void *stream) try {
    int64_t count;
    if (int rc = check_segments(segs, nsegs, staging, staging_bytes, &count)) return rc;
    if (!count) return CG_OK;
    uint8_t *stage = static_cast<uint8_t *>(staging);
    Job job(static_cast<int>(count));
    std::vector<Part> parts(static_cast<size_t>(count));
    int k = 0;
    for (int i = 0; i < nsegs; ++i) {
        const uint8_t *src = static_cast<const uint8_t *>(segs[i].host);
        for (int64_t a = 0; a < segs[i].bytes; a += kPiece, ++k) {
            job.pieces[k].dst = stage + a;
            job.pieces[k].src = src + a;
            job.pieces[k].bytes = segs[i].bytes - a < kPiece ? segs[i].bytes - a : kPiece;
            parts[k] = Part{static_cast<uint8_t *>(segs[i].device) + a, stage + a, job.pieces[k].bytes, k + 1};
        }
        stage += round_up(segs[i].bytes);
    }
    job.ready.store(k, std::memory_order_release);
    if (k > 1) helpers().add(&job);
    const cudaError_t err = send_parts(job, parts, static_cast<cudaStream_t>(stream));
    while (!job.taken()) job.work();  // only after an error: nobody may touch the job once it is gone
    if (k > 1) helpers().remove(&job);
    return err == cudaSuccess ? CG_OK : set_cuda_error(err);
} catch (const std::exception &) {
    return CG_E_CAPACITY;
}

extern "C" int cg_host_stage(const void *host, int64_t bytes, void *staging, int64_t staging_bytes, void **handle) try {
    if (!host || !staging || !handle) return CG_E_NULL;
    if (bytes <= 0 || (bytes + kPiece - 1) / kPiece > 0x7FFFFFFF) return CG_E_SHAPE;
    if (bytes > staging_bytes) return CG_E_CAPACITY;
    std::unique_ptr<Stage> s(new Stage(host, bytes, staging, staging_bytes));
    helpers().add(&s->job);
    *handle = s.release();
    return CG_OK;
} catch (const std::exception &) {
    return CG_E_CAPACITY;
}

extern "C" int cg_host_stage_ahead(const void *host, int64_t bytes, void *staging, int64_t staging_bytes, void *device_copy,
                                   void *stream, void **handle) try {
    if (!host || !staging || !handle || !device_copy) return CG_E_NULL;
    if (bytes <= 0 || (bytes + kPiece - 1) / kPiece > 0x7FFFFFFF) return CG_E_SHAPE;
    if (bytes > staging_bytes) return CG_E_CAPACITY;
    std::unique_ptr<Stage> s(new Stage(host, bytes, staging, staging_bytes));
    const cudaError_t e = cudaGetDevice(&s->device);
    if (e != cudaSuccess) return set_cuda_error(e);
    s->ahead = static_cast<uint8_t *>(device_copy);
    s->stream = static_cast<cudaStream_t>(stream);
    s->parts.resize(s->job.pieces.size());
    for (size_t k = 0; k < s->parts.size(); ++k) {
        const int64_t a = static_cast<int64_t>(k) * kPiece;
        s->parts[k] = Part{s->ahead + a, s->staging + a, s->job.pieces[k].bytes, static_cast<int>(k) + 1};
    }
    s->job.run_beside = Stage::send_ahead;
    s->job.beside_of = s.get();
    s->job.beside.store(1, std::memory_order_release);
    helpers().add(&s->job);
    *handle = s.release();
    return CG_OK;
} catch (const std::exception &) {
    return CG_E_CAPACITY;
}

// What follows a string that went ahead: its segments from the copy on the GPU, small ones from elsewhere through the free part
// of the staging memory.
static int spread_ahead(Stage &s, const cg_host_segment *segs, int nsegs) {
    s.job.take_beside();
    while (s.job.beside.load(std::memory_order_acquire) != 3)
        if (!s.job.work()) cg::spin_pause();
    if (s.error != cudaSuccess) return set_cuda_error(s.error);
    SpreadList list;
    int n = 0;
    int64_t longest = 0;
    const auto launch = [&]() -> int {
        if (!n) return CG_OK;
        const int64_t blocks = (longest + kSpreadThreads * 16 - 1) / (kSpreadThreads * 16);
        spread_kernel<<<dim3(static_cast<unsigned>(blocks < 2048 ? blocks : 2048), n), kSpreadThreads, 0, s.stream>>>(list);
        n = 0;
        longest = 0;
        return check_launch();
    };
    for (int i = 0; i < nsegs; ++i) {
        if (!segs[i].bytes) continue;
        const uint8_t *host = static_cast<const uint8_t *>(segs[i].host);
        const uintptr_t in = reinterpret_cast<uintptr_t>(host) - reinterpret_cast<uintptr_t>(s.host);
        if (in >= static_cast<uintptr_t>(s.bytes)) {
            memcpy(s.staging + s.spare, host, static_cast<size_t>(segs[i].bytes));
            const cudaError_t e = cudaMemcpyAsync(segs[i].device, s.staging + s.spare, static_cast<size_t>(segs[i].bytes), cudaMemcpyHostToDevice, s.stream);
            if (e != cudaSuccess) return set_cuda_error(e);
            s.spare += round_up(segs[i].bytes);
            continue;
        }
        list.dst[n] = static_cast<uint8_t *>(segs[i].device);
        list.src[n] = s.ahead + in;
        list.bytes[n] = segs[i].bytes;
        longest = segs[i].bytes > longest ? segs[i].bytes : longest;
        if (++n == kSpreadSegments)
            if (int rc = launch()) return rc;
    }
    return launch();
}

extern "C" int cg_host_stage_send(void *handle, const cg_host_segment *segs, int nsegs, void *stream) try {
    if (!handle || !segs) return CG_E_NULL;
    Stage &s = *static_cast<Stage *>(handle);
    if (s.ahead) {
        if (static_cast<cudaStream_t>(stream) != s.stream) return CG_E_SHAPE;
        int64_t spare = s.spare;  // all segments are looked at before anything is launched
        for (int i = 0; i < nsegs; ++i) {
            if (segs[i].bytes < 0) return CG_E_SHAPE;
            if (segs[i].bytes && (!segs[i].device || !segs[i].host)) return CG_E_NULL;
            const uintptr_t in = reinterpret_cast<uintptr_t>(segs[i].host) - reinterpret_cast<uintptr_t>(s.host);
            if (in >= static_cast<uintptr_t>(s.bytes)) {
                if (segs[i].bytes > s.room - spare) return CG_E_CAPACITY;
                spare += round_up(segs[i].bytes);
            } else if (segs[i].bytes > s.bytes - static_cast<int64_t>(in)) {
                return CG_E_SHAPE;
            }
        }
        return spread_ahead(s, segs, nsegs);
    }
    std::vector<Part> parts;
    for (int i = 0; i < nsegs; ++i) {
        if (segs[i].bytes < 0) return CG_E_SHAPE;
        if (segs[i].bytes && (!segs[i].device || !segs[i].host)) return CG_E_NULL;
        const uint8_t *host = static_cast<const uint8_t *>(segs[i].host);
        const uintptr_t in = reinterpret_cast<uintptr_t>(host) - reinterpret_cast<uintptr_t>(s.host);
        if (in >= static_cast<uintptr_t>(s.bytes)) {  // outside the byte string: to the free part, by the caller
            if (segs[i].bytes > s.room - s.spare) return CG_E_CAPACITY;
            memcpy(s.staging + s.spare, host, static_cast<size_t>(segs[i].bytes));
            parts.push_back(Part{static_cast<uint8_t *>(segs[i].device), s.staging + s.spare, segs[i].bytes, 0});
            s.spare += round_up(segs[i].bytes);
            continue;
        }
        if (segs[i].bytes > s.bytes - static_cast<int64_t>(in)) return CG_E_SHAPE;
        const int64_t at = static_cast<int64_t>(in);
        for (int64_t a = 0; a < segs[i].bytes;) {  // up to the end of the piece
            const int64_t k = (at + a) / kPiece, room = (k + 1) * kPiece - (at + a);
            const int64_t n = room < segs[i].bytes - a ? room : segs[i].bytes - a;
            parts.push_back(Part{static_cast<uint8_t *>(segs[i].device) + a, s.staging + at + a, n, static_cast<int>(k) + 1});
            a += n;
        }
    }
    const cudaError_t err = send_parts(s.job, parts, static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? CG_OK : set_cuda_error(err);
} catch (const std::exception &) {
    return CG_E_CAPACITY;
}

extern "C" int cg_host_stage_end(void *handle) {
    if (!handle) return CG_E_NULL;
    Stage *s = static_cast<Stage *>(handle);
    s->job.next.store(static_cast<int>(s->job.pieces.size()), std::memory_order_relaxed);  // what has not been sent is not wanted
    s->job.stop.store(true, std::memory_order_release);
    int wanted = 1;
    s->job.beside.compare_exchange_strong(wanted, 3, std::memory_order_acq_rel);
    helpers().remove(&s->job);
    delete s;
    return CG_OK;
}

namespace {
// events of this thread, made once per device and kept
struct Events {
    int device = -1;
    std::vector<cudaEvent_t> list;
    ~Events() {
        for (cudaEvent_t v : list) cudaEventDestroy(v);
    }
    cudaError_t want(size_t n) {
        int dev;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev != device) {
            for (cudaEvent_t v : list) cudaEventDestroy(v);
            list.clear();
            device = dev;
        }
        while (list.size() < n) {
            cudaEvent_t v;
            e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
            if (e != cudaSuccess) return e;
            list.push_back(v);
        }
        return cudaSuccess;
    }
};
constexpr int64_t kMaxUnits = 64;
}  // namespace

extern "C" int cg_host_download(const cg_host_segment *segs, int nsegs, void *staging, int64_t staging_bytes, int phase,
                                void *stream) try {
    int64_t count;
    if (phase < 0 || phase > 2) return CG_E_SHAPE;
    if (!segs || !staging) return CG_E_NULL;
    if (phase == 1) {  // host pointers come with the second phase
        std::vector<cg_host_segment> any(segs, segs + (nsegs > 0 ? nsegs : 0));
        for (auto &x : any) x.host = staging;
        if (int rc = check_segments(any.data(), nsegs, staging, staging_bytes, &count)) return rc;
    } else if (int rc = check_segments(segs, nsegs, staging, staging_bytes, &count)) {
        return rc;
    }
    if (!count) return CG_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    static thread_local Events events;
    const int n = static_cast<int>(count);
    // the transfers, in the order of the bytes; the events follow them
    struct Unit {
        int segment;
        int64_t at, bytes;
    };
    std::vector<Unit> units;
    std::vector<int64_t> start(static_cast<size_t>(nsegs), 0);  // of each segment in the staging memory
    for (int i = 1; i < nsegs; ++i) start[i] = start[i - 1] + round_up(segs[i - 1].bytes);
    int64_t left = 0, most = kMostBytes;
    for (int i = 0; i < nsegs; ++i) left += segs[i].bytes;
    while (left / most > kMaxUnits) most *= 2;
    for (int i = 0; i < nsegs; ++i)
        for (int64_t a = 0; a < segs[i].bytes;) {
            const int64_t part = part_of(left, kLastFetch, most), rest = segs[i].bytes - a;
            units.push_back({i, a, part < rest ? part : rest});
            a += units.back().bytes;
            left -= units.back().bytes;
        }
    cudaError_t err = events.want(units.size());
    if (err != cudaSuccess) return set_cuda_error(err);
    if (phase != 2) {
        uint8_t *stage = static_cast<uint8_t *>(staging);
        for (size_t u = 0; u < units.size() && err == cudaSuccess; ++u) {
            const Unit &t = units[u];
            err = cudaMemcpyAsync(stage + start[t.segment] + t.at, static_cast<const uint8_t *>(segs[t.segment].device) + t.at,
                                  static_cast<size_t>(t.bytes), cudaMemcpyDeviceToHost, st);
            if (err == cudaSuccess) err = cudaEventRecord(events.list[u], st);
        }
        if (err != cudaSuccess) {
            cudaStreamSynchronize(st);
            return set_cuda_error(err);
        }
        if (phase == 1) return CG_OK;
    }
    // Fresh memory is faulted in while it is written: 7,500 pages of 30 MB took the copying threads 1.4 ms.  So a
    // large result asks for 2 MB pages, and they are touched, each by one thread, while the transfers run.
    constexpr uintptr_t kHuge = 2 << 20;
    std::vector<std::pair<uint8_t *, int64_t>> touch;
    for (int i = 0; i < nsegs; ++i) {
        if (segs[i].bytes < kHugeFrom) continue;
        const uintptr_t dst = reinterpret_cast<uintptr_t>(segs[i].host), end = dst + static_cast<uintptr_t>(segs[i].bytes);
        const uintptr_t first = (dst + 4095) & ~uintptr_t{4095}, last = end & ~uintptr_t{4095};
        madvise(reinterpret_cast<void *>(first), last - first, MADV_HUGEPAGE);
        for (uintptr_t p = dst; p < end;) {
            // outside the whole 2 MB pages there are small ones to fault in one by one: less at a time
            const bool whole = p % kHuge == 0 && p + kHuge <= last;
            const uintptr_t stop = whole ? p + kHuge : (p / (kHuge / 16) + 1) * (kHuge / 16);
            const uintptr_t next = stop < end ? stop : end;
            touch.emplace_back(reinterpret_cast<uint8_t *>(p), static_cast<int64_t>(next - p));
            p = next;
        }
    }
    const int lead = static_cast<int>(touch.size());
    Job job(lead + n);
    for (int i = 0; i < lead; ++i) {
        job.pieces[i].dst = touch[i].first;
        job.pieces[i].src = nullptr;
        job.pieces[i].bytes = touch[i].second;
    }
    job.ready.store(lead, std::memory_order_release);
    std::vector<int> upto;  // pieces that may be taken once each transfer has arrived
    const uint8_t *stage = static_cast<const uint8_t *>(staging);
    int k = lead;
    for (const Unit &t : units) {
        for (int64_t a = 0; a < t.bytes; a += kPiece, ++k) {
            job.pieces[k].dst = static_cast<uint8_t *>(segs[t.segment].host) + t.at + a;
            job.pieces[k].src = stage + start[t.segment] + t.at + a;
            job.pieces[k].bytes = t.bytes - a < kPiece ? t.bytes - a : kPiece;
        }
        upto.push_back(k);
    }
    if (n > 1) helpers().add(&job);
    size_t arrived = 0;
    while (!job.taken()) {
        if (arrived < upto.size()) {
            const cudaError_t q = cudaEventQuery(events.list[arrived]);
            if (q == cudaSuccess) {
                job.ready.store(upto[arrived++], std::memory_order_release);
                continue;
            }
            if (q != cudaErrorNotReady) {
                err = q;
                break;
            }
        }
        if (!job.work()) cg::spin_pause();
    }
    if (err != cudaSuccess) job.next.store(lead + n, std::memory_order_relaxed);  // nothing more to take
    if (n > 1) helpers().remove(&job);
    return err == cudaSuccess ? CG_OK : set_cuda_error(err);
} catch (const std::exception &) {
    cudaStreamSynchronize(static_cast<cudaStream_t>(stream));  // transfers may be on their way to the staging memory
    return CG_E_CAPACITY;
}
