// Ray queries on host arrays (pt_trace_rays, pt_occluded).
//
// Rays and results pass through page-locked staging, one copy in and one out per chunk. Copies
// from and to the caller's pageable arrays, one per array, held these calls at 15 GB/s, 0.1 ms even
// for a single ray. Calls beyond four chunks are worked off by several host threads, each with its own
// stream and staging: a thread copies a chunk's rays into its staging, queues copy, kernel and
// copy back, and copies the results out while the other threads' chunks are on the bus and on
// the GPU. The staging is bounded (kQueryWorkers chunks) and borrowed from the process's pool. Large
// calls whose arrays overlap, or are page-locked already, are not cut up: whole_query copies each array once.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <vector>

#include "../../include/pathed.h"
#include "session.h"

namespace pt {

namespace {
// Rays per chunk, with 8 threads: 1M / 200k / 33k closest hits in ms at 8192 rays 2.6 / 0.64 / 0.21, at 16384 2.1 /
// 0.56 / 0.24, at 32768 2.0 / 0.8 / 0.29 (whole-array copies on one thread: 4.2 / 1.03 / 0.34). The staging, 0.9 MB per
// thread, takes about 4 ms to page-lock, once per process.
constexpr size_t kChunkRays = 16384;
// Up to here a call is one piece, staged by the calling thread: starting threads and their first CUDA call cost more
// than they save. 17k / 33k / 50k / 66k / 100k closest hits in ms in one piece 0.15 / 0.23 / 0.30 / 0.37 / 0.51, in
// chunks on several threads 0.17 / 0.37 / 0.46 / 0.36 / 0.36 (whole-array copies 0.22 / 0.27 / 0.36 / 0.41 / 0.55). The
// staging of such a piece stays within the pool's (kQueryWorkers chunks).
constexpr size_t kOnePiece = 4 * kChunkRays;
// Up to here the kernel reads and writes the staging itself: 42 us for one ray, 105 us before.
constexpr int kDirectRays = 2048;
constexpr size_t kInBytes = 32;     // origin, direction, tmin, tmax
constexpr size_t kFlagBytes = 16;   // overflow flag, work cursor
constexpr size_t kOutBytes = 24;    // type, primitive, material, t, barycentrics
size_t chunk_bytes(size_t n) { return (n * (kInBytes + kOutBytes) + kFlagBytes + 255) & ~(size_t)255; }

struct Array {  // one of a call's arrays, null where the call has none
    const void* p;
    size_t bytes;
};
struct Arrays {
    Array in[4], out[6];
    Arrays(const HostRays& r, const HostHits& h)
        : in{{r.o, 12 * (size_t)r.n}, {r.d, 12 * (size_t)r.n}, {r.tmin, 4 * (size_t)r.n}, {r.tmax, 4 * (size_t)r.n}},
          out{{h.prim_type, 4 * (size_t)r.n}, {h.prim_id, 4 * (size_t)r.n}, {h.mat_id, 4 * (size_t)r.n},
              {h.t, 4 * (size_t)r.n}, {h.bary, 8 * (size_t)r.n}, {h.occluded, 4 * (size_t)r.n}} {}
    // no array that is written shares memory with another one
    bool apart() const {
        for (int k = 0; k < 6; k++) {
            for (const Array& a : in)
                if (overlap(a, out[k])) return false;
            for (int i = 0; i < k; i++)
                if (overlap(out[i], out[k])) return false;
        }
        return true;
    }
    // the arrays' memory: every one page-locked; one of them device memory, which the host cannot read
    void memory(bool& locked, bool& device) const {
        locked = true;
        device = false;
        auto look = [&](const Array& a) {
            cudaPointerAttributes attr{};
            if (!a.p) return;
            if (cudaPointerGetAttributes(&attr, a.p) != cudaSuccess) cudaGetLastError();  // unknown: as any host memory
            locked = locked && attr.type == cudaMemoryTypeHost;
            device = device || attr.type == cudaMemoryTypeDevice;
        };
        for (const Array& a : in) look(a);
        for (const Array& a : out) look(a);
    }
    static bool overlap(const Array& a, const Array& b) {
        const char *x = static_cast<const char*>(a.p), *y = static_cast<const char*>(b.p);
        return x && y && x < y + b.bytes && y < x + a.bytes;
    }
};
}  // namespace

QueryStaging::~QueryStaging() {
    for (cudaStream_t s : streams)
        if (s) cudaStreamDestroy(s);
    if (host) cudaFreeHost(host);
}

QueryPool& QueryPool::get() {
    static QueryPool* p = new QueryPool;  // never destroyed: no CUDA calls while the process ends
    return *p;
}

std::unique_ptr<QueryStaging> QueryPool::take(int device) {
    {
        std::lock_guard<std::mutex> lock(m_);
        for (size_t i = 0; i < idle_.size(); i++)
            if (idle_[i]->device == device) {
                std::unique_ptr<QueryStaging> s = std::move(idle_[i]);
                idle_.erase(idle_.begin() + i);
                return s;
            }
    }
    return std::unique_ptr<QueryStaging>(new QueryStaging(device));
}

void QueryPool::give(std::unique_ptr<QueryStaging> s) {
    std::lock_guard<std::mutex> lock(m_);
    int idle = 0;
    for (const auto& i : idle_) idle += i->device == s->device;
    if (sessions_[s->device] > 0 && idle < kQueryStagings && s->host_bytes <= kQueryWorkers * chunk_bytes(kChunkRays))
        idle_.push_back(std::move(s));
}

void QueryPool::attach(int device) {
    std::lock_guard<std::mutex> lock(m_);
    sessions_[device]++;
}

void QueryPool::detach(int device) {
    std::vector<std::unique_ptr<QueryStaging>> gone;  // freed after the lock
    std::lock_guard<std::mutex> lock(m_);
    if (--sessions_[device] > 0) return;
    for (size_t i = idle_.size(); i-- > 0;)
        if (idle_[i]->device == device) {
            gone.push_back(std::move(idle_[i]));
            idle_.erase(idle_.begin() + i);
        }
}

cudaError_t QueryStaging::ensure(int workers, size_t bytes_each) {
    cudaError_t e;
    if ((size_t)workers * bytes_each > host_bytes) {
        if (host) cudaFreeHost(host);
        host = nullptr;
        host_bytes = 0;
        if ((e = cudaMallocHost(&host, workers * bytes_each))) return e;
        host_bytes = workers * bytes_each;
    }
    if ((e = dev.alloc(workers * bytes_each))) return e;
    while ((int)streams.size() < workers) {
        cudaStream_t st = nullptr;
        if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking))) return e;
        streams.push_back(st);
    }
    return cudaSuccess;
}

int Session::host_query(const HostRays& rays, const HostHits& out) {
    const Arrays arrays(rays, out);
    bool locked, device;
    arrays.memory(locked, device);  // 0.1 us per array
    if (device) return fail(PT_ERR_ARG, "device memory passed as a host array (pt_trace_rays_device takes it)");
    // a chunk's results are written while later chunks' rays are unread: only when no arrays overlap
    const bool apart = arrays.apart();
    if (!apart && (size_t)rays.n > kOnePiece) return whole_query(rays, out);
    // the bus reads and writes page-locked arrays as they are: 33k / 200k / 1M closest hits in ms 0.18 / 0.43 / 1.5,
    // staged 0.37 / 0.53 / 2.0; up to one chunk the staging's single copies win (10k: 0.10, one copy per array 0.12)
    if ((size_t)rays.n > kChunkRays && locked) return whole_query(rays, out);
    std::unique_ptr<QueryStaging> staging = QueryPool::get().take(device_);
    const int r = staged_query(rays, out, (size_t)rays.n <= kOnePiece ? kOnePiece : kChunkRays, *staging);
    // nothing of it is in use: every worker has waited for its stream; after an error it is freed
    if (r == PT_OK) QueryPool::get().give(std::move(staging));
    return r;
}

// The whole call at once: every array is copied by itself from and to the caller's memory, in stream
// order, so all rays are read before a result is written.
int Session::whole_query(const HostRays& rays, const HostHits& out) {
    const size_t n = (size_t)rays.n;
    const Arrays arrays(rays, out);
    int r;
    if ((r = check_cuda(d_scratch_.alloc(n * (kInBytes + kOutBytes) + kFlagBytes), "scratch"))) return r;
    char* g = d_scratch_.as<char>();
    float* f = reinterpret_cast<float*>(g);
    int* flags = reinterpret_cast<int*>(g + kInBytes * n);
    int* o = reinterpret_cast<int*>(g + kInBytes * n + kFlagBytes);
    int flag = 0;
    auto enqueue = [&]() -> cudaError_t {
        cudaError_t e;
        char* at = g;
        for (const Array& a : arrays.in) {
            if ((e = cudaMemcpyAsync(at, a.p, a.bytes, cudaMemcpyHostToDevice, stream_))) return e;
            at += a.bytes;
        }
        if ((e = cudaMemsetAsync(flags, 0, kFlagBytes, stream_))) return e;
        const StackShape stack = stack_shape(kMainStacks);
        e = out.occluded ? enqueue_occluded(scene_view(), stack, f, f + 3 * n, f + 6 * n, f + 7 * n, rays.n, o, flags, stream_)
                         : enqueue_trace_rays(scene_view(), stack, f, f + 3 * n, f + 6 * n, f + 7 * n, rays.n, o, o + n,
                                              o + 2 * n, reinterpret_cast<float*>(o + 3 * n),
                                              out.bary ? reinterpret_cast<float*>(o + 4 * n) : nullptr, flags, stream_);
        if (e != cudaSuccess) return e;
        at = reinterpret_cast<char*>(o);
        for (const Array& a : arrays.out) {
            if (!a.p) continue;
            if ((e = cudaMemcpyAsync(const_cast<void*>(a.p), at, a.bytes, cudaMemcpyDeviceToHost, stream_))) return e;
            at += a.bytes;
        }
        return cudaMemcpyAsync(&flag, flags, sizeof(int), cudaMemcpyDeviceToHost, stream_);
    };
    const cudaError_t e = enqueue();
    const cudaError_t s = cudaStreamSynchronize(stream_);  // also after an error: no copy may land after the return
    if ((r = check_cuda(e != cudaSuccess ? e : s, "ray query"))) return r;
    if (flag) return fail(PT_ERR_DEVICE, "traversal stack overflow reported by a kernel");
    return PT_OK;
}

// The call in chunks of at most `chunk_rays`, through `staging`.
int Session::staged_query(const HostRays& rays, const HostHits& out, size_t chunk_rays, QueryStaging& staging) {
    const size_t n = (size_t)rays.n;
    const bool any = out.occluded != nullptr;
    const size_t chunk = std::min(n, chunk_rays);
    const int chunks = (int)((n + chunk - 1) / chunk);
    const int threads = std::max(1, (int)std::thread::hardware_concurrency() / 2);
    const int workers = std::min({chunks, kQueryWorkers, threads});
    // whole chunks, so that longer and longer calls do not page-lock their staging anew each time
    const size_t each = chunk_bytes(chunk <= kChunkRays ? chunk : (chunk + kChunkRays - 1) / kChunkRays * kChunkRays);
    int r;
    if ((r = check_cuda(staging.ensure(workers, each), "query staging"))) return r;

    const SceneDevice sc = scene_view();
    const size_t deep = (size_t)std::max(0, stack_need(bvh_.width, bvh_.depth) - kStackShared);
    const int lanes = num_sms_ * kStackLanes / workers / 128 * 128;  // each worker's part of the stacks' global memory
    std::atomic<int> next{0};
    std::atomic<int> err{(int)cudaSuccess}, overflowed{0};
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(device_);
        char* h = static_cast<char*>(staging.host) + w * each;
        char* d = staging.dev.as<char>() + w * each;
        const cudaStream_t st = staging.streams[w];
        StackShape stack = stack_shape(kMainStacks);
        stack.spill_stride = lanes;
        if (stack.spill) stack.spill = static_cast<char*>(stack.spill) + (size_t)w * deep * lanes * sizeof(int2);
        for (int c; e == cudaSuccess && err.load() == (int)cudaSuccess && (c = next.fetch_add(1)) < chunks;) {
            const size_t at = c * chunk, m = std::min(chunk, n - at);
            // staging: o, d, tmin, tmax, flags, then the results
            std::memcpy(h, rays.o + 3 * at, 12 * m);
            std::memcpy(h + 12 * m, rays.d + 3 * at, 12 * m);
            std::memcpy(h + 24 * m, rays.tmin + at, 4 * m);
            std::memcpy(h + 28 * m, rays.tmax + at, 4 * m);
            std::memset(h + kInBytes * m, 0, kFlagBytes);
            const bool direct = m <= (size_t)kDirectRays && chunks == 1;
            const size_t in_bytes = kInBytes * m + kFlagBytes;
            const size_t out_bytes = any ? 4 * m : (out.bary ? 24 : 16) * m;
            char* g = direct ? h : d;
            if (!direct && (e = cudaMemcpyAsync(d, h, in_bytes, cudaMemcpyHostToDevice, st))) break;
            float* f = reinterpret_cast<float*>(g);
            int* flags = reinterpret_cast<int*>(g + kInBytes * m);
            int* o = reinterpret_cast<int*>(g + in_bytes);
            e = any ? enqueue_occluded(sc, stack, f, f + 3 * m, f + 6 * m, f + 7 * m, (int)m, o, flags, st)
                    : enqueue_trace_rays(sc, stack, f, f + 3 * m, f + 6 * m, f + 7 * m, (int)m, o, o + m, o + 2 * m,
                                         reinterpret_cast<float*>(o + 3 * m),
                                         out.bary ? reinterpret_cast<float*>(o + 4 * m) : nullptr, flags, st);
            if (e == cudaSuccess && !direct)
                e = cudaMemcpyAsync(h + kInBytes * m, d + kInBytes * m, kFlagBytes + out_bytes, cudaMemcpyDeviceToHost, st);
            const cudaError_t s = cudaStreamSynchronize(st);  // also after an error: nothing may still write the staging
            if (e != cudaSuccess || (e = s) != cudaSuccess) break;
            int flag;
            std::memcpy(&flag, h + kInBytes * m, sizeof(int));
            if (flag) overflowed.store(1);
            const char* res = h + in_bytes;
            if (any) {
                std::memcpy(out.occluded + at, res, 4 * m);
            } else {
                std::memcpy(out.prim_type + at, res, 4 * m);
                std::memcpy(out.prim_id + at, res + 4 * m, 4 * m);
                std::memcpy(out.mat_id + at, res + 8 * m, 4 * m);
                std::memcpy(out.t + at, res + 12 * m, 4 * m);
                if (out.bary) std::memcpy(out.bary + 2 * at, res + 16 * m, 8 * m);
            }
        }
        if (e != cudaSuccess) {
            int none = (int)cudaSuccess;
            err.compare_exchange_strong(none, (int)e);
        }
    };
    std::vector<std::thread> helpers;
    helpers.reserve(workers);
    for (int w = 1; w < workers; w++) {
        try {
            helpers.emplace_back(work, w);
        } catch (...) {
            break;  // no thread to be had: the others take its chunks
        }
    }
    work(0);
    for (std::thread& t : helpers) t.join();
    if ((r = check_cuda((cudaError_t)err.load(), "ray query"))) return r;
    if (overflowed.load()) return fail(PT_ERR_DEVICE, "traversal stack overflow reported by a kernel");
    return PT_OK;
}

}  // namespace pt
