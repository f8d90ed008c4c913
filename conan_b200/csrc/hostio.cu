// hostio.cu -- see hostio.cuh.
#include "hostio.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace conan {
namespace {

constexpr int MAX_DEVICES = 64;

struct Lane {
    cudaStream_t st = nullptr;
    void *buf = nullptr;
};

struct Plan {
    int device, R, n;
    bool dbl;
    FFTPair fft;
};

// Never destroyed: at process exit the CUDA context may be gone before it.
struct Caches {
    std::mutex mu;
    std::vector<Lane> idle[MAX_DEVICES];
    int lanes[MAX_DEVICES] = {};  // existing, idle or in use
    cudaMemPool_t pool[MAX_DEVICES] = {};
    std::vector<Plan> plans;  // idle, oldest first
};
Caches &caches() {
    static Caches *c = new Caches;
    return *c;
}

int current_device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= MAX_DEVICES) {
        cudaGetLastError();
        return -1;
    }
    return d;
}

void lane_destroy(Lane &l) {
    if (l.st) cudaStreamDestroy(l.st);
    if (l.buf) cudaFreeHost(l.buf);
    l = Lane{};
}

// Up to `want` lanes of the device; fewer (or none) when others hold them.
std::vector<Lane> lanes_take(int dev, int want) {
    std::vector<Lane> got;
    Caches &c = caches();
    std::lock_guard<std::mutex> lock(c.mu);
    while ((int)got.size() < want) {
        if (!c.idle[dev].empty()) {
            got.push_back(c.idle[dev].back());
            c.idle[dev].pop_back();
        } else if (c.lanes[dev] < HOSTIO_LANES) {
            Lane l;
            if (cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking) != cudaSuccess ||
                cudaHostAlloc(&l.buf, HOSTIO_CHUNK, cudaHostAllocDefault) != cudaSuccess) {
                cudaGetLastError();
                lane_destroy(l);
                break;
            }
            ++c.lanes[dev];
            got.push_back(l);
        } else {
            break;
        }
    }
    return got;
}

void lanes_return(int dev, std::vector<Lane> &l) {
    Caches &c = caches();
    std::lock_guard<std::mutex> lock(c.mu);
    c.idle[dev].insert(c.idle[dev].end(), l.begin(), l.end());
    l.clear();
}

bool page_locked(const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

// Copies `bytes` between host and device in chunks over the lanes, one host
// thread per lane taking the next chunk; everything has arrived on return.
cudaError_t lanes_copy(int dev, std::vector<Lane> &lanes, char *host, char *devp, size_t bytes, bool to_host,
                       cudaEvent_t after) {
    const size_t nc = (bytes + HOSTIO_CHUNK - 1) / HOSTIO_CHUNK;
    std::atomic<size_t> next{0};
    std::atomic<int> err{0};
    auto work = [&](const Lane &l) {
        cudaError_t e = cudaSetDevice(dev);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(l.st, after, 0);
        for (size_t c; e == cudaSuccess && !err.load() && (c = next.fetch_add(1)) < nc;) {
            const size_t o = c * HOSTIO_CHUNK, n = std::min(HOSTIO_CHUNK, bytes - o);
            if (!to_host) std::memcpy(l.buf, host + o, n);
            e = to_host ? cudaMemcpyAsync(l.buf, devp + o, n, cudaMemcpyDeviceToHost, l.st)
                        : cudaMemcpyAsync(devp + o, l.buf, n, cudaMemcpyHostToDevice, l.st);
            const cudaError_t s = cudaStreamSynchronize(l.st);  // also before the buffer goes back
            if (e == cudaSuccess) e = s;
            if (e == cudaSuccess && to_host) std::memcpy(host + o, l.buf, n);
        }
        if (e != cudaSuccess) err.store((int)e);
    };
    std::vector<std::thread> th;
    try {
        th.reserve(lanes.size());
        for (size_t i = 1; i < lanes.size(); ++i) th.emplace_back(work, std::cref(lanes[i]));
    } catch (...) {  // fewer threads than lanes: those that run take all chunks
    }
    work(lanes[0]);
    for (auto &t : th) t.join();
    return (cudaError_t)err.load();
}

int copy(void *host, void *devp, size_t bytes, bool to_host, cudaStream_t st) {
    // below four chunks the threads' start costs more than it saves (6 MB out
    // and in: 0.42 ms by the driver, 0.6 with three threads; 50 MB into fresh
    // pages 11 ms by the driver, 3.2 with eight)
    static const int cores = (int)std::thread::hardware_concurrency();  // a read of /sys
    const int want = (int)std::min<size_t>(std::min(HOSTIO_LANES, std::max(1, cores / 2)),
                                           bytes / HOSTIO_CHUNK);
    const int dev = want >= 4 ? current_device() : -1;
    if (dev >= 0 && !page_locked(host)) {
        std::vector<Lane> lanes = lanes_take(dev, want);
        if (lanes.size() >= 2) {
            cudaEvent_t after = nullptr;
            cudaError_t e = cudaEventCreateWithFlags(&after, cudaEventDisableTiming);
            if (e == cudaSuccess) e = cudaEventRecord(after, st);
            if (e == cudaSuccess) e = lanes_copy(dev, lanes, (char *)host, (char *)devp, bytes, to_host, after);
            if (after) cudaEventDestroy(after);
            lanes_return(dev, lanes);
            if (e != cudaSuccess) return set_error(CONAN_ERR_CUDA, "host copy: %s", cudaGetErrorString(e));
            return CONAN_OK;
        }
        lanes_return(dev, lanes);
    }
    if (to_host) CONAN_CUDA(cudaMemcpyAsync(host, devp, bytes, cudaMemcpyDeviceToHost, st));
    else CONAN_CUDA(cudaMemcpyAsync(devp, host, bytes, cudaMemcpyHostToDevice, st));
    return CONAN_OK;
}

}  // namespace

int copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    return copy(dst, const_cast<void *>(src), bytes, true, st);
}
int copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    return copy(const_cast<void *>(src), dst, bytes, false, st);
}

cudaError_t pool_alloc(void **p, size_t bytes, cudaStream_t st) {
    const int dev = current_device();
    cudaMemPool_t pool = nullptr;
    if (dev >= 0) {
        Caches &c = caches();
        std::lock_guard<std::mutex> lock(c.mu);
        if (!c.pool[dev]) {
            cudaMemPoolProps pr{};
            pr.allocType = cudaMemAllocationTypePinned;
            pr.location.type = cudaMemLocationTypeDevice;
            pr.location.id = dev;
            cudaError_t e = cudaMemPoolCreate(&c.pool[dev], &pr);
            if (e != cudaSuccess) {
                c.pool[dev] = nullptr;
                return e;
            }
            unsigned long long keep = HOSTIO_POOL_KEEP;
            cudaMemPoolSetAttribute(c.pool[dev], cudaMemPoolAttrReleaseThreshold, &keep);
        }
        pool = c.pool[dev];
    }
    if (!pool) return cudaErrorInvalidDevice;
    return alloc_retry([&] { return cudaMallocFromPoolAsync(p, bytes ? bytes : 16, pool, st); });
}
void pool_free(void *p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}

int plan_take(const Mesh &m, bool is_double, FFTPair *fft) {
    const int dev = current_device();
    {
        Caches &c = caches();
        std::lock_guard<std::mutex> lock(c.mu);
        for (size_t i = 0; i < c.plans.size(); ++i) {
            const Plan &p = c.plans[i];
            if (p.device == dev && p.R == m.R && p.n == m.n && p.dbl == is_double) {
                *fft = p.fft;
                c.plans.erase(c.plans.begin() + (long)i);
                return CONAN_OK;
            }
        }
    }
    return fft->create(m, is_double, 1);
}

void plan_return(const Mesh &m, bool is_double, FFTPair *fft) {
    if (!fft->r2c || !fft->c2r) {  // a pair that was not made
        fft->destroy();
        return;
    }
    FFTPair old;
    {
        Caches &c = caches();
        std::lock_guard<std::mutex> lock(c.mu);
        c.plans.push_back(Plan{current_device(), m.R, m.n, is_double, *fft});
        *fft = FFTPair{};
        if ((int)c.plans.size() > HOSTIO_PLANS) {
            old = c.plans.front().fft;
            c.plans.erase(c.plans.begin());
        }
    }
    old.destroy();
}

int release_caches() {
    Caches &c = caches();
    std::lock_guard<std::mutex> lock(c.mu);
    int was = 0;
    const bool have = cudaGetDevice(&was) == cudaSuccess;
    for (auto &p : c.plans) {
        if (have) cudaSetDevice(p.device);
        p.fft.destroy();
    }
    c.plans.clear();
    for (int d = 0; d < MAX_DEVICES; ++d) {
        if (!c.idle[d].empty() || c.pool[d]) cudaSetDevice(d);
        for (auto &l : c.idle[d]) {
            lane_destroy(l);
            --c.lanes[d];
        }
        c.idle[d].clear();
        if (c.pool[d]) cudaMemPoolTrimTo(c.pool[d], 0);
    }
    if (have) cudaSetDevice(was);
    cudaGetLastError();
    return CONAN_OK;
}

}  // namespace conan

extern "C" int conan_release_caches(void) { return conan::release_caches(); }
