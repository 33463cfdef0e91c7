// common.cu -- error state, CFA parsing and device queries shared by the
// imops_b200 entry points.
#include "common.cuh"

#include <cstdlib>
#include <cstring>
#include <atomic>
#include <mutex>
#include <thread>

namespace imops {

namespace {
thread_local std::string g_last_error;
}

void set_error(const std::string& msg) { g_last_error = msg; }
void clear_error() { g_last_error.clear(); }
const char* last_error() { return g_last_error.c_str(); }

int fail(int code, const std::string& msg) {
    set_error(msg);
    return code;
}

int cuda_status(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return IMOPS_OK;
    std::string m = std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    if (e == cudaErrorMemoryAllocation) return fail(IMOPS_ERR_OUT_OF_MEMORY, m);
    return fail(IMOPS_ERR_CUDA, m);
}

int parse_cfa(const char* pattern, int shift_x, int shift_y, CfaDev* out) {
    if (!pattern) return fail(IMOPS_ERR_INVALID_ARGUMENT, "CFA pattern is NULL");
    size_t n = std::strlen(pattern);
    int pw, ph;
    switch (n) {
        case 4: pw = 2; ph = 2; break;
        case 36: pw = 6; ph = 6; break;
        case 16: pw = 2; ph = 8; break;
        case 144: pw = 12; ph = 12; break;
        default:
            return fail(IMOPS_ERR_UNSUPPORTED_CFA, std::string("Unknown CFA size \"") + pattern + "\"");
    }
    uint8_t base[144];
    for (size_t i = 0; i < n; i++) {
        switch (pattern[i]) {
            case 'R': base[i] = 0; break;
            case 'G': base[i] = 1; break;
            case 'B': base[i] = 2; break;
            case 'E': case 'C': base[i] = 3; break;
            case 'M': base[i] = 4; break;
            case 'Y': base[i] = 5; break;
            default:
                return fail(IMOPS_ERR_UNSUPPORTED_CFA, std::string("Unknown CFA color \"") + pattern[i] + "\"");
        }
    }
    out->pw = pw;
    out->ph = ph;
    for (int r = 0; r < ph; r++)
        for (int c = 0; c < pw; c++) {
            int sr = ((r + shift_y) % ph + ph) % ph;
            int sc = ((c + shift_x) % pw + pw) % pw;
            out->col[r * pw + c] = base[sr * pw + sc];
        }
    return IMOPS_OK;
}

bool cfa_is_bayer(const CfaDev& c) {
    if (c.pw != 2 || c.ph != 2) return false;
    int g = 0, r = 0, b = 0;
    for (int i = 0; i < 4; i++) {
        g += c.col[i] == 1;
        r += c.col[i] == 0;
        b += c.col[i] == 2;
    }
    // greens on one diagonal: (0,0)&(1,1) or (0,1)&(1,0)
    bool diag = (c.col[0] == 1 && c.col[3] == 1) || (c.col[1] == 1 && c.col[2] == 1);
    return g == 2 && r == 1 && b == 1 && diag;
}

int sm_count() {
    static std::mutex mu;
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

namespace {
std::mutex g_caches_mu;
std::vector<StreamCache*>& caches() {
    static std::vector<StreamCache*> v;
    return v;
}
}  // namespace

StreamCache::StreamCache(const char* what) : what_(what) {
    std::lock_guard<std::mutex> lock(g_caches_mu);
    caches().push_back(this);
}

// Buffers are allocated and replaced in stream order (cudaMallocAsync /
// cudaFreeAsync on s): unlike cudaMalloc, neither waits for the work
// already queued on the device, so the first call on a stream, or a larger
// image, does not stall frames in flight on other streams.  Work on other
// streams that uses the buffer is ordered after s with events.
int StreamCache::get(cudaStream_t s, size_t bytes, void** out) {
    if (fault_injected("alloc"))
        return fail(IMOPS_ERR_OUT_OF_MEMORY, std::string("injected allocation failure (") + what_ + ")");
    int dev = 0;
    IMOPS_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    // a request without room leaves nothing behind: the stream's next one
    // allocates anew, and the runtime's last error is not for others to find
    auto allocate = [&](void** p) {
        const cudaError_t e = cudaMallocAsync(p, bytes, s);
        if (e != cudaSuccess) cudaGetLastError();
        return cuda_status(e, (std::string("cudaMallocAsync(") + what_ + ")").c_str());
    };
    std::lock_guard<std::mutex> lock(mu_);
    for (auto& e : v_)
        if (e.dev == dev && e.s == s) {
            if (e.bytes < bytes) {
                if (e.p) IMOPS_CUDA_TRY(cudaFreeAsync(e.p, s), "cudaFreeAsync");
                e.p = nullptr;
                e.bytes = 0;
                if (int rc = allocate(&e.p)) {
                    e.p = nullptr;
                    return rc;
                }
                e.bytes = bytes;
            }
            *out = e.p;
            return IMOPS_OK;
        }
    void* p = nullptr;
    if (int rc = allocate(&p)) return rc;
    v_.push_back({dev, s, p, bytes});
    *out = p;
    return IMOPS_OK;
}

void StreamCache::release_device(int dev) {
    std::lock_guard<std::mutex> lock(mu_);
    for (size_t k = 0; k < v_.size();) {
        if (v_[k].dev == dev) {
            if (v_[k].p) cudaFree(v_[k].p);
            v_.erase(v_.begin() + k);
        } else {
            k++;
        }
    }
}

// ---- side streams ----------------------------------------------------------------

namespace {

struct SideEntry {
    int dev;
    cudaStream_t s;
    SideStream ss;
};
std::mutex g_sides_mu;
std::vector<SideEntry> g_sides;

void destroy_side(SideStream& ss) {
    if (ss.side) cudaStreamDestroy(ss.side);
    if (ss.forked) cudaEventDestroy(ss.forked);
    if (ss.joined) cudaEventDestroy(ss.joined);
}

}  // namespace

int side_stream(cudaStream_t s, SideStream* out) {
    int dev = 0;
    IMOPS_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lock(g_sides_mu);
    int held = 0;
    for (const SideEntry& e : g_sides) {
        if (e.dev != dev) continue;
        if (e.s == s) {
            *out = e.ss;
            return IMOPS_OK;
        }
        held++;
    }
    SideStream ss;
    if (held >= SIDE_STREAMS) {
        ss.side = s;
        *out = ss;
        return IMOPS_OK;
    }
    cudaError_t e = cudaStreamCreateWithFlags(&ss.side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ss.forked, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ss.joined, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        destroy_side(ss);
        return cuda_status(e, "side stream");
    }
    g_sides.push_back({dev, s, ss});
    *out = ss;
    return IMOPS_OK;
}

int SideStream::fork(cudaStream_t s) const {
    if (side == s) return IMOPS_OK;
    IMOPS_CUDA_TRY(cudaEventRecord(forked, s), "cudaEventRecord(side fork)");
    IMOPS_CUDA_TRY(cudaStreamWaitEvent(side, forked, 0), "cudaStreamWaitEvent(side fork)");
    return IMOPS_OK;
}

int SideStream::record(cudaStream_t s) const {
    if (side != s) IMOPS_CUDA_TRY(cudaEventRecord(joined, side), "cudaEventRecord(side join)");
    return IMOPS_OK;
}

int SideStream::wait(cudaStream_t s) const {
    if (side != s) IMOPS_CUDA_TRY(cudaStreamWaitEvent(s, joined, 0), "cudaStreamWaitEvent(side join)");
    return IMOPS_OK;
}

// ---- downloads -----------------------------------------------------------------

namespace {

// Pinned chunks, of use to every device; the table is guarded, its memory is
// made and used by the call that holds the ring.
struct Ring {
    bool busy = false;
    void* slot[DOWNLOAD_SLOTS] = {};
};
std::mutex g_rings_mu;
Ring g_rings[DOWNLOAD_RINGS];

void free_slots(Ring& r) {
    for (void*& p : r.slot) {
        if (p) cudaFreeHost(p);
        p = nullptr;
    }
}

void give_back(Ring* r) {
    std::lock_guard<std::mutex> lock(g_rings_mu);
    r->busy = false;
}

// A ring that no call holds, rather one that has its memory; nullptr when all
// are held or there is no memory for one (the caller then copies directly).
Ring* take_ring() {
    Ring* ring = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_rings_mu);
        for (Ring& r : g_rings)
            if (!r.busy && (!ring || (r.slot[0] && !ring->slot[0]))) ring = &r;
        if (!ring) return nullptr;
        ring->busy = true;
    }
    if (ring->slot[0]) return ring;
    for (void*& p : ring->slot)
        if (cudaHostAlloc(&p, DOWNLOAD_CHUNK, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();  // not this call's failure: it has another way
            p = nullptr;
            free_slots(*ring);
            give_back(ring);
            return nullptr;
        }
    return ring;
}

// One call's events of the current device, one a slot.
struct SlotEvents {
    cudaEvent_t e[DOWNLOAD_SLOTS] = {};
    bool make() {
        for (cudaEvent_t& v : e)
            if (cudaEventCreateWithFlags(&v, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                v = nullptr;
                return false;
            }
        return true;
    }
    ~SlotEvents() {
        for (cudaEvent_t v : e)
            if (v) cudaEventDestroy(v);
    }
};

}  // namespace

int download(void* dst, const void* src, size_t bytes, cudaStream_t s, const char* what) {
    int dev = 0;
    IMOPS_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    Ring* ring = nullptr;
    cudaPointerAttributes to{}, from{};
    if (bytes > DOWNLOAD_LEAST && cudaPointerGetAttributes(&to, dst) == cudaSuccess &&
        to.type == cudaMemoryTypeUnregistered && cudaPointerGetAttributes(&from, src) == cudaSuccess &&
        from.type == cudaMemoryTypeDevice && from.device == dev)
        ring = take_ring();
    SlotEvents filled;
    if (ring && !filled.make()) {
        give_back(ring);
        ring = nullptr;
    }
    if (!ring) {
        IMOPS_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), what);
        IMOPS_CUDA_TRY(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        return IMOPS_OK;
    }
    const size_t chunks = (bytes + DOWNLOAD_CHUNK - 1) / DOWNLOAD_CHUNK;
    std::atomic<int> failed{(int)cudaSuccess};
    auto size_of = [&](size_t c) { return c + 1 < chunks ? DOWNLOAD_CHUNK : bytes - c * DOWNLOAD_CHUNK; };
    // slot i takes the chunks i, i + DOWNLOAD_SLOTS, ...
    auto queue = [&](int i, size_t c) {
        cudaError_t e = cudaMemcpyAsync(ring->slot[i], static_cast<const char*>(src) + c * DOWNLOAD_CHUNK, size_of(c),
                                        cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(filled.e[i], s);
        return e;
    };
    auto drain = [&](int i) {
        cudaError_t e = cudaSetDevice(dev);  // a helper's; the caller's current device already
        for (size_t c = i; c < chunks && e == cudaSuccess && failed.load() == (int)cudaSuccess; c += DOWNLOAD_SLOTS) {
            if ((e = cudaEventSynchronize(filled.e[i])) != cudaSuccess) break;
            std::memcpy(static_cast<char*>(dst) + c * DOWNLOAD_CHUNK, ring->slot[i], size_of(c));
            if (c + DOWNLOAD_SLOTS < chunks) e = queue(i, c + DOWNLOAD_SLOTS);
        }
        if (e != cudaSuccess) failed.store((int)e);
    };
    int queued = 0;
    for (; queued < DOWNLOAD_SLOTS && (size_t)queued < chunks; queued++) {
        const cudaError_t e = queue(queued, queued);
        if (e != cudaSuccess) {
            failed.store((int)e);
            break;
        }
    }
    std::thread helpers[DOWNLOAD_SLOTS];
    int started = 1;  // slot 0 is this thread's
    try {
        for (; started < queued; started++) helpers[started] = std::thread(drain, started);
    } catch (...) {
        // no thread (std::system_error) or no memory for one: this one drains the rest
    }
    if (queued > 0) drain(0);
    for (int i = started; i < queued; i++) drain(i);
    for (int i = 1; i < started; i++) helpers[i].join();
    // nothing of this call may still be writing to the ring
    const cudaError_t e = cudaStreamSynchronize(s);
    give_back(ring);
    IMOPS_CUDA_TRY((cudaError_t)failed.load(), what);
    IMOPS_CUDA_TRY(e, "cudaStreamSynchronize");
    return IMOPS_OK;
}

int release_working_sets(int dev) {
    IMOPS_CUDA_TRY(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    {
        std::lock_guard<std::mutex> lock(g_rings_mu);
        for (Ring& r : g_rings)
            if (!r.busy) free_slots(r);
    }
    {
        std::lock_guard<std::mutex> lock(g_sides_mu);
        for (size_t k = 0; k < g_sides.size();) {
            if (g_sides[k].dev == dev) {
                destroy_side(g_sides[k].ss);
                g_sides.erase(g_sides.begin() + k);
            } else {
                k++;
            }
        }
    }
    std::lock_guard<std::mutex> lock(g_caches_mu);
    for (StreamCache* c : caches()) c->release_device(dev);
    return IMOPS_OK;
}

static std::atomic<uint64_t> g_launches{0};

void note_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

bool fault_injected(const char* site) {
    const char* v = std::getenv("IMOPS_FAULT_INJECT");
    if (!v || !*v) return false;
    return std::strstr(v, site) != nullptr;
}

}  // namespace imops

extern "C" const char* imops_last_error(void) { return imops::last_error(); }

extern "C" uint64_t imops_launch_count(void) { return imops::g_launches.load(std::memory_order_relaxed); }

extern "C" const char* imops_version(void) { return "imops_b200 0.1.0 (sm_100a)"; }

extern "C" int imops_release_working_sets(void) {
    imops::clear_error();
    int dev = 0;
    IMOPS_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    return imops::release_working_sets(dev);
}
