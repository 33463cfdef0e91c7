// Downloads into pageable memory on the fake runtime, on two devices: what one
// device's downloads left serves the other's, a call that waits for pinned
// memory holds up no other, and threads that cannot be started are done without.
#include <chrono>
#include <condition_variable>
#include <new>
#include <thread>
#include <vector>

#include "fake_cuda.hpp"
#include "common.cuh"

using namespace std::chrono_literals;

// operator new that fails from its left_to_fail-th call of this thread on
static thread_local int left_to_fail = -1;
void* operator new(size_t n) {
    if (left_to_fail >= 0 && left_to_fail-- == 0) {
        left_to_fail = 0;
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static const size_t BYTES = 9 * imops::DOWNLOAD_CHUNK + 12345;
static std::atomic<size_t> largest{0};  // copy so far
static std::atomic<int> queued{0};      // copies by the caller of download, when counted

static void note_copy(void*, size_t bytes) {
    size_t was = largest;
    while (bytes > was && !largest.compare_exchange_weak(was, bytes)) {
    }
}

// Waits for a condition, five seconds at most.
template <class F>
static bool eventually(F f) {
    for (int k = 0; k < 5000 && !f(); k++) std::this_thread::sleep_for(1ms);
    return f();
}

struct Frame {
    void* dev = nullptr;
    std::vector<char> host;
    explicit Frame(int seed) : host(BYTES) {
        cudaMallocAsync(&dev, BYTES, nullptr);
        for (size_t k = 0; k < BYTES; k++) static_cast<char*>(dev)[k] = (char)(k * 31 + (k >> 20) + seed);
    }
    int get() { return imops::download(host.data(), dev, BYTES, nullptr, "test"); }
    bool same() const { return std::memcmp(host.data(), dev, BYTES) == 0; }
};

// Four downloads at once on device 0, then one on device 1.
static int other_device() {
    const int rings = imops::DOWNLOAD_RINGS, slots = imops::DOWNLOAD_SLOTS;
    fake::on_event_wait = [] { eventually([] { return fake::pinned >= imops::DOWNLOAD_RINGS * imops::DOWNLOAD_SLOTS; }); };
    std::vector<std::thread> ts;
    std::atomic<int> bad{0};
    for (int k = 0; k < rings; k++)
        ts.emplace_back([&, k] {
            cudaSetDevice(0);
            Frame f(k);
            if (f.get() != IMOPS_OK || !f.same()) bad++;
        });
    for (auto& t : ts) t.join();
    fake::on_event_wait = nullptr;
    EXPECT(bad == 0 && fake::pinned == rings * slots && largest <= imops::DOWNLOAD_CHUNK);
    cudaSetDevice(1);
    Frame f(9);
    EXPECT(f.get() == IMOPS_OK && f.same());
    EXPECT(largest <= imops::DOWNLOAD_CHUNK);  // not copied directly
    EXPECT(fake::pinned == rings * slots && fake::events == 0);
    EXPECT(imops::release_working_sets(1) == IMOPS_OK && fake::pinned == 0);
    return 0;
}

// A download whose pinned memory takes long to come: another is done before.
static int slow_pinned_memory() {
    static std::atomic<bool> waiting{false}, other_done{false}, in_time{false};
    fake::on_host_alloc = [] {
        if (waiting.exchange(true)) return;
        in_time = eventually([] { return other_done.load(); });
    };
    std::thread slow([] {
        Frame f(1);
        f.get();
    });
    EXPECT(eventually([] { return waiting.load(); }));
    Frame f(2);
    EXPECT(f.get() == IMOPS_OK && f.same());
    other_done = true;
    slow.join();
    fake::on_host_alloc = nullptr;
    EXPECT(in_time);
    return 0;
}

// The caller's thread finds no memory for its first, second, .. helper thread.
static int no_threads() {
    for (int started = 0; started < imops::DOWNLOAD_SLOTS; started++) {
        Frame f(started);
        static int fail_from;
        fail_from = started;
        queued = 0;
        fake::on_copy = [](void* dst, size_t bytes) {
            note_copy(dst, bytes);
            // the caller queues a copy a slot, then starts its helpers
            if (++queued == imops::DOWNLOAD_SLOTS) left_to_fail = fail_from;
        };
        int rc = -1;
        try {
            rc = f.get();
        } catch (const std::bad_alloc&) {
        }
        left_to_fail = -1;
        EXPECT(rc == IMOPS_OK && f.same());
    }
    fake::on_copy = note_copy;
    return 0;
}

int main(int argc, char** argv) {
    fake::on_copy = note_copy;
    const std::string which = argc > 1 ? argv[1] : "";
    if (which == "other_device") return other_device();
    if (which == "slow_pinned_memory") return slow_pinned_memory();
    if (which == "no_threads") return no_threads();
    return 2;
}
