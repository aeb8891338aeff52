// hostpipe.cu -- rows between pageable host memory and the device.
//
// Cell_par and the flux routine's arrays live in ordinary (pageable) host memory, mostly as rows of
// 64 bytes at a pitch of 128, or renumbered.  The driver copies such rows through one staging buffer
// of its own on one core: setb_set_state + setb_get_state of a 96^3 grid (57 MB each way) took 67 ms.
// Here a few threads gather rows into pinned slots (scatter them from there) while the copy engine
// moves other slots, so the transfer runs near the rate of the cores' memory copies or of the link.
// Memory that the driver already knows (pinned, managed) is copied by it directly, as is anything small.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "setb_internal.cuh"

namespace sb {
namespace {

constexpr size_t kSlotBytes = 512 << 10;
constexpr int kMaxThreads = 8;
// Slots kept for later transfers: 8 MiB of pinned memory at most, freed when no handle or batch is
// left (host_pool_release).  Transfers that overlap take more and give them back to the driver.
constexpr size_t kKeepSlots = 2 * kMaxThreads;

struct Pool {
    std::mutex mu;
    std::vector<void*> free;
    long long owners = 0;
};
Pool& pool() {
    static Pool* p = new Pool;   // never destroyed: calls may come from other threads at exit
    return *p;
}

void* take_slot() {
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (!p.free.empty()) {
            void* s = p.free.back();
            p.free.pop_back();
            return s;
        }
    }
    void* s = nullptr;
    if (cudaHostAlloc(&s, kSlotBytes, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return s;
}

void give_slot(void* s) {
    if (!s) return;
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (p.free.size() < kKeepSlots && p.free.capacity() >= kKeepSlots) {
            p.free.push_back(s);
            return;
        }
    }
    cudaFreeHost(s);
}

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

struct Rows {
    bool to_device;
    char* dev;
    size_t dpitch;
    char* host;
    size_t hpitch, width, n;
    const int32_t* perm;
    cudaStream_t stream;
    size_t per;                    // rows of a slot
    std::atomic<size_t> next{0};   // next chunk
    std::atomic<int> err{0};
};

template <size_t W>
void move_fixed(char* slot, size_t sp, char* host, size_t hp, size_t r0, size_t m, const int32_t* perm, bool in) {
    for (size_t r = 0; r < m; r++) {
        char* h = host + hp * (perm ? (size_t)perm[r0 + r] : r0 + r);
        if (in) std::memcpy(slot + sp * r, h, W);
        else std::memcpy(h, slot + sp * r, W);
    }
}
// Rows r0 .. r0 + m between a slot (row pitch `sp`) and host memory; `in`: into the slot.
void move_rows(const Rows& t, char* slot, size_t r0, size_t m, bool in) {
    const size_t sp = t.dpitch;
    if (!t.perm && t.hpitch == t.width && sp == t.width) {
        if (in) std::memcpy(slot, t.host + t.width * r0, t.width * m);
        else std::memcpy(t.host + t.width * r0, slot, t.width * m);
    } else if (t.width == 64) {
        move_fixed<64>(slot, sp, t.host, t.hpitch, r0, m, t.perm, in);
    } else if (t.width == 8) {
        move_fixed<8>(slot, sp, t.host, t.hpitch, r0, m, t.perm, in);
    } else {
        for (size_t r = 0; r < m; r++) {
            char* h = t.host + t.hpitch * (t.perm ? (size_t)t.perm[r0 + r] : r0 + r);
            if (in) std::memcpy(slot + sp * r, h, t.width);
            else std::memcpy(h, slot + sp * r, t.width);
        }
    }
}

// One thread's share: two slots, so one is gathered or scattered while the other's copy runs.
void work(Rows* t, int device, void* s0, void* s1) {
    cudaError_t e = cudaSetDevice(device);
    char* slot[2] = {static_cast<char*>(s0), static_cast<char*>(s1)};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (int b = 0; b < 2 && e == cudaSuccess; b++) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
    size_t first[2] = {0, 0}, count[2] = {0, 0};   // rows in flight in each slot
    const size_t chunks = (t->n + t->per - 1) / t->per;
    bool more = true;
    for (int b = 0; e == cudaSuccess && t->err.load() == 0; b ^= 1) {
        if (count[b]) {
            e = cudaEventSynchronize(ev[b]);
            if (e != cudaSuccess) break;
            if (!t->to_device) move_rows(*t, slot[b], first[b], count[b], false);
            count[b] = 0;
        }
        const size_t c = more ? t->next.fetch_add(1) : chunks;
        if (c >= chunks) {
            more = false;
            if (!count[b ^ 1]) break;
            continue;
        }
        const size_t r0 = c * t->per, m = std::min(t->per, t->n - r0);
        char* d = t->dev + t->dpitch * r0;
        // the last row of the device's rows may end at its payload
        const size_t bytes = t->dpitch * (m - 1) + t->width;
        if (t->to_device) {
            move_rows(*t, slot[b], r0, m, true);
            e = cudaMemcpyAsync(d, slot[b], bytes, cudaMemcpyHostToDevice, t->stream);
        } else {
            e = cudaMemcpyAsync(slot[b], d, bytes, cudaMemcpyDeviceToHost, t->stream);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ev[b], t->stream);
        first[b] = r0;
        count[b] = m;
    }
    if (e != cudaSuccess) t->err.store((int)e);
    for (int b = 0; b < 2; b++)
        if (ev[b]) cudaEventDestroy(ev[b]);
}

cudaError_t run_rows(Rows& t) {
    if (t.n == 0) return cudaSuccess;
    const size_t total = t.n * t.width;
    const bool direct = t.perm == nullptr && (total < (64u << 10) || t.dpitch > kSlotBytes || !pageable(t.host));
    if (direct) {
        if (t.to_device)
            return cudaMemcpy2DAsync(t.dev, t.dpitch, t.host, t.hpitch, t.width, t.n, cudaMemcpyHostToDevice, t.stream);
        return cudaMemcpy2DAsync(t.host, t.hpitch, t.dev, t.dpitch, t.width, t.n, cudaMemcpyDeviceToHost, t.stream);
    }
    t.per = std::max<size_t>(1, kSlotBytes / t.dpitch);
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const int hw = std::max(1u, std::thread::hardware_concurrency());
    const int want = (int)std::min<size_t>(std::min(kMaxThreads, hw), (total + (1u << 20) - 1) >> 20);
    void* slots[2 * kMaxThreads] = {};
    int pairs = 0;
    for (; pairs < want; pairs++) {
        slots[2 * pairs] = take_slot();
        slots[2 * pairs + 1] = take_slot();
        if (!slots[2 * pairs] || !slots[2 * pairs + 1]) break;
    }
    if (pairs == 0) {
        e = cudaErrorMemoryAllocation;
    } else {
        std::thread th[kMaxThreads];
        int started = 0;
        for (int k = 1; k < pairs; k++) {
            try {
                th[started] = std::thread(work, &t, device, slots[2 * k], slots[2 * k + 1]);
                started++;
            } catch (const std::system_error&) {   // no more threads: the others take its chunks
                break;
            }
        }
        work(&t, device, slots[0], slots[1]);
        for (int k = 0; k < started; k++) th[k].join();
        e = (cudaError_t)t.err.load();
        if (e != cudaSuccess) cudaStreamSynchronize(t.stream);   // no copy may still use a slot
    }
    for (void* s : slots) give_slot(s);
    return e;
}

}  // namespace

void host_pool_acquire() {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    p.owners++;
    try {
        p.free.reserve(kKeepSlots);
    } catch (const std::bad_alloc&) {   // nothing is kept then (give_slot)
    }
}

void host_pool_release() {
    std::vector<void*> drop;
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (--p.owners == 0) drop.swap(p.free);
    }
    for (void* s : drop) cudaFreeHost(s);
}

cudaError_t copy_rows_to_device(void* dev, const void* host, size_t hpitch, size_t width, size_t n,
                                const int32_t* perm, cudaStream_t s) {
    Rows t;
    t.to_device = true;
    t.dev = static_cast<char*>(dev);
    t.dpitch = width;
    t.host = const_cast<char*>(static_cast<const char*>(host));   // read only
    t.hpitch = hpitch;
    t.width = width;
    t.n = n;
    t.perm = perm;
    t.stream = s;
    return run_rows(t);
}

cudaError_t copy_rows_to_host(void* host, size_t hpitch, const void* dev, size_t dpitch, size_t width, size_t n,
                              const int32_t* perm, cudaStream_t s) {
    Rows t;
    t.to_device = false;
    t.dev = const_cast<char*>(static_cast<const char*>(dev));     // read only
    t.dpitch = dpitch;
    t.host = static_cast<char*>(host);
    t.hpitch = hpitch;
    t.width = width;
    t.n = n;
    t.perm = perm;
    t.stream = s;
    return run_rows(t);
}

}  // namespace sb
