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
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>

#include <cudaTypedefs.h>

#include "setb_internal.cuh"

namespace sb {
namespace {

template <typename F> F driver_entry(const char* name, unsigned version) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion(name, &p, version, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
        return reinterpret_cast<F>(p);
    cudaGetLastError();
    return nullptr;
}

// The calling thread's current context; null: none, or it cannot be told.
CUcontext current_context() {
    static const auto current = driver_entry<PFN_cuCtxGetCurrent_v4000>("cuCtxGetCurrent", 4000);
    CUcontext c = nullptr;
    return current && current(&c) == CUDA_SUCCESS ? c : nullptr;
}
// Makes the caller's context `c` (device `device`) current on a thread of the team.  The caller may have made
// it by the driver API; cudaSetDevice would take the device's primary one, where its stream does not exist.
cudaError_t enter_context(CUcontext c, int device) {
    static const auto set = driver_entry<PFN_cuCtxSetCurrent_v4000>("cuCtxSetCurrent", 4000);
    return c && set && set(c) == CUDA_SUCCESS ? cudaSuccess : cudaSetDevice(device);
}
// A context by an id that no other context of the process has had; 0: none, or it cannot be told.
unsigned long long context_id(CUcontext c) {
    static const auto id_of = driver_entry<PFN_cuCtxGetId_v12000>("cuCtxGetId", 12000);
    unsigned long long id = 0;
    return c && id_of && id_of(c, &id) == CUDA_SUCCESS ? id : 0;
}

constexpr size_t kSlotBytes = 512 << 10;
constexpr int kMaxThreads = 8;
// Slots kept for later transfers: 8 MiB of pinned memory a device at most, given back when its last handle
// or batch goes (host_pool_release; a program that makes flux calls alone keeps them).  Transfers that
// overlap take more and give them back at once.  A slot is used in the context it was allocated in alone: a
// reset of the device releases it, and the context that follows has another id.
constexpr int kKeepSlots = 2 * kMaxThreads;
constexpr int kMaxDevices = 64;   // devices beyond that keep none

struct Slot {
    void* p;
    unsigned long long ctx;
};
struct Pool {
    std::mutex mu;
    Slot free[kKeepSlots] = {};
    int n = 0;
    long long owners = 0;
};
Pool g_pools[kMaxDevices];

Pool* pool_of_device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return d >= 0 && d < kMaxDevices ? &g_pools[d] : nullptr;
}

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// `pool`, `ctx`: of the calling thread's device and context (null, 0: nothing is kept).
void* take_slot(Pool* pool, unsigned long long ctx) {
    if (pool && ctx) {
        std::lock_guard<std::mutex> lock(pool->mu);
        for (int k = pool->n - 1; k >= 0; k--)
            if (pool->free[k].ctx == ctx) {
                void* s = pool->free[k].p;
                pool->free[k] = pool->free[--pool->n];
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

void give_slot(Pool* pool, unsigned long long ctx, void* s) {
    if (!s) return;
    if (pool && ctx) {
        std::lock_guard<std::mutex> lock(pool->mu);
        // a place, or that of a slot that went with its context
        for (int k = 0; k < kKeepSlots; k++) {
            if (k < pool->n && (pool->free[k].ctx == ctx || !pageable(pool->free[k].p))) continue;
            pool->free[k] = Slot{s, ctx};
            pool->n = std::max(pool->n, k + 1);
            return;
        }
    }
    cudaFreeHost(s);
}

// The copies of one call, handed out in slot-sized chunks.
struct Team {
    const RowCopy* copy[kMaxRowCopies];
    size_t per[kMaxRowCopies];         // rows of a slot
    size_t end[kMaxRowCopies];         // chunks up to and including this copy
    int n = 0;
    cudaStream_t stream;
    std::atomic<size_t> next{0};
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
// Rows r0 .. r0 + m between a slot (row pitch as the device's) and host memory; `in`: into the slot.
void move_rows(const RowCopy& t, char* slot, size_t r0, size_t m, bool in) {
    char* host = static_cast<char*>(t.host);
    const size_t sp = t.dpitch;
    if (!t.perm && t.hpitch == t.width && sp == t.width) {
        if (in) std::memcpy(slot, host + t.width * r0, t.width * m);
        else std::memcpy(host + t.width * r0, slot, t.width * m);
    } else if (t.width == 64) {
        move_fixed<64>(slot, sp, host, t.hpitch, r0, m, t.perm, in);
    } else if (t.width == 8) {
        move_fixed<8>(slot, sp, host, t.hpitch, r0, m, t.perm, in);
    } else {
        for (size_t r = 0; r < m; r++) {
            char* h = host + t.hpitch * (t.perm ? (size_t)t.perm[r0 + r] : r0 + r);
            if (in) std::memcpy(slot + sp * r, h, t.width);
            else std::memcpy(h, slot + sp * r, t.width);
        }
    }
}

// One thread's share, in the caller's context: two slots, so one is gathered or scattered while the
// other's copy runs.
void work(Team* t, void* s0, void* s1) {
    cudaError_t e = cudaSuccess;
    char* slot[2] = {static_cast<char*>(s0), static_cast<char*>(s1)};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (int b = 0; b < 2 && e == cudaSuccess; b++) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
    const RowCopy* which[2] = {nullptr, nullptr};   // rows in flight in each slot
    size_t first[2] = {0, 0}, count[2] = {0, 0};
    bool more = true;
    for (int b = 0; e == cudaSuccess && t->err.load() == 0; b ^= 1) {
        if (count[b]) {
            e = cudaEventSynchronize(ev[b]);
            if (e != cudaSuccess) break;
            if (!which[b]->to_device) move_rows(*which[b], slot[b], first[b], count[b], false);
            count[b] = 0;
        }
        size_t c = more ? t->next.fetch_add(1) : t->end[t->n - 1];
        if (c >= t->end[t->n - 1]) {
            more = false;
            if (!count[b ^ 1]) break;
            continue;
        }
        int k = 0;
        while (c >= t->end[k]) k++;
        if (k) c -= t->end[k - 1];
        const RowCopy& y = *t->copy[k];
        const size_t r0 = c * t->per[k], m = std::min(t->per[k], y.n - r0);
        char* dev = static_cast<char*>(y.dev) + y.dpitch * r0;
        const size_t bytes = y.dpitch * (m - 1) + y.width;   // the last row may end at its payload
        if (y.to_device) {
            move_rows(y, slot[b], r0, m, true);
            e = cudaMemcpyAsync(dev, slot[b], bytes, cudaMemcpyHostToDevice, t->stream);
        } else {
            e = cudaMemcpyAsync(slot[b], dev, bytes, cudaMemcpyDeviceToHost, t->stream);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ev[b], t->stream);
        which[b] = &y;
        first[b] = r0;
        count[b] = m;
    }
    if (e != cudaSuccess) t->err.store((int)e);
    for (int b = 0; b < 2; b++)
        if (ev[b]) cudaEventDestroy(ev[b]);
}

// The same on a thread of its own.
void work_aside(Team* t, CUcontext ctx, int device, void* s0, void* s1) {
    const cudaError_t e = enter_context(ctx, device);
    if (e == cudaSuccess) work(t, s0, s1);
    else t->err.store((int)e);
}

// A copy the driver makes by itself: known memory, or too little to be worth a slot.
bool is_direct(const RowCopy& c) {
    return !c.perm && (c.n * c.width < (64u << 10) || c.dpitch > kSlotBytes || !pageable(c.host));
}

// Rows that are not renumbered, by the driver.  Rows without gaps are one row: as 8-byte rows the copy engine
// takes arrays of 100k faces in pinned memory in 6.0 ms a flux call, as one in 0.63 ms (1.5 million: 89 and 10.5 ms).
cudaError_t copy_direct(const RowCopy& c, cudaStream_t s) {
    const cudaMemcpyKind kind = c.to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    void* const dst = c.to_device ? c.dev : c.host;
    const void* const src = c.to_device ? c.host : c.dev;
    if (c.hpitch == c.width && c.dpitch == c.width) return cudaMemcpyAsync(dst, src, c.width * c.n, kind, s);
    return c.to_device ? cudaMemcpy2DAsync(dst, c.dpitch, src, c.hpitch, c.width, c.n, kind, s)
                       : cudaMemcpy2DAsync(dst, c.hpitch, src, c.dpitch, c.width, c.n, kind, s);
}

// The copy where no pinned slot can be had: by the driver, renumbered rows through a pageable buffer.
cudaError_t copy_unstaged(const RowCopy& c, cudaStream_t s) {
    if (!c.perm) return copy_direct(c, s);
    const size_t per = std::max<size_t>(1, kSlotBytes / c.dpitch);
    const std::unique_ptr<char[]> buf(new (std::nothrow) char[per * c.dpitch]);
    if (!buf) return cudaErrorMemoryAllocation;
    for (size_t r0 = 0; r0 < c.n; r0 += per) {
        const size_t m = std::min(per, c.n - r0), bytes = c.dpitch * (m - 1) + c.width;
        char* dev = static_cast<char*>(c.dev) + c.dpitch * r0;
        if (c.to_device) move_rows(c, buf.get(), r0, m, true);
        cudaError_t e = c.to_device ? cudaMemcpyAsync(dev, buf.get(), bytes, cudaMemcpyHostToDevice, s)
                                    : cudaMemcpyAsync(buf.get(), dev, bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return e;
        if (!c.to_device) move_rows(c, buf.get(), r0, m, false);
    }
    return cudaSuccess;
}

}  // namespace

void host_pool_acquire() {
    Pool* const pool = pool_of_device();
    if (!pool) return;
    std::lock_guard<std::mutex> lock(pool->mu);
    pool->owners++;
}

void host_pool_release() {
    Pool* const pool = pool_of_device();
    if (!pool) return;
    const unsigned long long ctx = context_id(current_context());
    void* drop[kKeepSlots];
    int n = 0;
    {
        std::lock_guard<std::mutex> lock(pool->mu);
        if (--pool->owners == 0)
            for (int k = pool->n - 1; k >= 0; k--)
                if (pool->free[k].ctx == ctx) {
                    drop[n++] = pool->free[k].p;
                    pool->free[k] = pool->free[--pool->n];
                }
    }
    for (int k = 0; k < n; k++) cudaFreeHost(drop[k]);
}

cudaError_t copy_rows(const RowCopy* list, int count, cudaStream_t s) {
    Team t;
    t.stream = s;
    size_t total = 0, chunks = 0;
    for (int k = 0; k < count; k++) {
        const RowCopy& c = list[k];
        if (c.n == 0) continue;
        if (c.to_device && c.dpitch != c.width) return cudaErrorInvalidValue;   // would write its row padding
        if (is_direct(c)) {
            const cudaError_t e = copy_direct(c, s);
            if (e != cudaSuccess) return e;
            continue;
        }
        if (t.n == kMaxRowCopies) return cudaErrorInvalidValue;
        t.copy[t.n] = &c;
        t.per[t.n] = std::max<size_t>(1, kSlotBytes / c.dpitch);
        chunks += (c.n + t.per[t.n] - 1) / t.per[t.n];
        t.end[t.n++] = chunks;
        total += c.n * c.width;
    }
    if (t.n == 0) return cudaSuccess;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
    const int want = (int)std::min<size_t>(std::min(kMaxThreads, hw), (total + (1u << 20) - 1) >> 20);
    void* slots[2 * kMaxThreads] = {};
    int pairs = 0;
    Pool* const pool = pool_of_device();
    CUcontext const current = current_context();
    const unsigned long long ctx = context_id(current);
    for (; pairs < want; pairs++) {
        slots[2 * pairs] = take_slot(pool, ctx);
        slots[2 * pairs + 1] = take_slot(pool, ctx);
        if (!slots[2 * pairs] || !slots[2 * pairs + 1]) break;
    }
    if (pairs == 0) {
        for (int k = 0; k < t.n && e == cudaSuccess; k++) e = copy_unstaged(*t.copy[k], s);
    } else {
        std::thread th[kMaxThreads];
        int started = 0;
        for (int k = 1; k < pairs; k++) {
            try {
                th[started] = std::thread(work_aside, &t, current, device, slots[2 * k], slots[2 * k + 1]);
                started++;
            } catch (const std::exception&) {   // no more threads: the others take its chunks
                break;
            }
        }
        work(&t, slots[0], slots[1]);
        for (int k = 0; k < started; k++) th[k].join();
        e = (cudaError_t)t.err.load();
        if (e != cudaSuccess) cudaStreamSynchronize(s);   // no copy may still use a slot
    }
    for (void* p : slots) give_slot(pool, ctx, p);
    return e;
}

cudaError_t copy_rows_to_device(void* dev, const void* host, size_t hpitch, size_t width, size_t n,
                                const int32_t* perm, cudaStream_t s) {
    const RowCopy c = row_copy_in(dev, host, hpitch, width, n, perm);
    return copy_rows(&c, 1, s);
}

cudaError_t copy_rows_to_host(void* host, size_t hpitch, const void* dev, size_t dpitch, size_t width, size_t n,
                              const int32_t* perm, cudaStream_t s) {
    const RowCopy c = row_copy_out(host, hpitch, dev, dpitch, width, n, perm);
    return copy_rows(&c, 1, s);
}

}  // namespace sb
