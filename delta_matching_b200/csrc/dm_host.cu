// Host-side plumbing of libdm_b200: pointer checks, TMA tensor maps, the per-device status word, build identity.
#include <stdarg.h>
#include <atomic>
#include <mutex>

#include "dm_host.h"
#include "dm_attn_common.cuh"

#include <algorithm>

namespace dmh {

// Pointers that have been verified once are remembered by the 2 MiB segment of the address space they lie in (with the device
// that owns them): CUDA reserves device address ranges in units of at least that size and never hands parts of them to host
// allocations, so a later pointer in the same segment needs no driver query.  Eight to fourteen queries per entry point were
// most of the host time of the small kernels.  A direct-mapped table of atomics: a stale or colliding entry only costs a query.
static std::atomic<uint64_t> g_seg_cache[512];

static bool seg_cached(const void* p, int dev) {
    const uint64_t seg = reinterpret_cast<uintptr_t>(p) >> 21;
    const uint64_t want = (seg << 8) | (uint64_t)(dev + 1);
    return g_seg_cache[(seg ^ (seg >> 9)) & 511].load(std::memory_order_relaxed) == want;
}
static void seg_remember(const void* p, int dev) {
    const uint64_t seg = reinterpret_cast<uintptr_t>(p) >> 21;
    g_seg_cache[(seg ^ (seg >> 9)) & 511].store((seg << 8) | (uint64_t)(dev + 1), std::memory_order_relaxed);
}

thread_local int CallScope::device = -1;

int current_device(int* dev, char* err, size_t errlen) {
    if (CallScope::active()) {
        *dev = CallScope::device;
        return DM_OK;
    }
    DM_CUDA(cudaGetDevice(dev));
    return DM_OK;
}

int check_device_ptr(const void* p, const char* name, char* err, size_t errlen) {
    if (CallScope::active()) return DM_OK;          // the composite entry point has checked it
    int dev = -1;
    DM_CUDA(cudaGetDevice(&dev));
    return check_device_ptr_on(p, name, dev, err, errlen);
}

int check_device_ptr_on(const void* p, const char* name, int dev, char* err, size_t errlen) {
    DM_REQUIRE(p != nullptr, DM_ERR_ARG, "%s is NULL", name);
    if (dev >= 0 && dev < 255 && seg_cached(p, dev)) return DM_OK;
    cudaPointerAttributes a;
    cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(err, errlen, DM_ERR_ARG, "%s is not a CUDA device pointer (%s)", name, cudaGetErrorString(e));
    }
    DM_REQUIRE(a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged, DM_ERR_ARG,
               "%s must be CUDA device memory (got a host pointer)", name);
    DM_REQUIRE(a.type == cudaMemoryTypeManaged || a.device == dev, DM_ERR_ARG,
               "%s lives on device %d but the current device is %d: every tensor must be on the same device", name, a.device, dev);
    if (a.type == cudaMemoryTypeDevice && dev >= 0 && dev < 255) seg_remember(p, dev);
    return DM_OK;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// The driver encodes a map in about 0.3 us, and a step needs fourteen.  A map is a pure function of its four arguments, and a
// caching allocator hands the same addresses out again, so each thread keeps its last maps in a small direct-mapped table.
namespace {
struct TmapSlot {
    const void* base = nullptr;
    uint64_t row_bytes = 0, rows = 0;
    uint32_t box_rows = 0;
    CUtensorMap map;
};
}  // namespace

int make_tmap_u8(CUtensorMap* out, const void* base, uint64_t row_bytes, uint64_t rows, uint32_t box_rows, char* err,
                 size_t errlen) {
    static thread_local TmapSlot slots[64];
    const uint64_t h = (reinterpret_cast<uintptr_t>(base) >> 8) * 0x9E3779B97F4A7C15ull + rows * 31 + box_rows;
    TmapSlot& slot = slots[h >> 58];
    if (slot.base == base && slot.row_bytes == row_bytes && slot.rows == rows && slot.box_rows == box_rows && base) {
        *out = slot.map;
        return DM_OK;
    }
    EncodeTiledFn fn = encode_fn();
    DM_REQUIRE(fn != nullptr, DM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the CUDA driver");
    DM_REQUIRE(aligned16(base), DM_ERR_ARG, "tensor base %p is not 16-byte aligned", base);
    DM_REQUIRE(row_bytes % 128 == 0 && box_rows >= 1 && box_rows <= 256, DM_ERR_ARG, "bad tensor-map geometry");
    cuuint64_t dims[2] = {row_bytes, rows};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {128, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    DM_REQUIRE(r == CUDA_SUCCESS, DM_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    slot.base = base;
    slot.row_bytes = row_bytes;
    slot.rows = rows;
    slot.box_rows = box_rows;
    slot.map = *out;
    return DM_OK;
}

bool register_pool_ok(int compiled_regs_per_thread, int threads, int regs_needed) {
    return compiled_regs_per_thread > 0 && threads > 0 && (int64_t)compiled_regs_per_thread * threads >= (int64_t)regs_needed;
}

int check_register_pool(const void* kernel, int threads, int regs_needed, char* err, size_t errlen) {
    cudaFuncAttributes a;
    DM_CUDA(cudaFuncGetAttributes(&a, kernel));
    DM_REQUIRE(register_pool_ok(a.numRegs, threads, regs_needed), DM_ERR_UNSUPPORTED,
               "this build of the kernel was compiled with %d registers per thread (%d threads), but its roles request %d in "
               "all: refusing to launch (a setmaxnreg.inc would never be satisfied)", a.numRegs, threads, regs_needed);
    return DM_OK;
}

int sm_count(int* sms, char* err, size_t errlen) {
    static std::atomic<int> cached[64] = {};
    int dev = 0;
    if (int rc = current_device(&dev, err, errlen)) return rc;
    if (dev >= 0 && dev < 64 && (*sms = cached[dev].load(std::memory_order_relaxed))) return DM_OK;
    DM_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
    if (dev >= 0 && dev < 64) cached[dev].store(*sms, std::memory_order_relaxed);
    return DM_OK;
}

static std::mutex g_status_mu;
static std::atomic<int*> g_status[64] = {};

int* device_status_word(char* err, size_t errlen) {
    int dev = 0;
    if (current_device(&dev, err, errlen) || dev < 0 || dev >= 64) {
        fail(err, errlen, DM_ERR_CUDA, "cudaGetDevice failed");
        return nullptr;
    }
    if (int* p = g_status[dev].load(std::memory_order_acquire)) return p;
    std::lock_guard<std::mutex> lk(g_status_mu);
    if (!g_status[dev].load(std::memory_order_relaxed)) {
        int* p = nullptr;
        if (cudaMalloc(&p, sizeof(int)) != cudaSuccess || cudaMemset(p, 0, sizeof(int)) != cudaSuccess) {
            fail(err, errlen, DM_ERR_CUDA, "cannot allocate the device status word");
            return nullptr;
        }
        g_status[dev].store(p, std::memory_order_release);
    }
    return g_status[dev].load(std::memory_order_relaxed);
}

// In two to five rounds of causal items the snake leaves the busiest CTA 4 to 15 % above the mean (3.5 rounds of one head of 65536 rows:
// 6 %; 8 heads of 5632: 11 %), and so does longest-first.  Packing comes to 1 or 2 %: the smallest capacity into which the
// items fit when every CTA in turn takes the longest that still fits it (multifit).  An item costs its tiles and two more: with half a
// tile the packings come out with CTAs of a dozen one-tile items, 83 against 67 us for pass 1 of B2 N2048 H16; with four or more the
// gain of the packed calls shrinks.  Forward and pass 1 take it; pass 2, whose items cost six or more tiles besides their own, lost
// as often as it won (B2 N3584 H8 24.1 -> 24.9 us).  Taken where the busiest CTA saves two tiles and 3 %: pass 1 / forward of one head
// of 65536 1560 -> 1490 / 952 -> 905 us, B5 N11264 H1 254 -> 240 / 157 -> 146, B4 N5632 H2 111 -> 102 / 69.0 -> 64.8, B2 N3072 H9
// 80.9 -> 77.4 / 50.4 -> 48.6, B10 N512 H12 31.1 -> 29.7 / 19.0 -> 18.5, B3 N2816 H7 78.2 -> 77.0 / 48.9 -> 48.5; with less to save
// (B4 N1024 H14: one tile of 22) the longer walks cost what the balance gives, 24.5 -> 24.9 us.  Packing ends at kWalkItems, the
// size of the list that travels with the kernel's parameters.  Beyond it there is less to gain: by the costs above the snake is
// within 3 % of the mean in 93 % of 635 shapes of 801 to 1300 items and in 98 % of 730 of 1301 to 2000 (148 CTAs, even numbers of blocks), but not
// in all: 50 heads of 18 blocks 5.8 %, 75 of 16 5.7 %, 149 of 16 5.2 %, 224 of 4 10 %.
namespace {
struct WalkPlanner {
    int heads, nblk, ctas;
    static int cost(int size) { return size + 2; }
    int snake() const {                              // tiles of the busiest CTA without a plan
        int load[dm::kWalkCtas] = {};
        int at = 0, step = 1;
        for (int size = nblk; size > 0; --size)
            for (int h = 0; h < heads; ++h) {
                load[at] += cost(size);
                if (at + step < 0 || at + step == ctas) step = -step;      // the round ends: the next one comes back
                else at += step;
            }
        return *std::max_element(load, load + ctas);
    }
    // Fills the CTAs up to `cap`; true if every item found a place.  `w` takes the lists.  `largest` finds the largest size
    // up to `s` of which an item is left (0: none) along links that skip the sizes used up and are shortened on the way, so that a
    // fill costs items and CTAs and not sizes times CTAs.
    bool fill(int cap, dm::PackedWalk* w) const {
        uint16_t used[dm::kWalkItems + 1], link[dm::kWalkItems + 1];
        for (int s = 0; s <= nblk; ++s) {
            used[s] = 0;
            link[s] = (uint16_t)s;
        }
        const auto largest = [&link](int s) {
            while (link[s] != s) s = link[s] = link[link[s]];
            return s;
        };
        int at = 0;
        for (int c = 0; c < ctas; ++c) {
            w->first[c] = (uint16_t)at;
            int room = cap;
            for (int size = largest(std::min(nblk, room - cost(0))); size > 0; size = largest(std::min(size, std::max(room - cost(0), 0)))) {
                const int n = std::min(heads - used[size], room / cost(size));
                for (int i = 0; i < n; ++i) w->item[at + i] = (uint16_t)((nblk - size) * heads + used[size] + i);
                at += n;
                room -= n * cost(size);
                used[size] = (uint16_t)(used[size] + n);
                if (used[size] == heads) link[size] = (uint16_t)(size - 1);
            }
        }
        w->first[ctas] = (uint16_t)at;
        return at == heads * nblk;
    }
    bool plan(dm::PackedWalk* w) const {
        int64_t total = 0;
        for (int size = 1; size <= nblk; ++size) total += (int64_t)heads * cost(size);
        const int busiest = snake(), limit = busiest - std::max(2, (busiest + 31) / 32);
        // The smallest capacity that does is, but for a few shapes, what the mean CTA or the longest item asks for, so the search goes up from
        // there in growing steps and halves the last one (the fit is not quite monotone; any capacity that does is right).
        int fails = std::max((int)((total + ctas - 1) / ctas), cost(nblk)) - 1, fits = 0, held = 0;
        for (int step = 1; !fits && fails < limit; step *= 2) {
            held = std::min(fails + step, limit);
            (fill(held, w) ? fits : fails) = held;
        }
        if (!fits) return false;
        while (fits - fails > 1) {
            held = (fits + fails) / 2;
            (fill(held, w) ? fits : fails) = held;
        }
        if (held != fits) fill(fits, w);
        for (int c = 1; c < ctas; ++c)          // an item for every CTA: those left without take the shortest, one each
            w->first[c] = (uint16_t)std::min((int)w->first[c], heads * nblk - (ctas - c));
        return true;
    }
};

// The answers for the shapes asked for last, the same for every thread and device (a plan is a pure function of the three numbers): forward and
// backward run on different threads, and a program with bucketed lengths comes back to some dozens of shapes.  Shapes with and without a
// plan have places of their own.  One that is not kept costs 2 to 10 us here (a fill that scanned every size for every CTA, once per step
// of a bisection, took 20 to 1300), a kept one 0.1.  Evaluation of many lengths in turn, each call waited for, eight shapes per thread and
// that fill / this: 15 lengths of one head of 38400 to 45568 rows 622 -> 409 us a call, 20 of two heads of 19456 to 24320 366 -> 244, 16 of
// eight heads of 4864 to 8704 146 -> 125.
struct WalkTable {
    static constexpr unsigned kKept = 64;
    std::mutex mu;
    uint32_t planned[kKept] = {}, refused[kKept] = {};
    dm::PackedWalk walk[kKept] = {};
    unsigned next_planned = 0, next_refused = 0;
};
WalkTable g_walks;

bool kept_walk(uint32_t key, dm::PackedWalk* out, bool* taken) {
    std::lock_guard<std::mutex> lk(g_walks.mu);
    for (unsigned i = 0; i < WalkTable::kKept; ++i) {
        if (g_walks.planned[i] == key) {
            *out = g_walks.walk[i];
            return *taken = true;
        }
        if (g_walks.refused[i] == key) {
            *taken = false;
            return true;
        }
    }
    return false;
}
void keep_walk(uint32_t key, const dm::PackedWalk& w, bool taken) {      // (two threads may keep the same answer twice)
    std::lock_guard<std::mutex> lk(g_walks.mu);
    if (taken) {
        const unsigned i = g_walks.next_planned++ % WalkTable::kKept;
        g_walks.planned[i] = key;
        g_walks.walk[i] = w;
    } else {
        g_walks.refused[g_walks.next_refused++ % WalkTable::kKept] = key;
    }
}
}  // namespace

bool plan_walk(int heads, int nblk, int ctas, dm::PackedWalk* out) {
    const int64_t n = (int64_t)heads * nblk;
    if (n <= ctas || n > dm::kWalkItems || ctas > dm::kWalkCtas) return false;
    static_assert(dm::kWalkItems < 1024 && dm::kWalkCtas < 1024, "a key holds ten bits of each");
    const uint32_t key = (uint32_t)heads | (uint32_t)nblk << 10 | (uint32_t)ctas << 20;
    bool taken;
    if (kept_walk(key, out, &taken)) return taken;
    *out = {};
    taken = WalkPlanner{heads, nblk, ctas}.plan(out);
    keep_walk(key, *out, taken);
    return taken;
}

}  // namespace dmh

extern "C" const char* dm_build_info(void) {
    return "libdm_b200 0.1.0; arch=sm_100a; numerics=Delta-Matching-128 v3 / Delta-Matching-256 v1 (tcgen05 realization); "
           "twins=none; bf16_dp=0; dbg=1";
}

extern "C" int dm_register_pool_ok(int32_t compiled_regs_per_thread, int32_t threads, int32_t regs_needed) {
    return dmh::register_pool_ok(compiled_regs_per_thread, threads, regs_needed) ? 1 : 0;
}

extern "C" int dm_walk_plan(int32_t heads, int32_t nblk, int32_t ctas, int32_t* first, int32_t* items) {
    if (heads <= 0 || nblk <= 0 || ctas <= 0 || !first || !items) return 0;
    dm::PackedWalk w;
    if (!dmh::plan_walk(heads, nblk, ctas, &w)) return 0;
    for (int c = 0; c <= ctas; ++c) first[c] = w.first[c];
    for (int i = 0; i < w.first[ctas]; ++i) items[i] = w.item[i];
    return 1;
}

extern "C" int dm_init(char* err, size_t errlen) {
    if (!dmh::device_status_word(err, errlen)) return DM_ERR_CUDA;
    int rc, sms = 0;
    if ((rc = dmh::sm_count(&sms, err, errlen))) return rc;
    if ((rc = dmh::prepare_fwd(err, errlen))) return rc;
    if ((rc = dmh::prepare_fwd256(err, errlen))) return rc;
    if ((rc = dmh::prepare_delta(err, errlen))) return rc;
    if ((rc = dmh::prepare_bwd1(err, errlen))) return rc;
    if ((rc = dmh::prepare_bwd1_d256(err, errlen))) return rc;
    return dmh::prepare_bwd2(err, errlen);
}

extern "C" int dm_device_status(int32_t* status, char* err, size_t errlen) {
    DM_REQUIRE(status != nullptr, DM_ERR_ARG, "status is NULL");
    int* w = dmh::device_status_word(err, errlen);
    if (!w) return DM_ERR_CUDA;
    DM_CUDA(cudaDeviceSynchronize());
    int v = 0;
    DM_CUDA(cudaMemcpy(&v, w, sizeof(int), cudaMemcpyDeviceToHost));
    DM_CUDA(cudaMemset(w, 0, sizeof(int)));
    *status = v;
    return DM_OK;
}
