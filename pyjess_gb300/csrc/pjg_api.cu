// pjg_api.cu — C ABI of libpjg (include/pjg.h): template / structure
// upload and the query pipeline.
//
// Pipeline of pjg_query (on one CUDA stream owned by the call):
//   k_params                      annulus radii for the query's r and s
//   k_candidate_counts            |C| and |R| of every (structure, signature)
//   k_struct_totals               candidate entries per structure
//   per structure chunk (bounded entry budget):
//     k_scan_*, k_block_counts    list offsets, culling blocks of CULL_BLK leaves
//     k_search_free               complete assignments of every pair, in any
//                                 order; requests the lists that tell a
//                                 pair's rows apart
//     k_candidates                lists in candidate order (of the pairs
//                                 taken in items of seeds), k_search_free on
//                                 those items
//     k_leaf_part, k_leaf_sorted, k_leaf_exact, k_mark_ordered
//                                 requested lists in kd leaf order
//     k_unit_order                the rows' places in their pair's stream
//     or, in the plain mode and with explicit leaf levels:
//     k_demand_levels             requests the lists of the first levels
//     k_search                    complete assignments, ordered per pair;
//                                 pairs that reach a list without leaf order
//                                 request it and are suspended, the lists are
//                                 ordered (as above) and a second k_search
//                                 round resumes them
//     k_superpose                 rmsd / rotation / centroids per row
//     k_order_counts, k_automaton, k_gather_hits
//                                 rows in (structure, template descending,
//                                 ordinal) order, the Query.__next__
//                                 automaton (src/pyjess/_jess.pyx:2197-2283)
//                                 per pair, hits and warnings compacted

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <unordered_map>
#include <mutex>
#include <numeric>
#include <atomic>
#include <string>
#include <thread>
#include <vector>

#include "../../include/pjg.h"
#include "pjg_common.cuh"
#include "pjg_kernels.cuh"

using namespace pjg;

namespace {

thread_local std::string g_error = "";

pjg_status fail(pjg_status st, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_error = buf;
    return st;
}

#define CUDA_TRY(expr)                                                                          \
    do {                                                                                        \
        cudaError_t _e = (expr);                                                                \
        if (_e != cudaSuccess) {                                                                \
            status = fail(_e == cudaErrorMemoryAllocation ? PJG_ERR_OOM : PJG_ERR_CUDA,         \
                          "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__,     \
                          __LINE__);                                                            \
            goto done;                                                                          \
        }                                                                                       \
    } while (0)

inline uint8_t up(uint8_t c) { return (c >= 'a' && c <= 'z') ? (uint8_t)(c & ~0x20) : c; }

inline uint32_t pack_upper(const uint8_t *b) {
    return (uint32_t)up(b[0]) | ((uint32_t)up(b[1]) << 8) | ((uint32_t)up(b[2]) << 16) |
           ((uint32_t)up(b[3]) << 24);
}

inline uint32_t pack_lit(const char *s) { return pack_upper((const uint8_t *)s); }

// Small device blocks kept between the queries that share a stream: by power
// of two from 256 B to 4 MiB, reused in stream order.  A query takes some 60
// buffers; from the allocator they cost it about 0.2 ms.
struct BlockCache {
    static constexpr int CLASSES = 15;
    std::vector<void *> idle[CLASSES];
    static int class_of(size_t bytes) {
        int c = 0;
        while (c < CLASSES && (size_t(256) << c) < bytes) c++;
        return c < CLASSES ? c : -1;
    }
};
// the cache of the query running on this thread (nullptr: none)
thread_local BlockCache *t_cache = nullptr;

// device buffer helper (stream ordered)
template <typename T>
struct DBuf {
    T *p = nullptr;
    size_t n = 0;
    int cls = -1;  // class of a cached block
};

template <typename T>
void dfree(DBuf<T> &b, cudaStream_t st) {
    if (b.p && b.cls >= 0) t_cache->idle[b.cls].push_back(b.p);
    else if (b.p) cudaFreeAsync(b.p, st);
    b.p = nullptr;
    b.n = 0;
    b.cls = -1;
}

template <typename T>
cudaError_t dalloc(DBuf<T> &b, size_t n, cudaStream_t st) {
    if (b.n >= n && b.p) return cudaSuccess;
    dfree(b, st);
    n = std::max<size_t>(n, 1);
    const size_t bytes = n * sizeof(T);
    const int c = t_cache ? BlockCache::class_of(bytes) : -1;
    if (c >= 0 && !t_cache->idle[c].empty()) {
        b.p = (T *)t_cache->idle[c].back();
        t_cache->idle[c].pop_back();
    } else {
        cudaError_t e = cudaMallocAsync((void **)&b.p, c >= 0 ? size_t(256) << c : bytes, st);
        if (e != cudaSuccess) {
            b.p = nullptr;
            return e;
        }
    }
    b.n = n;
    b.cls = c;
    return cudaSuccess;
}

// Keep the stream-ordered pool's memory mapped between calls (up to half the
// device) instead of returning it at every sync: the next call's buffers then
// need no new mappings.
void keep_pool(int device) {
    static std::mutex m;
    static bool done[256] = {};
    std::lock_guard<std::mutex> g(m);
    if (device < 0 || device >= 256 || done[device]) return;
    cudaMemPool_t pool;
    size_t fb = 0, tb = 0;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess && cudaMemGetInfo(&fb, &tb) == cudaSuccess) {
        uint64_t thr = tb / 2;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    cudaGetLastError();
    done[device] = true;
}

// What a call on a device needs and the next one can take over: a stream,
// events, a pinned buffer and the stream's small blocks.  Idle ones are kept
// (at most IDLE_MAX, with at most CACHE_MAX bytes of blocks each) while any
// template or structure handle lives; one call has one to itself.  One whose
// CUDA context has been reset is forgotten.
struct Scratch {
    static constexpr size_t PINNED = 1 << 20;
    int device = 0;
    unsigned long long ctx = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[8] = {};
    unsigned char *pinned = nullptr;
    BlockCache cache;

    cudaError_t create(int dev) {
        device = dev;
        ctx = bound_context_id(dev);
        cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        for (auto &v : ev)
            if (e == cudaSuccess) e = cudaEventCreate(&v);
        if (e == cudaSuccess) e = cudaMallocHost((void **)&pinned, PINNED);
        return e;
    }
    // blocks beyond `most` bytes back to the allocator, the largest first
    void trim(size_t most) {
        size_t held = 0;
        for (int c = 0; c < BlockCache::CLASSES; c++) held += cache.idle[c].size() * (size_t(256) << c);
        for (int c = BlockCache::CLASSES - 1; c >= 0; c--)
            while (held > most && !cache.idle[c].empty()) {
                cudaFreeAsync(cache.idle[c].back(), st);
                cache.idle[c].pop_back();
                held -= size_t(256) << c;
            }
    }
    void destroy() {
        if (st) {
            trim(0);
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
        for (auto &v : ev)
            if (v) cudaEventDestroy(v);
        if (pinned) cudaFreeHost(pinned);
    }
};

// Memory of handles and results (and of the arrays a structure upload needs
// meanwhile): a pool of their own on each device, which keeps a 64th of the
// device (PJG_OBJECT_KEEP bytes) beyond the live blocks for the next ones and
// gives the rest back to the device: at the next wait of any stream, and as
// soon as a block of OBJECT_PROMPT bytes is freed.  (Mapping memory anew costs:
// a query of 10 M pairs with 2.2 GB of hits took 218.8 ms with 256 MiB kept,
// 211.0 with 4.4 GB.  The pool of the queries' buffers keeps up to half the
// device.)
constexpr size_t OBJECT_PROMPT = 64 << 20;

struct ObjectPool {
    cudaMemPool_t pool = nullptr;
    unsigned long long ctx = 0;  // the context it belongs to
    size_t live = 0;             // bytes of its blocks
    size_t keep = 0;             // bytes it keeps beyond them
    uint64_t threshold = 0;      // what it may hold (set anew when live has
};                               //   moved by a quarter of `keep`)
std::mutex g_object_mutex;
ObjectPool g_object_pool[256];   // guarded by g_object_mutex

struct Block {
    void *p = nullptr;
    size_t bytes = 0;
    int device = 0;
    unsigned long long ctx = 0;

    cudaError_t alloc(size_t n, cudaStream_t st) {
        bytes = std::max<size_t>(n, 1);
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return e;
        if (device >= 256) return cudaErrorInvalidDevice;
        ctx = bound_context_id(device);
        std::lock_guard<std::mutex> g(g_object_mutex);
        ObjectPool &o = g_object_pool[device];
        if (!o.pool || o.ctx != ctx) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = device;
            o = ObjectPool{};
            e = cudaMemPoolCreate(&o.pool, &props);
            if (e != cudaSuccess) return e;
            o.ctx = ctx;
            size_t fb = 0, tb = 0;
            o.keep = cudaMemGetInfo(&fb, &tb) == cudaSuccess ? tb / 64 : 256 << 20;
        }
        if (const char *v = getenv("PJG_OBJECT_KEEP"))
            if (atoll(v) > 0) o.keep = (size_t)atoll(v);
        e = cudaMallocFromPoolAsync(&p, bytes, o.pool, st);
        if (e == cudaErrorMemoryAllocation) {
            // what the queries' pool holds unused may make the room
            cudaGetLastError();
            cudaMemPool_t q;
            if (cudaDeviceGetDefaultMemPool(&q, device) == cudaSuccess) cudaMemPoolTrimTo(q, 0);
            e = cudaMallocFromPoolAsync(&p, bytes, o.pool, st);
        }
        if (e != cudaSuccess) {
            p = nullptr;
            return e;
        }
        o.live += bytes;
        limit(o);
        return e;
    }
    // in the order of `st` (nullptr: now); nothing to do once its context is gone
    void free(cudaStream_t st = nullptr) {
        if (!p) return;
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev != device) cudaSetDevice(device);
        if (bound_context_id(device) == ctx) {
            cudaFreeAsync(p, st);
            if (bytes >= OBJECT_PROMPT && !st) cudaStreamSynchronize(nullptr);
            std::lock_guard<std::mutex> g(g_object_mutex);
            ObjectPool &o = g_object_pool[device];
            if (o.pool && o.ctx == ctx) {
                o.live -= bytes;
                limit(o);
                if (bytes >= OBJECT_PROMPT && !st) cudaMemPoolTrimTo(o.pool, o.live + o.keep);
            }
        }
        if (dev != device) cudaSetDevice(dev);
        p = nullptr;
    }

private:
    static void limit(ObjectPool &o) {
        const uint64_t most = o.live + o.keep;
        if (o.threshold <= most + o.keep / 4 && most <= o.threshold + o.keep / 4) return;
        o.threshold = most;
        cudaMemPoolSetAttribute(o.pool, cudaMemPoolAttrReleaseThreshold, &o.threshold);
    }
};

constexpr size_t IDLE_MAX = 8, CACHE_MAX = 64 << 20;
std::mutex g_scratch_mutex;
std::vector<Scratch *> g_idle;   // guarded by g_scratch_mutex
int g_handles = 0;               // live template and structure handles (guarded likewise)

// a scratch of the current device, idle; nullptr with *e set on failure
Scratch *acquire_scratch(int device, cudaError_t *e) {
    const unsigned long long ctx = bound_context_id(device);
    *e = cudaSuccess;
    {
        std::lock_guard<std::mutex> g(g_scratch_mutex);
        for (size_t i = g_idle.size(); i-- > 0;) {
            Scratch *x = g_idle[i];
            if (x->device != device) continue;
            g_idle.erase(g_idle.begin() + (long)i);
            if (ctx != 0 && x->ctx == ctx) return x;
            delete x;  // its context is gone, its stream and memory with it
        }
    }
    Scratch *x = new Scratch;
    *e = x->create(device);
    if (*e == cudaSuccess) return x;
    x->destroy();
    delete x;
    cudaGetLastError();  // (reported here; a later call does not meet it)
    return nullptr;
}

// back to the idle ones (its stream idle); `reuse` false: after an error
void release_scratch(Scratch *x, bool reuse) {
    if (!x) return;
    if (reuse) {
        x->trim(CACHE_MAX);
        std::lock_guard<std::mutex> g(g_scratch_mutex);
        if (g_handles > 0 && g_idle.size() < IDLE_MAX) {
            g_idle.push_back(x);
            return;
        }
    }
    x->destroy();
    delete x;
}

void handle_created() {
    std::lock_guard<std::mutex> g(g_scratch_mutex);
    g_handles++;
}

// the last handle gone: the idle scratch is given back
void handle_destroyed() {
    std::vector<Scratch *> out;
    {
        std::lock_guard<std::mutex> g(g_scratch_mutex);
        if (--g_handles == 0) out.swap(g_idle);
    }
    int dev = 0;
    if (!out.empty()) cudaGetDevice(&dev);
    const unsigned long long ctx = out.empty() ? 0 : bound_context_id(dev);
    for (Scratch *x : out) {
        // (another device's or context's: dropped with its context)
        if (x->device != dev) {
            cudaSetDevice(x->device);
            if (bound_context_id(x->device) == x->ctx) x->destroy();
            cudaSetDevice(dev);
        } else if (x->ctx == ctx) {
            x->destroy();
        }
        delete x;
    }
}

// Arrays uploaded into one device block: one allocation, and one copy through
// the pinned buffer when they fit it.
struct Upload {
    struct Item {
        void **dst;
        const void *src;  // nullptr: room only
        size_t bytes, at;
    };
    std::vector<Item> items;
    size_t total = 0;

    template <typename T, typename U>
    void add(T **dst, const U *src, size_t n) {
        static_assert(sizeof(T) == sizeof(U), "element size");
        const size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
        items.push_back({(void **)dst, n ? (const void *)src : nullptr, bytes, total});
        total += (bytes + 255) & ~size_t(255);
    }
    template <typename T>
    void add(T **dst, const std::vector<T> &v) {
        add(dst, v.data(), v.size());
    }
    template <typename T>
    void room(T **dst, size_t n) {
        items.push_back({(void **)dst, nullptr, std::max<size_t>(n, 1) * sizeof(T), total});
        total += (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~size_t(255);
    }
    // allocates `block` and fills it on x's stream (arrays with a source
    // first, so that they share one copy)
    cudaError_t run(Block *block, Scratch *x) {
        cudaError_t e = block->alloc(total, x->st);
        if (e != cudaSuccess) return e;
        size_t filled = 0;
        for (const Item &it : items) {
            *it.dst = (char *)block->p + it.at;
            if (it.src) filled = it.at + it.bytes;
        }
        if (filled <= Scratch::PINNED) {
            for (const Item &it : items)
                if (it.src) std::memcpy(x->pinned + it.at, it.src, it.bytes);
            return cudaMemcpyAsync(block->p, x->pinned, filled, cudaMemcpyHostToDevice, x->st);
        }
        for (const Item &it : items)
            if (it.src && e == cudaSuccess)
                e = cudaMemcpyAsync(*it.dst, it.src, it.bytes, cudaMemcpyHostToDevice, x->st);
        return e;
    }
};

// Host staging array of n elements left uninitialised (every element is
// written before use; a std::vector would zero it first).
template <typename T>
struct HostArray {
    std::unique_ptr<T[]> p;
    explicit HostArray(size_t n) : p(new T[std::max<size_t>(n, 1)]) {}
    T &operator[](size_t i) { return p[i]; }
    const T &operator[](size_t i) const { return p[i]; }
};

// Chemically equivalent atom pairs used by match mode 1 (see the oracle's
// same_position rule; pinned by the reference fixture for ASN OD1/ND2).
struct PartnerDef { const char *res; const char *a; const char *b; };
const PartnerDef PARTNER_TABLE[] = {
    {"ASP", "_OD1", "_OD2"}, {"GLU", "_OE1", "_OE2"}, {"ASN", "_OD1", "_ND2"},
    {"GLN", "_OE1", "_NE2"}, {"ARG", "_NH1", "_NH2"}, {"HIS", "_ND1", "_CD2"},
    {"HIS", "_CE1", "_NE2"}, {"PHE", "_CD1", "_CD2"}, {"PHE", "_CE1", "_CE2"},
    {"TYR", "_CD1", "_CD2"}, {"TYR", "_CE1", "_CE2"}, {"LEU", "_CD1", "_CD2"},
    {"VAL", "_CG1", "_CG2"},
};

uint32_t res_lit(const char *three) {
    uint8_t b[4] = {(uint8_t)three[0], (uint8_t)three[1], (uint8_t)three[2], 0};
    return pack_upper(b);
}

}  // namespace

// ---------------------------------------------------------------------------
// Handles

struct pjg_templates {
    int32_t T = 0, A = 0, nmax = 0, G = 0;
    std::vector<int32_t> atom_begin, param_begin, dim;
    // device
    int32_t *d_atom_begin = nullptr, *d_sig = nullptr, *d_key = nullptr, *d_param_begin = nullptr;
    double *d_pos = nullptr, *d_weight = nullptr, *d_dist = nullptr;
    int32_t *d_code = nullptr, *d_rule = nullptr, *d_mainchain = nullptr, *d_name_begin = nullptr,
            *d_res_begin = nullptr, *d_partner_begin = nullptr;
    uint32_t *d_names = nullptr, *d_resnames = nullptr, *d_partner_res = nullptr, *d_partner_name = nullptr;
    int64_t n_params = 0;
    int device = 0;
    // templates of more than 32 atoms (k_search_large in the search in order);
    // of them, those of at most 64 (order-free search) and the larger ones
    std::vector<int32_t> large, wide, huge;
    int32_t *d_large = nullptr, *d_wide = nullptr, *d_huge = nullptr;
    Block block;            // the device arrays
    bool counted = false;   // a live handle
};

struct pjg_structures {
    int32_t S = 0;
    int64_t N = 0;
    int32_t max_atoms = 0;
    double max_radius = 0.0;
    std::vector<int64_t> atom_base;
    int64_t *d_atom_base = nullptr;
    int32_t *d_atom_count = nullptr;
    double *d_xyz64 = nullptr;
    float4 *d_xyz32 = nullptr;
    uint32_t *d_name = nullptr, *d_resname = nullptr;
    int32_t *d_sorted = nullptr;
    int32_t *d_bucket_begin = nullptr, *d_bucket_lo = nullptr, *d_bucket_hi = nullptr;
    uint32_t *d_bucket_name = nullptr;
    uint32_t *d_lrank = nullptr, *d_urank = nullptr;  // [3][N] axis ranks
    int32_t *d_nh_begin = nullptr, *d_nh_count = nullptr;  // name histogram per bucket
    uint32_t *d_nh_name = nullptr;
    uint8_t *d_name_id = nullptr;                      // name index within the bucket
    // per distinct name of a bucket: where its atoms start (structure-local)
    // in nh_pos, which holds every structure's atoms grouped by (bucket,
    // name), each group in ResIndex order
    int32_t *d_nh_off = nullptr, *d_nh_pos = nullptr;
    // order-free search (FreeView): kinds of the set, per nh_* entry its kind,
    // points in nh_pos order, atoms in residue order
    int32_t n_kinds = 0, max_local_kinds = 0;
    uint32_t *d_kind_name = nullptr, *d_kind_res = nullptr;
    int32_t *d_nh_kind = nullptr, *d_res_pos = nullptr, *d_res_place = nullptr;
    float4 *d_kxyz = nullptr;
    uint16_t *d_res_kind = nullptr;
    int4 *d_res_range = nullptr;
    int device = 0;
    Block block;            // the device arrays
    bool counted = false;   // a live handle
};

// Hits and warnings of a query, on the device: contiguous arrays that grow
// (doubling) as chunks append to them.
struct HitStore {
    int64_t hits = 0, atoms = 0, warns = 0;           // in use
    int64_t cap_h = 0, cap_a = 0, cap_w = 0;          // allocated
    int32_t *structure = nullptr, *tpl = nullptr, *atoms_ = nullptr, *warn_structure = nullptr;
    int64_t *ordinal = nullptr, *atom_offset = nullptr, *warn_before = nullptr;
    double *rmsd = nullptr, *rot = nullptr, *centres = nullptr;

    Block block;                                      // the arrays

    // room for `h` more hits, `a` more atoms, `w` more warnings: twice what
    // there is, or, where that cannot be had, what is needed
    cudaError_t reserve(int64_t h, int64_t a, int64_t w, cudaStream_t st) {
        if (block.p && hits + h <= cap_h && atoms + a <= cap_a && warns + w <= cap_w) return cudaSuccess;
        auto bigger = [](int64_t need, int64_t cap) { return need <= cap ? cap : std::max<int64_t>(need, 2 * cap); };
        int64_t nh = bigger(hits + h, cap_h), na = bigger(atoms + a, cap_a), nw = bigger(warns + w, cap_w);
        Block fresh;
        Upload lay = layout(nh, na, nw);
        cudaError_t e = fresh.alloc(lay.total, st);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            nh = hits + h;
            na = atoms + a;
            nw = warns + w;
            lay = layout(nh, na, nw);
            e = fresh.alloc(lay.total, st);
        }
        if (e != cudaSuccess) return e;
        // (what each array holds, in the order of layout)
        const int64_t used[] = {4 * hits, 4 * hits, 8 * hits, 8 * hits, 72 * hits, 48 * hits, 8 * hits,
                                4 * atoms, 4 * warns, 8 * warns};
        for (size_t i = 0; i < lay.items.size(); i++) {
            const Upload::Item &it = lay.items[i];
            char *to = (char *)fresh.p + it.at;
            if (e == cudaSuccess && block.p && used[i] > 0)
                e = cudaMemcpyAsync(to, *it.dst, (size_t)used[i], cudaMemcpyDeviceToDevice, st);
            *it.dst = to;
        }
        block.free(st);
        block = fresh;
        cap_h = nh;
        cap_a = na;
        cap_w = nw;
        return e;
    }
    Upload layout(int64_t nh, int64_t na, int64_t nw) {
        Upload lay;
        lay.room(&structure, (size_t)nh);
        lay.room(&tpl, (size_t)nh);
        lay.room(&ordinal, (size_t)nh);
        lay.room(&rmsd, (size_t)nh);
        lay.room(&rot, 9 * (size_t)nh);
        lay.room(&centres, 6 * (size_t)nh);
        lay.room(&atom_offset, (size_t)nh + 1);
        lay.room(&atoms_, (size_t)na);
        lay.room(&warn_structure, (size_t)nw);
        lay.room(&warn_before, (size_t)nw);
        return lay;
    }
    // the segment view at the current ends
    HitSegment tail() const {
        return HitSegment{structure + hits, tpl + hits, ordinal + hits, rmsd + hits, rot + 9 * hits,
                          centres + 6 * hits, atom_offset + hits, atoms_ + atoms, warn_structure + warns,
                          warn_before + warns};
    }
    ~HitStore() { block.free(); }
};

struct pjg_results {
    HitStore store;
    pjg_stats stats{};
    int device = 0;
    // count-only query: store.hits/atoms/warns are counts, nothing is kept
    bool count_only = false;
    const pjg_structures *structures = nullptr;  // the set the query searched
};

namespace {

// Device-to-host copy of result arrays into caller memory.  Small copies
// are plain cudaMemcpy.  Large ones are split into equal byte ranges, one
// per host thread: each thread first touches every page of its range of the
// caller's arrays (freshly allocated arrays are not yet mapped, and taking
// those page faults is what limits such a copy; measured on a GB300 host,
// 2.25 GB into untouched pages 81 ms, into touched ones 12 ms), then copies
// its range with cudaMemcpy straight into them.

struct CopySeg {
    void *dst;
    const void *src;
    size_t bytes;
};

// bytes [lo, hi) of the concatenation of `segs`, by one thread
cudaError_t copy_range(const std::vector<CopySeg> &segs, size_t lo, size_t hi, int device) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    size_t base = 0;
    for (const CopySeg &sg : segs) {
        const size_t a = std::max(lo, base), b = std::min(hi, base + sg.bytes);
        if (a < b) {
            volatile char *d = (volatile char *)sg.dst + (a - base);
            for (size_t x = 0; x < b - a; x += 4096) d[x] = 0;
            d[b - a - 1] = 0;
        }
        base += sg.bytes;
    }
    base = 0;
    for (const CopySeg &sg : segs) {
        const size_t a = std::max(lo, base), b = std::min(hi, base + sg.bytes);
        if (a < b) {
            e = cudaMemcpy((char *)sg.dst + (a - base), (const char *)sg.src + (a - base), b - a,
                           cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) return e;
        }
        base += sg.bytes;
    }
    return cudaSuccess;
}

cudaError_t copy_out_all(const std::vector<CopySeg> &segs_in) {
    std::vector<CopySeg> segs;
    size_t total = 0;
    for (const CopySeg &sg : segs_in)
        if (sg.dst && sg.bytes) {
            segs.push_back(sg);
            total += sg.bytes;
        }
    if (total == 0) return cudaSuccess;
    int device = 0;
    cudaGetDevice(&device);
    unsigned hw = std::thread::hardware_concurrency();
    // one thread per MiB, up to 16 (or the host's cores)
    int threads = (int)std::min<size_t>(std::min<unsigned>(hw ? hw : 1, 16u), total >> 20);
    if (total <= Scratch::PINNED) {
        // small: every array into the pinned buffer in stream order, one wait
        cudaError_t e;
        Scratch *x = acquire_scratch(device, &e);
        if (x) {
            size_t at = 0;
            for (const CopySeg &sg : segs) {
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(x->pinned + at, sg.src, sg.bytes, cudaMemcpyDeviceToHost, x->st);
                at += sg.bytes;
            }
            const cudaError_t e2 = cudaStreamSynchronize(x->st);
            if (e == cudaSuccess) e = e2;
            at = 0;
            for (const CopySeg &sg : segs) {
                if (e == cudaSuccess) std::memcpy(sg.dst, x->pinned + at, sg.bytes);
                at += sg.bytes;
            }
            release_scratch(x, e == cudaSuccess);
        }
        return e;
    }
    if (threads <= 1) {
        for (const CopySeg &sg : segs) {
            cudaError_t e = cudaMemcpy(sg.dst, sg.src, sg.bytes, cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    const size_t slice = ((total + threads - 1) / threads + 4095) & ~size_t(4095);
    std::vector<cudaError_t> errs(threads, cudaSuccess);
    std::vector<std::thread> pool;
    for (int t = 0; t < threads; t++) {
        const size_t lo = std::min(total, (size_t)t * slice), hi = std::min(total, lo + slice);
        pool.emplace_back([&, t, lo, hi] { errs[t] = copy_range(segs, lo, hi, device); });
    }
    for (auto &th : pool) th.join();
    for (cudaError_t e : errs)
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t copy_out(void *dst, const void *src, size_t bytes) { return copy_out_all({{dst, src, bytes}}); }

}  // namespace

extern "C" {

const char *pjg_last_error(void) { return g_error.c_str(); }

pjg_status pjg_init(int32_t device) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0)
        return fail(PJG_ERR_NO_DEVICE, "no CUDA device: %s", e == cudaSuccess ? "count is 0" : cudaGetErrorString(e));
    if (device < 0 || device >= n) return fail(PJG_ERR_INVALID, "device %d out of range (%d devices)", device, n);
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(PJG_ERR_CUDA, "cudaSetDevice: %s", cudaGetErrorString(e));
    return PJG_OK;
}

// ---------------------------------------------------------------------------
// Templates

pjg_status pjg_templates_create(const pjg_template_set *set, pjg_templates **out) {
    pjg_status status = PJG_OK;
    if (!set || !out) return fail(PJG_ERR_INVALID, "null argument");
    if (set->n_templates < 0) return fail(PJG_ERR_INVALID, "negative template count");
    int T = set->n_templates;
    if (T > 0 && (!set->atom_offset)) return fail(PJG_ERR_INVALID, "null atom_offset");
    int A = T > 0 ? set->atom_offset[T] : 0;
    if (A > 0 && (!set->code || !set->res_seq || !set->chain || !set->xyz || !set->dist_weight ||
                  !set->name_offset || !set->resname_offset))
        return fail(PJG_ERR_INVALID, "null template atom array");
    pjg_templates *h = new pjg_templates;
    cudaGetDevice(&h->device);
    h->T = T;
    h->A = A;
    h->atom_begin.assign(set->atom_offset, set->atom_offset + T + 1);
    if (T == 0) h->atom_begin = {0};
    std::vector<int32_t> sig(A), key(A);
    std::vector<double> pos(3 * (size_t)A), weight(A);
    // signatures
    // signature ids by the bytes of (code, name count, names, residue names)
    std::unordered_map<std::string, int> sig_ids;
    sig_ids.reserve((size_t)A);
    std::vector<uint32_t> names, res, keyv;
    std::string keys;
    std::vector<int32_t> s_code, s_rule, s_main, s_nb{0}, s_rb{0}, s_pb{0};
    std::vector<uint32_t> s_names, s_res, s_pres, s_pname;
    for (int t = 0; t < T; t++) {
        int a0 = set->atom_offset[t], a1 = set->atom_offset[t + 1];
        if (a1 < a0) {
            delete h;
            return fail(PJG_ERR_INVALID, "template %d: decreasing atom offsets", t);
        }
        if (a1 - a0 > MAX_TEMPLATE_ATOMS) {
            delete h;
            return fail(PJG_ERR_INVALID, "template %d has %d atoms; at most %d are supported", t, a1 - a0,
                        MAX_TEMPLATE_ATOMS);
        }
        if (a1 - a0 > 32) {
            h->large.push_back(t);
            (a1 - a0 <= 64 ? h->wide : h->huge).push_back(t);
        }
        h->nmax = std::max(h->nmax, a1 - a0);
    }
    for (int a = 0; a < A; a++) {
        int code = set->code[a];
        bool valid = (code >= -1 && code <= 8) || (code >= 100 && code <= 107);
        if (!valid) {
            delete h;
            return fail(PJG_ERR_INVALID, "template atom %d: invalid match mode %d", a, code);
        }
        names.clear();
        res.clear();
        for (int q = set->name_offset[a]; q < set->name_offset[a + 1]; q++) names.push_back(pack_upper(set->names + 4 * q));
        for (int q = set->resname_offset[a]; q < set->resname_offset[a + 1]; q++) {
            uint32_t r = pack_upper(set->resnames + 4 * q);
            if (std::find(res.begin(), res.end(), r) == res.end()) res.push_back(r);
        }
        keyv.clear();
        keyv.push_back((uint32_t)code);
        keyv.push_back((uint32_t)names.size());
        keyv.insert(keyv.end(), names.begin(), names.end());
        keyv.insert(keyv.end(), res.begin(), res.end());
        keys.assign(reinterpret_cast<const char *>(keyv.data()), keyv.size() * sizeof(uint32_t));
        auto it = sig_ids.find(keys);
        int id;
        if (it == sig_ids.end()) {
            id = (int)s_code.size();
            sig_ids.emplace(keys, id);
            int mode = code >= 100 ? code - 100 : code;
            int rule = mode == -1 ? RULE_ANY : mode == 1 ? RULE_NAME_OR_PARTNER : mode == 2 ? RULE_NAME_OR_MAINCHAIN
                     : mode == 3 ? RULE_ELEMENT : RULE_NAME;
            s_code.push_back(code);
            s_rule.push_back(rule);
            int mc = 0;
            for (uint32_t nm : names)
                if (nm == pack_lit("_CA_") || nm == pack_lit("_N__") || nm == pack_lit("_O__")) mc = 1;
            s_main.push_back(mc);
            s_names.insert(s_names.end(), names.begin(), names.end());
            s_nb.push_back((int32_t)s_names.size());
            s_res.insert(s_res.end(), res.begin(), res.end());
            s_rb.push_back((int32_t)s_res.size());
            if (rule == RULE_NAME_OR_PARTNER) {
                for (uint32_t nm : names)
                    for (const PartnerDef &p : PARTNER_TABLE) {
                        if (nm == pack_lit(p.a)) {
                            s_pres.push_back(res_lit(p.res));
                            s_pname.push_back(pack_lit(p.b));
                        }
                        if (nm == pack_lit(p.b)) {
                            s_pres.push_back(res_lit(p.res));
                            s_pname.push_back(pack_lit(p.a));
                        }
                    }
            }
            s_pb.push_back((int32_t)s_pres.size());
        } else {
            id = it->second;
        }
        sig[a] = id;
        key[a] = make_key(set->res_seq[a], set->chain[2 * a + 1]);
        for (int d = 0; d < 3; d++) pos[3 * (size_t)a + d] = set->xyz[3 * (size_t)a + d];
        weight[a] = set->dist_weight[a];
    }
    h->G = (int32_t)s_code.size();
    // distance matrices (TessAtom_distance, patches/TessAtom.c.patch:229-244;
    // Template.__init__, src/pyjess/_jess.pyx:1894-1901)
    std::vector<double> dist;
    h->param_begin.push_back(0);
    for (int t = 0; t < T; t++) {
        int a0 = set->atom_offset[t], n = set->atom_offset[t + 1] - a0;
        size_t base = dist.size();
        dist.resize(base + (size_t)n * n, 0.0);
        for (int i = 0; i < n; i++)
            for (int j = i + 1; j < n; j++) {
                double acc = 0.0;
                for (int d = 0; d < 3; d++) {
                    double tmp = pos[3 * (size_t)(a0 + i) + d] - pos[3 * (size_t)(a0 + j) + d];
                    acc += tmp * tmp;
                }
                acc = std::sqrt(acc);
                dist[base + (size_t)i * n + j] = acc;
                dist[base + (size_t)j * n + i] = acc;
            }
        h->param_begin.push_back((int32_t)dist.size());
    }
    if (dist.size() > (size_t)INT32_MAX) {
        delete h;
        return fail(PJG_ERR_INVALID, "templates too large: %zu distance-matrix entries (at most %d)", dist.size(),
                    INT32_MAX);
    }
    h->n_params = (int64_t)dist.size();
    if (set->dim) h->dim.assign(set->dim, set->dim + T);
    {
        Upload up;
        up.add(&h->d_atom_begin, h->atom_begin);
        up.add(&h->d_sig, sig);
        up.add(&h->d_key, key);
        up.add(&h->d_param_begin, h->param_begin);
        up.add(&h->d_pos, pos);
        up.add(&h->d_weight, weight);
        up.add(&h->d_dist, dist);
        up.add(&h->d_code, s_code);
        up.add(&h->d_rule, s_rule);
        up.add(&h->d_mainchain, s_main);
        up.add(&h->d_name_begin, s_nb);
        up.add(&h->d_names, s_names);
        up.add(&h->d_res_begin, s_rb);
        up.add(&h->d_resnames, s_res);
        up.add(&h->d_partner_begin, s_pb);
        up.add(&h->d_partner_res, s_pres);
        up.add(&h->d_partner_name, s_pname);
        up.add(&h->d_large, h->large);
        up.add(&h->d_wide, h->wide);
        up.add(&h->d_huge, h->huge);
        keep_pool(h->device);
        cudaError_t e;
        Scratch *x = acquire_scratch(h->device, &e);
        if (e == cudaSuccess) e = up.run(&h->block, x);
        if (e == cudaSuccess) e = cudaStreamSynchronize(x->st);
        if (e == cudaSuccess) {
            handle_created();
            h->counted = true;
        }
        release_scratch(x, e == cudaSuccess);
        if (e != cudaSuccess) {
            status = fail(e == cudaErrorMemoryAllocation ? PJG_ERR_OOM : PJG_ERR_CUDA, "template upload: %s",
                          cudaGetErrorString(e));
            pjg_templates_destroy(h);
            return status;
        }
    }
    *out = h;
    return PJG_OK;
}

void pjg_templates_destroy(pjg_templates *h) {
    if (!h) return;
    h->block.free();
    if (h->counted) handle_destroyed();
    delete h;
}

// ---------------------------------------------------------------------------
// Structures

pjg_status pjg_structures_create(const pjg_structure_set *set, pjg_structures **out) {
    if (!set || !out) return fail(PJG_ERR_INVALID, "null argument");
    if (set->n_structures < 0) return fail(PJG_ERR_INVALID, "negative structure count");
    int S = set->n_structures;
    if (S > 0 && !set->atom_offset) return fail(PJG_ERR_INVALID, "null atom_offset");
    int64_t N = S > 0 ? set->atom_offset[S] : 0;
    if (N > 0 && (!set->xyz || !set->name || !set->resname || !set->chain || !set->res_seq || !set->serial))
        return fail(PJG_ERR_INVALID, "null structure atom array");
    pjg_structures *h = new pjg_structures;
    cudaGetDevice(&h->device);
    h->S = S;
    h->N = N;
    std::vector<int64_t> base(std::max(S, 0));
    std::vector<int32_t> count(std::max(S, 0));
    HostArray<float4> xyz32((size_t)N);
    HostArray<uint32_t> name((size_t)N), resname((size_t)N);
    HostArray<int32_t> sorted((size_t)N);
    HostArray<uint8_t> name_id((size_t)N);
    HostArray<int32_t> nh_pos((size_t)N);
    HostArray<uint16_t> local_kind((size_t)N);
    std::vector<int32_t> bucket_begin{0}, bucket_lo, bucket_hi;
    std::vector<uint32_t> bucket_name;
    for (int s = 0; s < S; s++) {
        int64_t b0 = set->atom_offset[s], b1 = set->atom_offset[s + 1];
        if (b1 < b0) {
            delete h;
            return fail(PJG_ERR_INVALID, "structure %d: decreasing atom offsets", s);
        }
        if (b1 - b0 > INT32_MAX / 2) {
            delete h;
            return fail(PJG_ERR_INVALID, "structure %d too large", s);
        }
        base[s] = b0;
        count[s] = (int)(b1 - b0);
        h->max_atoms = std::max(h->max_atoms, count[s]);
    }
    // per structure, on host threads: centroid-relative FP32 coordinates
    // with the residue key, packed names, and the ResIndex order (stable by
    // residue name, then serial) with its residue-name buckets
    struct Buckets {
        std::vector<uint32_t> name;
        std::vector<int32_t> lo, hi;
        std::vector<uint32_t> hname;  // distinct atom names of each bucket, sorted
        std::vector<int32_t> hcount, hbegin{0};
        std::vector<int32_t> hoff;    // start of each distinct name's atoms in nh_pos (structure-local)
        std::vector<int32_t> hkind;   // its kind (distinct residue and atom name), in the numbers of
        int thread = 0;               //   the host thread that met it
        double radius = 0.0;
        int64_t bad = -1;  // first atom with a non-finite coordinate
    };
    std::vector<Buckets> bk(std::max(S, 0));
    // kinds of the set: each host thread numbers those it meets, the numbers
    // are joined afterwards (a table shared by the threads, locked for each new
    // kind, made an upload of 16 structures 0.8 ms longer)
    struct ThreadKinds {
        std::unordered_map<uint64_t, int32_t> number;
        std::vector<uint64_t> key;
        int32_t of(uint32_t res, uint32_t nm) {
            const uint64_t k = ((uint64_t)res << 32) | nm;
            auto ins = number.emplace(k, (int32_t)key.size());
            if (ins.second) key.push_back(k);
            return ins.first->second;
        }
    };
    auto prepare = [&](int s, ThreadKinds &seen, int thread) {
        const int64_t b0 = base[s];
        const int n = count[s];
        Buckets &B = bk[s];
        B.thread = thread;
        for (int i = 0; i < n && B.bad < 0; i++)
            for (int d = 0; d < 3; d++)
                if (!std::isfinite(set->xyz[3 * (b0 + i) + d])) B.bad = i;
        if (B.bad >= 0) return;
        double c[3] = {0, 0, 0};
        for (int i = 0; i < n; i++)
            for (int d = 0; d < 3; d++) c[d] += set->xyz[3 * (b0 + i) + d];
        if (n > 0)
            for (int d = 0; d < 3; d++) c[d] /= (double)n;
        for (int i = 0; i < n; i++) {
            int64_t a = b0 + i;
            double dx = set->xyz[3 * a] - c[0], dy = set->xyz[3 * a + 1] - c[1], dz = set->xyz[3 * a + 2] - c[2];
            double r = std::sqrt(dx * dx + dy * dy + dz * dz);
            if (r > B.radius) B.radius = r;
            int32_t k = make_key(set->res_seq[a], set->chain[2 * a + 1]);
            float kf;
            std::memcpy(&kf, &k, 4);
            xyz32[a] = make_float4((float)dx, (float)dy, (float)dz, kf);
            name[a] = pack_upper(set->name + 4 * a);
            resname[a] = pack_upper(set->resname + 4 * a);
        }
        // ResIndex: stable order by (residue name, serial) -- a counting
        // sort by residue name (in byte order of the upper-cased name), then
        // a stable sort by serial of each bucket not already in serial order
        std::vector<int32_t> idx(n);
        {
            std::vector<std::pair<uint32_t, int32_t>> kinds;  // big-endian name, count
            std::vector<int32_t> kind(n);
            for (int i = 0; i < n; i++) {
                const uint8_t *r = set->resname + 4 * (b0 + i);
                const uint32_t k = ((uint32_t)up(r[0]) << 24) | ((uint32_t)up(r[1]) << 16) |
                                   ((uint32_t)up(r[2]) << 8) | up(r[3]);
                int q = 0;
                while (q < (int)kinds.size() && kinds[q].first != k) q++;
                if (q == (int)kinds.size()) kinds.push_back({k, 0});
                kinds[q].second++;
                kind[i] = q;
            }
            std::vector<int> by(kinds.size());
            std::iota(by.begin(), by.end(), 0);
            std::sort(by.begin(), by.end(), [&](int x, int y) { return kinds[x].first < kinds[y].first; });
            std::vector<int32_t> start(kinds.size());
            int acc = 0;
            for (int q : by) {
                start[q] = acc;
                acc += kinds[q].second;
            }
            std::vector<int32_t> fill = start;
            for (int i = 0; i < n; i++) idx[fill[kind[i]]++] = i;
            const int32_t *ser = set->serial + b0;
            for (size_t q = 0; q < kinds.size(); q++) {
                int32_t *lo = idx.data() + start[q], *hi = lo + kinds[q].second;
                bool ordered = true;
                for (int32_t *x = lo; x + 1 < hi && ordered; x++) ordered = ser[x[0]] <= ser[x[1]];
                if (!ordered) std::stable_sort(lo, hi, [&](int x, int y) { return ser[x] < ser[y]; });
            }
        }
        for (int i = 0; i < n; i++) {
            sorted[b0 + i] = idx[i];
            uint32_t rn = resname[b0 + idx[i]];
            if (i == 0 || rn != B.name.back()) {
                if (i > 0) B.hi.push_back(i);
                B.name.push_back(rn);
                B.lo.push_back(i);
            }
        }
        if (n > 0) B.hi.push_back(n);
        // per bucket: its distinct atom names and their counts
        std::vector<uint32_t> nm;
        for (size_t k = 0; k < B.name.size(); k++) {
            nm.clear();
            for (int i = B.lo[k]; i < B.hi[k]; i++) nm.push_back(name[b0 + idx[i]]);
            std::sort(nm.begin(), nm.end());
            const size_t h0 = B.hname.size();
            for (size_t i = 0; i < nm.size(); i++) {
                if (i == 0 || nm[i] != nm[i - 1]) {
                    B.hname.push_back(nm[i]);
                    B.hcount.push_back(0);
                    B.hkind.push_back(seen.of(B.name[k], nm[i]));
                }
                B.hcount.back()++;
            }
            B.hbegin.push_back((int32_t)B.hname.size());
            // the bucket's atoms grouped by name (groups in name order, each
            // in ResIndex order), from the bucket's first position
            std::vector<int32_t> fill(B.hname.size() - h0);
            for (size_t j = 0, acc = (size_t)B.lo[k]; j < fill.size(); j++) {
                fill[j] = (int32_t)acc;
                B.hoff.push_back((int32_t)acc);
                acc += (size_t)B.hcount[h0 + j];
            }
            for (int i = B.lo[k]; i < B.hi[k]; i++) {
                const int a = idx[i];
                const size_t id = std::lower_bound(B.hname.begin() + h0, B.hname.end(), name[b0 + a]) -
                                  (B.hname.begin() + h0);
                name_id[b0 + a] = (uint8_t)std::min<size_t>(id, 255);
                local_kind[b0 + a] = (uint16_t)std::min<size_t>(h0 + id, 65535);
                nh_pos[b0 + fill[id]++] = a;
            }
        }
    };
    const int nthreads = (int)std::max<unsigned>(1, std::min<unsigned>(32, std::thread::hardware_concurrency()));
    std::vector<ThreadKinds> met((size_t)std::max(1, std::min(nthreads, S)));
    {
        std::atomic<int> next{0};
        auto worker = [&](int i) {
            for (int s; (s = next.fetch_add(1)) < S;) prepare(s, met[i], i);
        };
        std::vector<std::thread> pool;
        for (int i = 1; i < (int)met.size(); i++) pool.emplace_back(worker, i);
        worker(0);
        for (auto &th : pool) th.join();
    }
    for (int s = 0; s < S; s++)
        if (bk[s].bad >= 0) {
            delete h;
            return fail(PJG_ERR_INVALID, "structure %d atom %lld: non-finite coordinate", s, (long long)bk[s].bad);
        }
    // the kinds' numbers in the set, per thread and its own number
    ThreadKinds all;
    std::vector<std::vector<int32_t>> kind_of(met.size());
    for (size_t i = 0; i < met.size(); i++)
        for (uint64_t k : met[i].key) kind_of[i].push_back(all.of((uint32_t)(k >> 32), (uint32_t)k));
    std::vector<uint32_t> kind_name, kind_res;
    for (uint64_t k : all.key) {
        kind_name.push_back((uint32_t)k);
        kind_res.push_back((uint32_t)(k >> 32));
    }
    std::vector<int32_t> nh_begin{0}, nh_count, nh_off, nh_kind;
    std::vector<uint32_t> nh_name;
    for (int s = 0; s < S; s++) {
        const Buckets &B = bk[s];
        for (size_t k = 0; k + 1 < B.hbegin.size(); k++) nh_begin.push_back((int32_t)nh_name.size() + B.hbegin[k + 1]);
        nh_name.insert(nh_name.end(), B.hname.begin(), B.hname.end());
        nh_count.insert(nh_count.end(), B.hcount.begin(), B.hcount.end());
        nh_off.insert(nh_off.end(), B.hoff.begin(), B.hoff.end());
        for (int32_t k : B.hkind) nh_kind.push_back(kind_of[(size_t)B.thread][(size_t)k]);
        h->max_local_kinds = std::max(h->max_local_kinds, (int32_t)B.hname.size());
    }
    h->n_kinds = (int32_t)kind_name.size();
    for (int s = 0; s < S; s++) {
        const Buckets &B = bk[s];
        h->max_radius = std::max(h->max_radius, B.radius);
        bucket_name.insert(bucket_name.end(), B.name.begin(), B.name.end());
        bucket_lo.insert(bucket_lo.end(), B.lo.begin(), B.lo.end());
        bucket_hi.insert(bucket_hi.end(), B.hi.begin(), B.hi.end());
        bucket_begin.push_back((int32_t)bucket_name.size());
    }
    h->atom_base = base;
    const size_t n1 = (size_t)std::max<int64_t>(N, 1);
    uint16_t *d_local_kind = nullptr;
    Upload up;
    up.add(&h->d_xyz64, set->xyz, 3 * (size_t)N);
    up.add(&h->d_atom_base, base);
    up.add(&h->d_atom_count, count);
    up.add(&h->d_xyz32, xyz32.p.get(), (size_t)N);
    up.add(&h->d_name, name.p.get(), (size_t)N);
    up.add(&h->d_resname, resname.p.get(), (size_t)N);
    up.add(&h->d_sorted, sorted.p.get(), (size_t)N);
    up.add(&h->d_bucket_begin, bucket_begin);
    up.add(&h->d_bucket_name, bucket_name);
    up.add(&h->d_bucket_lo, bucket_lo);
    up.add(&h->d_bucket_hi, bucket_hi);
    up.add(&h->d_nh_begin, nh_begin);
    up.add(&h->d_nh_name, nh_name);
    up.add(&h->d_nh_count, nh_count);
    up.add(&h->d_name_id, name_id.p.get(), (size_t)N);
    up.add(&h->d_nh_off, nh_off);
    up.add(&h->d_nh_pos, nh_pos.p.get(), (size_t)N);
    up.add(&h->d_kind_name, kind_name);
    up.add(&h->d_kind_res, kind_res);
    up.add(&h->d_nh_kind, nh_kind);
    up.add(&d_local_kind, local_kind.p.get(), (size_t)N);
    up.room(&h->d_lrank, 3 * n1);
    up.room(&h->d_urank, 3 * n1);
    up.room(&h->d_kxyz, n1);
    up.room(&h->d_res_pos, n1);
    up.room(&h->d_res_place, n1);
    up.room(&h->d_res_kind, n1);
    up.room(&h->d_res_range, n1);
    keep_pool(h->device);
    cudaError_t e;
    Scratch *x = acquire_scratch(h->device, &e);
    if (e == cudaSuccess) e = up.run(&h->block, x);
    if (e == cudaSuccess) {
        // axis ranks of every atom (the leaf-order sorted-axis path), and the
        // residue order and kind-ordered points of the order-free search
        // (the sorted tiles: a kept block where one is large enough)
        const size_t tile_bytes = (sizeof(unsigned long long) + sizeof(uint16_t)) * 4 * n1;
        DBuf<unsigned long long> kept;
        Block tiles;
        t_cache = &x->cache;
        const bool small = BlockCache::class_of(tile_bytes) >= 0;
        e = small ? dalloc(kept, tile_bytes / sizeof(unsigned long long) + 1, x->st) : tiles.alloc(tile_bytes, x->st);
        if (e == cudaSuccess) {
            unsigned long long *tile_key = small ? kept.p : (unsigned long long *)tiles.p;
            uint16_t *tile_idx = (uint16_t *)(tile_key + 4 * n1);
            launch_axis_ranks(x->st, S, h->max_atoms, h->d_atom_base, h->d_atom_count, h->d_xyz64, N, tile_key,
                              tile_idx, h->d_lrank, h->d_urank,
                              ResidueOrder{h->d_xyz32, h->d_nh_pos, d_local_kind, h->d_kxyz, h->d_res_pos,
                                           h->d_res_kind, h->d_res_range, h->d_sorted, h->d_res_place});
            e = cudaGetLastError();
        }
        tiles.free(x->st);
        dfree(kept, x->st);
        t_cache = nullptr;
        const cudaError_t e2 = cudaStreamSynchronize(x->st);
        if (e == cudaSuccess) e = e2;
    }
    if (e == cudaSuccess) {
        handle_created();
        h->counted = true;
    }
    release_scratch(x, e == cudaSuccess);
    if (e != cudaSuccess) {
        pjg_status st = fail(e == cudaErrorMemoryAllocation ? PJG_ERR_OOM : PJG_ERR_CUDA, "structure upload: %s",
                             cudaGetErrorString(e));
        pjg_structures_destroy(h);
        return st;
    }
    *out = h;
    return PJG_OK;
}

void pjg_structures_destroy(pjg_structures *h) {
    if (!h) return;
    h->block.free();
    if (h->counted) handle_destroyed();
    delete h;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Query

namespace {

__global__ void k_struct_totals(int32_t S, int32_t G, const int32_t *count, int64_t *totals) {
    int lane = threadIdx.x & 31;
    int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = warp; s < S; s += nw) {
        int64_t acc = 0;
        for (int g = lane; g < G; g += 32) acc += count[s * G + g];
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) totals[s] = acc;
    }
}

int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

// exclusive scan in[0..n) -> out[0..n), recursive over tile sums
// kernels launched by scan_exclusive on this thread (query statistics)
thread_local int t_scan_launches = 0;

template <typename T>
cudaError_t scan_exclusive(const T *in, int64_t n, int64_t *out, std::vector<DBuf<int64_t>> &tmp,
                           cudaStream_t st, int depth = 0) {
    if (n <= 0) return cudaSuccess;
    t_scan_launches += n > SCAN_TILE_ITEMS ? 2 : 1;
    const int TILE = SCAN_TILE_ITEMS;
    int64_t tiles = (n + TILE - 1) / TILE;
    if ((int)tmp.size() < 2 * (depth + 1)) tmp.resize(2 * (depth + 1));
    cudaError_t e = dalloc(tmp[2 * depth], (size_t)tiles, st);
    if (e != cudaSuccess) return e;
    e = dalloc(tmp[2 * depth + 1], (size_t)tiles, st);
    if (e != cudaSuccess) return e;
    int64_t *sums = tmp[2 * depth].p, *soff = tmp[2 * depth + 1].p;
    if constexpr (sizeof(T) == 4) launch_scan_tiles_i32(st, in, n, out, sums);
    else launch_scan_tiles_i64(st, in, n, out, sums);
    if (tiles > 1) {
        e = scan_exclusive<int64_t>(sums, tiles, soff, tmp, st, depth + 1);
        if (e != cudaSuccess) return e;
        launch_scan_add(st, out, n, soff);
    }
    return cudaGetLastError();
}

// bytes of an item's arrays: its place and result, rows before it, its list of
// segments, its levels, its counting bins, its counters
constexpr double ITEM_BYTES = 8 + 8 + 8 + 4 + 8 + 8 + 32;

// places in a query's block of counters: the statistics (Counter), the lists
// requested in a chunk, then what an attempt at a chunk's search adds up
enum : int {
    ZC_LEAF_USED = C_NUM,
    ZC_NFILL,
    ZC_ATTEMPT,
    ZC_ROWS = ZC_ATTEMPT,
    ZC_FREE,            // units, heavy pairs, their items, scratch, large units,
                        // spilled entries, units left to the leaf order, long
                        // units, items to search in order
    ZC_NWORK = ZC_FREE + 9,
    ZC_NSUSP,
    ZC_POOL,
    ZC_ITEM,            // the work queue (32 bits)
    ZC_TOTALS,          // hits, warnings, hit atoms, passing rows, long pairs
    ZC_LIVE = ZC_TOTALS + 5,
    ZC_SNAP = ZC_LIVE,  // the statistics before a chunk's search,
    ZC_CHUNK = ZC_SNAP + C_NUM,  // and before the chunk
    ZC_END = ZC_CHUNK + C_NUM
};

#if PJG_SEARCH_PROF
// Profile builds: append the query's search profile as one JSON line to the
// file named by PJG_PROF_OUT (nothing when unset).
void write_search_profile(const unsigned long long *d_prof, cudaStream_t st, const pjg_stats &stats) {
    static const char *names[SP_NUM] = {
        "pairs", "empty", "cyc_pair", "cyc_setup", "cyc_seed", "cyc_block", "cyc_prod", "cyc_emit",
        "loop_iters", "block_visits", "block_visits_l0", "chain_full", "chain_sibling", "g0_iters",
        "blocks_tested", "blocks_hit", "leaves_inbox", "batches", "batch_lanes", "child_block",
        "prod_batches", "prod_batches_l0", "prod_lanes", "child_prod", "fp64", "rows", "cyc_chain", "cyc_batch", "cyc_ctrl", "cyc_susp",
        "tail_ns", "pair_max_cyc"};
    unsigned long long h[SP_NUM] = {};
    if (cudaMemcpyAsync(h, d_prof, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return;
    const char *path = getenv("PJG_PROF_OUT");
    if (!path || !*path) return;
    FILE *f = fopen(path, "a");
    if (!f) return;
    fprintf(f, "{\"ms_expansion\": %.3f, \"partials\": %lld, \"search_rounds\": %d", stats.ms_expansion,
            (long long)stats.partials, stats.search_rounds);
    for (int i = 0; i < SP_NUM; i++) fprintf(f, ", \"%s\": %llu", names[i], h[i]);
    static const char *lnames[LP_CLASS] = {"lists", "entries", "handed", "cyc_list", "cyc_load", "cyc_sort",
                                           "cyc_count", "cyc_seg", "cyc_write", "sort_nodes", "sort_words",
                                           "count_pairs"};
    unsigned long long lh[LP_NUM] = {};
    leaf_profile_read(lh, st);
    cudaStreamSynchronize(st);
    fprintf(f, ", \"leaf_order\": {");
    for (int i = 0; i < LP_CLASS; i++) fprintf(f, "%s\"%s\": %llu", i ? ", " : "", lnames[i], lh[i]);
    const char *cls[3] = {"class_lists", "class_entries", "class_cycles"};
    for (int k = 0; k < 3; k++) {
        fprintf(f, ", \"%s\": [", cls[k]);
        for (int c = 0; c < 7; c++) fprintf(f, "%s%llu", c ? ", " : "", lh[LP_CLASS + 7 * k + c]);
        fprintf(f, "]");
    }
    fprintf(f, "}}\n");
    fclose(f);
}
#endif

}  // namespace

// ---------------------------------------------------------------------------
// Execution tuning (process-wide, read at the start of each query)

namespace {
std::mutex g_tuning_mutex;
// (leaf_levels 0: the order-free search first; what it leaves, and chunks it
// does not take, are searched in order with ORDER_LEVELS)
constexpr pjg_tuning TUNING_DEFAULTS = {0, 64, 4096, 1, LEAF_RANK_MAX, -1};
constexpr int ORDER_LEVELS = 4;
pjg_tuning g_tuning = TUNING_DEFAULTS;

pjg_tuning current_tuning() {
    std::lock_guard<std::mutex> g(g_tuning_mutex);
    return g_tuning;
}
}  // namespace

extern "C" pjg_status pjg_set_tuning(const pjg_tuning *t) {
    pjg_tuning d = TUNING_DEFAULTS;
    if (t) {
        if (t->leaf_levels < -1 || t->leaf_levels > 64) return fail(PJG_ERR_INVALID, "leaf_levels %d", t->leaf_levels);
        if (t->block_min < 0 || t->block_min > 65535) return fail(PJG_ERR_INVALID, "block_min %d", t->block_min);
        if (t->tile_cap != 0 && (t->tile_cap < 32 || t->tile_cap > 16384))
            return fail(PJG_ERR_INVALID, "tile_cap %d", t->tile_cap);
        if (t->pair_grain < 0 || t->pair_grain > 64) return fail(PJG_ERR_INVALID, "pair_grain %d", t->pair_grain);
        if (t->leaf_rank_max < 0 || t->leaf_rank_max > LEAF_FAST_MAX)
            return fail(PJG_ERR_INVALID, "leaf_rank_max %d", t->leaf_rank_max);
        if (t->leaf_reach < -1 || t->leaf_reach > 64) return fail(PJG_ERR_INVALID, "leaf_reach %d", t->leaf_reach);
        if (t->leaf_levels) d.leaf_levels = t->leaf_levels;
        if (t->block_min) d.block_min = t->block_min;
        if (t->tile_cap) d.tile_cap = t->tile_cap;
        if (t->pair_grain) d.pair_grain = t->pair_grain;
        if (t->leaf_rank_max) d.leaf_rank_max = t->leaf_rank_max;
        if (t->leaf_reach) d.leaf_reach = t->leaf_reach;
    }
    std::lock_guard<std::mutex> g(g_tuning_mutex);
    g_tuning = d;
    return PJG_OK;
}

extern "C" pjg_status pjg_get_tuning(pjg_tuning *t) {
    if (!t) return fail(PJG_ERR_INVALID, "null argument");
    *t = current_tuning();
    return PJG_OK;
}

extern "C" pjg_status pjg_device_name(char *buf, int32_t len) {
    if (!buf || len <= 0) return fail(PJG_ERR_INVALID, "null or empty buffer");
    int dev = 0;
    cudaDeviceProp prop;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaGetDeviceProperties(&prop, dev);
    if (e != cudaSuccess) {
        buf[0] = 0;
        return fail(PJG_ERR_NO_DEVICE, "no CUDA device: %s", cudaGetErrorString(e));
    }
    snprintf(buf, (size_t)len, "%s", prop.name);
    return PJG_OK;
}

extern "C" pjg_status pjg_query(const pjg_templates *tp, const pjg_structures *sp, const pjg_query_params *P,
                                pjg_results **out) {
    pjg_status status = PJG_OK;
    if (!tp || !sp || !P || !out) return fail(PJG_ERR_INVALID, "null argument");
    if (P->ignore_chain < 0 || P->ignore_chain > 2) return fail(PJG_ERR_INVALID, "invalid ignore_chain %d", P->ignore_chain);
    if (P->max_candidates < -1) return fail(PJG_ERR_INVALID, "invalid max_candidates %d", P->max_candidates);
    if (P->mode < 0 || P->mode > 2) return fail(PJG_ERR_INVALID, "invalid mode %d", P->mode);
    if (P->count_only < 0 || P->count_only > 1) return fail(PJG_ERR_INVALID, "invalid count_only %d", P->count_only);
    if (!std::isfinite(P->distance_cutoff) || !std::isfinite(P->max_dynamic_distance))
        return fail(PJG_ERR_INVALID, "non-finite distance parameters");

    pjg_results *res = new pjg_results;
    cudaGetDevice(&res->device);
    res->count_only = P->count_only != 0;
    res->structures = sp;
    const int T = tp->T, S = sp->S, G = tp->G;
    const bool fp32 = P->mode == PJG_MODE_BATCHED_FP32;
    cudaStream_t st = nullptr;
    Scratch *scratch = nullptr;
    cudaEvent_t *ev = nullptr;
    // the query's counters, in one device block (offsets ZC_*): what a round
    // adds up is zeroed by one copy and read back by one
    DBuf<unsigned long long> d_z;
    unsigned long long *hz = nullptr;  // its host copy (pinned)
    struct {
        unsigned long long *p;
    } d_counters{}, d_ccount{}, d_rtotals{}, d_nwork{}, d_nsusp{}, d_nfill{}, d_pool_used{}, d_leaf_used{}, d_free_n{};
    struct {
        int32_t *p;
    } d_pair_counter{};
    DBuf<AnnulusParam> d_params;
    // order-free search: kinds of each signature, units of rows, heavy pairs
    // and their items, frontiers of the items, keys of large units
    DBuf<uint32_t> d_sig_bits, d_kind_masks;
    DBuf<RowUnit> d_units;
    DBuf<HeavyPair> d_heavy_pairs;
    DBuf<unsigned long long> d_item_stats, d_row_key;
    DBuf<int2> d_items, d_results;
    DBuf<int64_t> d_item_base, d_bin_off;
    DBuf<int32_t> d_bins, d_arena_atom, d_row_scratch, d_item_head, d_large_units, d_long_pairs, d_pending;
    DBuf<unsigned long long> d_item_branch;
    DBuf<SpilledEntry> d_spill_a, d_spill_b;
    DBuf<float4> d_arena_xyz;
    DBuf<uint16_t> d_arena_parent;
    DBuf<int32_t> d_count, d_scanned, d_cand_atom, d_leaf_atom;
    DBuf<int64_t> d_offset, d_totals, d_boff;
    DBuf<int32_t> d_nblk;
    DBuf<int64_t> d_exact_list, d_sorted_list;
    DBuf<unsigned long long> d_exact_count, d_sorted_count;
    DBuf<float4> d_blk_lo, d_blk_hi;
    DBuf<float4> d_leaf_xyz, d_leaf_xyz2;
    DBuf<int32_t> d_leaf_atom2;
    DBuf<int64_t> d_leaf_off;
    DBuf<int32_t> d_c_pair, d_c_atoms, d_pair_rows, d_cnt_q;
    DBuf<int64_t> d_c_ord, d_off_q;
    // lists ordered on demand: per-list state, requested lists, suspended pairs
    DBuf<int32_t> d_lstate;
    DBuf<int64_t> d_work;
    // lists filled on demand
    DBuf<int32_t> d_fill_state;
    DBuf<int64_t> d_fill_work;
    DBuf<Suspended> d_susp_a, d_susp_b;
    DBuf<unsigned char> d_pool_a, d_pool_b;
    // costliest pairs first: cost buckets, heavy flags and list, histogram
    DBuf<uint8_t> d_pcost, d_hflag;
    DBuf<int32_t> d_heavy;
    DBuf<unsigned long long> d_hbins;
    int64_t pool_cap = 0;
    // requested lists sharing one leaf order (table and worklists)
    DBuf<unsigned long long> d_ls_key, d_ls_n;
    DBuf<int32_t> d_ls_rep, d_ls_slot;
    DBuf<int64_t> d_ls_rep_work, d_ls_dup, d_ls_left;
    DBuf<uint8_t> d_ls_ok;
    DBuf<double> d_c_rmsd;
    DBuf<unsigned long long> d_prof;  // search profile (profile builds)
    // per complete row, in reference order
    DBuf<double> d_r_rmsd, d_r_rot, d_r_cen;
    DBuf<int32_t> d_r_nan, d_r_hit, d_r_warn, d_r_hatoms;
    DBuf<int64_t> d_r_src, d_r_hidx, d_r_widx, d_r_aidx;
    std::vector<DBuf<int64_t>> scan_tmp;
    int64_t passing = 0;
    const int stride = std::max(tp->nmax, 1);
    unsigned long long counters[C_NUM] = {};
    float ms = 0.f;
    double ms_cand = 0, ms_exp = 0, ms_sup = 0, ms_total = 0, ms_search = 0;
    int launches = 0, chunks = 0, search_rounds = 0, row_splits = 0;
    t_scan_launches = 0;
    int64_t suspensions = 0;
    // levels whose lists are put in kd leaf order before the search (deeper
    // lists when a pair's frontier first reaches them): the tuning's
    // leaf_levels, or PJG_LEAF_LEVELS when set; a negative value orders
    // every list up front.  The plain per-structure path orders every list
    // up front: with one structure a chunk, the host round trip of each
    // extra search round costs more than the ordering it saves.
    const pjg_tuning tune = current_tuning();
    int demand_levels = P->mode == PJG_MODE_PLAIN_FP64 ? -1 : tune.leaf_levels ? tune.leaf_levels : ORDER_LEVELS;
    {
        const char *v = getenv("PJG_LEAF_LEVELS");
        if (v && *v && P->mode != PJG_MODE_PLAIN_FP64) demand_levels = atoi(v);
    }
    // every pair searched without order first (k_search_free): the batched
    // modes, unless the levels to order up front are chosen explicitly
    FreeView fv{sp->n_kinds, (sp->n_kinds + 31) / 32, sp->d_kind_name, sp->d_kind_res, nullptr,
                (sp->max_local_kinds + 31) / 32, nullptr, sp->d_nh_kind, sp->d_kxyz, sp->d_res_pos, sp->d_res_kind,
                sp->d_res_range};
    bool free_first = P->mode != PJG_MODE_PLAIN_FP64 && tune.leaf_levels == 0 &&
                            !getenv("PJG_LEAF_LEVELS") && sp->max_local_kinds <= FREE_MAX_KINDS &&
                            (int64_t)G * fv.kind_words <= (1ll << 28);
    // few enough atoms and signatures for one chunk whatever the lists hold:
    // their total is not read back (order-free search: the lists are filled on
    // demand, and then their total is)
    constexpr int64_t LEAST_ENTRIES = 48ll << 20;
    bool few_entries = free_first && sp->N * (int64_t)G <= LEAST_ENTRIES && !getenv("PJG_ENTRY_BUDGET");
    // the lists' kind masks (up to 128 B a list, as the structure of the most
    // kinds needs) of the whole set in the pass that counts the lists, when
    // they take no more than mask_budget bytes; else chunk by chunk, so many
    // structures at a time (1,000 x 4,000 pairs: 0.2 GB and 3.0 ms in one pass)
    int64_t mask_budget = 2ll << 30;
    if (const char *v = getenv("PJG_MASK_BUDGET"))
        if (atoll(v) > 0) mask_budget = atoll(v);
    const int64_t mask_bytes = 4ll * G * fv.mask_words;  // a structure's
    bool masks_whole = free_first && (double)mask_bytes * S <= (double)mask_budget;
    // most structures a chunk may take for the order-free search's buffers: by
    // the masks, and for now (smaller once they did not fit, growing again)
    int mask_cap = INT32_MAX;
    if (free_first && !masks_whole)
        mask_cap = (int)std::max<int64_t>(
            1, std::min<int64_t>(INT32_MAX, mask_budget / std::max<int64_t>(mask_bytes, 1)));
    int free_cap = mask_cap;
    std::vector<int64_t> totals(S);

    if (T == 0 || S == 0) {
        *out = res;
        return PJG_OK;
    }
    {
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev != tp->device || dev != sp->device) {
            delete res;
            return fail(PJG_ERR_INVALID, "templates, structures and the calling thread use different devices");
        }
    }
    keep_pool(res->device);
    {
        cudaError_t e;
        scratch = acquire_scratch(res->device, &e);
        if (!scratch) {
            delete res;
            return fail(e == cudaErrorMemoryAllocation ? PJG_ERR_OOM : PJG_ERR_CUDA, "query set-up: %s",
                        cudaGetErrorString(e));
        }
        st = scratch->st;
        ev = scratch->ev;
        hz = reinterpret_cast<unsigned long long *>(scratch->pinned);
        t_cache = &scratch->cache;
    }
#if PJG_SEARCH_PROF
    leaf_profile_reset(st);
#endif
    CUDA_TRY(cudaEventRecord(ev[0], st));

    {
        // guard band: the requested width, widened if the FP32 rounding bound
        // of the largest structure needs more.  Coordinates are stored
        // relative to the structure's centroid, so each is within about
        // 2^-24 R of its FP64 value (R = largest distance from the centroid)
        // and the error of an FP32 squared distance d^2 is below
        // 2^-24 (10.4 R d + 4 d^2); a band g in distance covers a band of
        // about 2 b g in squared distance at radius b, so g must exceed
        // 2^-24 (5.2 R + 2 b), with b at most 2 R + 1 for any pair of atoms
        // (plus the tolerance) inside a structure.
        double g = P->guard_band > 0 ? P->guard_band : 1e-4;
        double bound = 2.0 * std::ldexp(1.0, -24) * (5.2 * sp->max_radius + 2.0 * (2.0 * sp->max_radius + 1.0));
        if (bound > g) g = bound;
        CUDA_TRY(dalloc(d_params, (size_t)std::max<int64_t>(tp->n_params, 1), st));
        launch_params(st, T, tp->d_atom_begin, tp->d_param_begin, tp->d_dist, tp->d_weight,
                      P->distance_cutoff, P->max_dynamic_distance, g, fp32, d_params.p);
        launches++;
        CUDA_TRY(cudaGetLastError());
    }
    CUDA_TRY(dalloc(d_z, ZC_END, st));
    CUDA_TRY(cudaMemsetAsync(d_z.p, 0, ZC_END * sizeof(unsigned long long), st));
    d_counters.p = d_z.p;
    d_leaf_used.p = d_z.p + ZC_LEAF_USED;
    d_nfill.p = d_z.p + ZC_NFILL;
    d_ccount.p = d_z.p + ZC_ROWS;
    d_free_n.p = d_z.p + ZC_FREE;
    d_nwork.p = d_z.p + ZC_NWORK;
    d_nsusp.p = d_z.p + ZC_NSUSP;
    d_pool_used.p = d_z.p + ZC_POOL;
    d_pair_counter.p = reinterpret_cast<int32_t *>(d_z.p + ZC_ITEM);
    d_rtotals.p = d_z.p + ZC_TOTALS;

    {
        // pass 1: list lengths for every (structure, signature)
        int64_t W = (int64_t)S * G;
        CUDA_TRY(dalloc(d_count, (size_t)W, st));
        CUDA_TRY(dalloc(d_scanned, (size_t)W, st));
        CUDA_TRY(dalloc(d_totals, (size_t)S, st));
        ChunkView cv{S, sp->d_atom_base, sp->d_atom_count, sp->d_xyz64, sp->d_xyz32, sp->d_name, sp->d_resname,
                     sp->d_sorted, sp->d_bucket_begin, sp->d_bucket_name, sp->d_bucket_lo, sp->d_bucket_hi,
                     sp->N, sp->d_lrank, sp->d_urank, sp->d_nh_begin, sp->d_nh_name, sp->d_nh_count,
                     sp->d_name_id, sp->d_nh_off, sp->d_nh_pos};
        SigView sv{G, tp->d_code, tp->d_rule, tp->d_mainchain, tp->d_name_begin, tp->d_names, tp->d_res_begin,
                   tp->d_resnames, tp->d_partner_begin, tp->d_partner_res, tp->d_partner_name};
        int blocks = (int)std::min<int64_t>((W + 7) / 8, (int64_t)sm_count() * 32);
        if (free_first) {
            // (no room for the signatures' kinds: the search in order)
            cudaError_t e = dalloc(d_sig_bits, (size_t)G * fv.kind_words, st);
            if (e == cudaSuccess && masks_whole) e = dalloc(d_kind_masks, (size_t)W * fv.mask_words, st);
            if (e == cudaErrorMemoryAllocation) {
                cudaGetLastError();
                free_first = few_entries = false;
                free_cap = mask_cap = INT32_MAX;
            } else {
                CUDA_TRY(e);
            }
        }
        if (free_first) {
            fv.sig_bits = d_sig_bits.p;
            launch_sig_kinds(st, sv, fv, d_sig_bits.p);
            launch_list_kinds(st, cv, sv, fv, d_count.p, d_scanned.p, masks_whole ? d_kind_masks.p : nullptr);
            launches++;
        } else {
            launch_candidates(st, std::max(blocks, 1), false, cv, sv, d_count.p, d_scanned.p, nullptr, nullptr);
        }
        launches++;
        CUDA_TRY(cudaGetLastError());
        if (!few_entries) {
            k_struct_totals<<<std::max(1, std::min(S, sm_count() * 8)), 256, 0, st>>>(S, G, d_count.p, d_totals.p);
            launches++;
            CUDA_TRY(cudaGetLastError());
            CUDA_TRY(cudaMemcpyAsync(totals.data(), d_totals.p, sizeof(int64_t) * S, cudaMemcpyDeviceToHost, st));
            CUDA_TRY(cudaStreamSynchronize(st));
        }
    }

    {
        // chunks of structures under an entry budget.  A candidate entry
        // costs at most ENTRY_BYTES: its atom in candidate order (4), block
        // boxes (32 B a block of CULL_BLK leaves), per-list arrays (~1) and,
        // once its list is put in leaf order, its atom and FP32 point in
        // leaf order (20; allocated as lists are requested).  The budget
        // takes 60% of the free device memory (counting memory the
        // stream-ordered pool holds unused) at that worst case, at least 48M
        // entries, which leaves room for growing the leaf arrays (old and new
        // copies live at once while they grow).  Fewer, larger chunks leave
        // fewer kernel tails and search rounds.  PJG_ENTRY_BUDGET overrides
        // it.
        constexpr double ENTRY_BYTES = 25.0 + 32.0 / CULL_BLK;
        int64_t ENTRY_BUDGET = LEAST_ENTRIES;
        if (!few_entries) {
            size_t free_b = 0, total_b = 0;
            if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) {
                cudaMemPool_t pool;
                if (cudaDeviceGetDefaultMemPool(&pool, res->device) == cudaSuccess) {
                    uint64_t reserved = 0, used = 0;
                    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
                        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
                        reserved > used)
                        free_b += (size_t)(reserved - used);
                }
                cudaGetLastError();
                ENTRY_BUDGET = std::max<int64_t>(ENTRY_BUDGET, (int64_t)((double)free_b * 0.6 / ENTRY_BYTES));
            }
            const char *v = getenv("PJG_ENTRY_BUDGET");
            if (v && atoll(v) > 0) ENTRY_BUDGET = atoll(v);
        }
        const int max_chunk = P->mode == PJG_MODE_PLAIN_FP64 ? 1 : 4096;
        // structures a chunk may take; halved when a chunk's complete rows
        // outgrow the memory of the per-row stages (see below), then sized
        // from the rows a structure of the last chunk produced
        int chunk_cap = max_chunk;
        const bool cut_inline = !P->best_match && P->max_candidates >= 0;
        // device bytes a complete row takes: its record in the row buffers
        // (grown with a quarter of headroom) and the per-row stages after the
        // search (superposition, automaton, compaction and the hits they may
        // append)
        // (order-free search: a unit a row, and for the units put in order by
        // their lists' leaves a key, five words of scratch and three places)
        const double row_buf_bytes = 12.0 + 4.0 * stride + (cut_inline ? 8.0 : 0.0) +
                                     (free_first ? (double)sizeof(RowUnit) : 0.0);
        const double row_stage_bytes = 360.0 + 4.0 * stride + (free_first ? 40.0 : 0.0);
        // memory a chunk's rows may use: free device memory, memory the
        // stream-ordered pool holds unused, and the row buffers and per-row
        // arrays of the previous chunk (reused)
        auto row_memory = [&]() -> double {
            double a = 0.0;
            size_t free_b = 0, total_b = 0;
            if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) a = (double)free_b;
            cudaMemPool_t pool;
            if (cudaDeviceGetDefaultMemPool(&pool, res->device) == cudaSuccess) {
                uint64_t reserved = 0, used = 0;
                if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
                    cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
                    reserved > used)
                    a += (double)(reserved - used);
            }
            cudaGetLastError();
            a += (double)(d_c_pair.n * 4 + d_c_ord.n * 8 + d_c_atoms.n * 4 + d_c_rmsd.n * 8);
            a += (double)(d_units.n * sizeof(RowUnit) + d_row_key.n * 8 + d_row_scratch.n * 4 + d_pending.n * 4 +
                          d_large_units.n * 4);
            a += (double)(d_r_rmsd.n * 8 + d_r_rot.n * 8 + d_r_cen.n * 8 + d_r_nan.n * 4 + d_r_src.n * 8 +
                          d_r_hit.n * 4 + d_r_warn.n * 4 + d_r_hatoms.n * 4 + d_r_hidx.n * 8 + d_r_widx.n * 8 +
                          d_r_aidx.n * 8);
            return a;
        };
        // rows a chunk may produce (PJG_ROW_BUDGET sets it)
        auto row_budget = [&]() -> int64_t {
            const char *v = getenv("PJG_ROW_BUDGET");
            if (v && atoll(v) > 0) return atoll(v);
            return (int64_t)(0.7 * row_memory() / (row_buf_bytes * 1.25 + row_stage_bytes));
        };
        // best_match with max_candidates: a pair stops after max_candidates
        // + 2 complete rows, so a structure yields at most T times that; the
        // chunks are sized from this bound before any search (no chunk then
        // needs a split)
        int bound_cap = max_chunk;
        if (P->best_match && P->max_candidates >= 0 && max_chunk > 1) {
            const double per = (double)T * ((double)P->max_candidates + 2.0);
            bound_cap = (int)std::max(1.0, std::min((double)max_chunk, (double)row_budget() / per));
            chunk_cap = bound_cap;
        }
        // items a chunk may hold: their arrays in an eighth of the memory its
        // rows may use (PJG_ITEM_BUDGET sets it)
        auto item_budget = [&](int64_t n) -> int64_t {
            const char *v = getenv("PJG_ITEM_BUDGET");
            if (v && atoll(v) > 0) return atoll(v);
            if (n <= 1 << 22) return INT32_MAX;
            return std::min<int64_t>(INT32_MAX, (int64_t)(row_memory() / 8 / ITEM_BYTES));
        };
        int ordered_from = -1;  // a structure searched in order: alone it outgrows the order-free search
        int s0 = 0;
        int64_t c_cap = 1 << 20;
        CUDA_TRY(dalloc(d_c_pair, c_cap, st));
        CUDA_TRY(dalloc(d_c_ord, c_cap, st));
        CUDA_TRY(dalloc(d_c_atoms, (size_t)c_cap * stride, st));
        if (cut_inline) CUDA_TRY(dalloc(d_c_rmsd, c_cap, st));
        while (s0 < S) {
            int s1 = s0;
            int64_t entries = 0;
            while (s1 < S && (s1 == s0 || (entries + totals[s1] <= ENTRY_BUDGET && s1 - s0 < std::min(chunk_cap, free_cap)))) {
                entries += totals[s1];
                s1++;
            }
            chunks++;
            const double ms_search_chunk0 = ms_search;
            // host statistics and device counters before this chunk (restored
            // if it is redone on fewer structures)
            const int search_rounds0 = search_rounds;
            const int64_t suspensions0 = suspensions;
            const size_t stats_bytes = C_NUM * sizeof(unsigned long long);
            CUDA_TRY(cudaMemcpyAsync(d_z.p + ZC_CHUNK, d_counters.p, stats_bytes, cudaMemcpyDeviceToDevice, st));
            const int Sc = s1 - s0;
            const int64_t Wc = (int64_t)Sc * G;
            ChunkView cv{Sc, sp->d_atom_base + s0, sp->d_atom_count + s0, sp->d_xyz64, sp->d_xyz32, sp->d_name,
                         sp->d_resname, sp->d_sorted, sp->d_bucket_begin + s0, sp->d_bucket_name, sp->d_bucket_lo,
                         sp->d_bucket_hi, sp->N, sp->d_lrank, sp->d_urank, sp->d_nh_begin, sp->d_nh_name,
                         sp->d_nh_count, sp->d_name_id, sp->d_nh_off, sp->d_nh_pos};
            SigView sv{G, tp->d_code, tp->d_rule, tp->d_mainchain, tp->d_name_begin, tp->d_names, tp->d_res_begin,
                       tp->d_resnames, tp->d_partner_begin, tp->d_partner_res, tp->d_partner_name};
            int32_t *cnt_c = d_count.p + (int64_t)s0 * G;
            int32_t *scn_c = d_scanned.p + (int64_t)s0 * G;
            CUDA_TRY(cudaEventRecord(ev[1], st));
            const int64_t n_pairs = (int64_t)Sc * T;
            bool free_chunk = free_first && n_pairs <= INT32_MAX - (1 << 20) && s0 != ordered_from;
            if (free_chunk && masks_whole) {
                fv.kind_masks = d_kind_masks.p + (int64_t)s0 * G * fv.mask_words;
            } else if (free_chunk) {
                const cudaError_t e = dalloc(d_kind_masks, (size_t)Wc * fv.mask_words, st);
                if (e == cudaErrorMemoryAllocation) {
                    cudaGetLastError();
                    free_chunk = false;
                } else {
                    CUDA_TRY(e);
                    fv.kind_masks = d_kind_masks.p;
                    launch_list_kinds(st, cv, sv, fv, cnt_c, scn_c, d_kind_masks.p);
                    launches++;
                }
            }
            int64_t leaf_filled = 0;  // leaf entries of the lists ordered so far
            const int fill_blocks = std::max(1, (int)std::min<int64_t>((Wc + 7) / 8, (int64_t)sm_count() * 32));
            TemplateView tv{T, tp->nmax, tp->d_atom_begin, tp->d_sig, tp->d_pos, tp->d_key, tp->d_param_begin,
                            d_params.p};
            CandView cd{G, cnt_c, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
            const int64_t *leaf_off = nullptr;
            // kd leaf order: up front for the lists of the first
            // `demand_levels` levels of every pair that can run, later (between
            // search rounds) for each deeper list a pair's frontier reaches;
            // a negative value orders every list of the chunk up front
            LeafDemand dm{};
            dm.n_suspended = d_nsusp.p;
            dm.n_work = d_nwork.p;
            dm.leaf_used = d_leaf_used.p;
            dm.n_fill = d_nfill.p;
            dm.pool_used = d_pool_used.p;
            const int leaf_blocks =
                std::max(1, (int)std::min<int64_t>((Wc + LEAF_WARPS - 1) / LEAF_WARPS, (int64_t)sm_count() * 32));
            // room in the leaf arrays for `need` entries (the lists ordered so
            // far keep their places)
            auto ensure_leaf = [&](int64_t need) -> cudaError_t {
                if (need <= (int64_t)d_leaf_atom.n) return cudaSuccess;
                const size_t cap2 = (size_t)std::max<int64_t>(need + need / 4, (int64_t)d_leaf_atom.n * 3 / 2);
                cudaError_t e = dalloc(d_leaf_atom2, cap2, st);
                if (e == cudaSuccess) e = dalloc(d_leaf_xyz2, cap2, st);
                if (e != cudaSuccess) return e;
                if (leaf_filled > 0) {
                    e = cudaMemcpyAsync(d_leaf_atom2.p, d_leaf_atom.p, (size_t)leaf_filled * sizeof(int32_t),
                                        cudaMemcpyDeviceToDevice, st);
                    if (e == cudaSuccess)
                        e = cudaMemcpyAsync(d_leaf_xyz2.p, d_leaf_xyz.p, (size_t)leaf_filled * sizeof(float4),
                                            cudaMemcpyDeviceToDevice, st);
                    if (e != cudaSuccess) return e;
                }
                std::swap(d_leaf_atom, d_leaf_atom2);
                std::swap(d_leaf_xyz, d_leaf_xyz2);
                dfree(d_leaf_atom2, st);
                dfree(d_leaf_xyz2, st);
                cd.leaf_atom = d_leaf_atom.p;
                cd.leaf_xyz = d_leaf_xyz.p;
                return cudaSuccess;
            };
            // lists of the same atoms share one leaf order (demand mode only:
            // there the leaf offsets are a separate, writable array)
            ListShare ls{};
            bool share_on = false;
            auto order_requested = [&](bool few = false) -> cudaError_t {
                if (dm.fill_state) {
                    // the requested lists not filled yet
                    launch_candidates(st, fill_blocks, true, cv, sv, nullptr, nullptr, d_offset.p, d_cand_atom.p,
                                      dm.work, dm.n_work, dm.fill_state, true);
                    launches++;
                }
                if (few) {
                    launch_leaf_order_few(st, cv, G, cnt_c, d_offset.p, d_boff.p, d_cand_atom.p, leaf_off,
                                          d_leaf_atom.p, d_leaf_xyz.p, d_blk_lo.p, d_blk_hi.p, d_sorted_list.p,
                                          d_sorted_count.p, d_exact_list.p, d_exact_count.p, d_counters.p, dm.work,
                                          dm.n_work);
                    launches += LEAF_FEW_LAUNCHES;
                } else if (share_on) {
                    // key every requested list, order one list per key, point
                    // the others at its leaves, order those whose atoms differ
                    const cudaError_t e0 = cudaMemsetAsync(ls.n, 0, 3 * sizeof(unsigned long long), st);
                    if (e0 != cudaSuccess) return e0;
                    launch_list_keys(st, sm_count() * 16, G, cnt_c, d_offset.p, d_cand_atom.p, dm.work, dm.n_work,
                                     ls, d_counters.p);
                    launch_list_reps(st, sm_count() * 16, dm.work, dm.n_work, ls);
                    launch_leaf_order(st, leaf_blocks, cv, G, cnt_c, d_offset.p, d_boff.p, d_cand_atom.p, leaf_off,
                                      d_leaf_atom.p, d_leaf_xyz.p, d_blk_lo.p, d_blk_hi.p, d_sorted_list.p,
                                      d_sorted_count.p, Wc, d_exact_list.p, d_exact_count.p, d_counters.p,
                                      ls.rep_work, ls.n, tune.leaf_rank_max, ls.part_ok, 0);
                    launch_list_share(st, sm_count() * 8, cv, G, cnt_c, d_offset.p, d_cand_atom.p, d_leaf_off.p,
                                      d_boff.p, ls, d_counters.p);
                    launch_leaf_order(st, leaf_blocks, cv, G, cnt_c, d_offset.p, d_boff.p, d_cand_atom.p, leaf_off,
                                      d_leaf_atom.p, d_leaf_xyz.p, d_blk_lo.p, d_blk_hi.p, d_sorted_list.p,
                                      d_sorted_count.p, Wc, d_exact_list.p, d_exact_count.p, d_counters.p,
                                      ls.left_work, ls.n + 2, tune.leaf_rank_max, ls.part_ok, 0);
                    launches += 2 * LEAF_ORDER_LAUNCHES + 3;
                } else {
                    launch_leaf_order(st, leaf_blocks, cv, G, cnt_c, d_offset.p, d_boff.p, d_cand_atom.p, leaf_off,
                                      d_leaf_atom.p, d_leaf_xyz.p, d_blk_lo.p, d_blk_hi.p, d_sorted_list.p,
                                      d_sorted_count.p, Wc, d_exact_list.p, d_exact_count.p, d_counters.p, dm.work,
                                      dm.n_work, tune.leaf_rank_max);
                    launches += LEAF_ORDER_LAUNCHES;
                }
                if (dm.state) {
                    launch_mark_ordered(st, sm_count() * 4, dm);
                    launches++;
                }
                return cudaGetLastError();
            };
            // the chunk's lists: offsets, culling blocks, room for their atoms
            // in candidate order and in leaf order, and the state of those
            // put in leaf order on demand.  The order-free search needs none
            // of it before a pair is split into items or rows are left to
            // the leaf order.
            bool lists_ready = false;
            auto setup_lists = [&]() -> cudaError_t {
                if (lists_ready) return cudaSuccess;
                lists_ready = true;
                cudaError_t e = cudaSuccess;
                auto room = [&](auto &buf, int64_t n) {
                    if (e == cudaSuccess) e = dalloc(buf, (size_t)std::max<int64_t>(n, 1), st);
                };
                auto fill = [&](void *p, int v, size_t bytes) {
                    if (e == cudaSuccess) e = cudaMemsetAsync(p, v, bytes, st);
                };
                room(d_offset, Wc);
                room(d_nblk, Wc);
                room(d_boff, Wc);
                if (e == cudaSuccess) e = scan_exclusive(cnt_c, Wc, d_offset.p, scan_tmp, st);
                if (e != cudaSuccess) return e;
                // culling blocks of CULL_BLK leaves: counts, offsets, total
                launch_block_counts(st, Wc, cnt_c, d_nblk.p);
                launches++;
                e = scan_exclusive(d_nblk.p, Wc, d_boff.p, scan_tmp, st);
                int64_t last[3] = {};  // offset and blocks of the last list, its block count and length
                int32_t lastn[2] = {};
                auto back = [&](void *to, const void *from, size_t bytes) {
                    if (e == cudaSuccess) e = cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToHost, st);
                };
                back(&last[0], d_offset.p + Wc - 1, 8);
                back(&last[1], d_boff.p + Wc - 1, 8);
                back(&lastn[0], cnt_c + Wc - 1, 4);
                back(&lastn[1], d_nblk.p + Wc - 1, 4);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                const int64_t all = last[0] + lastn[0], nblocks = last[1] + lastn[1];
                room(d_blk_lo, nblocks);
                room(d_blk_hi, nblocks);
                room(d_cand_atom, all);
                // leaf-order arrays: every entry when every list is ordered
                // up front, else half of them to start with (order-free
                // search: few; grown on demand; PJG_LEAF_CAPACITY sets the
                // starting size)
                int64_t cap0 = demand_levels < 0 ? all
                               : free_chunk      ? 1 << 18
                                                 : std::max<int64_t>(all / 2, 1 << 20);
                const char *v = getenv("PJG_LEAF_CAPACITY");
                if (demand_levels >= 0 && v && atoll(v) > 0) {
                    cap0 = atoll(v);
                    dfree(d_leaf_atom, st);
                    dfree(d_leaf_xyz, st);
                }
                room(d_leaf_atom, cap0);
                room(d_leaf_xyz, (int64_t)d_leaf_atom.n);
                room(d_exact_list, Wc);
                room(d_exact_count, 1);
                room(d_sorted_list, (int64_t)LEAF_LISTS * Wc);
                room(d_sorted_count, LEAF_LISTS);
                if (demand_levels >= 0) room(d_leaf_off, Wc);
                if (e != cudaSuccess) return e;
                leaf_off = demand_levels < 0 ? d_offset.p : d_leaf_off.p;
                cd = CandView{G, cnt_c, d_offset.p, d_cand_atom.p, leaf_off, d_leaf_atom.p, d_leaf_xyz.p,
                              d_boff.p, d_blk_lo.p, d_blk_hi.p};
                if (demand_levels < 0) {
                    // every list filled and put in leaf order up front
                    launch_candidates(st, fill_blocks, true, cv, sv, nullptr, nullptr, d_offset.p, d_cand_atom.p);
                    launches++;
                    return cudaGetLastError();
                }
                // otherwise only the lists a search reads are filled: the
                // level-0 list of each pair that needs it and each list put in
                // leaf order (just before it is)
                room(d_lstate, Wc);
                room(d_work, Wc);
                room(d_fill_state, Wc);
                room(d_fill_work, Wc);
                fill(d_lstate.p, 0, (size_t)Wc * sizeof(int32_t));
                fill(d_fill_state.p, 0, (size_t)Wc * sizeof(int32_t));
                if (e != cudaSuccess) return e;
                dm.state = d_lstate.p;
                dm.work = d_work.p;
                dm.leaf_offset = d_leaf_off.p;
                dm.fill_state = d_fill_state.p;
                dm.fill_work = d_fill_work.p;
                {
                    // the list-sharing table: twice the chunk's lists, a power
                    // of two (without the memory, every list is ordered)
                    int64_t cap = 1;
                    while (cap < 2 * Wc) cap <<= 1;
                    room(d_ls_key, cap);
                    room(d_ls_rep, cap);
                    room(d_ls_slot, Wc);
                    room(d_ls_rep_work, Wc);
                    room(d_ls_dup, Wc);
                    room(d_ls_left, Wc);
                    room(d_ls_n, 3);
                    room(d_ls_ok, Wc);
                    if (e == cudaSuccess) {
                        fill(d_ls_key.p, 0, (size_t)cap * sizeof(unsigned long long));
                        fill(d_ls_rep.p, 0xFF, (size_t)cap * sizeof(int32_t));
                        fill(d_ls_ok.p, 0, (size_t)Wc);
                    }
                    // PJG_LIST_SHARING=0 orders every list itself
                    const char *w = getenv("PJG_LIST_SHARING");
                    share_on = e == cudaSuccess && !(w && w[0] == '0');
                    if (e != cudaSuccess) {
                        cudaGetLastError();
                        dfree(d_ls_key, st);
                        dfree(d_ls_rep, st);
                        dfree(d_ls_slot, st);
                        dfree(d_ls_rep_work, st);
                        dfree(d_ls_dup, st);
                        dfree(d_ls_left, st);
                        dfree(d_ls_ok, st);
                    }
                    ls.key = d_ls_key.p;
                    ls.rep = d_ls_rep.p;
                    ls.mask = cap - 1;
                    ls.slot = d_ls_slot.p;
                    ls.rep_work = d_ls_rep_work.p;
                    ls.dup_work = d_ls_dup.p;
                    ls.left_work = d_ls_left.p;
                    ls.n = d_ls_n.p;
                    ls.part_ok = d_ls_ok.p;
                }
                return cudaSuccess;
            };
            if (n_pairs > INT32_MAX) {
                status = fail(PJG_ERR_CAPACITY, "too many pairs in one chunk");
                goto done;
            }
            // (lists requested in this chunk and the attempt's counters)
            CUDA_TRY(cudaMemsetAsync(d_leaf_used.p, 0, (ZC_LIVE - ZC_LEAF_USED) * sizeof(unsigned long long), st));
            if (!free_chunk || !tp->huge.empty()) CUDA_TRY(setup_lists());
            if (demand_levels < 0) {
                CUDA_TRY(order_requested());
            } else {
                CUDA_TRY(dalloc(d_susp_a, (size_t)n_pairs, st));
                if (!free_chunk) CUDA_TRY(dalloc(d_susp_b, (size_t)n_pairs, st));
                if (pool_cap == 0 && !free_chunk) {
                    // saved search states of suspended pairs, one pool per
                    // round in turn: a sixteenth of the free memory each,
                    // 64 MiB to 4 GiB (a pair that finds its pool full is
                    // rerun from its start instead; pairs the order-free
                    // search leaves are never suspended)
                    size_t free_b = 0, total_b = 0;
                    int64_t cap = 64ll << 20;
                    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess)
                        cap = std::max<int64_t>(cap, std::min<int64_t>(4ll << 30, (int64_t)(free_b / 16)));
                    const char *v = getenv("PJG_STATE_POOL");
                    if (v && atoll(v) >= 0) cap = atoll(v);
                    pool_cap = std::max<int64_t>(cap, 16);
                    CUDA_TRY(dalloc(d_pool_a, (size_t)pool_cap, st));
                    CUDA_TRY(dalloc(d_pool_b, (size_t)pool_cap, st));
                }
                dm.pool_cap = pool_cap;
                // the costliest pairs are searched first (a pair can take
                // milliseconds; started last, it alone would run on while the
                // other warps idle): the level demand estimates each pair's
                // cost, and the pairs of the top cost buckets, at most two
                // (PJG_HEAVY_PER_WARP) per resident search warp, are taken
                // before the others
                const char *hw = getenv("PJG_HEAVY_PER_WARP");
                const int64_t per_warp = hw && atoi(hw) > 0 ? atoi(hw) : 2;
                const int64_t heavy_target = per_warp * 2 * sm_count() * SEARCH_WARPS;
                const char *hf = getenv("PJG_HEAVY_FIRST");
                const bool heavy_on = !free_chunk && (int64_t)n_pairs >= 8 * heavy_target &&
                                      (int64_t)n_pairs <= (int64_t)INT32_MAX - heavy_target &&
                                      !(hf && atoi(hf) == 0);
                dm.pair_cost = nullptr;
                dm.heavy = nullptr;
                if (heavy_on) {
                    CUDA_TRY(dalloc(d_pcost, (size_t)n_pairs, st));
                    CUDA_TRY(dalloc(d_hflag, (size_t)n_pairs, st));
                    CUDA_TRY(dalloc(d_heavy, (size_t)heavy_target, st));
                    CUDA_TRY(dalloc(d_hbins, 66, st));
                    CUDA_TRY(cudaMemsetAsync(d_hbins.p, 0, 66 * sizeof(unsigned long long), st));
                    dm.pair_cost = d_pcost.p;
                }
                // (order-free first: only the lists of templates over 64 atoms)
                if (!free_chunk || !tp->huge.empty()) {
                    launch_demand_levels(st, sm_count() * 16, tv, cd, (int32_t)n_pairs,
                                         free_chunk ? -1 : demand_levels, P->reorder, free_chunk ? 64 : 32, dm);
                    if (heavy_on) {
                        launch_heavy_pairs(st, (int32_t)n_pairs, d_pcost.p, d_hbins.p, heavy_target, d_hflag.p,
                                           d_heavy.p);
                        dm.heavy = d_heavy.p;
                        dm.n_heavy = d_hbins.p + 64;
                        dm.heavy_flag = d_hflag.p;
                        launches += 2;
                    }
                    // the level-0 lists the pairs read in candidate order
                    launch_candidates(st, fill_blocks, true, cv, sv, nullptr, nullptr, d_offset.p, d_cand_atom.p,
                                      dm.fill_work, dm.n_fill, nullptr, false);
                    launches += 2;
                    unsigned long long used = 0;
                    CUDA_TRY(cudaMemcpyAsync(&used, d_leaf_used.p, sizeof used, cudaMemcpyDeviceToHost, st));
                    CUDA_TRY(cudaStreamSynchronize(st));
                    CUDA_TRY(ensure_leaf((int64_t)used));
                    CUDA_TRY(order_requested());
                    leaf_filled = (int64_t)used;
                }
            }
            CUDA_TRY(cudaEventRecord(ev[2], st));
            SearchArgs sa;
            sa.n_pairs = Sc * T;
            sa.ignore_chain = P->ignore_chain;
            sa.reorder = P->reorder;
            sa.best_match = P->best_match;
            sa.max_candidates = P->max_candidates;
            {
                // shared memory per warp: pair state + tiles of >= 64
                // entries for every level but the last (k_search takes
                // templates of up to 32 atoms)
                int levels = std::max(1, std::min(tp->nmax, 32) - 1);
                size_t entry = sp->max_atoms > 65535 ? 8 : 4;
                size_t need = search_state_bytes() + entry * 64 * (size_t)levels;
                sa.warp_smem = (int)((std::max<size_t>(need, search_state_bytes() + 5376) + 15) & ~size_t(15));
            }
            sa.cut_inline = cut_inline ? 1 : 0;
            sa.rmsd_threshold = P->rmsd_threshold;
            sa.prof = nullptr;
            sa.block_min = tune.block_min;
            sa.tile_cap = tune.tile_cap;
            sa.pair_grain = tune.pair_grain;
            sa.leaf_reach = tune.leaf_reach;
#if PJG_SEARCH_PROF
            if (!d_prof.p) {
                CUDA_TRY(dalloc(d_prof, SP_NUM, st));
                CUDA_TRY(cudaMemsetAsync(d_prof.p, 0, SP_NUM * sizeof(unsigned long long), st));
            }
            sa.prof = d_prof.p;
#endif
            {
                const char *b = getenv("PJG_KERNEL_BUDGET_S");
                double sec = b ? atof(b) : 120.0;
                if (!(sec > 0)) sec = 120.0;
                sa.budget_ns = (uint64_t)(sec * 1e9);
            }
            bool wide = sp->max_atoms > 65535;
            // counters before this chunk's search, restored if it must rerun
            CUDA_TRY(cudaMemcpyAsync(d_z.p + ZC_SNAP, d_counters.p, stats_bytes, cudaMemcpyDeviceToDevice, st));
            CUDA_TRY(dalloc(d_pair_rows, (size_t)n_pairs, st));
            // room before the first attempt (a rerun of the search costs a
            // whole chunk): two complete rows a pair, or, with best_match
            // and max_candidates, the most a pair can produce (max_candidates
            // + 2) when the row budget takes that
            int64_t want_rows = 2 * n_pairs;
            if (P->best_match && P->max_candidates >= 0) {
                const int64_t bound = n_pairs * ((int64_t)P->max_candidates + 2);
                const int64_t budget = row_budget();
                if (bound <= budget) {
                    // (the items of a pair in flight when its first
                    // max_candidates + 2 rows are there add to them)
                    want_rows = std::max(want_rows, free_chunk ? std::min(budget, 2 * bound) : bound);
                } else if (Sc > 1) {
                    // with the chunk's own lists in memory its bound no
                    // longer fits: take fewer structures before searching
                    chunk_cap = std::max(1, (int)((double)Sc * (double)budget / (double)bound));
                    bound_cap = std::min(bound_cap, chunk_cap);
                    chunks--;
                    row_splits++;
                    CUDA_TRY(cudaMemcpyAsync(d_counters.p, d_z.p + ZC_CHUNK, stats_bytes, cudaMemcpyDeviceToDevice,
                                             st));
                    continue;
                }
            }
            if (c_cap < want_rows) {
                c_cap = want_rows;
                CUDA_TRY(dalloc(d_c_pair, c_cap, st));
                CUDA_TRY(dalloc(d_c_ord, c_cap, st));
                CUDA_TRY(dalloc(d_c_atoms, (size_t)c_cap * stride, st));
                if (cut_inline) CUDA_TRY(dalloc(d_c_rmsd, c_cap, st));
            }
            // set when the chunk's complete rows cannot be held: the chunk is
            // redone on half its structures
            bool split = false;
            bool invalid_rows = false;  // rows without a place: of pairs k_search took over, past a cut
            // set when the order-free search's own buffers cannot be held: the
            // chunk is redone on fewer structures (free_fit of them), a single
            // structure in order
            bool free_full = false;
            double free_fit = 0.5;
            auto no_room = [&](cudaError_t e) -> bool {
                if (e != cudaErrorMemoryAllocation) return false;
                cudaGetLastError();
                return free_full = true;
            };
            for (int attempt = 0; attempt < 8; attempt++) {
                if (attempt > 0)
                    CUDA_TRY(cudaMemsetAsync(d_z.p + ZC_ATTEMPT, 0,
                                             (ZC_LIVE - ZC_ATTEMPT) * sizeof(unsigned long long), st));
                CUDA_TRY(cudaMemsetAsync(d_pair_rows.p, 0, (size_t)n_pairs * sizeof(int32_t), st));
                CompleteRows cr{d_ccount.p, c_cap, stride, d_c_pair.p, d_c_ord.p, d_c_atoms.p,
                                cut_inline ? d_c_rmsd.p : nullptr, d_pair_rows.p};
                int grid = sm_count() * 8;
                unsigned long long nc = 0;
                // search rounds: every pair, then the pairs suspended at a
                // list that had no leaf order (ordered in between), until
                // no pair is suspended
                dm.resume = nullptr;
                dm.n_resume = 0;
                dm.pool_in = nullptr;
                // units, heavy pairs, their items, (scratch, large units,) spilled entries,
                // units left to the leaf order, long units, items to search in order
                unsigned long long free_n[9] = {};
                FreeWork fw{};
                Suspended *next_out = d_susp_a.p, *spare = d_susp_b.p;
                unsigned char *pool_next = d_pool_a.p, *pool_spare = d_pool_b.p;
                for (int round = 0;; round++) {
                    dm.suspended = next_out;
                    dm.pool_out = pool_next;
                    // requested lists, suspended pairs, pool and work queue
                    // (the first order-free round: zeroed with the attempt)
                    if (round > 0 || !free_chunk || !tp->huge.empty())
                        CUDA_TRY(cudaMemsetAsync(d_nwork.p, 0, (ZC_TOTALS - ZC_NWORK) * sizeof(unsigned long long),
                                                 st));
                    CUDA_TRY(cudaEventRecord(ev[6], st));
                    if (round == 0 && free_chunk) {
                        cudaError_t er = dalloc(d_units, (size_t)c_cap, st);
                        if (er == cudaSuccess) er = dalloc(d_heavy_pairs, (size_t)n_pairs, st);
                        if (no_room(er)) break;
                        CUDA_TRY(er);
                        fw.item_seeds = P->max_candidates >= 0        ? FREE_ITEM_CUT
                                        : n_pairs <= FREE_FEW_PAIRS ? FREE_ITEM_FEW
                                                                    : FREE_ITEM;
                        fw.scratch_used = d_free_n.p + 3;
                        fw.n_large_units = d_free_n.p + 4;
                        fw.n_spilled = d_free_n.p + 5;
                        fw.n_pending = d_free_n.p + 6;
                        fw.n_long_units = d_free_n.p + 7;
                        fw.n_failed = d_free_n.p + 8;
                        fw.units = d_units.p;
                        fw.n_units = d_free_n.p;
                        fw.heavy = d_heavy_pairs.p;
                        fw.n_heavy = d_free_n.p + 1;
                        CUDA_TRY(launch_search_free(st, fp32, cv, tv, cd, fv, sa, d_pair_counter.p, scn_c, cr,
                                                    d_counters.p, dm, fw));
                        if (!tp->wide.empty()) {
                            FreeWork ww = fw;
                            ww.wide = tp->d_wide;
                            ww.n_wide = (int32_t)tp->wide.size();
                            CUDA_TRY(cudaMemsetAsync(d_pair_counter.p, 0, sizeof(int32_t), st));
                            CUDA_TRY(launch_search_free(st, fp32, cv, tv, cd, fv, sa, d_pair_counter.p, scn_c, cr,
                                                        d_counters.p, dm, ww));
                            launches++;
                        }
                    } else {
                        CUDA_TRY(launch_search(st, grid, wide, fp32, cv, tv, cd, sa, d_pair_counter.p, scn_c, cr,
                                               d_counters.p, dm));
                    }
                    launches++;
                    // pairs of templates over 32 atoms (over 64: the others
                    // are searched without order), every list of theirs
                    // ordered before this round; later, those left to it
                    const bool left = free_chunk && round > 0;
                    const auto &big = free_chunk && !left ? tp->huge : tp->large;
                    if ((round == 0 || left) && !big.empty()) {
                        CUDA_TRY(cudaMemsetAsync(d_pair_counter.p, 0, sizeof(int32_t), st));
                        CUDA_TRY(launch_search_large(st, cv, tv, cd, sa, free_chunk && !left ? tp->d_huge : tp->d_large,
                                                     (int32_t)big.size(), d_pair_counter.p, scn_c, cr, d_counters.p,
                                                     dm.state, left ? dm.resume : nullptr, left ? dm.n_resume : 0));
                        launches++;
                    }
                    CUDA_TRY(cudaEventRecord(ev[7], st));
                    CUDA_TRY(cudaGetLastError());
                    unsigned long long ns = 0, used = 0;
                    auto read_back = [&]() -> cudaError_t {
                        cudaError_t e = cudaMemcpyAsync(hz, d_z.p, ZC_LIVE * sizeof(unsigned long long),
                                                        cudaMemcpyDeviceToHost, st);
                        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                        nc = hz[ZC_ROWS];
                        ns = dm.state || free_chunk ? hz[ZC_NSUSP] : 0;
                        used = hz[ZC_LEAF_USED];
                        if (round == 0)
                            for (int i = 0; i < 9; i++) free_n[i] = hz[ZC_FREE + i];
                        float m = 0.f;
                        if (e == cudaSuccess) e = cudaEventElapsedTime(&m, ev[6], ev[7]);
                        ms_search += m;
                        return e;
                    };
                    CUDA_TRY(read_back());
                    search_rounds++;
                    if (round == 0 && free_chunk && (free_n[1] || ns)) {
                        // level-0 lists, in candidate order, of the pairs taken
                        // in items and of those left to k_search, whose other
                        // lists are to be put in leaf order
                        CUDA_TRY(setup_lists());
                        launch_free_requests(st, tv, cd, P->reorder, dm, d_heavy_pairs.p, (int32_t)free_n[1],
                                             dm.suspended, 0, (int32_t)ns);
                        launches++;
                        launch_candidates(st, fill_blocks, true, cv, sv, nullptr, nullptr, d_offset.p, d_cand_atom.p,
                                          dm.fill_work, dm.n_fill, nullptr, false);
                        launches++;
                    }
                    if (round == 0 && free_chunk && free_n[1]) {
                        // the heavy pairs in items of seeds, block 0
                        // of every pair first
                        const int32_t nh = (int32_t)free_n[1];
                        const int64_t ns1 = (int64_t)ns;
                        const int64_t ni = (int64_t)free_n[2];
                        const int64_t nbins = (sp->max_atoms + fw.item_seeds - 1) / fw.item_seeds;
                        const int64_t most_items = item_budget(ni);
                        if (ni > most_items) {
                            free_full = true;
                            free_fit = 0.9 * (double)most_items / (double)ni;
                            break;
                        }
                        int64_t warps = 0;
                        cudaError_t er = heavy_warps(fp32, ni, &warps);
                        auto room = [&](auto &buf, int64_t n) {
                            if (er == cudaSuccess) er = dalloc(buf, (size_t)n, st);
                        };
                        room(d_bins, 2 * nbins);
                        room(d_bin_off, nbins);
                        room(d_items, ni);
                        room(d_results, ni);
                        room(d_item_base, ni);
                        room(d_item_head, ni);
                        room(d_item_branch, ni);
                        room(d_spill_a, SPILL_CAP);
                        room(d_item_stats, 4 * ni);
                        room(d_arena_xyz, warps * HEAVY_CAP);
                        room(d_arena_atom, warps * HEAVY_CAP);
                        room(d_arena_parent, 2 * warps * HEAVY_CAP);
                        if (no_room(er)) break;
                        CUDA_TRY(er);
                        CUDA_TRY(cudaMemsetAsync(d_bins.p, 0, 2 * (size_t)nbins * sizeof(int32_t), st));
                        CUDA_TRY(cudaMemsetAsync(d_results.p, 0xFF, (size_t)ni * sizeof(int2), st));
                        CUDA_TRY(cudaMemsetAsync(d_item_head.p, 0xFF, (size_t)ni * sizeof(int32_t), st));
                        CUDA_TRY(cudaMemsetAsync(d_item_branch.p, 0, (size_t)ni * sizeof(unsigned long long), st));
                        CUDA_TRY(cudaMemsetAsync(d_item_stats.p, 0, 4 * (size_t)ni * sizeof(unsigned long long), st));
                        CUDA_TRY(cudaMemsetAsync(d_pair_counter.p, 0, sizeof(int32_t), st));
                        launch_heavy_bins(st, nh, d_heavy_pairs.p, d_bins.p);
                        CUDA_TRY(scan_exclusive(d_bins.p, nbins, d_bin_off.p, scan_tmp, st));
                        launch_heavy_items(st, nh, d_heavy_pairs.p, d_bin_off.p, d_bins.p + nbins, d_items.p);
                        fw.items = d_items.p;
                        fw.n_items = (int32_t)ni;
                        fw.results = d_results.p;
                        fw.item_stats = d_item_stats.p;
                        fw.item_base = d_item_base.p;
                        fw.arena_xyz = d_arena_xyz.p;
                        fw.arena_atom = d_arena_atom.p;
                        fw.arena_parent = d_arena_parent.p;
                        fw.item_head = d_item_head.p;
                        fw.item_branch = d_item_branch.p;
                        fw.spilled_out = d_spill_a.p;
                        fw.spill_cap = SPILL_CAP;
                        // every item, and again for those of wide templates
                        auto search_items = [&](int64_t w) -> cudaError_t {
                            cudaError_t e = launch_search_heavy(st, fp32, w, cv, tv, cd, fv, sa, d_pair_counter.p, cr,
                                                                d_counters.p, dm, fw);
                            if (e != cudaSuccess || tp->wide.empty()) return e;
                            FreeWork ww = fw;
                            ww.wide = tp->d_wide;
                            ww.n_wide = (int32_t)tp->wide.size();
                            e = cudaMemsetAsync(d_pair_counter.p, 0, sizeof(int32_t), st);
                            if (e != cudaSuccess) return e;
                            launches++;
                            return launch_search_heavy(st, fp32, w, cv, tv, cd, fv, sa, d_pair_counter.p, cr,
                                                       d_counters.p, dm, ww);
                        };
                        CUDA_TRY(cudaEventRecord(ev[6], st));
                        CUDA_TRY(search_items(warps));
                        CUDA_TRY(cudaEventRecord(ev[7], st));
                        launches += 3;
                        CUDA_TRY(cudaGetLastError());
                        CUDA_TRY(read_back());
                        // entries whose children outgrew the frontier, level
                        // by level at most as deep as a template
                        for (int pass = 0; free_n[5] > 0 && hz[C_ERROR] == 0; pass++) {
                            if (pass > std::min(tp->nmax, 64)) {
                                status = fail(PJG_ERR_CAPACITY, "spilled entries did not converge");
                                goto done;
                            }
                            fw.n_items = (int32_t)free_n[5];
                            if (pass > 0) std::swap(d_spill_a, d_spill_b);
                            CUDA_TRY(heavy_warps(fp32, fw.n_items, &warps));
                            room(d_spill_b, SPILL_CAP);
                            room(d_arena_xyz, warps * HEAVY_CAP);
                            room(d_arena_atom, warps * HEAVY_CAP);
                            room(d_arena_parent, 2 * warps * HEAVY_CAP);
                            if (no_room(er)) break;
                            CUDA_TRY(er);
                            fw.spilled_in = d_spill_a.p;
                            fw.spilled_out = d_spill_b.p;
                            CUDA_TRY(cudaMemsetAsync(fw.n_spilled, 0, sizeof(unsigned long long), st));
                            CUDA_TRY(cudaMemsetAsync(d_pair_counter.p, 0, sizeof(int32_t), st));
                            fw.arena_xyz = d_arena_xyz.p;
                            fw.arena_atom = d_arena_atom.p;
                            fw.arena_parent = d_arena_parent.p;
                            CUDA_TRY(cudaEventRecord(ev[6], st));
                            CUDA_TRY(search_items(warps));
                            CUDA_TRY(cudaEventRecord(ev[7], st));
                            launches++;
                            CUDA_TRY(cudaGetLastError());
                            CUDA_TRY(read_back());
                        }
                        if (free_full) break;
                        launch_heavy_rows(st, nh, fw, sa, d_item_base.p, d_pair_rows.p, dm, d_counters.p);
                        launches++;
                        CUDA_TRY(cudaGetLastError());
                        // (rows of items past the cut, and of pairs that go to
                        // k_search, have no place)
                        invalid_rows = invalid_rows || P->max_candidates >= 0 || free_n[8];
                        if (free_n[8]) {
                            const double ms0 = ms_search;
                            CUDA_TRY(read_back());
                            ms_search = ms0;
                        }
                        if ((int64_t)ns > ns1) {
                            // pairs that an item left to k_search (their level-0
                            // lists are filled)
                            launch_free_requests(st, tv, cd, P->reorder, dm, nullptr, 0, dm.suspended, (int32_t)ns1,
                                                 (int32_t)ns);
                            launches++;
                            CUDA_TRY(cudaGetLastError());
                        }
                    }
                    if (round == 0 && free_chunk && free_n[0] && (int64_t)nc <= c_cap) {
                        // the rows found without order, in the reference's;
                        // units it leaves wait for their lists' leaf order
                        const cudaError_t er = dalloc(d_pending, 2 * (size_t)free_n[0], st);
                        if (no_room(er)) break;
                        CUDA_TRY(er);
                        fw.pending = d_pending.p;
                        fw.long_units = d_pending.p + free_n[0];
                        CUDA_TRY(launch_unit_order_direct(st, (int64_t)free_n[0], cv, tv, cd, sv, fv, sp->d_res_place,
                                                          P->reorder, fw, cr));
                        launches += 2;
                        const double ms0 = ms_search;
                        CUDA_TRY(read_back());
                        if (free_n[6]) {
                            CUDA_TRY(setup_lists());
                            launch_pending_requests(st, (int64_t)free_n[6], tv, cd, P->reorder, dm, fw);
                            launches++;
                        }
                        if (free_n[6] || ns) CUDA_TRY(read_back());
                        ms_search = ms0;
                    } else if (round == 0 && free_chunk && ns) {
                        const double ms0 = ms_search;
                        CUDA_TRY(read_back());
                        ms_search = ms0;
                    }
                    if (ns == 0 && (!free_chunk || (int64_t)used <= leaf_filled)) break;
                    if (round > 80) {
                        status = fail(PJG_ERR_CAPACITY, "leaf order on demand did not converge");
                        goto done;
                    }
                    suspensions += (int64_t)ns;
                    // the lists the suspended pairs reached, then those pairs
                    CUDA_TRY(ensure_leaf((int64_t)used));
                    CUDA_TRY(order_requested(free_chunk && (int64_t)used - leaf_filled <= LEAF_FEW_ENTRIES));
                    leaf_filled = (int64_t)used;
                    if (ns == 0) break;
                    dm.resume = next_out;
                    dm.n_resume = (int32_t)ns;
                    dm.pool_in = pool_next;
                    if (round == 0 && free_chunk) {
                        CUDA_TRY(dalloc(d_susp_b, (size_t)n_pairs, st));
                        spare = d_susp_b.p;
                    }
                    std::swap(next_out, spare);
                    std::swap(pool_next, pool_spare);
                }
                if (free_full) break;
                if ((int64_t)nc <= c_cap) {
                    if (free_chunk && free_n[6]) {
                        cudaError_t er = dalloc(d_row_key, (size_t)nc, st);
                        if (er == cudaSuccess) er = dalloc(d_row_scratch, 5 * (size_t)nc, st);
                        if (er == cudaSuccess) er = dalloc(d_large_units, (size_t)free_n[6], st);
                        if (no_room(er)) break;
                        CUDA_TRY(er);
                        fw.row_key = d_row_key.p;
                        fw.row_scratch = d_row_scratch.p;
                        fw.large_units = d_large_units.p;
                        launch_unit_order(st, (int64_t)free_n[6], cv, tv, cd, sv, sp->d_res_place, P->reorder,
                                          sa.budget_ns, d_counters.p, fw, cr);
                        launches++;
                        CUDA_TRY(cudaGetLastError());
                    }
                    break;
                }
                // the row buffer was too small: grow and run the chunk again
                // (the search counters of the failed attempt are rolled back;
                // lists ordered meanwhile stay ordered).  Rows beyond the
                // chunk's row budget, or a growth that fails, split the chunk
                // instead (down to one structure).
                if (Sc > 1 && (int64_t)nc > row_budget()) {
                    split = true;
                    break;
                }
                c_cap = (int64_t)nc + nc / 4 + 1024;
                {
                    cudaError_t eg = dalloc(d_c_pair, c_cap, st);
                    if (eg == cudaSuccess) eg = dalloc(d_c_ord, c_cap, st);
                    if (eg == cudaSuccess) eg = dalloc(d_c_atoms, (size_t)c_cap * stride, st);
                    if (eg == cudaSuccess && cut_inline) eg = dalloc(d_c_rmsd, c_cap, st);
                    if (eg == cudaErrorMemoryAllocation && Sc > 1) {
                        cudaGetLastError();
                        c_cap = std::min<int64_t>({(int64_t)d_c_pair.n, (int64_t)d_c_ord.n,
                                                   (int64_t)(d_c_atoms.n / stride)});
                        if (cut_inline) c_cap = std::min<int64_t>(c_cap, (int64_t)d_c_rmsd.n);
                        split = true;
                        break;
                    }
                    CUDA_TRY(eg);
                }
                {
                    // (the leaf order's statistics and an error stay)
                    unsigned long long cur[C_NUM], snap[C_NUM];
                    CUDA_TRY(cudaMemcpyAsync(cur, d_counters.p, sizeof cur, cudaMemcpyDeviceToHost, st));
                    CUDA_TRY(cudaMemcpyAsync(snap, d_z.p + ZC_SNAP, sizeof snap, cudaMemcpyDeviceToHost, st));
                    CUDA_TRY(cudaStreamSynchronize(st));
                    for (int c : {C_LEAF_EXACT, C_LEAF_SORTED, C_LEAF_REPLAY, C_LEAF_LISTS, C_LEAF_ENTRIES, C_LEAF_SHARED, C_ERROR})
                        snap[c] = cur[c];
                    CUDA_TRY(cudaMemcpyAsync(d_counters.p, snap, sizeof snap, cudaMemcpyHostToDevice, st));
                    CUDA_TRY(cudaStreamSynchronize(st));
                }
            }
            if (free_full) {
                if (Sc > 1) free_cap = std::max(1, std::min(Sc / 2, (int)(free_fit * Sc)));
                else ordered_from = s0;
                chunks--;
                row_splits++;
                search_rounds = search_rounds0;
                suspensions = suspensions0;
                ms_search = ms_search_chunk0;
                CUDA_TRY(cudaMemcpyAsync(d_counters.p, d_z.p + ZC_CHUNK, stats_bytes, cudaMemcpyDeviceToDevice, st));
                continue;
            }
            CUDA_TRY(cudaEventRecord(ev[3], st));
            {
                // superposition of every complete row into its slot in
                // reference order, Query.__next__ per pair, compaction of
                // the hits and warnings into this chunk's segment
                const int64_t rows = (int64_t)hz[ZC_ROWS];  // (as read back last)
                // the per-row stages below hold ~360 + 4 * stride bytes a
                // complete row: when the chunk's rows need more than 70% of
                // the memory they may use, or the row buffers could not hold
                // them, the chunk is redone on half its structures
                const bool many_rows = split || rows > (1 << 20) || getenv("PJG_ROW_BUDGET");
                const int64_t budget_now = many_rows ? row_budget() : INT64_MAX;
                if (Sc > 1 && (split || rows > budget_now)) {
                    // at most half the structures, fewer when the rows seen
                    // say so (rows scale with the structures of a chunk)
                    const double fit = 0.8 * (double)Sc * (double)budget_now / (double)std::max<int64_t>(rows, 1);
                    chunk_cap = std::max(1, std::min(Sc / 2, (int)fit));
                    chunks--;
                    row_splits++;
                    search_rounds = search_rounds0;
                    suspensions = suspensions0;
                    ms_search = ms_search_chunk0;
                    CUDA_TRY(cudaMemcpyAsync(d_counters.p, d_z.p + ZC_CHUNK, stats_bytes, cudaMemcpyDeviceToDevice,
                                             st));
                    continue;
                }
                CompleteRows cr{d_ccount.p, c_cap, stride, d_c_pair.p, d_c_ord.p, d_c_atoms.p,
                                cut_inline ? d_c_rmsd.p : nullptr, d_pair_rows.p};
                if (rows > 0) {
                    CUDA_TRY(dalloc(d_cnt_q, (size_t)n_pairs, st));
                    CUDA_TRY(dalloc(d_off_q, (size_t)n_pairs, st));
                    launch_order_counts(st, n_pairs, T, d_pair_rows.p, d_cnt_q.p);
                    CUDA_TRY(scan_exclusive(d_cnt_q.p, n_pairs, d_off_q.p, scan_tmp, st));
                    CUDA_TRY(dalloc(d_r_rmsd, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_rot, (size_t)rows * 9, st));
                    CUDA_TRY(dalloc(d_r_cen, (size_t)rows * 6, st));
                    CUDA_TRY(dalloc(d_r_nan, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_src, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_hit, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_warn, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_hatoms, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_hidx, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_widx, (size_t)rows, st));
                    CUDA_TRY(dalloc(d_r_aidx, (size_t)rows, st));
                    RowResults rr{d_off_q.p, T, d_r_rmsd.p, d_r_nan.p, d_r_rot.p, d_r_cen.p, d_r_src.p};
                    int blocks = (int)std::min<int64_t>((rows + 127) / 128, (int64_t)sm_count() * 24);
                    launch_superpose(st, blocks, cv, tv, cr, rr);
                    CUDA_TRY(dalloc(d_long_pairs, (size_t)std::min<int64_t>(n_pairs, rows), st));
                    if (invalid_rows) {
                        // (rows of a pair that k_search took over, or past a cut, have no slot)
                        CUDA_TRY(cudaMemsetAsync(d_r_hit.p, 0, (size_t)rows * sizeof(int32_t), st));
                        CUDA_TRY(cudaMemsetAsync(d_r_warn.p, 0, (size_t)rows * sizeof(int32_t), st));
                        CUDA_TRY(cudaMemsetAsync(d_r_hatoms.p, 0, (size_t)rows * sizeof(int32_t), st));
                    }
                    launch_automaton(st, n_pairs, T, tp->d_atom_begin, d_cnt_q.p, d_off_q.p, rr, P->max_candidates,
                                     P->best_match, P->rmsd_threshold, d_r_hit.p, d_r_warn.p, d_r_hatoms.p,
                                     d_rtotals.p, d_long_pairs.p, d_rtotals.p + 4);
                    CUDA_TRY(scan_exclusive(d_r_hit.p, rows, d_r_hidx.p, scan_tmp, st));
                    CUDA_TRY(scan_exclusive(d_r_warn.p, rows, d_r_widx.p, scan_tmp, st));
                    CUDA_TRY(scan_exclusive(d_r_hatoms.p, rows, d_r_aidx.p, scan_tmp, st));
                    CUDA_TRY(cudaMemcpyAsync(hz, d_z.p, ZC_LIVE * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                             st));
                    CUDA_TRY(cudaStreamSynchronize(st));
                    const unsigned long long *tot = hz + ZC_TOTALS;
                    passing += (int64_t)tot[3];
                    if (P->count_only) {
                        // counts only: the hits and warnings are not kept
                        res->store.hits += (int64_t)tot[0];
                        res->store.atoms += (int64_t)tot[2];
                        res->store.warns += (int64_t)tot[1];
                    } else if (tot[0] + tot[1] > 0) {
                        HitStore &hs = res->store;
                        CUDA_TRY(hs.reserve((int64_t)tot[0], (int64_t)tot[2], (int64_t)tot[1], st));
                        launch_gather_hits(st, rows, T, s0, hs.atoms, tp->d_atom_begin, cr, rr, d_r_hit.p,
                                           d_r_warn.p, d_r_hidx.p, d_r_widx.p, d_r_aidx.p, P->best_match, hs.tail());
                        CUDA_TRY(cudaGetLastError());
                        hs.hits += (int64_t)tot[0];
                        hs.atoms += (int64_t)tot[2];
                        hs.warns += (int64_t)tot[1];
                    }
                    launches += 9;
                }
                CUDA_TRY(cudaEventRecord(ev[4], st));
                float m1 = 0, m2 = 0, m3 = 0;
                if (s1 == S) {
                    // (the last chunk: with the query's end)
                    CUDA_TRY(cudaMemcpyAsync(hz, d_z.p, ZC_LIVE * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                             st));
                    CUDA_TRY(cudaEventRecord(ev[5], st));
                    CUDA_TRY(cudaStreamSynchronize(st));
                } else {
                    CUDA_TRY(cudaEventSynchronize(ev[4]));
                }
                cudaEventElapsedTime(&m1, ev[1], ev[2]);
                cudaEventElapsedTime(&m2, ev[2], ev[3]);
                cudaEventElapsedTime(&m3, ev[3], ev[4]);
                // search launches count as expansion; the leaf order run
                // between search rounds counts with the candidate lists
                ms_cand += m1 + (m2 - (float)(ms_search - ms_search_chunk0));
                ms_exp += ms_search - ms_search_chunk0;
                ms_sup += m3;
                // next chunk: as many structures as the row budget takes at
                // this chunk's rows per structure (a dense chunk early in the
                // set does not keep every later chunk small)
                if (s1 == S) {
                } else if (rows > 0 && max_chunk > 1) {
                    const double per = (double)rows / (double)Sc;
                    const double fit = 0.8 * (double)row_budget() / per;
                    chunk_cap = (int)std::max(1.0, std::min((double)max_chunk, fit));
                } else {
                    chunk_cap = max_chunk;
                }
                chunk_cap = std::max(chunk_cap, std::min(bound_cap, max_chunk));
                free_cap = free_cap < mask_cap / 2 ? 2 * free_cap : mask_cap;
            }
            s0 = s1;
        }
    }
    std::memcpy(counters, hz, sizeof counters);
    cudaEventElapsedTime(&ms, ev[0], ev[5]);
    ms_total = ms;
    if (counters[C_ERROR] == 3) {
        status = fail(PJG_ERR_TIMEOUT, "search kernel exceeded its time budget (PJG_KERNEL_BUDGET_S)");
        goto done;
    }
    if (counters[C_ERROR]) {
        const unsigned long long c = counters[C_ERROR];
        status = fail(PJG_ERR_CAPACITY, "kernel reported error %llu (%s)", c,
                      c == 2 ? "template too large for the frontier tile"
                      : c == 4 ? "leaf order: too many small subtrees" : c == 5 ? "leaf order: partition did not converge"
                      : c == 7 ? "a list of a template over 32 atoms had no kd leaf order"
                      : "leaf order: inconsistent node partition");
        goto done;
    }

    res->stats.pairs = (int64_t)counters[C_PAIRS];
    res->stats.candidate_entries = (int64_t)counters[C_CAND];
    res->stats.partials = (int64_t)counters[C_PARTIALS];
    res->stats.complete = (int64_t)counters[C_COMPLETE];
    res->stats.passing = passing;
    res->stats.hits = res->store.hits;
    res->stats.fp64_rechecks = (int64_t)counters[C_RECHECK];
    res->stats.leaf_exact = (int64_t)counters[C_LEAF_EXACT];
    res->stats.leaf_sorted = (int64_t)counters[C_LEAF_SORTED];
    res->stats.leaf_replays = (int64_t)counters[C_LEAF_REPLAY];
    res->stats.bytes_candidates = (int64_t)counters[C_BYTES_CAND];
    res->stats.bytes_expansion = (int64_t)counters[C_BYTES_EXP];
    // per hit: its atoms, rmsd, rotation and centroids
    res->stats.bytes_superposition = 4 * res->store.atoms + (8 + 72 + 48) * res->store.hits;
    res->stats.ms_candidates = ms_cand;
    res->stats.ms_expansion = ms_exp;
    res->stats.ms_superposition = ms_sup;
    res->stats.ms_total = ms_total;
    res->stats.launches = launches + t_scan_launches;
    res->stats.chunks = chunks;
    res->stats.leaf_lists = (int64_t)counters[C_LEAF_LISTS];
    res->stats.leaf_entries = (int64_t)counters[C_LEAF_ENTRIES];
    res->stats.suspensions = suspensions;
    res->stats.search_rounds = search_rounds;
    res->stats.row_splits = row_splits;
    res->stats.leaf_shared = (int64_t)counters[C_LEAF_SHARED];
#if PJG_SEARCH_PROF
    if (d_prof.p) write_search_profile(d_prof.p, st, res->stats);
#endif

done:
    if (st) {
        dfree(d_sig_bits, st); dfree(d_kind_masks, st); dfree(d_units, st); dfree(d_heavy_pairs, st);
        dfree(d_item_stats, st); dfree(d_row_key, st); dfree(d_items, st); dfree(d_results, st);
        dfree(d_item_base, st); dfree(d_bin_off, st); dfree(d_bins, st); dfree(d_arena_atom, st);
        dfree(d_row_scratch, st); dfree(d_arena_xyz, st); dfree(d_arena_parent, st); dfree(d_item_head, st);
        dfree(d_large_units, st); dfree(d_long_pairs, st); dfree(d_pending, st); dfree(d_item_branch, st); dfree(d_spill_a, st);
        dfree(d_spill_b, st);
        dfree(d_params, st); dfree(d_count, st); dfree(d_scanned, st); dfree(d_cand_atom, st);
        dfree(d_leaf_atom, st); dfree(d_offset, st); dfree(d_totals, st);
        dfree(d_leaf_xyz, st); dfree(d_leaf_atom2, st); dfree(d_leaf_xyz2, st); dfree(d_leaf_off, st);
       
        dfree(d_c_pair, st); dfree(d_c_atoms, st); dfree(d_pair_rows, st);
        dfree(d_cnt_q, st); dfree(d_c_ord, st); dfree(d_off_q, st); dfree(d_c_rmsd, st); dfree(d_boff, st);
        dfree(d_nblk, st); dfree(d_blk_lo, st); dfree(d_blk_hi, st); dfree(d_exact_list, st);
        dfree(d_exact_count, st); dfree(d_sorted_list, st); dfree(d_sorted_count, st);
        dfree(d_r_rmsd, st); dfree(d_r_rot, st); dfree(d_r_cen, st); dfree(d_r_nan, st); dfree(d_r_hit, st);
        dfree(d_r_warn, st); dfree(d_r_hatoms, st); dfree(d_r_src, st); dfree(d_r_hidx, st); dfree(d_r_widx, st);
        dfree(d_r_aidx, st); dfree(d_lstate, st); dfree(d_work, st);
        dfree(d_pcost, st); dfree(d_hflag, st); dfree(d_heavy, st); dfree(d_hbins, st);
        dfree(d_susp_a, st); dfree(d_susp_b, st); dfree(d_pool_a, st); dfree(d_pool_b, st);
        dfree(d_prof, st);
        dfree(d_fill_state, st); dfree(d_fill_work, st);
        dfree(d_ls_key, st); dfree(d_ls_n, st); dfree(d_ls_rep, st); dfree(d_ls_slot, st);
        dfree(d_ls_rep_work, st); dfree(d_ls_dup, st); dfree(d_ls_left, st); dfree(d_ls_ok, st);
        dfree(d_z, st);
        for (auto &b : scan_tmp) dfree(b, st);
        t_cache = nullptr;
        const cudaError_t e = cudaStreamSynchronize(st);
        release_scratch(scratch, e == cudaSuccess && status != PJG_ERR_CUDA);
    }
    if (status != PJG_OK) {
        delete res;
        return status;
    }
    *out = res;
    return PJG_OK;
}

extern "C" {

int64_t pjg_results_count(const pjg_results *r) { return r ? r->store.hits : 0; }

int64_t pjg_results_atom_count(const pjg_results *r) { return r ? r->store.atoms : 0; }

pjg_status pjg_results_copy(const pjg_results *r, int32_t *structure, int32_t *template_index, int64_t *ordinal,
                            double *rmsd, double *rotation, double *centres, int64_t *atom_offset, int32_t *atoms) {
    if (!r) return fail(PJG_ERR_INVALID, "null results");
    if (r->count_only) return fail(PJG_ERR_INVALID, "the results of a count-only query hold no hits");
    const HitStore &hs = r->store;
    const size_t n = (size_t)hs.hits;
    if (atom_offset) atom_offset[n] = hs.atoms;
    if (n == 0) return PJG_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != r->device) cudaSetDevice(r->device);
    cudaError_t e = copy_out_all({{structure, hs.structure, 4 * n},
                                  {template_index, hs.tpl, 4 * n},
                                  {ordinal, hs.ordinal, 8 * n},
                                  {rmsd, hs.rmsd, 8 * n},
                                  {rotation, hs.rot, 72 * n},
                                  {centres, hs.centres, 48 * n},
                                  {atom_offset, hs.atom_offset, 8 * n},
                                  {atoms, hs.atoms_, 4 * (size_t)hs.atoms}});
    if (prev != r->device) cudaSetDevice(prev);
    if (e != cudaSuccess) return fail(PJG_ERR_CUDA, "results copy: %s", cudaGetErrorString(e));
    return PJG_OK;
}

int64_t pjg_results_warning_count(const pjg_results *r) { return r ? r->store.warns : 0; }

pjg_status pjg_results_superposed(const pjg_results *r, const pjg_structures *s, double *xyz) {
    if (!r || !s) return fail(PJG_ERR_INVALID, "null argument");
    if (r->count_only) return fail(PJG_ERR_INVALID, "the results of a count-only query hold no hits");
    if (s != r->structures) return fail(PJG_ERR_INVALID, "structures differ from the ones the query searched");
    const HitStore &hs = r->store;
    if (hs.atoms == 0) return PJG_OK;
    if (!xyz) return fail(PJG_ERR_INVALID, "null output");
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != r->device) cudaSetDevice(r->device);
    const size_t bytes = (size_t)hs.atoms * 3 * sizeof(double);
    double *d_out = nullptr;
    cudaError_t e;
    Scratch *x = acquire_scratch(r->device, &e);
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&d_out, bytes, x->st);
    if (e == cudaSuccess) {
        launch_superposed_atoms(x->st, hs.hits, hs.atoms, hs.structure, hs.atom_offset, hs.atoms_, hs.rot, hs.centres,
                                s->d_atom_base, s->d_xyz64, d_out);
        e = cudaGetLastError();
    }
    if (x) {
        cudaError_t e2 = cudaStreamSynchronize(x->st);
        if (e == cudaSuccess) e = e2;
        if (e == cudaSuccess) e = copy_out(xyz, d_out, bytes);
        if (d_out) cudaFreeAsync(d_out, x->st);
        e2 = cudaStreamSynchronize(x->st);
        if (e == cudaSuccess) e = e2;
        release_scratch(x, e == cudaSuccess);
    }
    if (prev != r->device) cudaSetDevice(prev);
    if (e != cudaSuccess) return fail(PJG_ERR_CUDA, "superposed atoms: %s", cudaGetErrorString(e));
    return PJG_OK;
}

pjg_status pjg_results_warnings(const pjg_results *r, int32_t *structure, int64_t *hits_before) {
    if (!r) return fail(PJG_ERR_INVALID, "null results");
    if (r->count_only) return fail(PJG_ERR_INVALID, "the results of a count-only query hold no warnings");
    const HitStore &hs = r->store;
    if (hs.warns == 0) return PJG_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != r->device) cudaSetDevice(r->device);
    cudaError_t e = copy_out(structure, hs.warn_structure, 4 * (size_t)hs.warns);
    if (e == cudaSuccess) e = copy_out(hits_before, hs.warn_before, 8 * (size_t)hs.warns);
    if (prev != r->device) cudaSetDevice(prev);
    if (e != cudaSuccess) return fail(PJG_ERR_CUDA, "warnings copy: %s", cudaGetErrorString(e));
    return PJG_OK;
}

pjg_status pjg_results_stats(const pjg_results *r, pjg_stats *stats) {
    if (!r || !stats) return fail(PJG_ERR_INVALID, "null argument");
    *stats = r->stats;
    return PJG_OK;
}

void pjg_results_destroy(pjg_results *r) {
    if (!r) return;
    int prev = 0;
    cudaGetDevice(&prev);
    const bool other = r->store.cap_h + r->store.cap_w > 0 && prev != r->device;
    if (other) cudaSetDevice(r->device);
    delete r;
    if (other) cudaSetDevice(prev);
}

}  // extern "C"
