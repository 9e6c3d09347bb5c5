// xtg_plancache.cpp — reuse of planned launch sequences.
//
// Parsing, type inference, broadcasting, dimension collapsing and kernel
// selection depend only on the call's arguments (tree, leaf arrays including
// their addresses — alignment decides vector widths —, destination,
// reduction descriptor) and on the options.  A call records the launches it
// makes (kernel, grid, block, dynamic shared memory, parameter block); the
// next call with byte-identical arguments replays them, allocating fresh
// split-reduction scratch and patching its address into the parameter
// blocks.  Serving loops that evaluate the same request shapes over and over
// skip the host-side planning entirely.
#include <algorithm>
#include <cstring>
#include <list>
#include <memory>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "xtg_plan.h"

namespace xtgh {

namespace {

struct Plan {
    std::vector<unsigned char> key;
    std::vector<RecLaunch> launches;
    size_t scratch_bytes = 0;
};

struct Cache {
    std::mutex mu;
    std::unordered_map<uint64_t, std::vector<std::shared_ptr<Plan>>> map;
    size_t count = 0;
};
Cache& cache() {
    static Cache c;
    return c;
}

// FNV-1a over 8-byte words (the tail byte by byte): keys are a few hundred
// bytes and are hashed on every call.
uint64_t fnv(const std::vector<unsigned char>& v) {
    uint64_t h = 1469598103934665603ull;
    const size_t n = v.size(), nw = n / 8;
    for (size_t i = 0; i < nw; ++i) {
        uint64_t w;
        memcpy(&w, v.data() + 8 * i, 8);
        h ^= w;
        h *= 1099511628211ull;
        h ^= h >> 29;
    }
    for (size_t i = nw * 8; i < n; ++i) {
        h ^= v[i];
        h *= 1099511628211ull;
    }
    return h;
}

// Appends to a key whose buffer is already long enough.
struct KeyWriter {
    unsigned char* at;
    void bytes(const void* p, size_t n) {
        memcpy(at, p, n);
        at += n;
    }
    template <class T> void put(const T& v) { bytes(&v, sizeof v); }
    void array(const xtg_array& a) {
        put(a.data);
        put(a.dtype);
        put(a.rank);
        const size_t r = (size_t)std::max(0, std::min(a.rank, (int32_t)XTG_MAX_RANK));
        bytes(a.shape, r * sizeof a.shape[0]);
        bytes(a.strides, r * sizeof a.strides[0]);
    }
};
constexpr size_t kArrayKey = 16 + 2 * XTG_MAX_RANK * sizeof(int64_t);

}  // namespace

bool plan_cache_enabled() { return !hot_opts().dry_run && hot_opts().plan_cache; }

std::vector<unsigned char>& plan_key(int kind, const xtg_expr* e, const xtg_reduce_desc* rd, const xtg_array* out,
                                     int32_t a0, int32_t a1, int64_t a2, const xtg_array* const* more, int n_more) {
    // one buffer per thread, reused: no allocation on the replay path
    static thread_local std::vector<unsigned char> k;
    const int nn = std::max(0, std::min(e->n_nodes, (int32_t)XTG_MAX_NODES));
    const int nl = std::max(0, std::min(e->n_leaves, (int32_t)XTG_MAX_LEAVES));
    k.resize(256 + nn * sizeof(xtg_node) + sizeof(xtg_reduce_desc) + (nl + 1 + n_more) * kArrayKey);
    KeyWriter w{k.data()};
    w.put(kind);
    w.put(opt_generation());
    w.put(e->n_nodes);
    w.put(e->n_leaves);
    w.bytes(e->nodes, nn * sizeof(xtg_node));
    for (int i = 0; i < nl; ++i) w.array(e->leaves[i]);
    if (rd) {
        w.put(rd->op);
        w.put(rd->n_axes);
        w.bytes(rd->axes, (size_t)std::max(0, std::min(rd->n_axes, (int32_t)XTG_MAX_RANK)) * sizeof rd->axes[0]);
        w.put(rd->keep_dims);
        w.put(rd->has_initial);
        w.put(rd->initial);
        w.put(rd->acc_dtype);
        w.put(rd->precision);
        w.put(rd->ddof);
    }
    w.put(a0);
    w.put(a1);
    w.put(a2);
    w.array(*out);
    for (int i = 0; i < n_more; ++i) {
        w.put((int32_t)(more[i] != nullptr));
        if (more[i]) w.array(*more[i]);
    }
    k.resize((size_t)(w.at - k.data()));
    return k;
}

// Replays a cached plan for `key`; false if there is none.
bool plan_replay(const std::vector<unsigned char>& key, cudaStream_t s, xtg_status* st) {
    std::shared_ptr<Plan> p;
    const uint64_t h = fnv(key);
    {
        Cache& c = cache();
        std::lock_guard<std::mutex> lk(c.mu);
        auto it = c.map.find(h);
        if (it == c.map.end()) return false;
        for (auto& cand : it->second)
            if (cand->key == key) p = cand;
        if (!p) return false;
    }
    void* scratch = nullptr;
    if (p->scratch_bytes) {
        *st = scratch_alloc(&scratch, p->scratch_bytes, s);
        if (*st != XTG_OK) return true;
    }
    unsigned char buf[8192];
    *st = XTG_OK;
    for (const RecLaunch& l : p->launches) {
        const void* params = l.params.data();
        if (l.scratch_off >= 0) {
            if (l.params.size() > sizeof buf) {
                *st = fail(XTG_ERR_INVALID, "parameter block too large");
                break;
            }
            memcpy(buf, l.params.data(), l.params.size());
            void* mine = (char*)scratch + l.scratch_base;
            memcpy(buf + l.scratch_off, &mine, sizeof mine);
            params = buf;
        }
        *st = launch_raw(l.k, l.grid, l.block, params, l.params.size(), s, l.smem, -1);
        if (*st != XTG_OK) break;
    }
    if (scratch) {
        xtg_status fs = scratch_free(scratch, s);
        if (*st == XTG_OK) *st = fs;
    }
    return true;
}

void plan_store(const std::vector<unsigned char>& key, Recorder& rec) {
    if (rec.nocache) return;
    auto p = std::make_shared<Plan>();
    p->key = key;
    p->launches = std::move(rec.launches);
    p->scratch_bytes = rec.scratch_bytes;
    for (auto& l : p->launches)
        if (l.scratch_off >= 0 && !p->scratch_bytes) return;
    Cache& c = cache();
    std::lock_guard<std::mutex> lk(c.mu);
    if (c.count >= (size_t)opt("plan.cache_max", 16384)) {
        c.map.clear();
        c.count = 0;
    }
    c.map[fnv(p->key)].push_back(p);
    ++c.count;
}

}  // namespace xtgh
