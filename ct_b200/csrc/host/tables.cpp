// Process-wide caches of the filter tables (twiddles + kernel spectrum) per
// (device, W, pad, filter) and of the Feldkamp weight tables per device and
// detector geometry, shared by the operator layer, the facade and batches.
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <tuple>
#include <vector>

#include "../ctb_internal.h"

namespace ctb {

namespace {
struct Key {
    int dev, W, pad, filter;
    bool operator<(const Key& o) const { return std::tie(dev, W, pad, filter) < std::tie(o.dev, o.W, o.pad, o.filter); }
};
std::mutex g_mtx;
std::map<Key, FilterTables> g_tables;
}  // namespace

int filter_tables(int W, int pad, int filter, cudaStream_t s, FilterTables* out) {
    int dev = 0;
    CTB_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_mtx);
    const Key key{dev, W, pad, filter};
    auto it = g_tables.find(key);
    if (it != g_tables.end()) {
        *out = it->second;
        return CTB_OK;
    }
    FilterTables t;
    t.M = filter_transform_length(W, pad);
    if (t.M == 0) {
        set_global_error("detector width exceeds the largest supported FFT length");
        return CTB_ERR_UNSUPPORTED;
    }
    while ((1 << t.logM) < t.M) ++t.logM;
    float2* tw = nullptr;
    float* K = nullptr;
    CTB_CUDA_TRY(cudaMalloc(&tw, sizeof(float2) * filter_twiddle_count(t.M)));
    CTB_CUDA_TRY(cudaMalloc(&K, sizeof(float) * t.M));
    const int st = filter_build_tables(W, pad, filter, t.M, tw, K, s);
    if (st != CTB_OK) return st;
    CTB_CUDA_TRY(cudaStreamSynchronize(s));
    t.tw = tw;
    t.K = K;
    g_tables[key] = t;
    *out = t;
    return CTB_OK;
}

namespace {
uint32_t bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
struct WeightTable {
    float* p = nullptr;
    size_t bytes = 0;
};
// (device, W, H, D, uPre, vPre) -> weight table
using PreKey = std::tuple<int, int, int, uint32_t, uint32_t, uint32_t>;
std::map<PreKey, std::shared_ptr<WeightTable>> g_pre;
size_t g_pre_bytes = 0;
// above this the tables that nobody holds are freed first
constexpr size_t kPreBudget = size_t(512) << 20;

int pre_table(const PreKey& key, size_t n, bool build, const std::function<int(float*)>& make, const float** out,
              std::shared_ptr<const void>* pin) {
    *out = nullptr;
    auto it = g_pre.find(key);
    if (it == g_pre.end()) {
        if (!build) return CTB_OK;
        const size_t bytes = n * sizeof(float);
        if (g_pre_bytes + bytes > kPreBudget) {
            // A holder (a call that has not launched yet, a batch, a captured graph) keeps its
            // table; cudaFree waits for launched work that may still read the others. Holders
            // take their references under g_mtx, so a count of 1 (the cache's) stays 1 here.
            for (auto i = g_pre.begin(); i != g_pre.end();) {
                if (i->second.use_count() > 1) {
                    ++i;
                    continue;
                }
                cudaFree(i->second->p);
                g_pre_bytes -= i->second->bytes;
                i = g_pre.erase(i);
            }
        }
        auto t = std::make_shared<WeightTable>();
        if (cudaMalloc(&t->p, bytes) != cudaSuccess) {
            cudaGetLastError();
            return CTB_OK;  // no table: the filter evaluates per pixel
        }
        t->bytes = bytes;
        const int st = make(t->p);
        if (st != CTB_OK) {
            cudaFree(t->p);
            return st;
        }
        it = g_pre.emplace(key, std::move(t)).first;
        g_pre_bytes += bytes;
    }
    *out = it->second->p;
    *pin = it->second;
    return CTB_OK;
}
}  // namespace

int pre_tables(FilterArgs* a, cudaStream_t s, bool build, std::shared_ptr<const void>* pin) {
    int dev = 0;
    CTB_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_mtx);
    const PreKey k{dev, a->W, a->H, bits(a->D), bits(a->uPre), bits(a->vPre)};
    return pre_table(k, size_t(a->W) * weight_rows(a->H), build, [&](float* t) {
        int r = build_weight_table(*a, t, s);
        if (r == CTB_OK) r = cuda_status(cudaStreamSynchronize(s), "weight table");
        return r;
    }, &a->wt, pin);
}

bool keep_for_graph(cudaGraph_t graph, const std::shared_ptr<const void>& pin) {
    using Pin = std::shared_ptr<const void>;
    Pin* held = new (std::nothrow) Pin(pin);
    if (!held) return false;
    // (the destructor runs on a thread of the driver's and may call nothing of CUDA: it
    // drops a reference that is never the last, since the cache holds one)
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, held, [](void* p) { delete static_cast<Pin*>(p); }, 1,
                             cudaUserObjectNoDestructorSync) != cudaSuccess) {
        cudaGetLastError();
        delete held;
        return false;
    }
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaGetLastError();
        cudaUserObjectRelease(obj, 1);
        return false;
    }
    return true;
}

}  // namespace ctb
