// itlbm_resplan.cu -- host side of the resident kernel: which boxes it takes, in which tiles, and its
// exchange memory (itlbm_resident.cu).
#include "itlbm_resident.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace itlbm {

namespace {

int npk_of(int prec, int shape) {
    return 2 * (prec == ITLBM_PREC_F32_FOLD ? 3 : 5) * res_half_perimeter(res_nodes(shape));
}
int pk_of(int prec) { return prec == ITLBM_PREC_F64 ? 2 : 1; }
size_t phi_bytes(int prec) { return prec == ITLBM_PREC_F64 ? 16 : 8; }

constexpr int MAX_DEVICES = 32;
struct Device {
    std::once_flag once;
    int sms = 0;  // 0: no cooperative launches
    // resident CTAs per SM by storage form and configuration, each asked when a plan comes to it: the question loads
    // the kernel, and all sixteen kept the first case of a process waiting for 5 ms
    std::once_flag asked[3][NRES];
    int ctas[3][NRES] = {};
    std::atomic<int> loaded{0};
};
Device g_dev[MAX_DEVICES];

Device *device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= MAX_DEVICES) return nullptr;
    Device &v = g_dev[d];
    std::call_once(v.once, [&] {
        int coop = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, d);
        if (!coop || cudaDeviceGetAttribute(&v.sms, cudaDevAttrMultiProcessorCount, d) != cudaSuccess) v.sms = 0;
    });
    return v.sms ? &v : nullptr;
}
int ctas_per_sm(Device &v, int prec, int shape) {
    std::call_once(v.asked[prec][shape], [&] {
        v.ctas[prec][shape] = res_occupancy(prec, shape);
        v.loaded += v.ctas[prec][shape] > 0;
    });
    return v.ctas[prec][shape];
}

std::mutex g_flag_lock;
int *g_flags = nullptr;
std::vector<int> g_flag_free;
constexpr int NFLAGS = 1 << 14;

}  // namespace

int res_capacity(int prec, int shape) {
    Device *v = device();
    return v ? ctas_per_sm(*v, prec, shape) * v->sms : 0;
}

bool res_whole_device(cudaStream_t st) {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuStreamGetGreenCtx", &f, 12040, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        return true;  // a driver without them
    }
    CUgreenCtx g = nullptr;
    return ((decltype(&cuStreamGetGreenCtx))f)((CUstream)st, &g) == CUDA_SUCCESS && g == nullptr;
}

itlbm_plan res_describe(int prec, const ResPlan &p) {
    Device *v = device();
    if (!v || p.shape < 0) return itlbm_plan{};
    return itlbm_plan{p.bx, p.by, res_threads(p.shape), res_nodes(p.shape), ctas_per_sm(*v, prec, p.shape)};
}

namespace {

int up(int a, int b) { return (a + b - 1) / b; }

// The tiling of an nx x ny box by configuration `shape` with the least cost(tiles, w, h), then the smallest
// tiles, then the shortest edge; w and h of the largest tile.
template <class COST>
double best_tiling(int prec, int nx, int ny, int shape, ResPlan &p, COST cost) {
    const int nodes = res_nodes(shape), wh = res_half_perimeter(nodes), cap = res_capacity(prec, shape);
    double least = 0;
    int size = 0, edge = 0;
    p = ResPlan();
    if (nx < RES_MIN_SIDE || ny < RES_MIN_SIDE || (long long)nx * ny > (long long)cap * nodes) return 0;
    // Tiles at least HMAX wide, so that a halo lies in the tiles beside; begins of tiles in 32 bits.  Of the counts
    // that give the same largest tile only the smallest is looked at (the cost does not fall with the tiles): a
    // 256 x 256 F2 box took 0.4 ms over all of them, a case's creation in all 1.3.
    for (int bx = 1; bx <= nx / HMAX && bx <= std::min(cap, 65535) && (long long)bx * nx < 1LL << 31;) {
        const int w = up(nx, bx), hmax = std::min(nodes / w, wh - w);
        if (hmax >= HMAX)
            for (int by = up(ny, hmax); by <= std::min(ny / HMAX, cap / bx) && by <= 65535 && (long long)by * ny < 1LL << 31;) {
                const int h = up(ny, by);
                const double v = cost(bx * by, w, h);
                if (p.shape < 0 || v < least || (v == least && (w * h < size || (w * h == size && w + h < edge)))) {
                    least = v;
                    size = w * h;
                    edge = w + h;
                    p.shape = shape;
                    p.bx = bx;
                    p.by = by;
                    p.tiles = bx * by;
                }
                if (h == 1) break;
                by = up(ny, h - 1);
            }
        if (w == 1) break;
        bx = up(nx, w - 1);
    }
    return least;
}

}  // namespace

// A case alone.  The smallest configuration that holds it: few warps share an SM, and each step ends the
// sooner (us per step, P3, 64 / 128 / 256 threads: FP64 100^2 3.6 / 3.8 / 5.4, FP32 100^2 2.70 / 2.75 / 3.2,
// 256^2 3.46 / 3.42 / 3.9, fold 256^2 2.86 / 2.90 / 3.0; k_step 7.1, 5.1, 6.6, 5.8), in the fewest tiles, or
// with 256 threads in as many as leave the fewest warps on the fullest SM (FP64 200^2 5.96 against 6.20).
// FP64 F1 / F2 also pass over the ring-1 region, a second time when it has more nodes than the CTA threads:
// there the configuration and tiling with the fewest warps on the fullest SM, the region's counted half
// (a second pass, one more), as long as the SMs are not full: F2 100^2 4.84 against 5.19, 150^2 5.45 / 6.0,
// 200^2 7.8 / 9.75.  (FP32 takes the inner nodes of the region while it waits; balanced in the same way
// 150^2 boxes are slower, F1 3.22 against 3.04, fold F2 2.78 / 2.69, 100^2 ones within 2 %.)
ResPlan res_plan_single(int prec, int tipo, int nx, int ny) {
    const Device *v = device();
    if (!v) return ResPlan();
    const bool ring = (tipo == ITLBM_OP_F1 || tipo == ITLBM_OP_F2) && prec == ITLBM_PREC_F64;
    ResPlan best;
    double least = 0;
    for (int shape = 0; shape < NRES; shape++) {
        constexpr double factor[NRES] = {1.0, 1.05, 1.1, 1.15, 1.2, 1.3, 1.4, 1.5, 1.6};  // same work per step
        const int threads = res_threads(shape);
        ResPlan p;
        const double c = factor[shape] * best_tiling(prec, nx, ny, shape, p, [&](int tiles, int w, int h) {
                             if (!ring && threads < 256) return (double)tiles;
                             const int region = (w + 2) * (h + 2);
                             return up(tiles, v->sms) *
                                    (up(w * h, 32) + (ring ? 0.5 * up(region, 32) + (region > threads ? 1.0 : 0.0) : 0.0));
                         });
        if (p.shape < 0) continue;
        if (!ring) return p;
        if (best.shape < 0 || c < least) {
            best = p;
            least = c;
        }
    }
    return best;
}

// In a batch the CTAs are all taken: what counts is the time of a step over the cases that run side by side.
// That time is about that of the exchange, worth some ten warps a CTA, and of the tile's own warps.
// Small cases fill what larger ones leave; of one that takes more than a sixth of the CTAs only whole
// ones fit side by side, and slightly smaller tiles may fill the same CTAs (fold F2 256 x 256: 24.7 G
// updates/s in 256 tiles, 27.2 in 296).
// An FP64 case of which only one fits at a time in tiles of 256 threads takes the smallest configuration that
// holds it, as a case alone does (sweeps of twelve boxes of 200 to 256 nodes a side 38.7 -> 31.3 ms, P3 36.2 ->
// 28.5); smaller ones gain more by company (60 to 200 nodes a side in 160 or 192 threads 20.5 ms, in 256 16.2), and
// so do the FP32 forms (12 x 200 to 330: two nodes a thread 22.3 ms, one 23.8).
ResPlan res_plan_batch(int prec, int nx, int ny) {
    auto plan = [&](int shape) {
        const int cap = res_capacity(prec, shape);
        ResPlan p;
        best_tiling(prec, nx, ny, shape, p, [&](int tiles, int w, int h) {
            return (10 + up(w * h, 32)) / (6 * tiles <= cap ? (double)cap / tiles : (double)(cap / tiles));
        });
        return p;
    };
    const int first = prec == ITLBM_PREC_F64 ? RES_256 : RES_256x2;
    if (prec == ITLBM_PREC_F64 && 2 * (long long)nx * ny > (long long)res_capacity(prec, RES_256) * res_nodes(RES_256))
        for (int shape = RES_160; shape < RES_256; shape++) {
            const ResPlan p = plan(shape);
            if (p.shape >= 0) return p;
        }
    for (int shape = first; shape < NRES; shape++) {
        const ResPlan p = plan(shape);
        if (p.shape >= 0) return p;
    }
    return ResPlan();
}

double res_min_nodes(int prec, int shape) {
    return prec == ITLBM_PREC_F64 ? 0.65 * res_capacity(prec, shape) * res_nodes(shape) : prec == ITLBM_PREC_F32 ? 60e3 : 180e3;
}

ResQueues res_queues(const std::vector<ResCase> &cases, int ctas) {
    ResQueues Q;
    std::vector<std::vector<ResTile>> queue(ctas);
    std::vector<std::pair<double, int>> load(ctas);  // when the CTA is free, and which
    for (int c = 0; c < ctas; c++) load[c] = {0.0, c};
    int order = 0;
    for (const ResCase &k : cases) {
        const int n = k.plan.tiles, peers = (int)Q.slots.size();
        // a case starts when its last CTA is free: the earliest ones
        if (order) std::partial_sort(load.begin(), load.begin() + n, load.end());
        const double end = load[n - 1].first + k.cost;
        for (int t = 0; t < n; t++) {
            const int c = load[t].second;
            Q.slots.push_back(c);
            queue[c].push_back(ResTile{k.case_id, t, peers, order, (unsigned short)k.plan.bx, (unsigned short)k.plan.by});
            load[t].first = end;
        }
        Q.length = std::max(Q.length, end);
        order++;
    }
    Q.first.push_back(0);
    for (const auto &q : queue) {
        Q.tiles.insert(Q.tiles.end(), q.begin(), q.end());
        Q.first.push_back((int)Q.tiles.size());
    }
    return Q;
}

cudaError_t res_queues_upload(ResArgs &a, const ResQueues &q, void *mem, cudaStream_t st) {
    std::vector<char> all(q.bytes());
    size_t at = 0;
    auto put = [&](const void *src, size_t n) {
        const size_t o = at;
        std::memcpy(all.data() + at, src, n);
        at += n;
        return (char *)mem + o;
    };
    a.tiles = (const ResTile *)put(q.tiles.data(), sizeof(ResTile) * q.tiles.size());
    a.first = (const int *)put(q.first.data(), sizeof(int) * q.first.size());
    a.queued = q.tiles.size() + 1 > q.first.size();
    a.slots = (const int *)put(q.slots.data(), sizeof(int) * q.slots.size());
    const cudaError_t e = cudaMemcpyAsync(mem, all.data(), at, cudaMemcpyHostToDevice, st);
    const cudaError_t w = cudaStreamSynchronize(st);  // pageable copies may return before they have read
    return e == cudaSuccess ? w : e;
}

size_t res_exchange_bytes(int prec, int shape, int slots) {
    return (size_t)slots * (2 * (npk_of(prec, shape) * pk_of(prec) * 16 + res_nodes(shape) * phi_bytes(prec)) + sizeof(unsigned)) + sizeof(unsigned);
}
void res_exchange_bind(ResArgs &a, void *base, int prec, int shape, int slots) {
    a.packs = (uint4 *)base;
    a.phis = (char *)base + (size_t)2 * slots * npk_of(prec, shape) * pk_of(prec) * 16;
    a.done = (unsigned *)((char *)a.phis + (size_t)2 * slots * res_nodes(shape) * phi_bytes(prec));
    a.finished = a.done + slots;
    a.nslots = slots;
    a.polls = RES_POLLS;
}

int *res_flag_get() {
    std::lock_guard<std::mutex> g(g_flag_lock);
    if (!g_flags) {
        if (cudaHostAlloc((void **)&g_flags, sizeof(int) * NFLAGS, cudaHostAllocMapped | cudaHostAllocPortable) !=
            cudaSuccess) {
            cudaGetLastError();
            g_flags = nullptr;
            return nullptr;
        }
        for (int i = NFLAGS - 1; i >= 0; i--) g_flag_free.push_back(i);
    }
    if (g_flag_free.empty()) return nullptr;
    int *f = g_flags + g_flag_free.back();
    g_flag_free.pop_back();
    *f = 0;
    return f;
}
void res_flag_put(int *f) {
    if (!f) return;
    std::lock_guard<std::mutex> g(g_flag_lock);
    g_flag_free.push_back((int)(f - g_flags));
}

}  // namespace itlbm

// Not in include/itlbm.h: for tests, the configurations loaded so far on the current device.
extern "C" int itlbm_internal_configurations(void) {
    itlbm::Device *v = itlbm::device();
    return v ? v->loaded.load() : 0;
}
