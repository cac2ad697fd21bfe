// itlbm_resplan.cu -- host side of the resident kernel: which boxes it takes, in which tiles, and its
// exchange memory (itlbm_resident.cu).
#include "itlbm_resident.h"

#include <algorithm>
#include <cstdlib>
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
    int sms = 0;
    int ctas[3][NRES] = {};  // resident CTAs per SM by storage form and configuration
};
Device g_dev[MAX_DEVICES];

const Device *device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= MAX_DEVICES) return nullptr;
    Device &v = g_dev[d];
    std::call_once(v.once, [&] {
        int coop = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, d);
        if (!coop || cudaDeviceGetAttribute(&v.sms, cudaDevAttrMultiProcessorCount, d) != cudaSuccess) return;
        for (int prec = 0; prec < 3; prec++)
            for (int shape = 0; shape < NRES; shape++) v.ctas[prec][shape] = res_occupancy(prec, shape);
    });
    return &v;
}

std::mutex g_flag_lock;
int *g_flags = nullptr;
std::vector<int> g_flag_free;
constexpr int NFLAGS = 1 << 14;

}  // namespace

int res_capacity(int prec, int shape) {
    const Device *v = device();
    return v ? v->ctas[prec][shape] * v->sms : 0;
}

int res_tiling(int nx, int ny, int shape, int &bx, int &by) {
    const int nodes = res_nodes(shape), wh = res_half_perimeter(nodes);
    long long best = 0;
    int best_wh = 0;
    // tiles at least HMAX wide, so that a halo lies in the tiles beside
    for (int b = 1; b <= nx / HMAX && b <= 65535 && (long long)b * nx < 1LL << 31; b++) {
        const int w = (nx + b - 1) / b;
        const int hmax = std::min(nodes / w, wh - w);
        if (hmax < HMAX) continue;
        const int v = (ny + hmax - 1) / hmax;
        if (v > 65535 || ny / v < HMAX || (long long)v * ny >= 1LL << 31) continue;
        const int h = (ny + v - 1) / v;
        const long long n = (long long)b * v;
        if (best == 0 || n < best || (n == best && w + h < best_wh)) {
            best = n;
            best_wh = w + h;
            bx = b;
            by = v;
        }
        if (w <= HMAX) break;
    }
    return best > (1 << 20) ? 0 : (int)best;
}

namespace {
ResPlan plan_of(int prec, int nx, int ny, int shape) {
    ResPlan p;
    if (nx < RES_MIN_SIDE || ny < RES_MIN_SIDE || (long long)nx * ny > 1 << 20) return p;
    const int n = res_tiling(nx, ny, shape, p.bx, p.by);
    if (n > 0 && n <= res_capacity(prec, shape)) {
        p.tiles = n;
        p.shape = shape;
    }
    return p;
}
}  // namespace

ResPlan res_plan_single(int prec, int nx, int ny) {
    // The smallest tile whose count fits: the fewer warps an SM runs, the sooner each step ends.  Measured
    // on B200, us per step, P3, tiles of 64 / 128 / 256 nodes: FP64 100^2 6.3 / 6.3 / 8.4; FP32 100^2
    // 2.65 / 2.75 / 3.64, 256^2 3.43 / 3.57 / 4.45; fold 256^2 2.86 / 2.89 / 3.12, 380^2 256 threads with
    // one node each 4.0, with two 5.7 (k_step: 11.8; 6.8, 8.2; 8.2, 9.3).
    for (const int shape : {RES_64, RES_128, RES_256, RES_256x2}) {
        const ResPlan p = plan_of(prec, nx, ny, shape);
        if (p.shape >= 0) return p;
    }
    return ResPlan();
}

ResPlan res_plan_batch(int prec, int nx, int ny) {
    return plan_of(prec, nx, ny, prec == ITLBM_PREC_F32_FOLD ? RES_256x2 : RES_256);
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
    char *p = (char *)mem;
    a.tiles = (const ResTile *)p;
    cudaError_t e = cudaMemcpyAsync(p, q.tiles.data(), sizeof(ResTile) * q.tiles.size(), cudaMemcpyHostToDevice, st);
    p += sizeof(ResTile) * q.tiles.size();
    a.first = (const int *)p;
    if (e == cudaSuccess) e = cudaMemcpyAsync(p, q.first.data(), sizeof(int) * q.first.size(), cudaMemcpyHostToDevice, st);
    p += sizeof(int) * q.first.size();
    a.slots = (const int *)p;
    if (e == cudaSuccess) e = cudaMemcpyAsync(p, q.slots.data(), sizeof(int) * q.slots.size(), cudaMemcpyHostToDevice, st);
    return e;
}

size_t res_exchange_bytes(int prec, int shape, int slots) {
    return (size_t)slots * (2 * (npk_of(prec, shape) * pk_of(prec) * 16 + res_nodes(shape) * phi_bytes(prec)) + sizeof(unsigned));
}
void res_exchange_bind(ResArgs &a, void *base, int prec, int shape, int slots) {
    a.packs = (uint4 *)base;
    a.phis = (char *)base + (size_t)2 * slots * npk_of(prec, shape) * pk_of(prec) * 16;
    a.done = (unsigned *)((char *)a.phis + (size_t)2 * slots * res_nodes(shape) * phi_bytes(prec));
    a.nslots = slots;
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
