// itlbm_resident.h -- the resident multi-step kernel (itlbm_resident.cu): its launch arguments, its
// tile configurations and the rule that chooses one for a case.
#pragma once

#include "itlbm_internal.h"

#include <vector>

namespace itlbm {

// Tile configurations, by threads: 64 and 128 with registers to spare (boxes that leave the SMs half empty
// anyway), 256 for many tiles per SM, and for the box sizes beyond: FP32 with four CTAs per SM instead of
// three (D), the fold with two nodes per thread (x2), with three and with four CTAs per SM.
enum { RES_64 = 0, RES_128 = 1, RES_256 = 2, RES_256D = 3, RES_256x2 = 4, RES_256x2D = 5, NRES = 6 };
__host__ __device__ constexpr int res_threads(int shape) { return shape == RES_64 ? 64 : (shape == RES_128 ? 128 : 256); }
__host__ __device__ constexpr int res_nodes(int shape) { return shape >= RES_256x2 ? 512 : res_threads(shape); }
// Largest w + h of a tile of that many nodes: 32 x 16, 32 x 8, 16 x 8, 8 x 8.
__host__ __device__ constexpr int res_half_perimeter(int nodes) {
    return nodes == 512 ? 48 : (nodes == 256 ? 40 : (nodes == 128 ? 24 : 16));
}

// A tile of a launch: its case, which of the case's bx x by tiles it is, where the CTAs (exchange slots) of
// the case's tiles are listed, and the case's place in the order the queues follow.
struct ResTile {
    int case_id, tile, peers, order;
    unsigned short bx, by;
};

struct ResArgs {
    const CaseDev *cases;
    const ResTile *tiles;   // the queues of the CTAs, one after the other
    const int *first;       // CTA b takes tiles [first[b], first[b + 1])
    const int *slots;       // CTA of each tile of each case, from ResTile::peers on
    unsigned *done;         // per CTA: the last tag of the last tile it finished
    uint4 *packs;      // exchange of populations: 2 parities x slots x NPK x PK packs
    void *phis;        // exchange of rho^N: 2 parities x slots x NODES entries of 8 (FP32) or 16 bytes
    int *err;          // set when a wait ran out
    int nslots;        // CTAs the exchange memory is laid out for (>= the grid)
    unsigned tag0;     // the case of order o uses the tags tag0 + o nsteps + 1 ..., used by no earlier launch
    int k0, nsteps, aux_k;
};

template <class S, bool FOLD, int SHAPE>
struct ResCfg {
    static constexpr int NT = res_threads(SHAPE), R = res_nodes(SHAPE) / NT;  // threads, nodes per thread
    static constexpr int NP = FOLD ? NK : NV;          // planes per colour
    static constexpr int ND = FOLD ? 3 : 5;            // of which leave through one side
    static constexpr int NODES = res_nodes(SHAPE);
    static constexpr int WH = res_half_perimeter(NODES);
    static constexpr int PS = NODES + 2 * WH;          // stride of a plane: the nodes, and w + 1 elements on each side
    static constexpr int RING = NODES + 2 * WH + 4;    // largest (w + 2)(h + 2)
    static constexpr int PHIN = NODES + 4 * WH + 16;   // largest (w + 4)(h + 4)
    static constexpr int NPK = 2 * ND * WH;            // exchanged nodes x planes of one tile
    static constexpr int NRING = 4 * WH + 16;          // halo nodes at reach 2
    static constexpr int PK = sizeof(S) == 8 ? 2 : 1;  // packs per exchanged plane: both colours in FP32
    static constexpr int SMEM = (int)sizeof(S) * (2 * NP * PS + PHIN) + 4 * (NPK + NRING) + 2 * NPK;
    // CTAs per SM the registers are sized for.  Measured on B200: FP32 with three CTAs of 256 threads (80
    // registers, no spills) runs sweeps of 100 x 100 boxes at 24.0 G updates/s, with four (64, spills) at
    // 20.6; the fold's P3 410 x 410 with two nodes per thread takes 4.8 us per step with three, 7.3 with four.
    static constexpr bool F64 = sizeof(S) == 8;
    static constexpr int MIN_CTAS = SHAPE == RES_64 ? (F64 ? 4 : 8) : SHAPE == RES_128 ? (F64 ? 2 : 4) :
                                    F64 ? 2 : ((SHAPE == RES_256 && !FOLD) || SHAPE == RES_256x2) ? 3 : 4;
    // The case's parameters in shared memory, or read through the cache where registers are so short that
    // what the compiler then keeps of them is spilled (FP64 sweep 9.2 against 9.6 G updates/s, FP32 380 x 380
    // 6.6 against 6.2 us per step; elsewhere 2 % faster).
    static constexpr bool OWN_CASE = !(SHAPE == RES_256D || (F64 && SHAPE == RES_256));
    static_assert(10 * RING <= 2 * NP * PS, "ring-1 auxiliaries in the planes' place");
    static_assert(PHIN <= 1024, "element of phi in 10 bits");
};

int res_occupancy_f64(int prec, int shape);
int res_occupancy_f32(int prec, int shape);
cudaError_t res_launch_f64(int prec, int shape, const ResArgs &a, int grid, cudaStream_t st);
cudaError_t res_launch_f32(int prec, int shape, const ResArgs &a, int grid, cudaStream_t st);
inline int res_occupancy(int prec, int shape) {
    return prec == ITLBM_PREC_F64 ? res_occupancy_f64(prec, shape) : res_occupancy_f32(prec, shape);
}
inline cudaError_t res_launch(int prec, int shape, const ResArgs &a, int grid, cudaStream_t st) {
    return prec == ITLBM_PREC_F64 ? res_launch_f64(prec, shape, a, grid, st) : res_launch_f32(prec, shape, a, grid, st);
}


// Steps a call must ask for to take the resident kernel, and the most one launch runs.  Its launch
// costs 20 us (tables, first loads) where a k_step launch costs 8, so it gains from about four steps on:
// call and synchronisation on a 100^2 drop, k_step / resident, 4 steps: FP64 53 / 52, FP32 34 / 37, fold
// 39 / 29 us; 6 steps: 76 / 64, 46 / 42, 56 / 34 us.
constexpr int RES_MIN_STEPS = 6;
constexpr int RES_MAX_STEPS = 4096;


// How a case is held on chip: the tile configuration and the bx x by tiles, or shape < 0 when the box
// has more tiles than the device holds at once (or sides below RES_MIN_SIDE).
constexpr int RES_MIN_SIDE = 8;
struct ResPlan {
    int shape = -1, bx = 0, by = 0, tiles = 0;
};
// CTAs of configuration `shape` the current device holds at once (0: no cooperative launch).
int res_capacity(int prec, int shape);
ResPlan res_plan_single(int prec, int tipo, int nx, int ny);  // one case alone on the device
ResPlan res_plan_batch(int prec, int nx, int ny);   // one of many cases that share it
// The queues of a launch: cases in order, each on the least loaded of `ctas` CTAs.  A CTA's load is the time its queue ends, with `cost` the time of one tile.
struct ResCase {
    ResPlan plan;
    int case_id;
    double cost;
};
struct ResQueues {
    std::vector<ResTile> tiles;
    std::vector<int> first, slots;
    size_t bytes() const { return sizeof(ResTile) * tiles.size() + sizeof(int) * (first.size() + slots.size()); }
};
ResQueues res_queues(const std::vector<ResCase> &cases, int ctas);
// The queues copied to device memory of bytes() bytes, on a stream, and bound to the launch arguments.
cudaError_t res_queues_upload(ResArgs &a, const ResQueues &q, void *mem, cudaStream_t st);
// Bytes of exchange memory for `slots` CTAs, and its binding in a block of that many bytes.
size_t res_exchange_bytes(int prec, int shape, int slots);
void res_exchange_bind(ResArgs &a, void *base, int prec, int shape, int slots);
// A word the resident kernel sets when a wait runs out, in pinned host memory the device writes
// (process-wide pool; nullptr when it cannot be had), and its return.
int *res_flag_get();
void res_flag_put(int *f);

}  // namespace itlbm
