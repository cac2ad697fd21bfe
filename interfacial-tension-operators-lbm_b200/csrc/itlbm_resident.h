// itlbm_resident.h -- the resident multi-step kernel (itlbm_resident.cu): its launch arguments, its
// tile configurations and the rule that chooses one for a case.
#pragma once

#include "itlbm_internal.h"

#include <vector>

namespace itlbm {

// Tile configurations, by threads: 64, 128 and (FP64) 160, 192 and 224 with registers to spare, for boxes that
// leave the SMs half empty anyway, 256 for many tiles per SM, with two nodes per thread (x2, the FP32 forms) and, for the box sizes
// beyond, four (x4, the fold) or four CTAs per SM at 64 registers (D, FP32).
enum { RES_64 = 0, RES_128, RES_160, RES_192, RES_224, RES_256, RES_256x2, RES_256D, RES_256x4, NRES };
__host__ __device__ constexpr int res_threads(int shape) {
    return shape == RES_64 ? 64 : shape == RES_128 ? 128 : shape == RES_160 ? 160 : shape == RES_192 ? 192 : shape == RES_224 ? 224 : 256;
}
__host__ __device__ constexpr int res_nodes(int shape) { return shape == RES_256x4 ? 1024 : (shape == RES_256x2 ? 512 : res_threads(shape)); }
// Largest w + h of a tile of that many nodes: 32 x 32, 32 x 16, 32 x 8, 32 x 7, 24 x 8, 20 x 8, 16 x 8, 8 x 8,
// a little more for 192 and 160.
__host__ __device__ constexpr int res_half_perimeter(int nodes) {
    return nodes == 1024 ? 64 : nodes == 512 ? 48 : nodes == 224 ? 39 : nodes == 192 ? 34 : nodes == 160 ? 30 : (nodes == 256 ? 40 : (nodes == 128 ? 24 : 16));
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
    unsigned *done;         // per CTA: the last tag of the last tile it finished, or the one before the first of its tile
    unsigned *finished;     // tiles finished in this exchange memory, over all CTAs and launches
    int polls;              // of `done`, after which a wait for a CTA runs out unless tiles are being finished
    int queued;             // whether a CTA of the launch has more than one tile
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
    // CTAs per SM the registers are sized for, measured on B200: FP32 sweeps with one node per thread in three
    // CTAs of 80 registers run at 24.0 G updates/s (100 x 100 boxes), in four of 64, which spill, at 20.6; two
    // nodes per thread in two CTAs of 128 registers at 24.3, and 25.5 against 23.2 on 192 x 192 boxes (F2 21.2
    // against 18.6).  Fold: two nodes in three CTAs 40.7 against 38.2, a 410 x 410 step 4.8 us against 7.3 in
    // four; four nodes in two CTAs, 500 x 500, 6.4 us against 7.8 for two in four.  FP64: one node in two CTAs of
    // 128 registers 9.5, two nodes in one CTA 8.8; for a case alone fewer threads of more registers where they
    // suffice (200 x 200 P3 4.8 us in 160 threads, 5.85 in 256; 230 x 230 F2 7.6 in 192, 8.9 in 256).
    static constexpr bool F64 = sizeof(S) == 8;
    static constexpr int MIN_CTAS = SHAPE == RES_64 ? (F64 ? 4 : 8) : SHAPE == RES_128 ? (F64 ? 2 : 4) :
                                    F64 ? 2 : SHAPE == RES_256D ? 4 : SHAPE == RES_256x4 ? 2 :
                                    FOLD ? (SHAPE == RES_256 ? 4 : 3) : (SHAPE == RES_256 ? 3 : 2);
    // The case's parameters in shared memory, or read through the cache where registers are so short that
    // what the compiler then keeps of them is spilled (FP64 sweep 9.2 against 9.6 G updates/s, FP32 380 x 380
    // 6.6 against 6.2 us per step; elsewhere 2 % faster).
    static constexpr bool OWN_CASE = !(SHAPE == RES_256D || (F64 && SHAPE == RES_256));
    static_assert(10 * RING <= 2 * NP * PS, "ring-1 auxiliaries in the planes' place");
    static constexpr int EB = NP * PS <= 8192 ? 13 : 14;  // bits of an element of a pack
    static_assert(NP * PS <= 1 << EB, "element of a pack");
    static constexpr int HB = PHIN <= 1024 ? 10 : 11;     // bits of an element of phi
    static_assert(PHIN <= 1 << HB, "element of phi");
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


// Steps a call must ask for to take the resident kernel, and the most one launch runs.  Its launch costs 20 us
// (tables, first loads) where a k_step launch costs 8, so most boxes gain from about five steps on, the largest from
// seven or eight: call and synchronisation, us, k_step / resident, 6 steps: FP64 40 x 40 51.6 / 41.4, 100 x 100
// 52.3 / 46.5, F2 256 x 256 86.7 / 73.8; FP32 100 x 100 40.6 / 42.1, 256 x 256 49.1 / 44.0, 380 x 380 70.1 / 72.3; fold
// 100 x 100 42.8 / 33.9, 500 x 500 68.3 / 75.9; 10 steps: 77.7 / 55.1, 80.6 / 60.1, 136.8 / 108.1; 61.5 / 52.3,
// 75.5 / 56.8, 110.3 / 94.2; 64.8 / 43.0, 107.5 / 101.3.
constexpr int RES_MIN_STEPS = 6;
constexpr int RES_MAX_STEPS = 4096;
// Polls without a finished tile, each a trip to L2: some 3 s.  The longest that a tile takes is RES_MAX_STEPS
// steps, below 0.1 s.
constexpr int RES_POLLS = 1 << 23;
// Sub-steps a batch's replay must have: its tables keep the GPU busy with k_step, and a resident tile's first loads
// and tables are hidden by nothing.  Tables / resident, G updates/s, 150 mixed cases of 64 to 512 nodes a side and 100
// of 64 to 256: FP64 10 steps 7.25 / 6.85 and 6.4 / 5.7, 20 steps 7.25 / 7.24 and 6.4 / 6.7; FP32 20 steps 14.8 / 15.0
// and 12.8 / 15.4 (600 cases 15.2 / 14.9), 40 steps 14.5 / 16.4 and 12.8 / 17.2; fold 20 steps 28.9 / 25.7 and
// 24.3 / 25.9, 40 steps 28.9 / 28.8 and 24.2 / 27.4, 80 steps 28.0 / 30.7 and 24.3 / 30.4.
inline int res_min_replay(int prec) { return prec == ITLBM_PREC_F32_FOLD ? 40 : 24; }
// Nodes that a batch's launch must hold per unit of its queues' length (the time of one tile), where the batch has
// cases for the work tables too: added to these, a node costs what it does at their full rate (FP64 7.4 G updates/s,
// FP32 12, fold 22), while a launch takes as long for one tile as for all its places (4.3 to 7 us per step by FP64
// configuration, 4.1 and 3.6 us).  One FP32 512 x 512 box and m others, ms per 500 steps with all in the tables / the
// others resident first: FP64 1 x 64^2 8.9 / 11.3, 4 x 100^2 (40 000 nodes, one unit) 11.1 / 12.0, 16 x 64^2 (65 500, one)
// 12.4 / 12.2, 16 x 100^2 21.2 / 18.7, 1 x 200^2 (40 000 in smaller tiles) 10.7 / 10.9, 4 x 200^2 18.5 / 17.5; FP32
// 1 x 64^2 8.7 / 10.7, 4 x 100^2 10.3 / 10.8, 16 x 64^2 10.4 / 10.7, 4 x 200^2 15.7 / 13.5; fold 1 x 64^2 9.0 / 10.3,
// 4 x 200^2 10.4 / 11.2, 16 x 100^2 (160 000, one) 11.1 / 11.2, 16 x 200^2 18.6 / 18.3.  (Run beside the tables instead
// of before them, small launches gain a little on that, 1 x 64^2 fold 8.7, but both slow down when they share SMs:
// 4 x 100^2 FP64 13.5, beside an FP32 1024 x 1024 box 51 against 35.)
double res_min_nodes(int prec, int shape);


// How a case is held on chip: the tile configuration and the bx x by tiles, or shape < 0 when the box
// has more tiles than the device holds at once (or sides below RES_MIN_SIDE).
constexpr int RES_MIN_SIDE = 8;
struct ResPlan {
    int shape = -1, bx = 0, by = 0, tiles = 0;
};
// CTAs of configuration `shape` the current device holds at once (0: no cooperative launch).
int res_capacity(int prec, int shape);
// Whether a stream has all the device's SMs: not one of a green context.
bool res_whole_device(cudaStream_t st);
// A plan as the C ABI reports it.
itlbm_plan res_describe(int prec, const ResPlan &p);
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
    double length = 0;  // when the last queue ends
    size_t bytes() const { return sizeof(ResTile) * tiles.size() + sizeof(int) * (first.size() + slots.size()); }
};
ResQueues res_queues(const std::vector<ResCase> &cases, int ctas);
// The queues copied to device memory of bytes() bytes, on a stream that is then waited for, and bound to the
// launch arguments.
cudaError_t res_queues_upload(ResArgs &a, const ResQueues &q, void *mem, cudaStream_t st);
// Bytes of exchange memory for `slots` CTAs, and its binding in a block of that many bytes.
size_t res_exchange_bytes(int prec, int shape, int slots);
void res_exchange_bind(ResArgs &a, void *base, int prec, int shape, int slots);
// A word the resident kernel sets when a wait runs out, in pinned host memory the device writes
// (process-wide pool; nullptr when it cannot be had), and its return.
int *res_flag_get();
void res_flag_put(int *f);

}  // namespace itlbm
