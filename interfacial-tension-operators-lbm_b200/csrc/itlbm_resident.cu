// itlbm_resident.cu -- many time steps in one launch, the state of every case held on chip.
//
// k_step (itlbm_step.cu) reads and writes the whole state in HBM every step, and a box of a few
// hundred nodes a side cannot hide what that costs: on B200 one FP64 step of a 100 x 100 drop takes
// 7.1 us (3.4 here), of which the launch, the dependent loads of the tile's descriptors and the two round
// trips for the node and halo loads are most.  Here a CTA keeps one tile of one case for all the steps of a
// launch: its populations live in shared memory, and per step only what crosses a tile's edge goes
// through L2, to the CTAs that hold the neighbouring tiles.  All CTAs are resident at once (a
// cooperative launch), since they wait for one another.
//
// Step of a tile of w x h nodes, R per thread (one; two or four in some FP32 and fold configurations):
//   1. each thread takes its node's planes from shared memory, forms rho^N, and posts it when the
//      node lies within the stencil's reach of the tile's edge;
//   2. the halo's rho^N are taken from the tiles that own those nodes;
//      (for class P the relaxation, which needs no gradient, comes before that wait);
//   3. gradient, force, collision (itlbm_node.cuh), and the push of every plane to x + c_i in shared
//      memory;
//   4. what left the tile is posted, and what enters it is taken from its neighbours.
// In a plane the nodes follow one another row by row without gaps, so a push is the same shift of the
// element for every thread and the warp's accesses hit distinct banks whatever the tile's width (planes
// with ghost columns cost half as many wavefronts again: 380 x 380 FP32 P3 6.6 us per step against 6.2).
// A value that leaves the tile lands, by the same shift, where one will enter (or in the padding), and is
// posted from there before that one is written.
// The values go as 16-byte packs {values, tag} written and read whole (relaxed b128 accesses), so a
// pack is its own flag: the reader polls the pack until its tag is that of the step, and no fence
// and no second round trip is needed.  Packs are double-buffered by the parity of the step: a
// neighbour posts step k + 2 only after it took what this tile posted at k + 1, which this tile did
// after it had taken everything of step k.
// A launch may hold more tiles than the device does at once: each CTA takes the tiles of its queue one
// after the other.  All queues follow one order of the cases, so the first unfinished case always has
// all its CTAs, and no wait is circular.
// A CTA that comes to a case before its neighbours waits until these are through the cases before it, which
// can take as long as those do; so a tile first waits for the tiles beside it to have begun, as long as any
// tile of the launch is being finished, and only then steps, in exchanges that take microseconds.
// Every wait is bounded: a wait that runs out sets *err and the CTA returns at the end of its step,
// as do its neighbours in turn.
//
// The tile's shape is free within a configuration's nodes and half perimeter (best_tiling in itlbm_resplan.cu): a
// 100 x 100 FP64 box alone is 13 x 13 tiles of 8 x 8 nodes at most.  A node's arithmetic does not depend on the tile, so the results are those of k_step to the
// bit.
#include "itlbm_node.cuh"
#include "itlbm_resident.h"

#include <algorithm>
#include <climits>

namespace itlbm {

namespace {

constexpr int SPIN_LIMIT = 1 << 21;  // polls of an exchange, each a trip to L2: about a second

// planes that leave a tile through a side (0 +x, 1 -x, 2 +y, 3 -y): the axis ones, then the two
// diagonals
template <bool FOLD>
__device__ __forceinline__ constexpr int side_plane(int side, int d) {
    constexpr int t19[20] = {1, 11, 13, 7, 9, 2, 12, 14, 8, 10, 3, 16, 18, 7, 10, 4, 15, 17, 8, 9};
    constexpr int t9[12] = {1, 5, 7, 2, 6, 8, 3, 5, 8, 4, 6, 7};
    return FOLD ? t9[side * 3 + d] : t19[side * 5 + d];
}
// in-plane velocity of plane d of a side: the axis, and for the last two d the diagonal's other part
template <bool FOLD>
__device__ __forceinline__ void side_dir(int side, int d, int &ex, int &ey) {
    constexpr int NA = FOLD ? 1 : 3;
    const int s = (side & 1) ? -1 : 1;
    // side_plane: +x {.., (1,1), (1,-1)}; -x {.., (-1,-1), (-1,1)}; +y {.., (1,1), (-1,1)}; -y {.., (-1,-1), (1,-1)}
    const int t = d < NA ? 0 : (d == NA ? s : -s);
    ex = side < 2 ? s : t;
    ey = side < 2 ? t : s;
}

__device__ __forceinline__ void st_pack(uint4 *p, unsigned long long lo, unsigned long long hi) {
    asm volatile("{ .reg .b128 v; mov.b128 v, {%1, %2}; st.relaxed.gpu.global.b128 [%0], v; }" ::"l"(p), "l"(lo), "l"(hi)
                 : "memory");
}
__device__ __forceinline__ void ld_pack(const uint4 *p, unsigned long long &lo, unsigned long long &hi) {
    asm volatile("{ .reg .b128 v; ld.relaxed.gpu.global.b128 v, [%2]; mov.b128 {%0, %1}, v; }" : "=l"(lo), "=l"(hi) : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st_pair(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_pair(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned *p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_word(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void count_word(unsigned *p) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ unsigned long long pair_of(unsigned a, unsigned b) {
    return (unsigned long long)a | ((unsigned long long)b << 32);
}

// Polls of up to MI items a thread: `load(u)` reads item u, `take(u)` uses it if it has come and says so.
// False when the wait ran out.  (A delay before the first poll changes nothing, several polls under way at once
// lengthen the wait by the trips of those not needed any more.)
template <int MI, class LOAD, class TAKE>
__device__ __forceinline__ bool poll_items(unsigned pend, LOAD load, TAKE take) {
    if (!pend) return true;
    for (int spins = 0; spins < SPIN_LIMIT; spins++) {
#pragma unroll
        for (int u = 0; u < MI; u++)
            if (pend >> u & 1u) load(u);
#pragma unroll
        for (int u = 0; u < MI; u++)
            if ((pend >> u & 1u) && take(u)) pend &= ~(1u << u);
        if (!pend) return true;
    }
    return false;
}

// Waits until the CTA of `done` has come as far as tag.  False when it has not after a.polls polls during which no
// tile was finished.
__device__ __forceinline__ bool wait_for(const ResArgs &a, const unsigned *done, unsigned tag) {
    unsigned finished = 0;
    for (int polls = 0; (int)(ld_word(done) - tag) < 0;)
        if (++polls >= a.polls) {
            const unsigned now = ld_word(a.finished);
            if (now == finished) return false;
            finished = now;
            polls = 0;
        }
    return true;
}

// first coordinate of tile t of n nodes cut into b tiles (best_tiling keeps the product in 32 bits)
__device__ __forceinline__ int tile_begin(int t, int n, int b) { return (int)((unsigned)t * (unsigned)n / (unsigned)b); }

// Of a CTA's tile: its case, its place and size, and what the loop needs of them.
struct Geo {
    int tipo, x0, y0, w, h;
    float rho0;
    int nring, npacks;  // halo nodes; packs that leave (and enter), with those that the corners leave out
    int nsteps, cur0;   // steps of this launch, the buffer it starts from
    int keep_step;      // the step whose force and gradient are kept
    unsigned tag0;      // the tags of this tile's steps are tag0 + 1 ...
    int slot[9];        // exchange slots of the tile (4) and the eight beside it, row by row
    int tx[3], ty[3], begin_x[3], begin_y[3], size_x[3], size_y[3];  // the tile's column and row and the ones beside them
};

template <class S, bool FOLD, int SHAPE>
__global__ void __launch_bounds__(res_threads(SHAPE), (ResCfg<S, FOLD, SHAPE>::MIN_CTAS)) k_resident(const __grid_constant__ ResArgs a) {
    using C = ResCfg<S, FOLD, SHAPE>;
    constexpr int NT = C::NT, R = C::R;
    constexpr int NP = C::NP, ND = C::ND, PS = C::PS, PAD = C::WH, PK = C::PK;
    constexpr bool F64 = std::is_same<S, double>::value;
    using PhiPack = std::conditional_t<F64, uint4, unsigned long long>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S *const pop = reinterpret_cast<S *>(smem_raw);             // [2 NP][PS]: node t = ly w + lx of a plane at PAD + t
    S *const phi = pop + 2 * NP * PS;                           // (w + 4) x (h + 4)
    unsigned *const rcv = reinterpret_cast<unsigned *>(phi + C::PHIN);  // packs that enter: source << EB | element
    unsigned *const hal = rcv + C::NPK;                         // halo nodes: source << HB | element of phi
    unsigned short *const snd = reinterpret_cast<unsigned short *>(hal + C::NRING);  // element of each pack that leaves
    // F1 / F2: the ring-1 gradient and auxiliaries, in the planes' place between their load and the push
    S *const ringg = pop, *const ringa = pop + 3 * C::RING;

    // What is the same for all threads sits in shared memory and is read where it is used: kept in
    // registers it would cost the 64-register forms spills, which a thousand threads per SM cannot
    // hold in the cache that the shared memory leaves.
    __shared__ Geo g;
    __shared__ std::conditional_t<C::OWN_CASE, CaseDev, const CaseDev *> own_case;
    auto the_case = [&]() -> const CaseDev & {
        if constexpr (C::OWN_CASE) return own_case;
        else return *own_case;
    };
    const int tid = threadIdx.x;
    int bad = 0;
    const int qend = a.first[blockIdx.x + 1];
    for (int qi = a.first[blockIdx.x]; qi < qend; qi++) {
    {
        const ResTile rt = a.tiles[qi];
        const CaseDev &dc = a.cases[rt.case_id];
        const int nsteps = min(a.nsteps, dc.chunk_len - a.k0);
        if (nsteps <= 0) continue;  // and so do its other tiles
        if constexpr (C::OWN_CASE) {
            for (int i = tid; i < (int)(sizeof(CaseDev) / sizeof(int)); i += NT) ((int *)&own_case)[i] = ((const int *)&dc)[i];
        } else if (tid == 0) own_case = &dc;
        __syncthreads();
        const CaseDev &c = the_case();
        const int bx = rt.bx, by = rt.by, H = c.halo;
        const int ty = rt.tile / bx, tx = rt.tile - ty * bx;
        if (tid < 6) {  // the tile's column and row and the ones beside them
            const bool col = tid < 3;
            const int d = col ? tid : tid - 3, b = col ? bx : by, n = col ? c.nx : c.ny;
            int t = (col ? tx : ty) + d - 1;
            t += t < 0 ? b : (t == b ? -b : 0);
            const int x = tile_begin(t, n, b);
            (col ? g.tx : g.ty)[d] = col ? t : t * bx;
            (col ? g.begin_x : g.begin_y)[d] = x;
            (col ? g.size_x : g.size_y)[d] = tile_begin(t + 1, n, b) - x;
        }
        const int wm = (c.nx + bx - 1) / bx, hm = (c.ny + by - 1) / by;  // largest tile of the case
        const int nxs = ND * hm, nitems = 2 * ND * (hm + wm);
        __syncthreads();
        if (tid >= 32 && tid < 41) g.slot[tid - 32] = a.slots[rt.peers + g.ty[(tid - 32) / 3] + g.tx[(tid - 32) % 3]];
        const int w = g.size_x[1], h = g.size_y[1], PP = w + 4;
        const int nring = 2 * H * (w + h + 2 * H);
        if (tid == 0) {
            g.tipo = c.tipo;
            g.rho0 = c.pf.rho0;
            g.x0 = g.begin_x[1];
            g.y0 = g.begin_y[1];
            g.w = w;
            g.h = h;
            g.nring = nring;
            g.npacks = nitems * PK;
            g.nsteps = nsteps;
            g.cur0 = (c.parity0 + a.k0) & 1;
            g.tag0 = a.tag0 + (unsigned)rt.order * (unsigned)a.nsteps;
            g.keep_step = c.aux == nullptr ? -1 : (c.aux_at_end ? c.chunk_len - 1 : a.aux_k) - a.k0;
        }

        __syncthreads();
        // the packs of the exchange: index = side offset + d * length + position along the side, the
        // same for every tile of the case
        for (int j = tid; j < nitems; j += NT) {
            const bool xs = j < 2 * nxs;
            const int L = xs ? hm : wm, r = xs ? j : j - 2 * nxs, dl = r / L, pos = r - dl * L;
            const int side = (xs ? 0 : 2) + (dl >= ND ? 1 : 0), d = dl >= ND ? dl - ND : dl;
            const int plane = side_plane<FOLD>(side, d);
            int ex, ey;
            side_dir<FOLD>(side, d, ex, ey);
            // leaving: source (lx, ly) in this tile; a diagonal that leaves through a corner goes by its x side
            int lx = xs ? (ex > 0 ? w - 1 : 0) : pos, ly = xs ? pos : (ey > 0 ? h - 1 : 0);
            bool ok = pos < (xs ? h : w) && (xs || (unsigned)(lx + ex) < (unsigned)w);
            snd[j] = ok ? (unsigned short)(plane * PS + PAD + (ly + ey) * w + lx + ex) : (unsigned short)0xFFFF;
            // entering: destination (lx, ly) in this tile, from the tile beside it that holds (lx - ex, ly - ey)
            lx = xs ? (ex > 0 ? 0 : w - 1) : pos;
            ly = xs ? pos : (ey > 0 ? 0 : h - 1);
            ok = pos < (xs ? h : w) && (xs || (unsigned)(lx - ex) < (unsigned)w);
            unsigned v = 0xFFFFFFFFu;
            if (ok) {
                const int sx = lx - ex, sy = ly - ey;
                const int ix = sx < 0 ? 0 : (sx >= w ? 2 : 1), iy = sy < 0 ? 0 : (sy >= h ? 2 : 1);
                const int spos = xs ? (iy == 0 ? g.size_y[0] - 1 : (iy == 2 ? 0 : sy)) : sx;
                v = ((unsigned)(g.slot[iy * 3 + ix] * C::NPK + j - pos + spos) << C::EB) |
                    (unsigned)(plane * PS + PAD + ly * w + lx);
            }
            rcv[j] = v;
        }
        // the halo nodes of rho^N, row by row around the tile
        for (int j = tid; j < nring; j += NT) {
            const int B = w + 2 * H, nb = H * B;
            int px, py;  // relative to the tile's first node
            if (j < 2 * nb) {
                const int q = j / B;
                py = q < H ? q - H : h + q - H;
                px = j - q * B - H;
            } else {
                const int r = j - 2 * nb, k = r & (2 * H - 1);
                py = H == 1 ? r >> 1 : r >> 2;
                px = k < H ? k - H : w + k - H;
            }
            const int ix = px < 0 ? 0 : (px >= w ? 2 : 1), iy = py < 0 ? 0 : (py >= h ? 2 : 1);
            const int sx = px < 0 ? px + g.size_x[0] : (px >= w ? px - w : px);
            const int sy = py < 0 ? py + g.size_y[0] : (py >= h ? py - h : py);
            const int node = sy * g.size_x[ix] + sx;
            hal[j] = ((unsigned)(g.slot[iy * 3 + ix] * C::NODES + node) << C::HB) |
                     (unsigned)((py + 2) * PP + px + 2);
        }
    }
    __syncthreads();

    // the thread's nodes, t = tid + r NT: whether there is one, whether it lies within the stencil's reach
    // of the tile's edge, and its row
    unsigned me[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const CaseDev &c = the_case();
        const int t = tid + r * NT, w = g.w, h = g.h, H = c.halo;
        me[r] = 0;
        if (t < w * h) {
            const int ly = t / w, lx = t - ly * w;
            const bool edge = lx < H || lx >= w - H || ly < H || ly >= h - H;
            const bool inner = lx > 0 && lx < w - 1 && ly > 0 && ly < h - 1;
            me[r] = 0x80000000u | (edge ? 0x40000000u : 0u) | (inner ? 0x20000000u : 0u) | (unsigned)ly;
            const S *src = (const S *)c.buf[g.cur0] + node_off(c, g.x0 + lx, g.y0 + ly);
#pragma unroll
            for (int q = 0; q < 2 * NP; q++) pop[q * PS + PAD + t] = src[q * PLANE];
        }
    }
    // F1 / F2 in FP32: the thread's node of the two outermost layers of the ring-1 region, row << 16 | element: the
    // nodes that need the halo's rho^N.  The others' gradients are taken while those are on their way.  (B200, us
    // per step: FP32 F2 333 x 207 4.12 -> 3.94, fold F2 150 x 150 2.85 -> 2.78.  FP64 has too few registers to gain
    // by it, and where one pass covers the region two are slower: F1 200 x 200 6.45 -> 6.8.)
    constexpr bool INNER_FIRST = !F64;
    // Class F: the moments too are taken while the halo's rho^N are on their way (FP64 F1 200 x 200 6.45 -> 6.28,
    // FP32 F2 333 x 207 3.94 -> 3.86).
    constexpr bool EARLY_MOMENTS = !FOLD;
    unsigned rim = 0xFFFFFFFFu;
    if (INNER_FIRST && (g.tipo == ITLBM_OP_F1 || g.tipo == ITLBM_OP_F2)) {
        static_assert(4 * C::WH <= NT, "a thread per node of the rim");
        const int w = g.w, h = g.h, PW = w + 2, r = tid - 4 * PW;
        if (tid < 4 * (w + h)) {
            const int j = tid / PW, k = r & 3;
            const int qy = r < 0 ? (j < 2 ? j : h - 2 + j) : 2 + (r >> 2), qx = r < 0 ? tid - j * PW : (k < 2 ? k : w - 2 + k);
            rim = (unsigned)qy << 16 | (unsigned)(qy * PW + qx);
        }
    }
    // the node's element of phi, with its halo of two nodes, and of the ring-1 region
    auto phi_el = [&](int r) { return tid + r * NT + (int)(me[r] & 0xFFFFu) * 4 + 2 * g.w + 10; };
    auto ring_el = [&](int r) { return tid + r * NT + (int)(me[r] & 0xFFFFu) * 2 + g.w + 3; };
    // the node's element in a state buffer
    auto home = [&](int r) {
        const int t = tid + r * NT, ly = t / g.w, lx = t - ly * g.w;
        return node_off(the_case(), g.x0 + lx, g.y0 + ly);
    };
    // where CTAs take several tiles, those of the tiles beside this one have begun it too (or finished the case before)
    if (a.queued) {
        if (tid == 0) st_word(a.done + blockIdx.x, g.tag0);
        if (tid < 9 && !wait_for(a, a.done + g.slot[tid], g.tag0)) bad = 1;
        if (__syncthreads_or(bad)) {
            if (tid == 0) *a.err = 1;
            return;
        }
    }
    // the buffer the launch does not end in: a site that is streamed unchanged waits there
    auto spare = [&]() { return (S *)the_case().buf[(g.cur0 ^ (g.nsteps & 1)) ^ 1]; };
    __syncthreads();

    for (int s = 0; s < g.nsteps; s++) {
        const unsigned tag = g.tag0 + (unsigned)s + 1u;
        uint4 *const pk = a.packs + ((tag & 1u) ? (size_t)a.nslots * (C::NPK * PK) : 0);
        PhiPack *const ph = (PhiPack *)a.phis + ((tag & 1u) ? (size_t)a.nslots * C::NODES : 0);

        // ---- 1: the node's planes and rho^N ----------------------------------------------------
        S f[R][NP], sa[R], sb[R];
        double sbd[R];
        Recolour<S, FOLD> rc[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            sa[r] = S(0);
            sb[r] = S(0);
            sbd[r] = 0.0;
            if (me[r]) {
                S va[NP], vb[NP];
#pragma unroll
                for (int i = 0; i < NP; i++) va[i] = pop[i * PS + PAD + tid + r * NT];
#pragma unroll
                for (int i = 0; i < NP; i++) vb[i] = pop[(NP + i) * PS + PAD + tid + r * NT];
#pragma unroll
                for (int i = 0; i < NP; i++) sa[r] = sa[r] + va[i];
#pragma unroll
                for (int i = 0; i < NP; i++) sb[r] = sb[r] + vb[i];
                const S p = phase_of(sa[r], sb[r], g.rho0);
                phi[phi_el(r)] = p;
                if (me[r] & 0x40000000u) {
                    const unsigned o = blockIdx.x * C::NODES + tid + r * NT;
                    if constexpr (F64) st_pack(ph + o, (unsigned long long)__double_as_longlong(p), tag);
                    else st_pair(ph + o, pair_of(__float_as_uint(p), tag));
                }
                bool keep;  // a site that will be streamed unchanged (rho <= 1e-30)
                if constexpr (F64) keep = !(sa[r] + sb[r] > 1.0e-30);
                else keep = !(g.rho0 + sa[r] > 1.0e-30f);
                if (keep) {
                    S *tmp = spare() + home(r);
#pragma unroll
                    for (int i = 0; i < NP; i++) {
                        tmp[i * PLANE] = va[i];
                        tmp[(NP + i) * PLANE] = vb[i];
                    }
                }
                if constexpr (!F64) {
#pragma unroll
                    for (int i = 0; i < NP; i++) sbd[r] += (double)vb[i];
                }
#pragma unroll
                for (int i = 0; i < NP; i++) f[r][i] = F64 ? va[i] + vb[i] : va[i];
                // what needs no force, while the halo's rho^N are on their way: for class P the relaxation too
                if (EARLY_MOMENTS || g.tipo < ITLBM_OP_F1) {
                    const CaseDev &c = the_case();
                    CaseDev::F32Par pf{};
                    if constexpr (!F64) pf = load_pf(c);
                    node_moments<S, FOLD>(pf, f[r], sa[r], sb[r], rc[r]);
                    if (!EARLY_MOMENTS || g.tipo < ITLBM_OP_F1)
                        node_relax<false, S, FOLD>(c, pf, f[r], sa[r], sb[r], S(0), S(0), S(0), rc[r]);
                }
            }
        }

        const int tipo = g.tipo, PW = g.w + 2, PP = g.w + 4;
        const bool force = tipo >= ITLBM_OP_F1, ring = tipo == ITLBM_OP_F1 || tipo == ITLBM_OP_F2;
        auto ring_node = [&](int q, int at) {
            const S *p = phi + at;
            ring_aux_node<S>(the_case(), tipo, [&](int dx, int dy) { return p[dy * PP + dx]; }, ringg + q * 3, ringa + q * AUXS);
        };
        if (INNER_FIRST && ring) {
            __syncthreads();
#pragma unroll
            for (int r = 0; r < R; r++)
                if (me[r] & 0x20000000u) ring_node(ring_el(r), phi_el(r));
        }

        // ---- 2: the halo's rho^N ----------------------------------------------------------------
        {
            constexpr int MI = (C::NRING + NT - 1) / NT;
            unsigned pend = 0, e[MI];
#pragma unroll
            for (int u = 0; u < MI; u++) {
                e[u] = 0;
                if (tid + u * NT < g.nring) {
                    e[u] = hal[tid + u * NT];
                    pend |= 1u << u;
                }
            }
            unsigned long long lo[MI], hi[MI];
            if (!poll_items<MI>(
                    pend,
                    [&](int u) {
                        if constexpr (F64) ld_pack(ph + (e[u] >> C::HB), lo[u], hi[u]);
                        else {
                            lo[u] = ld_pair(ph + (e[u] >> C::HB));
                            hi[u] = lo[u] >> 32;
                        }
                    },
                    [&](int u) {
                        if ((unsigned)hi[u] != tag) return false;
                        S *const d = phi + (e[u] & ((1u << C::HB) - 1u));
                        if constexpr (F64) *d = __longlong_as_double((long long)lo[u]);
                        else *d = __uint_as_float((unsigned)lo[u]);
                        return true;
                    }))
                bad = 1;
        }
        __syncthreads();

        // ---- 3: gradient, force, collision, push --------------------------------------------------
        const CaseDev &c = the_case();
        if (ring) {
            if constexpr (INNER_FIRST) {
                if (rim != 0xFFFFFFFFu) ring_node((int)(rim & 0xFFFFu), (int)((rim & 0xFFFFu) + (rim >> 16) * 2) + PP + 1);
            } else {
                const int nq = PW * (g.h + 2), M = (65536 + PW - 1) / PW;  // q / PW by multiply and shift, exact for q < 65536 / PW
                for (int q = tid; q < nq; q += NT) ring_node(q, q + ((q * M) >> 16) * 2 + PP + 1);
            }
            __syncthreads();
        }
        CaseDev::F32Par pf{};
        if constexpr (!F64) pf = load_pf(c);
        S gmx[R], gmy[R], gmz[R], Fx[R], Fy[R], Fz[R];
#pragma unroll
        for (int r = 0; r < R; r++)
            if (me[r]) {
                const S *p = phi + phi_el(r);
                const int o = ring ? ring_el(r) : 0;
                const S *q = ringa + o * AUXS;
                node_force<S>(c, tipo, pf, [&](int dx, int dy) { return p[dy * PP + dx]; },
                              [&](int dx, int dy) { return q + (dy * PW + dx) * AUXS; }, ringg + o * 3, gmx[r], gmy[r],
                              gmz[r], Fx[r], Fy[r], Fz[r]);
                if (!EARLY_MOMENTS && force) node_moments<S, FOLD>(pf, f[r], sa[r], sb[r], rc[r]);
                if (force) node_relax<true, S, FOLD>(c, pf, f[r], sa[r], sb[r], Fx[r], Fy[r], Fz[r], rc[r]);
            }
        if (ring) __syncthreads();  // the push overwrites the auxiliaries
#pragma unroll
        for (int r = 0; r < R; r++)
            if (me[r]) {
                S *const own = pop + PAD + tid + r * NT;
                S *const at[3] = {own - g.w, own, own + g.w};
                auto push = [&](auto Q, S v) {
                    constexpr int q = decltype(Q)::value, i = q % NP;
                    constexpr int ex = FOLD ? kx(i) : cx(i), ey = FOLD ? ky(i) : cy(i);
                    at[ey + 1][q * PS + ex] = v;
                };
                if constexpr (F64) gradient_size(gmx[r], gmy[r], gmz[r], rc[r]);
                if (!rc[r].skip) {
                    if (force) node_finish<true, S, FOLD>(c, pf, f[r], sa[r], gmx[r], gmy[r], gmz[r], rc[r]);
                    else node_finish<false, S, FOLD>(c, pf, f[r], sa[r], gmx[r], gmy[r], gmz[r], rc[r]);
                    node_split<S, FOLD>(pf, f[r], sbd[r], rc[r], push);
                } else {
                    const S *tmp = spare() + home(r);
                    sfor<0, 2 * NP>([&](auto Q) { push(Q, tmp[decltype(Q)::value * PLANE]); });
                }
                if (s == g.keep_step)
                    keep_aux(c, g.x0 + (tid + r * NT) % g.w, g.y0 + (tid + r * NT) / g.w, Fx[r], Fy[r], Fz[r], gmx[r], gmy[r], gmz[r]);
            }

        __syncthreads();

        // ---- 4: what crosses the tile's edges -----------------------------------------------------
        {
            constexpr int MI = (C::NPK * PK + NT - 1) / NT;
            unsigned pend = 0, e[MI];
#pragma unroll
            for (int u = 0; u < MI; u++) {
                const int j = tid + u * NT;
                e[u] = j < g.npacks ? snd[j / PK] : 0xFFFFu;
            }
#pragma unroll
            for (int u = 0; u < MI; u++) {
                const int j = tid + u * NT;
                if (e[u] == 0xFFFFu) continue;
                uint4 *const o = pk + (size_t)(blockIdx.x * C::NPK) * PK + j;
                if constexpr (F64) st_pack(o, (unsigned long long)__double_as_longlong(pop[e[u] + (j % PK) * NP * PS]), tag);
                else st_pack(o, pair_of(__float_as_uint(pop[e[u]]), __float_as_uint(pop[e[u] + NP * PS])), tag);
            }
            __syncthreads();  // what enters takes the places of what left
#pragma unroll
            for (int u = 0; u < MI; u++) {
                const int j = tid + u * NT;
                e[u] = j < g.npacks ? rcv[j / PK] : 0xFFFFFFFFu;
                if (e[u] != 0xFFFFFFFFu) pend |= 1u << u;
            }
            unsigned long long lo[MI], hi[MI];
            if (!poll_items<MI>(
                    pend,
                    [&](int u) {
                        ld_pack(pk + (size_t)(e[u] >> C::EB) * PK + (tid + u * NT) % PK, lo[u], hi[u]);
                    },
                    [&](int u) {
                        if ((unsigned)hi[u] != tag) return false;
                        S *const d = pop + (e[u] & ((1u << C::EB) - 1u));
                        if constexpr (F64) d[((tid + u * NT) % PK) * NP * PS] = __longlong_as_double((long long)lo[u]);
                        else {
                            d[0] = __uint_as_float((unsigned)lo[u]);
                            d[NP * PS] = __uint_as_float((unsigned)(lo[u] >> 32));
                        }
                        return true;
                    }))
                bad = 1;
        }
        if (__syncthreads_or(bad)) {
            if (tid == 0) *a.err = 1;
            return;
        }
    }

    // the state at the top of the next step
#pragma unroll
    for (int r = 0; r < R; r++)
        if (me[r]) {
            S *dst = (S *)the_case().buf[g.cur0 ^ (g.nsteps & 1)] + home(r);
#pragma unroll
            for (int q = 0; q < 2 * NP; q++) dst[q * PLANE] = pop[q * PS + PAD + tid + r * NT];
        }
    // Before its next tile writes into its exchange slot, the CTA knows that the tiles beside this one have
    // taken what it posted last: each says so when it is done.
    const unsigned last = g.tag0 + (unsigned)g.nsteps;
    if (tid == 0) {
        st_word(a.done + blockIdx.x, last);
        count_word(a.finished);
    }
    if (qi + 1 < qend && tid < 9 && !wait_for(a, a.done + g.slot[tid], last)) bad = 1;
    if (__syncthreads_or(bad)) {
        if (tid == 0) *a.err = 1;
        return;
    }
    }
}

template <class S, bool FOLD, int SHAPE>
struct Entry {
    using C = ResCfg<S, FOLD, SHAPE>;
    // resident CTAs per SM, asked once per device (the query also sets the shared-memory limit)
    static int occupancy() {
        int n = 0;
        if (cudaFuncSetAttribute(k_resident<S, FOLD, SHAPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_resident<S, FOLD, SHAPE>, C::NT, C::SMEM) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        // the packed table entries hold so many slots
        int d = 0, sms = 1;
        cudaGetDevice(&d);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d);
        const long long most = std::min((1ll << (32 - C::EB)) / C::NPK, (1ll << (32 - C::HB)) / C::NODES);
        while (n > 0 && (long long)n * sms > most) n--;
        return n;
    }
    static cudaError_t launch(const ResArgs &a, int grid, cudaStream_t st) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(C::NT);
        cfg.dynamicSmemBytes = C::SMEM;
        cfg.stream = st;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, k_resident<S, FOLD, SHAPE>, a);
    }
};

}  // namespace

// Compiled twice, like itlbm_step.cu: FP64 without FMA contraction, and the FP32 forms.
#ifdef ITLBM_STEP_F64
#define RES_SWITCH(prec, shape, what)                            \
    switch (shape) {                                             \
        case RES_64: return Entry<double, false, RES_64>::what;   \
        case RES_128: return Entry<double, false, RES_128>::what; \
        case RES_160: return Entry<double, false, RES_160>::what; \
        case RES_192: return Entry<double, false, RES_192>::what; \
        case RES_224: return Entry<double, false, RES_224>::what; \
        case RES_256: return Entry<double, false, RES_256>::what; \
    }
int res_occupancy_f64(int prec, int shape) {
    RES_SWITCH(prec, shape, occupancy())
    return 0;
}
cudaError_t res_launch_f64(int prec, int shape, const ResArgs &a, int grid, cudaStream_t st) {
    RES_SWITCH(prec, shape, launch(a, grid, st))
    return cudaErrorInvalidValue;
}
#else
#define RES_SWITCH(prec, shape, what)                                    \
    if (prec == ITLBM_PREC_F32) switch (shape) {                         \
        case RES_64: return Entry<float, false, RES_64>::what;           \
        case RES_128: return Entry<float, false, RES_128>::what;         \
        case RES_256: return Entry<float, false, RES_256>::what;         \
        case RES_256x2: return Entry<float, false, RES_256x2>::what;     \
        case RES_256D: return Entry<float, false, RES_256D>::what;       \
    }                                                                    \
    else switch (shape) {                                                \
        case RES_64: return Entry<float, true, RES_64>::what;            \
        case RES_128: return Entry<float, true, RES_128>::what;          \
        case RES_256: return Entry<float, true, RES_256>::what;          \
        case RES_256x2: return Entry<float, true, RES_256x2>::what;      \
        case RES_256x4: return Entry<float, true, RES_256x4>::what;    \
    }
int res_occupancy_f32(int prec, int shape) {
    RES_SWITCH(prec, shape, occupancy())
    return 0;
}
cudaError_t res_launch_f32(int prec, int shape, const ResArgs &a, int grid, cudaStream_t st) {
    RES_SWITCH(prec, shape, launch(a, grid, st))
    return cudaErrorInvalidValue;
}
#endif

}  // namespace itlbm
