// itlbm_node.cuh -- the update of one node, shared by the two step kernels (itlbm_step.cu, one step
// per launch with the state in HBM; itlbm_resident.cu, many steps per launch with the state on chip).
// Both call these functions, so a node's update is the same arithmetic whichever kernel runs it.
#pragma once

#include "itlbm_site.cuh"

namespace itlbm {

// Stride of the per-node auxiliary values in shared memory: 7, odd, so that the 32 lanes reading one
// component of consecutive nodes hit distinct banks (a stride of 6 words, or 12 for doubles, puts two
// lanes on each bank).
constexpr int AUXS = 7;

// rho^N from the two colour sums.  FP64: (rho_R - rho_B) / (rho_R + rho_B), Imm_OPS.cpp:255-258.
// FP32: the sums are sum e_i (rho - rho0) and sum d_i (rho_R - rho_B).
__device__ __forceinline__ double phase_of(double rR, double rB, float) {
    return (rR - rB) / (rR + rB);
}
__device__ __forceinline__ float phase_of(float drho, float D, float rho0) {
    return D / (rho0 + drho);
}

// F1 / F2: gradient g[3] and normal or stress aux[AUXS] of a ring-1 node from the staged phase field.
template <class S, class PHI>
__device__ __forceinline__ void ring_aux_node(const CaseDev &c, int tipo, PHI phi_at, S *g, S *aux) {
    S g0, g1, g2;
    if constexpr (std::is_same<S, float>::value) {
        // FP32 (both storage forms): the in-plane class forms, g_z = 0 on the slab
        mediator_grad_fold(phi_at, g0, g1);
        g0 = -g0;  // the isotropic gradient
        g1 = -g1;
        g2 = 0.f;
        if (tipo == ITLBM_OP_F1) aux_normal_plane(g0, g1, aux);
        else aux_stress_plane(g0, g1, c.pf.sigma, aux);
    } else {
        iso_grad_at<S>(phi_at, g0, g1, g2);
        if (tipo == ITLBM_OP_F1) aux_normal(g0, g1, g2, aux);
        else aux_stress(g0, g1, g2, (S)c.sigma, aux);
    }
    g[0] = g0;
    g[1] = g1;
    g[2] = g2;
}

// Mediator momentum and class-F force of a node.  phi_at(dx, dy) is the staged phase field around
// it, aux_at(dx, dy) points at the ring-1 auxiliaries (F1 / F2) and g at the node's ring-1 gradient.
template <class S, class PHI, class AUX>
__device__ __forceinline__ void node_force(const CaseDev &c, int tipo, const CaseDev::F32Par &pf, PHI phi_at,
                                           AUX aux_at, const S *g, S &gmx, S &gmy, S &gmz, S &Fx, S &Fy, S &Fz) {
    if constexpr (std::is_same<S, float>::value) {
        if (tipo == ITLBM_OP_F1 || tipo == ITLBM_OP_F2) {  // the ring-1 gradient is its exact negative
            gmx = -g[0];
            gmy = -g[1];
        } else mediator_grad_fold(phi_at, gmx, gmy);  // FP32: class form, g_z = 0 on the slab
        gmz = S(0);
    } else mediator_grad_at<S>(phi_at, gmx, gmy, gmz);
    Fx = S(0);
    Fy = S(0);
    Fz = S(0);
    if (tipo == ITLBM_OP_F1) {
        S kappa;
        if constexpr (std::is_same<S, float>::value) kappa = curvature_plane(aux_at);
        else kappa = curvature_at<S>(aux_at);
        S sig;
        if constexpr (std::is_same<S, float>::value) sig = pf.sigma;
        else sig = c.sigma;
        const S hs = (S(0.5) * sig) * kappa;
        Fx = hs * g[0];
        Fy = hs * g[1];
        Fz = hs * g[2];
    } else if (tipo == ITLBM_OP_F2) {
        if constexpr (std::is_same<S, float>::value) stress_div_plane(aux_at, Fx, Fy);
        else stress_div_at<S>(aux_at, Fx, Fy, Fz);
    } else if (tipo == ITLBM_OP_F3) {
        S g0, g1, g2, mu;
        if constexpr (std::is_same<S, float>::value) {
            g0 = -gmx;  // the isotropic gradient is the exact negative of the mediator momentum
            g1 = -gmy;
            g2 = -gmz;
            mu = chem_pot_fold(phi_at, pf.kf, pf.bf);
        } else {
            iso_grad_at<S>(phi_at, g0, g1, g2);
            mu = chem_pot_at<S>(phi_at, (S)c.kf, (S)c.bf);
        }
        Fx = mu * g0;
        Fy = mu * g1;
        Fz = mu * g2;
    }
}

// What the collision carries from its first part to its second.
template <class S, bool FOLD>
using Recolour = std::conditional_t<std::is_same<S, double>::value, Recolour64, std::conditional_t<FOLD, RecolourFold, Recolour32>>;

// What the collision takes from the node's populations alone (nothing in the fold: with its few moments apart the
// compiler contracts other products of the relaxation in one kernel than in the other).
template <class S, bool FOLD, int NP>
__device__ __forceinline__ void node_moments(const CaseDev::F32Par &pf, const S (&f)[NP], S sa, S sb, Recolour<S, FOLD> &rc) {
    if constexpr (std::is_same<S, double>::value) moments_f64(f, rc);
    else if constexpr (!FOLD) moments_f32(f, sa, sb, pf, rc);
}

// First part of the collision of a node, after node_moments: f (the totals, or their deviations in FP32) relaxed, from the
// colour sums and the force.  rc.skip is set, and f left, when rho <= 1e-30: such a site is streamed
// unchanged (Operadores_tensao.cpp:347).
template <bool FORCE, class S, bool FOLD, int NP>
__device__ __forceinline__ void node_relax(const CaseDev &c, const CaseDev::F32Par &pf, S (&f)[NP], S sa, S sb, S Fx, S Fy,
                                           S Fz, Recolour<S, FOLD> &rc) {
    if constexpr (FOLD) relax_fold<FORCE>(f, sa, sb, Fx, Fy, pf, rc);
    else if constexpr (std::is_same<S, double>::value) relax_f64<FORCE>(f, sa, sb, Fx, Fy, Fz, c, rc);
    else relax_f32<FORCE>(f, sa, Fx, Fy, Fz, pf, rc);
}

// Second part, for a node that is not skipped: perturbation and the recolouring's coefficients.
template <bool FORCE, class S, bool FOLD, int NP>
__device__ __forceinline__ void node_finish(const CaseDev &c, const CaseDev::F32Par &pf, S (&f)[NP], S sa, S gmx, S gmy,
                                            S gmz, Recolour<S, FOLD> &rc) {
    if constexpr (FOLD) finish_fold<FORCE>(f, sa, gmx, gmy, pf, rc);
    else if constexpr (std::is_same<S, double>::value) finish_f64<FORCE>(f, gmx, gmy, gmz, c, rc);
    else finish_f32<FORCE>(f, sa, gmx, gmy, gmz, pf, rc);
}

// The recolouring split: every post-collision plane out through st(plane, value) with the plane a
// compile-time constant: colour 0 (f_R or e) in [0, NP), colour 1 (f_B or d) in [NP, 2 NP).
template <class S, bool FOLD, int NP, class ST>
__device__ __forceinline__ void node_split(const CaseDev::F32Par &pf, const S (&f)[NP], double sbd,
                                           const Recolour<S, FOLD> &rc, ST st) {
    if constexpr (FOLD) {
        double dsum = 0.0;
        sfor<0, 4>([&](auto M) {
            constexpr int K = 2 * decltype(M)::value + 1;
            float dK, dJ;
            split_fold_pair<K>(rc, f[K], f[K + 1], shift_of<kx(K)>(pf), shift_of<kx(K + 1)>(pf), dK, dJ);
            dsum += (double)dK;
            dsum += (double)dJ;
            st(std::integral_constant<int, K>{}, f[K]);
            st(std::integral_constant<int, NK + K>{}, dK);
            st(std::integral_constant<int, K + 1>{}, f[K + 1]);
            st(std::integral_constant<int, NK + K + 1>{}, dJ);
        });
        st(std::integral_constant<int, 0>{}, f[0]);
        st(std::integral_constant<int, NK>{}, (float)(sbd - dsum));
    } else if constexpr (std::is_same<S, double>::value) {
        st(std::integral_constant<int, 0>{}, rc.cR * f[0]);
        st(std::integral_constant<int, NV>{}, rc.cB * f[0]);
        sfor<0, 9>([&](auto M) {
            constexpr int i = 2 * decltype(M)::value + 1;
            double r, b, rj, bj;
            split64_pair<i>(rc, f[i], f[i + 1], r, b, rj, bj);
            st(std::integral_constant<int, i>{}, r);
            st(std::integral_constant<int, NV + i>{}, b);
            st(std::integral_constant<int, i + 1>{}, rj);
            st(std::integral_constant<int, NV + i + 1>{}, bj);
        });
    } else {
        // d_0 is the complement of the moving d_i against the incoming D, both summed in
        // FP64: the d_i are O(w_i rho), so FP32 sums would round by ~1e-8 rho per node and
        // step, coherently over uniform regions, and drift the colour masses (1e-6 in 2000
        // steps); in FP64 the only rounding left is that of d_0 itself.
        double dsum = 0.0;
        sfor<0, 9>([&](auto M) {
            constexpr int i = 2 * decltype(M)::value + 1;
            float di, dj;
            split32_pair<i>(rc, f[i], f[i + 1], shift_of<cx(i)>(pf), shift_of<cx(i + 1)>(pf), di, dj);
            dsum += (double)di;
            dsum += (double)dj;
            st(std::integral_constant<int, i>{}, f[i]);
            st(std::integral_constant<int, NV + i>{}, di);
            st(std::integral_constant<int, i + 1>{}, f[i + 1]);
            st(std::integral_constant<int, NV + i + 1>{}, dj);
        });
        st(std::integral_constant<int, 0>{}, f[0]);
        st(std::integral_constant<int, NV>{}, (float)(sbd - dsum));
    }
}

// Force and mediator gradient of a diagnostic step, kept for the diagnostics.
template <class S>
__device__ __forceinline__ void keep_aux(const CaseDev &c, int x, int y, S Fx, S Fy, S Fz, S gmx, S gmy, S gmz) {
    const long long o = aux_off(c, x, y);
    const long long n = c.aux_stride;
    c.aux[o] = (double)Fx;
    c.aux[n + o] = (double)Fy;
    c.aux[2 * n + o] = (double)Fz;
    c.aux[3 * n + o] = sqrt((double)gmx * gmx + (double)gmy * gmy + (double)gmz * gmz);
}

}  // namespace itlbm
