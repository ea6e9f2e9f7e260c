// SLIC sweep kernels, generic over a model policy M (see physics_fp64.cuh).
//
// One sweep updates every cell once: U_i <- U_i + (dt/dx)(F_{i-1/2} - F_{i+1/2}) with the SLIC interface
// flux F = FORCE(evolve(L-side of right cell), evolve(R-side of left cell)).  The reference evaluates each
// interface flux twice (once per neighbour, Solvers/secondordersolver.cpp:146-161) and the half-step
// evolved edge states four times; here every cell's conserved vector, every evolved edge state and every
// interface flux is computed exactly once per sweep (plus a 1-3 % halo) -- the values are pure functions
// of the same inputs, so the result is unchanged.
//
// X sweep (along the contiguous column index): a block owns LPB row segments of P cells; the stages
// (conserve -> evolve edges -> FORCE -> update) exchange neighbours through shared memory.
// Y sweep (along rows): each thread owns one column and marches down a segment of TY rows keeping a
// sliding window of the stencil in registers; a warp reads 32 consecutive doubles per plane-row.
#pragma once

#include <type_traits>
#include <utility>

#include "exact_div.cuh"
#include "vg_common.cuh"

namespace vg {

// Models whose conversions and fluxes are templates over a division policy (exact_div.cuh) name SHARED_DIV; the others
// divide as the compiler does.
template <class M, class = void>
struct shared_div {
    static constexpr bool value = false;
};
template <class M>
struct shared_div<M, decltype((void)M::SHARED_DIV)> {
    static constexpr bool value = M::SHARED_DIV;
};
// Models compiled once more for p_inf == 0 and no limiter bias (M::Plain) say in which of the two forms they are.
template <class M, class = void>
struct plain_set {
    static constexpr bool value = false;
};
template <class M>
struct plain_set<M, decltype((void)M::PLAIN_SET)> {
    static constexpr bool value = M::PLAIN_SET;
};
// pick: f(M::Plain{}) where the model has that form and the launch's parameters allow it, f(M{}) otherwise; each: f of all forms
template <class M, class = void>
struct plain_form {
    template <class F>
    static auto pick(const SweepArgs&, F f) {
        return f(M{});
    }
    template <class F>
    static void each(F f) {
        f(M{});
    }
};
template <class M>
struct plain_form<M, std::enable_if_t<!plain_set<M>::value && plain_set<typename M::Plain>::value>> {
    template <class F>
    static auto pick(const SweepArgs& a, F f) {
        return a.bias == 0.0 && M::plain(a.params) ? f(typename M::Plain{}) : f(M{});
    }
    template <class F>
    static void each(F f) {
        f(M{});
        f(typename M::Plain{});
    }
};

template <class M, class D>
__device__ __forceinline__ void cons_by(const double* W, const typename M::P& q, double* U, D& dv) {
    if constexpr (shared_div<M>::value) M::cons(W, q, U, dv);
    else M::cons(W, q, U);
}
template <class M, class D>
__device__ __forceinline__ void setcons_by(const double* U, const typename M::P& q, double* W, D& dv) {
    if constexpr (shared_div<M>::value) M::setcons(U, q, W, dv);
    else M::setcons(U, q, W);
}
template <class M, int AXIS, class D>
__device__ __forceinline__ void flux_by(const double* U, const typename M::P& q, double* F, D& dv) {
    if constexpr (shared_div<M>::value) M::template flux<AXIS>(U, q, F, dv);
    else M::template flux<AXIS>(U, q, F);
}

// SlopeLimiters::computeSlopeLimiter (Solvers/slopelimiters.cpp:7-74)
__device__ __forceinline__ double limiter_f64(double r, double w, int id) {
    if (id == 0) {
        if (r < 0.0) return 0.0;
        if (r < 0.5) return 2.0 * r;
        if (r < 1.0) return 1.0;
        return std_min(std_min(r, 2.0 / ((1.0 - w) + ((1.0 + w) * r))), 2.0);
    } else if (id == 1) {
        if (r < 0.0) return 0.0;
        return std_min((2.0 * r) / (1.0 + r), 2.0 / ((1.0 - w) + ((1.0 + w) * r)));
    }
    if (r < 0.0) return 0.0;
    if (r < 1.0) return r;
    return std_min(1.0, 2.0 / ((1.0 - w) + ((1.0 + w) * r)));
}

// The same without branches for |w| <= 1 and a ratio r of nonzero numbers of magnitudes in [1e-5, 2^513): every quotient
// is formed, and the ones that the reference's branch does not reach are not used.  r is compared with 0, 1/2 and 1 by
// its upper word (the constants' lower words are zero).  For r >= 1 the second divisor is at least 2 to within a
// rounding, so xi_R stays below 2 and the reference's outer minimum with 2 cannot bite.
// UNBIASED (w == 0): the divisor is 1 + r exactly as the reference rounds it, both quotients of van Leer's limiter share its
// reciprocal, and xi_R <= 1 <= r for r >= 1 decides the other minima.
template <int ID, bool UNBIASED>
__device__ __forceinline__ double limiter_shared(double r, double w) {
    const int hi = __double2hiint(r);
    const bool low = hi < 0x3ff00000;
    double phi;
    if constexpr (UNBIASED) {
        const double b = 1.0 + r, y = SharedDiv::reciprocal(b);
        const double xi = SharedDiv::quotient(2.0, b, y);
        if constexpr (ID == 0) phi = low ? (hi < 0x3fe00000 ? 2.0 * r : 1.0) : xi;
        else if constexpr (ID == 1) phi = std_min(SharedDiv::quotient(2.0 * r, b, y), xi);
        else phi = low ? r : xi;
    } else {
        const double xi = SharedDiv::known(2.0, (1.0 - w) + ((1.0 + w) * r));
        if constexpr (ID == 0) phi = low ? (hi < 0x3fe00000 ? 2.0 * r : 1.0) : std_min(r, xi);
        else if constexpr (ID == 1) phi = std_min(SharedDiv::known(2.0 * r, 1.0 + r), xi);
        else phi = low ? r : std_min(1.0, xi);
    }
    return hi < 0 ? 0.0 : phi;
}

// |d| < floor5 by the bit patterns (which order as the magnitudes do; a NaN is above): the FP64 pipe is what the sweeps run
// out of
__device__ __forceinline__ double floored(double d, double floor5) {
    const unsigned long long m = (unsigned long long)__double_as_longlong(d) & 0x7fffffffffffffffULL;
    return m < (unsigned long long)__double_as_longlong(floor5) ? floor5 : d;
}

// Edge values u -+ s / 2 of N components, s of SlopeLimiters::computeSlopeVector (Solvers/slopelimiters.cpp:217-246).
// With shared reciprocals the limiter is chosen outside the loop, so that the components' chains of divisions overlap.
template <int ID, int N, bool UNBIASED>
__device__ __forceinline__ void slopes_of(const double* uL, const double* u, const double* uR, const SweepConst& k,
                                          double* s, SharedDiv& dv) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        const double dm = u[i] - uL[i], dp = uR[i] - u[i];
        const double num = floored(dm, k.floor5), den = floored(dp, k.floor5);
        dv.note_below(dm);
        dv.note_below(dp);
        s[i] = ((k.cm * dm) + (k.cp * dp)) * limiter_shared<ID, UNBIASED>(SharedDiv::known(num, den), k.bias);
    }
}
template <int N, bool UNBIASED, bool>
__device__ __forceinline__ void edge_values(const double* uL, const double* u, const double* uR, const SweepConst& k,
                                            double* xl, double* xr, SharedDiv& dv) {
    double s[N];
    if (k.limiter == 0) slopes_of<0, N, UNBIASED>(uL, u, uR, k, s, dv);
    else if (k.limiter == 1) slopes_of<1, N, UNBIASED>(uL, u, uR, k, s, dv);
    else slopes_of<2, N, UNBIASED>(uL, u, uR, k, s, dv);
#pragma unroll
    for (int i = 0; i < N; i++) {
        xl[i] = u[i] - (0.5 * s[i]);
        xr[i] = u[i] + (0.5 * s[i]);
    }
}
// With the compiler's division.
template <int N>
__device__ __forceinline__ void edge_values_ieee(const double* uL, const double* u, const double* uR, const SweepConst& k,
                                                 int limiter, double* xl, double* xr) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        const double dm = u[i] - uL[i], dp = uR[i] - u[i];
        double s = (k.cm * dm) + (k.cp * dp);
        double num = dm, den = dp;
        if (fabs(num) < k.floor5) num = k.floor5;
        if (fabs(den) < k.floor5) den = k.floor5;
        s = s * limiter_f64(num / den, k.bias, limiter);
        xl[i] = u[i] - (0.5 * s);
        xr[i] = u[i] + (0.5 * s);
    }
}
template <int N, bool UNBIASED, bool IN_LOOP>
__device__ __forceinline__ void edge_values(const double* uL, const double* u, const double* uR, const SweepConst& k,
                                            double* xl, double* xr, IeeeDiv&) {
    if (IN_LOOP) edge_values_ieee<N>(uL, u, uR, k, k.limiter, xl, xr);
    else if (k.limiter == 0) edge_values_ieee<N>(uL, u, uR, k, 0, xl, xr);
    else if (k.limiter == 1) edge_values_ieee<N>(uL, u, uR, k, 1, xl, xr);
    else edge_values_ieee<N>(uL, u, uR, k, 2, xl, xr);
}
// whether the branch-free limiter covers this bias
__device__ __forceinline__ bool bias_shared(double w) { return fabs(w) <= 1.0; }

// Solvers::evolveStateByHalf{X,Y}TimeStep for both sides of one cell (Solvers/solvers.cpp:454-466,
// :502-514, :550-565): returns the conserved vectors of the two evolved edge states after the reference's
// primitive round trip (setConservedVariableVector then computeConservedVariableVector).
template <class M, int AXIS, bool IN_LOOP, class D>
__device__ __forceinline__ void evolve_edges_by(const double* uL, const double* u, const double* uR, const SweepConst& k,
                                                const typename M::P& q, double* ua_left_side, double* ua_right_side, D& dv,
                                                bool want_left = true, bool want_right = true) {
    constexpr int NU = M::NU;
    double xl[NU], xr[NU], fl[NU], fr[NU];
    edge_values<NU, plain_set<M>::value, IN_LOOP>(uL, u, uR, k, xl, xr, dv);
    flux_by<M, AXIS>(xl, q, fl, dv);
    flux_by<M, AXIS>(xr, q, fr, dv);
    double a[NU], b[NU];
#pragma unroll
    for (int i = 0; i < NU; i++) {
        double ev = k.half_r * (fl[i] - fr[i]);
        a[i] = xl[i] + ev;
        b[i] = xr[i] + ev;
    }
    double w[M::NW];
    if (want_left) {
        setcons_by<M>(a, q, w, dv);
        cons_by<M>(w, q, ua_left_side, dv);
    }
    if (want_right) {
        setcons_by<M>(b, q, w, dv);
        cons_by<M>(w, q, ua_right_side, dv);
    }
}

// FirstOrderSolver::compute{X,Y}FORCEFlux (Solvers/firstordersolver.cpp:173-230) on the conserved vectors
// of the left state ua and right state ub.
template <class M, int AXIS, class D>
__device__ __forceinline__ void force_flux_by(const double* ua, const double* ub, const SweepConst& k,
                                              const typename M::P& q, double* F, D& dv) {
    constexpr int NU = M::NU;
    double fa[NU], fb[NU], uri[NU], fri[NU];
    flux_by<M, AXIS>(ua, q, fa, dv);
    flux_by<M, AXIS>(ub, q, fb, dv);
#pragma unroll
    for (int i = 0; i < NU; i++) uri[i] = 0.5 * ((ua[i] + ub[i]) + (k.r * (fa[i] - fb[i])));
    flux_by<M, AXIS>(uri, q, fri, dv);
#pragma unroll
    for (int i = 0; i < NU; i++) {
        double lf = 0.5 * ((fa[i] + fb[i]) + (k.rinv * (ua[i] - ub[i])));
        F[i] = 0.5 * (lf + fri[i]);
    }
}

// The stages of a sweep as its kernels call them: the shared-reciprocal form, and again with the compiler's division
// where an operand left the proven range (a call out of line, so that the common path holds no second copy of it).
template <class M, int AXIS>
__device__ __noinline__ void evolve_edges_ieee(const double* in, const SweepConst* k, const typename M::P* q, double* out) {
    IeeeDiv dv;
    evolve_edges_by<M, AXIS, true>(in, in + M::NU, in + 2 * M::NU, *k, *q, out, out + M::NU, dv);
}
template <class M, int AXIS>
__device__ __noinline__ void force_flux_ieee(const double* in, const SweepConst* k, const typename M::P* q, double* F) {
    IeeeDiv dv;
    force_flux_by<M, AXIS>(in, in + M::NU, *k, *q, F, dv);
}
template <class M>
__device__ __noinline__ void cons_ieee(const double* W, const typename M::P* q, double* U) {
    IeeeDiv dv;
    cons_by<M>(W, *q, U, dv);
}
template <class M>
__device__ __noinline__ void setcons_ieee(const double* U, const typename M::P* q, double* W) {
    IeeeDiv dv;
    setcons_by<M>(U, *q, W, dv);
}

// How a sweep with the compiler's division saves registers, in a shape that caps them (CAPPED) or not.  Measured on 2048^2 Euler
// multiphysics (X with 80 registers | Y with 96, 45 rows | Y uncapped, 56 rows) and MHD intermediate (Y, 56 rows), ms:
//   the limiter chosen outside the loop over the components   0.762 | 0.991 | 1.140    1.733
//   chosen for each component (IN_LOOP)                        0.734 | 0.978 | 1.161    1.796
//   outside, and each row fetched one step ahead (AHEAD)             | 1.023 | 1.095    1.803
//   the same, and both edges formed where one is read (BOTH)   0.788 | 1.023 | 1.064    1.786
// So short states (the first model) save all they can where registers are capped and nothing where they are not; longer ones
// have no use for a cap, and gain from the limiter's place alone.
template <class M, bool CAPPED>
struct ieee_form {
    static constexpr bool SHORT = M::NU <= 9;
    static constexpr bool IN_LOOP = SHORT && CAPPED, AHEAD = SHORT && !CAPPED, BOTH = SHORT && !CAPPED;
};

template <class M, int AXIS, bool CAPPED = false>
__device__ __forceinline__ void evolve_edges(const double* uL, const double* u, const double* uR, const SweepConst& k,
                                             const typename M::P& q, double* ua_left_side, double* ua_right_side,
                                             bool want_left = true, bool want_right = true) {
    if constexpr (shared_div<M>::value) {
        SharedDiv dv;
        const bool shared = bias_shared(k.bias);
        if (shared) evolve_edges_by<M, AXIS, false>(uL, u, uR, k, q, ua_left_side, ua_right_side, dv);
        if (!shared || !dv.ok()) {
            constexpr int NU = M::NU;
            double in[3 * NU], out[2 * NU];
            SweepConst kc = k;
            typename M::P qc = q;
#pragma unroll
            for (int i = 0; i < NU; i++) {
                in[i] = uL[i];
                in[NU + i] = u[i];
                in[2 * NU + i] = uR[i];
            }
            evolve_edges_ieee<M, AXIS>(in, &kc, &qc, out);
#pragma unroll
            for (int i = 0; i < NU; i++) {
                ua_left_side[i] = out[i];
                ua_right_side[i] = out[NU + i];
            }
        }
    } else {
        using F = ieee_form<M, CAPPED>;
        IeeeDiv dv;
        evolve_edges_by<M, AXIS, F::IN_LOOP>(uL, u, uR, k, q, ua_left_side, ua_right_side, dv, F::BOTH || want_left,
                                             F::BOTH || want_right);
    }
}

template <class M, int AXIS>
__device__ __forceinline__ void force_flux(const double* ua, const double* ub, const SweepConst& k,
                                           const typename M::P& q, double* F) {
    if constexpr (shared_div<M>::value) {
        SharedDiv dv;
        force_flux_by<M, AXIS>(ua, ub, k, q, F, dv);
        if (!dv.ok()) {
            constexpr int NU = M::NU;
            double in[2 * NU], out[NU];
            SweepConst kc = k;
            typename M::P qc = q;
#pragma unroll
            for (int i = 0; i < NU; i++) {
                in[i] = ua[i];
                in[NU + i] = ub[i];
            }
            force_flux_ieee<M, AXIS>(in, &kc, &qc, out);
#pragma unroll
            for (int i = 0; i < NU; i++) F[i] = out[i];
        }
    } else {
        IeeeDiv dv;
        force_flux_by<M, AXIS>(ua, ub, k, q, F, dv);
    }
}

template <class M>
__device__ __forceinline__ void cons_of(const double* W, const typename M::P& q, double* U) {
    if constexpr (shared_div<M>::value) {
        SharedDiv dv;
        cons_by<M>(W, q, U, dv);
        if (!dv.ok()) {
            double w[M::NW], u[M::NU];
            typename M::P qc = q;
#pragma unroll
            for (int i = 0; i < M::NW; i++) w[i] = W[i];
            cons_ieee<M>(w, &qc, u);
#pragma unroll
            for (int i = 0; i < M::NU; i++) U[i] = u[i];
        }
    } else {
        M::cons(W, q, U);
    }
}

// W holds the cell's own values of the fields that setConservedVariableVector leaves alone
template <class M>
__device__ __forceinline__ void setcons_of(const double* U, const typename M::P& q, double* W) {
    if constexpr (shared_div<M>::value) {
        SharedDiv dv;
        setcons_by<M>(U, q, W, dv);
        if (!dv.ok()) {
            double w[M::NW], u[M::NU];
            typename M::P qc = q;
#pragma unroll
            for (int i = 0; i < M::NU; i++) u[i] = U[i];
#pragma unroll
            for (int i = 0; i < M::NW; i++) w[i] = W[i];
            setcons_ieee<M>(u, &qc, w);
#pragma unroll
            for (int i = 0; i < M::NW; i++) W[i] = w[i];
        }
    } else {
        M::setcons(U, q, W);
    }
}

__device__ __forceinline__ SweepConst sweep_const(const SweepArgs& a, double& ts) {
    SweepConst k;
    if (a.ctrl) {
        ts = a.ctrl->dt * a.dt_scale;
        k.r = a.ctrl->kr[a.kslot];
        k.rinv = a.ctrl->krinv[a.kslot];
        k.half_r = a.ctrl->khalf_r[a.kslot];
    } else {
        ts = a.dt_host * a.dt_scale;
        k.r = a.r_host;
        k.rinv = a.rinv_host;
        k.half_r = a.half_r_host;
    }
    k.cm = 0.5 * (1.0 + a.bias);
    k.cp = 0.5 * (1.0 - a.bias);
    k.bias = a.bias;
    k.floor5 = a.floor5;
    k.limiter = a.limiter;
    return k;
}

template <class M>
__device__ __forceinline__ void load_w(const SweepArgs& a, long idx, double* W) {
#pragma unroll
    for (int v = 0; v < M::NW; v++) W[v] = a.in[v * a.plane + idx];
}

template <class M>
__device__ __forceinline__ void store_w(const SweepArgs& a, long idx, const double* W) {
#pragma unroll
    for (int v = 0; v < M::NW; v++) a.out[v * a.plane + idx] = W[v];
}

// Fields setConservedVariableVector leaves alone keep the cell's own values, as when the reference updates the
// cell object in place (Solvers/firstordersolver.cpp:428-433): HPR's J (planes 14-16) when the material is not
// thermal (HPR/hprstatevector.cpp:78-103), and the HPR two-material models' J when neither material is (planes 14-16
// of the reduced model, HPR/Multiphysics/hprreducedstatevector.cpp:111-152; 13-15 of the intermediate model,
// hprintermediatestatevector.cpp:112-159).  Models with heat flux name its first plane in J_PLANE; a model whose
// materials keep their heat fluxes separately (the HPR multiphysics model) has its own keep_cold.
template <class M, class = void>
struct heat_flux_plane {
    static constexpr int value = -1;
};
template <class M>
struct heat_flux_plane<M, decltype((void)M::J_PLANE)> {
    static constexpr int value = M::J_PLANE;
};
template <class M, class = void>
struct cold_fields {
    __device__ static void keep(const SweepArgs& a, long idx, const typename M::P& q, double* W) {
        constexpr int j0 = heat_flux_plane<M>::value;
        if constexpr (j0 >= 0) {
            if (!q.thermal)
                for (int v = j0; v < j0 + 3; v++) W[v] = a.in[v * a.plane + idx];
        }
    }
};
template <class M>
struct cold_fields<M, decltype((void)&M::keep_cold)> {
    __device__ static void keep(const SweepArgs& a, long idx, const typename M::P& q, double* W) {
        M::keep_cold(a, idx, q, W);
    }
};
template <class M>
__device__ __forceinline__ void keep_fields(const SweepArgs& a, long idx, const typename M::P& q, double* W) {
    cold_fields<M>::keep(a, idx, q, W);
}

// Whether a state of model M must have a positive pressure: models with a positive_pressure(q) member decide
// (HPR: only its gas equation of state); every other model requires it.
template <class M, class = void>
struct pressure_rule {
    __device__ static bool positive(const typename M::P&) { return true; }
};
template <class M>
struct pressure_rule<M, decltype((void)&M::positive_pressure)> {
    __device__ static bool positive(const typename M::P& q) { return M::positive_pressure(q); }
};

// The pressure at or below which a state has no real sound speed: -p_inf for the stiffened-gas models whose
// parameters carry p_inf (c^2 = gamma (p + p_inf) / rho, Euler/eulerequationofstate.cpp:23-29), 0 for the others.
template <class P, class = void>
struct pressure_floor {
    __device__ static double of(const P&) { return 0.0; }
};
template <class P>
struct pressure_floor<P, decltype((void)std::declval<P>().pinf)> {
    __device__ static double of(const P& q) { return -q.pinf; }
};

template <class M>
__device__ __forceinline__ bool bad_state(const double* W, const typename M::P& q) {
    double rho = M::density(W), p = M::pressure(W);
    if (!pressure_rule<M>::positive(q)) return !(rho > 0.0) || !isfinite(rho) || !isfinite(p);
    return !(rho > 0.0) || !(p > pressure_floor<typename M::P>::of(q)) || !isfinite(rho) || !isfinite(p);
}

// The wave speed of a stored cell into the running maximum.  Its quotients and roots are a tenth of an Euler cell's sweep in
// the exact form, and 43 us of a 190 us MHD X sweep in the mixed one (2048^2), so models with a cheap bound (wave_below) form
// it only where the cell may exceed what the accumulator held when the block began.  The maximum stays the same number.
// 4096^2 Euler, 20 steps: 42.6 -> 42.0 ms (mixed 17.7 -> 17.4); 2048^2 MHD, 60 steps: 63.4 -> 62.2 ms (mixed 37.6 -> 36.4).  The
// two-material Euler model's pair of bounds gained nothing (23.4 -> 23.6 ms at 2048^2) and is left out.
template <class M, class = void>
struct has_wave_bound {
    static constexpr bool value = false;
};
template <class M>
struct has_wave_bound<M, decltype((void)&M::wave_below)> {
    static constexpr bool value = true;
};
template <class M>
__device__ __forceinline__ void raise_wave(const double* W, const typename M::P& q, int dims, double floor, double& wave) {
    if constexpr (has_wave_bound<M>::value) {
        if (M::wave_below(W, q, dims, floor)) return;
    }
    const double s = M::wave(W, q, dims);
    if (s > wave) wave = s;
}
// In grids of a few waves of blocks the look at the accumulator is latency for nothing (130 x 97, 100 steps: 1.84 ms without
// it, 1.87 with); from 4096 blocks on most of them begin after others have ended.
template <class M>
__device__ __forceinline__ bool wave_bounded(const SweepArgs& a) {
    return has_wave_bound<M>::value && a.accumulate_wave && (unsigned)(gridDim.x * gridDim.y) >= 4096u;
}
// the accumulator's value so far, read past L1 (other blocks raise it), in one thread of the block
__device__ __forceinline__ double wave_so_far(const SweepArgs& a, bool bounded) {
    return bounded && threadIdx.x == 0 ? __longlong_as_double((long long)__ldcg(a.wave_acc)) : 0.0;
}

// ----------------------------------------------------------------------------------------- X sweep
template <class M, int P, int LPB, int MINB>
__global__ void __launch_bounds__(P* LPB, MINB) sweep_x_kernel(SweepArgs a) {
    constexpr int NU = M::NU, NW = M::NW;
    constexpr int NT = P * LPB;
    __shared__ double Us[NU][LPB][P + 2];
    __shared__ double Es[NU][LPB][P];
    __shared__ double Fs[NU][LPB][P];
    __shared__ double wave_floor;

    const int p = threadIdx.x % P, l = threadIdx.x / P;
    const int row = blockIdx.y * LPB + l;
    const int len = a.nx;
    const int s0 = blockIdx.x * (P - 2);           // first output cell of this segment
    const int cell = s0 - 1 + p;                   // cell owned by this thread (halo at p = 0, P-1)
    const bool row_ok = row < a.ny;
    const bool out_ok = row_ok && p >= 1 && p <= P - 2 && cell < len;
    const long rowbase = (long)(row_ok ? row : 0) * a.pitch;

    if (a.ctrl && !a.ctrl->active) {               // step past the end: carry the state over unchanged
        if (out_ok)
            for (int v = 0; v < NW; v++) a.out[v * a.plane + rowbase + cell] = a.in[v * a.plane + rowbase + cell];
        return;
    }
    double ts;
    const SweepConst k = sweep_const(a, ts);
    const typename M::P q = M::params(a.params, a.ctrl ? a.ctrl->ch : a.ch_host);

    const bool bounded = wave_bounded<M>(a);
    const double so_far = wave_so_far(a, bounded);
    // stage 1: conserved vectors of cells s0-2 .. s0+P-1 (slot = cell - s0 + 2)
    auto conserve = [&](int slot) {
        int c = ghost_index(s0 - 2 + slot, len, a.periodic);
        double W[NW], U[NU];
        load_w<M>(a, rowbase + c, W);
        cons_of<M>(W, q, U);
#pragma unroll
        for (int v = 0; v < NU; v++) Us[v][l][slot] = U[v];
    };
    conserve(p + 1);
    if (p == 0) conserve(0);
    if (p == P - 1) conserve(P + 1);
    if (threadIdx.x == 0) wave_floor = so_far;
    __syncthreads();

    // stage 2: evolved edge states of the owned cell
    double ub[NU];  // conserved left-side edge state of the owned cell (right state of interface cell-1/2)
    {
        double uL[NU], u[NU], uR[NU], ua[NU];
#pragma unroll
        for (int v = 0; v < NU; v++) {
            uL[v] = Us[v][l][p];
            u[v] = Us[v][l][p + 1];
            uR[v] = Us[v][l][p + 2];
        }
        evolve_edges<M, 0, (MINB > 1)>(uL, u, uR, k, q, ub, ua, p >= 1, p <= P - 2);
#pragma unroll
        for (int v = 0; v < NU; v++) Es[v][l][p] = ua[v];
    }
    __syncthreads();

    // stage 3: FORCE flux at the interface left of the owned cell
    if (p >= 1) {
        double ua[NU], F[NU];
#pragma unroll
        for (int v = 0; v < NU; v++) ua[v] = Es[v][l][p - 1];
        force_flux<M, 0>(ua, ub, k, q, F);
#pragma unroll
        for (int v = 0; v < NU; v++) Fs[v][l][p] = F[v];
    }
    __syncthreads();

    // stage 4: conservative update (FirstOrderSolver::computeFORCEUpdate, Solvers/firstordersolver.cpp:428-433)
    double wave = 0.0;
    if (out_ok) {
        double Un[NU], W[NW];
#pragma unroll
        for (int v = 0; v < NU; v++) Un[v] = Us[v][l][p + 1] + (k.r * (Fs[v][l][p] - Fs[v][l][p + 1]));
        keep_fields<M>(a, rowbase + cell, q, W);
        setcons_of<M>(Un, q, W);
        store_w<M>(a, rowbase + cell, W);
        if (bad_state<M>(W, q)) atomicOr(a.err, ERR_STATE);
        if (a.accumulate_wave) raise_wave<M>(W, q, a.dims, wave_floor, wave);
    }
    if (a.accumulate_wave) block_max_to<NT>(wave, a.wave_acc, bounded);
    if (a.advance_time && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        a.ctrl->t += a.ctrl->dt;
        a.ctrl->it += 1;
    }
}

// ----------------------------------------------------------------------------------------- Y sweep
template <class M, int TX, int TY, int MINB>
__global__ void __launch_bounds__(TX, MINB) sweep_y_kernel(SweepArgs a) {
    constexpr int NU = M::NU, NW = M::NW;
    const int col = blockIdx.x * TX + threadIdx.x;
    const bool col_ok = col < a.nx;
    const int len = a.ny;
    const int ty = a.ty_rows > 0 ? a.ty_rows : TY;
    const int r0 = blockIdx.y * ty;
    const int r1 = min(r0 + ty, len);
    const int c = col_ok ? col : 0;

    if (a.ctrl && !a.ctrl->active) {
        if (col_ok)
            for (int r = r0; r < r1; r++)
                for (int v = 0; v < NW; v++) a.out[v * a.plane + (long)r * a.pitch + c] = a.in[v * a.plane + (long)r * a.pitch + c];
        return;
    }
    double ts;
    const SweepConst k = sweep_const(a, ts);
    const typename M::P q = M::params(a.params, a.ctrl ? a.ctrl->ch : a.ch_host);

    auto conserve = [&](int r, double* U) {
        int rr = ghost_index(r, len, a.periodic);
        double W[NW];
        load_w<M>(a, (long)rr * a.pitch + c, W);
        cons_of<M>(W, q, U);
    };

    constexpr bool CAPPED = MINB > 1;
    constexpr bool AHEAD = shared_div<M>::value || ieee_form<M, CAPPED>::AHEAD;  // each row is fetched one step ahead of its use
    double um1[NU], u0[NU], up1[NU], ua_prev[NU], f_prev[NU], dummy[NU], next[AHEAD ? NW : 1];
    double wave = 0.0;
    auto fetch = [&](int r) {
        if constexpr (AHEAD) load_w<M>(a, (long)ghost_index(r, len, a.periodic) * a.pitch + c, next);
    };
    conserve(r0 - 2, up1);   // temporarily holds row r0-2
    conserve(r0 - 1, um1);
    conserve(r0, u0);
    fetch(r0 + 1);
    evolve_edges<M, 1, CAPPED>(up1, um1, u0, k, q, dummy, ua_prev, false, true);   // right edge of row r0-1
    for (int r = r0; r <= r1; r++) {
        if constexpr (AHEAD) cons_of<M>(next, q, up1);
        else conserve(r + 1, up1);
        fetch(r + 2);
        double ub[NU], ua_next[NU];
        evolve_edges<M, 1, CAPPED>(um1, u0, up1, k, q, ub, ua_next, true, r < r1);
        double F[NU];
        force_flux<M, 1>(ua_prev, ub, k, q, F);     // flux at r - 1/2
        if (r > r0 && col_ok) {                      // update row r-1 with fluxes at r-3/2 and r-1/2
            double Un[NU], W[NW];
#pragma unroll
            for (int v = 0; v < NU; v++) Un[v] = um1[v] + (k.r * (f_prev[v] - F[v]));
            keep_fields<M>(a, (long)(r - 1) * a.pitch + c, q, W);
            setcons_of<M>(Un, q, W);
            store_w<M>(a, (long)(r - 1) * a.pitch + c, W);
            if (bad_state<M>(W, q)) atomicOr(a.err, ERR_STATE);
            if (a.accumulate_wave) {
                double s = M::wave(W, q, 2);
                if (s > wave) wave = s;
            }
        }
#pragma unroll
        for (int v = 0; v < NU; v++) {
            f_prev[v] = F[v];
            ua_prev[v] = ua_next[v];
            um1[v] = u0[v];
            u0[v] = up1[v];
        }
    }
    if (a.accumulate_wave) block_max_to<TX>(wave, a.wave_acc);
    if (a.advance_time && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        a.ctrl->t += a.ctrl->dt;
        a.ctrl->it += 1;
    }
}

// ------------------------------------------------------------------------------- CFL and time step
// Maximum wave speed of the current state into ctrl->smax_next (grid-stride, block reduce, one atomic per
// block; the maximum of exact values does not depend on the order, unlike the reference's racy OpenMP max).
template <class M, int NT>
__global__ void __launch_bounds__(NT) max_wave_kernel(const double* __restrict__ in, long plane, long pitch, int nx, int ny,
                                                      Ctrl* ctrl, SweepArgs a) {
    const typename M::P q = M::params(a.params, 0.0);
    double best = 0.0;
    long n = (long)nx * ny;
    for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) {
        long r = i / nx, cidx = i - r * nx;
        double W[M::NW];
#pragma unroll
        for (int v = 0; v < M::NW; v++) W[v] = in[v * plane + r * pitch + cidx];
        double s = M::wave(W, q, a.dims);
        if (s > best) best = s;
    }
    block_max_to<NT>(best, &ctrl->smax_next);
}

// Solvers::computeStableTimeStep{,2D} (Solvers/solvers.cpp:388-452): dt = CFL * (dx / S), x0.2 for the first six
// steps, clamped to t_end.  In 2D S also covers the default-constructed corner ghosts of insertBoundaryCells2D
// (Solvers/solvers.cpp:92).  For MHD, c_h = S for this step (Solvers/mhdsecondordersolver.cpp:513-515).
template <class M>
__global__ void step_begin_kernel(Ctrl* c, SweepArgs a) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int it = c->it;
    int active = (c->t < c->t_end) && (it < c->max_steps);
    c->active = active;
    double S = __longlong_as_double((long long)c->smax_next);
    if (c->dims == 2) {
        double W[M::NW];
        M::default_state(W);
        const typename M::P q = M::params(a.params, 0.0);
        double sd = M::wave(W, q, 2);
        if (sd > S) S = sd;
    }
    if (active) {
        double dt = c->cfl * (c->dx / S);
        if (it <= 5) dt *= 0.2;
        if ((c->t + dt) > c->t_end) dt = c->t_end - c->t;
        c->dt = dt;
        c->ch = a.ch_fixed ? a.ch_host : S;
        for (int i = 0; i < 2; i++) {
            sweep_scale(dt * (i == 0 ? 0.5 : 1.0), c->dx, c->kr[i], c->krinv[i], c->khalf_r[i]);
            c->kr_f[i] = (float)c->kr[i];
            c->krinv_f[i] = (float)c->krinv[i];
            c->khalf_r_f[i] = (float)c->khalf_r[i];
        }
    }
    c->smax_next = 0ull;
}

// Copy of the host-visible result of vg_max_wave_speed: S including corner ghosts.
template <class M>
__global__ void max_wave_finish_kernel(Ctrl* c, SweepArgs a, double* out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double S = __longlong_as_double((long long)c->smax_next);
    if (c->dims == 2) {
        double W[M::NW];
        M::default_state(W);
        const typename M::P q = M::params(a.params, 0.0);
        double sd = M::wave(W, q, 2);
        if (sd > S) S = sd;
    }
    *out = S;
}

}  // namespace vg
