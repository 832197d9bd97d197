// heat.cu — P5, the implicit flux-limited radiative diffusion step (crates/sr-physics/src/reference/heat.rs:453-592).
//
// One backward-Euler step in the heat potential u = a_r T⁴ with the Levermore–Pomraning law frozen at the pass start.
// Newton passes linearise T(u); each pass is one SPD 5-point system A u = b, solved here by iterative refinement:
// the residual r = b - A x and the update x += s e in FP64 (s the residual's rms scale), the correction from an FP32
// preconditioned CG on A e = r/s with FP64 dot products, preconditioned by the FP32 multigrid V-cycle (mg.cu) or
// Jacobi. The passes stop by the reference's two rules (the heat moved, the largest cell change); the commit closes the
// heat balance with δ (heat.rs:521-536), or past the ceiling commits by limited fluxes (heat.rs:545-592).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <vector>

#include "heat.cuh"
#include "learned.cuh"
#include "mg.cuh"
#include "reduce.cuh"

namespace {

constexpr int RED_THREADS = 256;
constexpr double kFirstPassTol = 0.1;  // the first Newton pass's relative residual (and the loosest any pass asks)
constexpr double kTrustedPassTol = 1e-5;  // passes this loose end on their FP32 solve's own test
constexpr int kMaxRefinements = 16;    // FP64 refinement sweeps per Newton pass
constexpr int MAX_PART = 1184;    // most CTAs of a grid-stride heat kernel: one wave (148 SMs x 8), few partials to sum
constexpr int PART_CAP = 148 * 16;  // partials per reduced value (the learned preconditioner's grids are the largest)
// Device scalars. The kernels read Δt, the refinement's scale, δ and the PCG round's state from here (never from
// launch arguments), so a captured graph of the implicit step replays for any step. The fused MG/Jacobi rounds keep
// <r, z> of this round (S_RZN, from the preconditioner application that opens it) and of the last (S_RZP), and which
// direction buffer is current (S_PAR); the flexible (learned) rounds use S_RZ0/S_RZ1.
enum Slot { S_HEAT0, S_NGAS, S_DT, S_RR, S_BB, S_GAM, S_HM, S_MOVED, S_VIOL, S_UB, S_TB, S_R32, S_PQ, S_RRI, S_RZ0, S_RZ1,
            S_ZRO, S_MGRZ, S_BETA, S_RAD, S_GAIN, S_HELD, S_RZP, S_RZN, S_PAR, S_SCALE, S_ISCALE, S_DELTA,
            S_COUNT };

// Where a kernel's grid sum goes: the partials buffer, the ticket counter and the device scalar(s).
struct Red {
    double* part;
    unsigned* counter;
    double* out;
};

struct HeatConst {
    int w, h;
    double gm1, mu, t_floor, sigma_vac, sigma_floor, a_r, c_sb, kappa0, k_cond, chi;
    int limiter_on;
    int ref;  // reference mode: the sides of heat_cells_kernel's reference branch (C = Σ/μ of each cell)
};

// ---- the implicit step under device control (MG and Jacobi preconditioners)
//
// The host-driven step (heat_step's Newton loop, solve_pass's FP64 refinement, inner_pcg's rounds) decides from
// read-back scalars. Here the same decisions are taken on the device, inside one captured CUDA graph, and steer its
// conditional nodes: an IF around the step (no gas, pinned temperature or Δt <= 0 leave only the fluxes), a WHILE over
// the refinements of all Newton passes (an FP64 residual, an inner solve, and after a pass's last the Newton update), a
// WHILE over an inner solve's PCG rounds (the residual tested after every round: no host round trip, no predicted
// cadence), an IF around a new system's coarsening, and IFs choosing the commit. Entering a body costs 4 to 8 us, more
// than most of its kernels, so a kernel that may have nothing to do this time (the inner solve's scaling and correction,
// the Newton update) reads that and leaves instead of having a body of its own (a WHILE of passes around a WHILE of
// refinements, an IF around each inner solve and each Newton update: 2048², three steps, 30.5 -> 29.9 ms). A decision is
// taken by the thread that has just written the sums it reads, the last CTA's of the kernel whose grid sum it is
// (ctl_run): decisions in one-thread kernels of their own cost 3.5 us each with their launch gap, 250 of them in three
// 2048² steps and 1,050 in four 512² reference-mode steps. No launch argument changes from step to step: Δt, the scale, δ
// and the round state live in the device scalars.

// The graph's conditional bodies.
enum CtlBody { B_MAIN, B_SKIP, B_LOOP, B_ROUND, B_COARSEN, B_CONV, B_LIM, B_COUNT };

struct HeatCtl {
    // configuration (host-written)
    double tol, nheat, ncell, inner_floor;
    int max_passes, max_rounds, pin;
    // the step
    double heat0, n_gas;
    double dt;  // the Δt it covers; 0 where there was nothing to solve
    int passes, rounds, refinements, converged, ok;
    double pass_tol, moved_prev, rel;
    // the pass's refinement and its inner solve
    int ref, reached, it, max_it;
    double prev, eta, rr0;
    int newton;  // the loop body's Newton update has work this time
    // the commit
    double delta, radiated;
    // how often each body ran since the host last counted (for the launch count)
    unsigned long long runs[B_COUNT];
};

struct CtlHandles {
    cudaGraphConditionalHandle h[B_COUNT];
};

// A kernel's part in the control: the block (null: the host decides), the step's Δt and the conditional handles.
struct Ctl {
    HeatCtl* c;
    const double* dt;
    CtlHandles hd;
};

enum CtlPhase { C_BEGIN, C_NEWTON_BEGIN, C_REFINE, C_INNER_BEGIN, C_ROUND, C_NEWTON, C_DELTA, C_LIMITED };

__device__ __forceinline__ void ctl_set(const Ctl& k, int body, bool on, bool count_entry) {
    cudaGraphSetConditional(k.hd.h[body], on ? 1u : 0u);
    if (on && count_entry) k.c->runs[body]++;
}

// The commit follows: the converged one, or past the ceiling (or a breakdown) the limited one.
__device__ __forceinline__ void ctl_commit(const Ctl& k) {
    ctl_set(k, B_CONV, k.c->converged != 0, true);
    ctl_set(k, B_LIM, !k.c->converged, true);
}

__device__ __forceinline__ void ctl_pass_begin(const Ctl& k) {
    k.c->passes++;
    k.c->ref = 0;
    k.c->prev = INFINITY;
    ctl_set(k, B_LOOP, true, false);
}

// The pass's solve is done: its Newton update, unless the solve broke down.
__device__ __forceinline__ void ctl_refine_end(const Ctl& k) {
    k.c->newton = k.c->ok;
    if (!k.c->ok) {
        ctl_set(k, B_LOOP, false, false);
        ctl_commit(k);
    }
}

// The inner solve is done (its correction x += scale e follows).
__device__ __forceinline__ void ctl_inner_end(const Ctl& k) {
    HeatCtl* c = k.c;
    bool more = c->ok != 0;
    if (c->ok) {
        c->rounds += c->it;
        c->refinements++;
        // an intermediate pass (its tolerance far above the FP32 solve's floor) trusts the solve that reached its
        // reduction; the final pass is always verified by another FP64 residual
        if (c->reached && c->pass_tol >= kTrustedPassTol) {
            c->rel *= c->eta;
            more = false;
        }
    }
    if (++c->ref >= kMaxRefinements) more = false;
    if (more) ctl_set(k, B_LOOP, true, false);
    else ctl_refine_end(k);
}

// One decision, by one thread, after the sums it reads are in the scalars.
__device__ __noinline__ void ctl_run(const Ctl& k, double* scal, int phase) {
    HeatCtl* c = k.c;
    switch (phase) {
        case C_BEGIN: {  // after Σ C T⁰ and the gas cells
            scal[S_DT] = *k.dt;
            c->heat0 = scal[S_HEAT0];
            c->n_gas = scal[S_NGAS];
            const bool skip = c->pin || c->n_gas == 0.0 || !(scal[S_DT] > 0.0);
            c->dt = skip ? 0.0 : scal[S_DT];
            c->passes = c->rounds = c->refinements = 0;
            c->converged = skip ? 1 : 0;
            c->ok = 1;
            c->rel = c->delta = c->radiated = 0.0;
            ctl_set(k, B_MAIN, !skip, true);
            ctl_set(k, B_SKIP, skip, true);
            break;
        }
        case C_NEWTON_BEGIN: {  // after the first system (its two bounds in S_UB, S_TB)
            c->pass_tol = fmax(c->tol, kFirstPassTol);
            c->moved_prev = 0.0;
            const bool go = c->max_passes > 0 && c->max_rounds > 0;
            ctl_set(k, B_COARSEN, go, true);
            ctl_set(k, B_LOOP, go, false);
            if (go) ctl_pass_begin(k);
            else ctl_commit(k);
            break;
        }
        case C_REFINE: {  // after the FP64 residual: stop, or scale the residual for an inner solve
            c->runs[B_LOOP]++;
            c->newton = 0;
            const double rr = scal[S_RR], bb = scal[S_BB], gam = scal[S_GAM], hm = scal[S_HM];
            bool go = false;
            if (!isfinite(rr) || !isfinite(bb) || !isfinite(gam) || !isfinite(hm)) {
                c->ok = 0;
            } else {
                c->rel = bb > 0.0 ? sqrt(rr / bb) : 0.0;
                const double tol = c->pass_tol, ub = scal[S_UB], tb = scal[S_TB];
                double worst = c->rel / tol;
                if (ub > 0.0) worst = fmax(worst, sqrt(gam / ub) / tol);
                if (tb > 0.0) worst = fmax(worst, sqrt(hm / tb) / tol);
                if (!(worst <= 1.0 || rr == 0.0) && !(worst > 0.5 * c->prev) && c->rounds < c->max_rounds) {
                    c->prev = worst;
                    const double scale = sqrt(rr / fmax(1.0, c->n_gas));
                    scal[S_SCALE] = scale;
                    scal[S_ISCALE] = 1.0 / scale;
                    c->eta = fmin(0.5, fmax(c->inner_floor, 0.5 / worst));
                    c->max_it = c->max_rounds - c->rounds;
                    go = true;
                }
            }
            if (!go) {
                scal[S_SCALE] = scal[S_ISCALE] = 0.0;
                ctl_set(k, B_ROUND, false, false);
                ctl_refine_end(k);
            }
            break;
        }
        case C_INNER_BEGIN: {  // after the scaled residual
            ctl_set(k, B_COARSEN, false, true);  // this pass's is done
            scal[S_BETA] = 0.0;
            scal[S_PAR] = 0.0;
            c->rr0 = scal[S_R32];
            c->it = 0;
            c->reached = 0;
            const bool go = c->rr0 > 0.0 && c->max_it > 0;
            ctl_set(k, B_ROUND, go, false);
            if (!go) ctl_inner_end(k);
            break;
        }
        case C_ROUND: {  // after a round: rotate its state, test the residual
            c->runs[B_ROUND]++;
            c->it++;
            scal[S_RZP] = scal[S_RZN];
            scal[S_BETA] = 1.0;
            scal[S_PAR] = scal[S_PAR] != 0.0 ? 0.0 : 1.0;
            const double pq = scal[S_PQ], rr = scal[S_RRI];
            bool more = true;
            if (!(pq > 0.0) || !isfinite(pq) || !isfinite(rr)) {
                c->ok = 0;  // a breakdown: the solve's correction is dropped
                scal[S_SCALE] = 0.0;
                more = false;
            } else if (rr <= c->eta * c->eta * c->rr0) {
                c->reached = 1;
                more = false;
            } else if (c->it >= c->max_it) {
                more = false;
            }
            ctl_set(k, B_ROUND, more, false);
            if (!more) ctl_inner_end(k);
            break;
        }
        case C_NEWTON: {  // after the update and the next system: stop, or the next pass's tolerance and coarsening
            const double rel_moved = c->heat0 > 0.0 ? scal[S_MOVED] / c->heat0 : 0.0;
            bool more;
            if (rel_moved <= c->nheat && scal[S_VIOL] == 0.0 && c->pass_tol <= c->tol) {
                c->converged = 1;
                more = false;
            } else {
                // the next pass is solved to tol once it is expected to move less than nheat (the passes' observed
                // contraction times this pass's move), since only a pass solved to tol can end them
                const double ratio = c->moved_prev > 0.0 ? fmin(1.0, fmax(0.01, rel_moved / c->moved_prev)) : 0.1;
                c->moved_prev = rel_moved;
                c->pass_tol = fmax(c->tol, fmin(kFirstPassTol, rel_moved));
                if (ratio * rel_moved <= c->nheat) c->pass_tol = c->tol;
                more = c->passes < c->max_passes && c->rounds < c->max_rounds;
            }
            ctl_set(k, B_COARSEN, more, true);
            ctl_set(k, B_LOOP, more, false);
            if (more) ctl_pass_begin(k);
            else ctl_commit(k);
            break;
        }
        case C_DELTA: {  // after the commit's sums (heat.rs:521-531)
            const double rad = scal[S_RAD], gain = scal[S_GAIN], held = scal[S_HELD];
            c->delta = -(gain + rad) / held;
            c->radiated = rad;
            scal[S_DELTA] = c->delta;
            break;
        }
        case C_LIMITED:
            c->radiated = scal[S_RAD];
            break;
    }
}

__device__ __forceinline__ double u_of(const HeatConst& K, double t) {
    return K.chi > 0.0 ? t : K.a_r * ((t * t) * (t * t));
}
__device__ __forceinline__ double t_of(const HeatConst& K, double u) {
    return K.chi > 0.0 ? u : sqrt(sqrt(u / K.a_r));
}
__device__ __forceinline__ double dt_du(const HeatConst& K, double t) {
    return K.chi > 0.0 ? 1.0 : 1.0 / (4.0 * K.a_r * ((t * t) * t));
}

// eos.rs:118-131 in f64 on the device tables (u at the node, Δ ln u to the next): u(x) = u_i exp(frac Δ_i)
__device__ __forceinline__ double cold_u64(const float* u, const float* d, double x) {
    if (!(x > 0.0)) return 0.0;
    const double pos = (log(x) + 18.420680743952367) * (511.0 / 36.841361487904734);
    if (pos < 0.0) {
        const double r = x * 1e8;
        return (double)u[0] * r * r;
    }
    int i = (int)pos;
    i = i > 510 ? 510 : i;
    return (double)u[i] * exp((pos - (double)i) * (double)d[i]);
}

// ---- step set-up: the sides (heat.rs:215-226), the faces' D_f (heat.rs:263-294), Σ_f k over the vacuum faces
__global__ void heat_cells_kernel(HeatConst K, HeatRef RF, const float* __restrict__ U, const float* __restrict__ kappa,
                                  uint8_t* gas, double* t0, double* C, float* kap, float* sig, double* t, Red R,
                                  const __grid_constant__ Ctl ctl) {
    const size_t n = (size_t)K.w * K.h;
    double acc = 0.0, ngas = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double s = U[i];
        if (RF.on) {
            // reference/heat.rs:215-231 with the registry's composition (registry.rs:145-154)
            const double za[10] = {2.0, 0.75, 7.0 / 12.0, 9.0 / 16.0, 11.0 / 20.0, 13.0 / 24.0, 15.0 / 28.0,
                                   17.0 / 32.0, 27.0 / 56.0, 1.0};
            const double ze[10] = {1.0, 0.5, 0.5, 0.5, 0.5, 0.5, 0.5, 0.5, 26.0 / 56.0, 0.0};
            double inv_mu = 0.0, ye = 0.0, x0 = 0.0, x1 = 0.0, xn = 0.0;
            for (int k = 0; k < 10; k++) {
                const double x = U[(4 + k) * n + i];
                inv_mu += x * za[k];
                ye += x * ze[k];
                if (k == 0) x0 = x;
                if (k == 1) x1 = x;
                if (k == 9) xn = x;
            }
            const double mu = 1.0 / inv_mu, z_met = 1.0 - x0 - x1 - xn;
            double T;
            const bool g = s >= K.sigma_vac;
            if (!g) {
                T = K.t_floor;
            } else {
                const double mx = U[n + i], my = U[2 * n + i], e = U[3 * n + i];
                double cold = 0.0;
                if (RF.cold_e) cold += cold_u64(RF.table, RF.table + 512, ye * s);
                if (RF.cold_n) cold += cold_u64(RF.table + 1024, RF.table + 1536, xn * s);
                const double raw = e / s - 0.5 * (mx * mx + my * my) / (s * s) - cold / s;
                const double floor = K.t_floor / mu;
                T = mu * (raw < floor ? floor : raw);
            }
            kap[i] = (float)(K.kappa0 * (1.0 + x0) + (T < RF.t_dust ? RF.kappa_dust * z_met : 0.0));
            gas[i] = g ? 1 : 0;
            t0[i] = T;
            sig[i] = g ? (float)s : (float)K.sigma_floor;
            C[i] = (g ? s : K.sigma_floor) * inv_mu;
            t[i] = T;
            if (g) {
                acc += C[i] * T;
                ngas += 1.0;
            }
            continue;
        }
        const float k = kappa ? kappa[i] : (float)K.kappa0;
        kap[i] = k;
        if (s < K.sigma_vac) {
            gas[i] = 0;
            t0[i] = K.t_floor;
            sig[i] = (float)K.sigma_floor;
            C[i] = K.sigma_floor / (K.mu * K.gm1);
            t[i] = K.t_floor;
            continue;
        }
        const double mx = U[n + i], my = U[2 * n + i], e = U[3 * n + i];
        const double kinetic = 0.5 * (mx * mx + my * my) / (s * s);
        const double raw = e / s - kinetic;
        const double floor = K.t_floor / K.mu / K.gm1;
        const double eps = raw < floor ? floor : raw;
        const double T = K.mu * K.gm1 * eps;
        gas[i] = 1;
        t0[i] = T;
        sig[i] = (float)s;
        C[i] = s / (K.mu * K.gm1);
        t[i] = T;
        acc += C[i] * T;
        ngas += 1.0;
    }
    const double v[2] = {acc, ngas};
    const bool last = grid_sum_last<2>(v, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_HEAT0, C_BEGIN);
}

struct Side {
    bool gas;
    double t, s, kappa, c;
};

__device__ __forceinline__ Side side_at(const HeatConst& K, const uint8_t* gas, const double* t0, const float* kap,
                                        const float* sig, const double* C, size_t i) {
    Side o;
    o.gas = gas[i];
    o.t = t0[i];
    o.s = sig[i];
    o.kappa = kap[i];
    o.c = C[i];
    return o;
}

__device__ __forceinline__ Side vacuum_beyond(const HeatConst& K, const Side& g) {
    Side o;
    o.gas = false;
    o.t = K.t_floor;
    o.s = K.sigma_floor;
    o.kappa = g.kappa;
    o.c = K.ref ? K.sigma_floor * (g.c / g.s) : K.sigma_floor / (K.mu * K.gm1);  // the gas side's μ
    return o;
}

__device__ __forceinline__ double diffusivity(const HeatConst& K, const Side& a, const Side& b) {
    if (!a.gas && !b.gas) return 0.0;
    if (K.chi > 0.0) return K.chi * (0.5 * (a.c + b.c));
    const double ta2 = a.t * a.t, tb2 = b.t * b.t;
    const double era = K.a_r * (ta2 * ta2), erb = K.a_r * (tb2 * tb2);
    const double face_er = 0.5 * (era + erb);
    const double ks = 0.5 * (a.kappa * a.s + b.kappa * b.s);
    const double r = face_er > 0.0 ? fabs(erb - era) / (ks * face_er) : 0.0;
    const double lam = K.limiter_on ? (2.0 + r) / (6.0 + 3.0 * r + r * r) : 1.0 / 3.0;
    const double radiative = K.c_sb * lam / ks;
    const double conduction =
        K.k_cond != 0.0 ? K.k_cond / (K.a_r * (a.t + b.t) * (a.t * a.t + b.t * b.t)) : 0.0;
    return radiative + conduction;
}

__device__ __forceinline__ double face_coef(const HeatConst& K, const Side* a, const Side* b) {
    Side A, B;
    if (a && b) {
        if (a->gas || b->gas) {
            A = a->gas ? *a : vacuum_beyond(K, *b);
            B = b->gas ? *b : vacuum_beyond(K, *a);
        } else {
            A = *a;
            B = *a;
        }
    } else if (a) {
        A = *a;
        B = vacuum_beyond(K, *a);
    } else {
        A = vacuum_beyond(K, *b);
        B = *b;
    }
    return diffusivity(K, A, B);
}

__global__ void heat_faces_kernel(HeatConst K, const uint8_t* __restrict__ gas, const double* __restrict__ t0,
                                  const float* __restrict__ kap, const float* __restrict__ sig,
                                  const double* __restrict__ C, double* kx, double* ky) {
    const int w = K.w, h = K.h;
    const size_t nx = (size_t)(w + 1) * h, ny = (size_t)w * (h + 1);
    for (size_t f = (size_t)blockIdx.x * blockDim.x + threadIdx.x; f < nx + ny; f += (size_t)gridDim.x * blockDim.x) {
        Side a, b;
        bool ha, hb;
        if (f < nx) {
            int x, y;
            split_index(f, (w + 1), x, y);
            ha = x > 0;
            hb = x < w;
            if (ha) a = side_at(K, gas, t0, kap, sig, C, (size_t)y * w + x - 1);
            if (hb) b = side_at(K, gas, t0, kap, sig, C, (size_t)y * w + x);
            kx[f] = face_coef(K, ha ? &a : nullptr, hb ? &b : nullptr);
        } else {
            const size_t g = f - nx;
            int x, y;
            split_index(g, w, x, y);
            ha = y > 0;
            hb = y < h;
            if (ha) a = side_at(K, gas, t0, kap, sig, C, (size_t)(y - 1) * w + x);
            if (hb) b = side_at(K, gas, t0, kap, sig, C, (size_t)y * w + x);
            ky[g] = face_coef(K, ha ? &a : nullptr, hb ? &b : nullptr);
        }
    }
}

__global__ void heat_ksum_kernel(HeatConst K, const uint8_t* __restrict__ gas, const double* __restrict__ kx,
                                 const double* __restrict__ ky, double* kvac) {
    const int w = K.w, h = K.h;
    const size_t n = (size_t)w * h;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!gas[i]) {
            kvac[i] = 0.0;
            continue;
        }
        int x, y;
        split_index(i, w, x, y);
        const double k[4] = {kx[(size_t)y * (w + 1) + x], kx[(size_t)y * (w + 1) + x + 1], ky[(size_t)y * w + x],
                             ky[(size_t)(y + 1) * w + x]};
        const bool nb[4] = {x > 0 && gas[i - 1], x + 1 < w && gas[i + 1], y > 0 && gas[i - w],
                            y + 1 < h && gas[i + w]};
        double v = 0.0;
        for (int f = 0; f < 4; f++)
            if (!nb[f]) v += k[f];
        kvac[i] = v;
    }
}

// ---- a Newton pass's system at the iterate (heat.rs:476-489): the mass term c = c_i + Σ_vac D_f (the diagonal less the
// couplings to gas neighbours, so that A x = c x + Σ D (x_i - x_j) is evaluated without cancellation) and the right-hand
// side. Both follow from a cell's C, T, T⁰ and Σ_vac D_f: the kernels that need them in f64 form them from those (as
// many bytes read as the stored pair would take, and none written), and only level 0's FP32 copy of c is stored.
struct CellSystem {
    double heat, slope, c, rhs;
};
__device__ __forceinline__ CellSystem cell_system(const HeatConst& K, double inv_dt, double u_vac, double C, double t,
                                                  double t0, double kvac) {
    CellSystem s;
    s.heat = C * inv_dt;
    s.slope = dt_du(K, t);
    const double ci = s.heat * s.slope;
    s.c = ci + kvac;
    s.rhs = ci * u_of(K, t) - s.heat * (t - t0) + kvac * u_vac;
    return s;
}

// The first pass's system: level 0's c, the iterate x = u(T), and partials of the two measures' bounds, Σ c_i u² and
// Σ (C/Δt) T² (heat.rs:480-487).
__global__ void heat_system_kernel(HeatConst K, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                                   const double* __restrict__ C, const double* __restrict__ t,
                                   const double* __restrict__ kvac, float* c0, double* x, Red R, const __grid_constant__ Ctl ctl) {
    const size_t n = (size_t)K.w * K.h;
    const double dt = scal[S_DT];
    double ub = 0.0, tb = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!gas[i]) {
            c0[i] = 1.0f;
            x[i] = 0.0;
            continue;
        }
        const double heat = C[i] / dt, ti = t[i], ui = u_of(K, ti);
        const double ci = heat * dt_du(K, ti);
        c0[i] = (float)(ci + kvac[i]);
        x[i] = ui;
        ub += ci * ui * ui;
        tb += heat * ti * ti;
    }
    const double v[2] = {ub, tb};
    const bool last = grid_sum_last<2>(v, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_UB, C_NEWTON_BEGIN);
}

// r = b - A x in FP64, A x = c x + Σ_gas D (x_i - x_j), with partials of <r, r>, <b, b> and the reference's two
// measures (heat.rs:413-447): rᵀD⁻¹r and the heat measure Σ (C/Δt)(r (dT/du) / D_ii)².
// A thread walks down `rows` rows of a column (as spmv_dir_kernel does, and by the same rule): the iterate above and below
// and the couplings between rows stay in registers, those across come from the next lanes, and the next row's operands
// are in flight behind this row's arithmetic (a thread a cell: five loads of x and of the mask and two of each coupling;
// 512²: 12.9 -> 11.0 us; 2048², beside the coarsening: 75).
__global__ void __launch_bounds__(RED_THREADS, 2)
    heat_residual64_kernel(HeatConst K, int rows, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                           const double* __restrict__ kvac, const double* __restrict__ kx,
                           const double* __restrict__ ky, const double* __restrict__ C, const double* __restrict__ t,
                           const double* __restrict__ t0, const double* __restrict__ x, double* __restrict__ r, Red R,
                           const __grid_constant__ Ctl ctl) {
    const int w = K.w, h = K.h, lane = threadIdx.x & 31;
    const int at = blockIdx.x * RED_THREADS + threadIdx.x, bands = (h + rows - 1) / rows;
    const bool live = at < w * bands;
    const int band = live ? at / w : 0, xx = live ? at - band * w : 0, y0 = band * rows;
    const double inv_dt = 1.0 / scal[S_DT], u_vac = u_of(K, K.t_floor);
    double rr = 0.0, bb = 0.0, gg = 0.0, hh = 0.0;
    // what lane 0 lacks on its left and lane 31 on its right
    const int side = lane == 0 ? (xx > 0 ? -1 : 0) : (lane == 31 && xx + 1 < w ? 1 : 0);
    struct Below {  // of the row below the one in work
        double x, xs;
        int g, gs;
    };
    auto below_at = [&](int y) {
        const size_t i = (size_t)min(y, h - 1) * w + xx;
        Below b;
        b.x = x[i];
        b.g = gas[i];
        b.xs = side ? x[i + side] : 0.0;
        b.gs = side ? gas[i + side] : 0;
        return b;
    };
    struct Cell {
        double kv, t0, C, t, kl, kr, kd;
    };
    auto cell_at = [&](int y) {
        const size_t i = (size_t)min(y, h - 1) * w + xx, f = (size_t)min(y, h - 1) * (w + 1) + xx;
        Cell c;
        c.kv = kvac[i];
        c.t0 = t0[i];
        c.C = C[i];
        c.t = t[i];
        c.kl = kx[f];
        c.kr = lane == 31 || xx + 1 == w ? kx[f + 1] : 0.0;
        c.kd = ky[i + w];
        return c;
    };
    double xu = y0 > 0 ? x[(size_t)(y0 - 1) * w + xx] : 0.0, ku = ky[(size_t)y0 * w + xx];
    int gu = y0 > 0 && gas[(size_t)(y0 - 1) * w + xx];
    Below c = below_at(y0), dn = below_at(y0 + 1);
    Cell k = cell_at(y0);
    for (int q = 0; q < rows; q++) {
        const int y = y0 + q;
        Below nb = dn;
        Cell nk = k;
        if (q + 1 < rows) {  // rows past the last are the last again, and leave nothing
            nb = below_at(y + 2);
            nk = cell_at(y + 1);
        }
        double xl = __shfl_up_sync(0xffffffffu, c.x, 1), xr = __shfl_down_sync(0xffffffffu, c.x, 1);
        double kr = __shfl_down_sync(0xffffffffu, k.kl, 1);
        int gl = __shfl_up_sync(0xffffffffu, c.g, 1), gr = __shfl_down_sync(0xffffffffu, c.g, 1);
        if (lane == 0) {
            xl = c.xs;
            gl = c.gs;
        }
        if (lane == 31) {
            xr = c.xs;
            gr = c.gs;
        }
        if (lane == 31 || xx + 1 == w) kr = k.kr;
        if (xx == 0) gl = 0;
        if (xx + 1 == w) gr = 0;
        const bool gd = y + 1 < h && dn.g;
        if (live && y < h) {
            const size_t i = (size_t)y * w + xx;
            if (!c.g) {
                r[i] = 0.0;
            } else {
                const double xi = c.x;
                const CellSystem S = cell_system(K, inv_dt, u_vac, k.C, k.t, k.t0, k.kv);
                double s = S.c * xi, d = S.c;
                if (gl) {
                    s += k.kl * (xi - xl);
                    d += k.kl;
                }
                if (gr) {
                    s += kr * (xi - xr);
                    d += kr;
                }
                if (gu) {
                    s += ku * (xi - xu);
                    d += ku;
                }
                if (gd) {
                    s += k.kd * (xi - dn.x);
                    d += k.kd;
                }
                const double ri = S.rhs - s;
                r[i] = ri;
                rr += ri * ri;
                bb += S.rhs * S.rhs;
                const double rd = ri / d;  // FP64 divisions are what this kernel has few of to spend
                gg += ri * rd;
                const double e = rd * S.slope;
                hh += S.heat * e * e;
            }
        }
        xu = c.x;
        gu = c.g;
        ku = k.kd;
        c = dn;
        dn = nb;
        k = nk;
    }
    const double v[4] = {rr, bb, gg, hh};
    const bool last = grid_sum_last<4>(v, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_RR, C_REFINE);
}

__global__ void scale_kernel(size_t n, const double* __restrict__ r64, const double* __restrict__ scal, float* r32,
                             float* e32, Red R, const __grid_constant__ Ctl ctl) {
    const double inv_scale = scal[S_ISCALE];
    if (inv_scale == 0.0) return;  // the captured loop: no inner solve this time
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float v = (float)(r64[i] * inv_scale);
        r32[i] = v;
        e32[i] = 0.0f;
        acc += (double)v * v;
    }
    const bool last = grid_sum_last1(acc, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_R32, C_INNER_BEGIN);
}

constexpr int ILP = 4;  // cells a thread takes a grid stride apart, all of their loads issued before the arithmetic

// q = A p on level 0's FP32 operator in difference form, c p_i + Σ d (p_i - p_j); partials of <p, q>. ILP cells per
// thread, loads first (masked cells have c = 1 and no couplings; the mask selects afterwards).
__global__ void spmv_kernel(MgLevel L, const float* __restrict__ p, float* __restrict__ q, Red R) {
    const int w = L.w, h = L.h;
    const size_t n = (size_t)w * h, stride = (size_t)gridDim.x * blockDim.x;
    double acc = 0.0;
    for (size_t base = (size_t)blockIdx.x * blockDim.x + threadIdx.x; base < n; base += ILP * stride) {
        float pv[ILP], v[ILP];
#pragma unroll
        for (int u = 0; u < ILP; u++) {
            const size_t i = base + u * stride;
            pv[u] = 0.0f;
            v[u] = 0.0f;
            if (i < n) {
                int x, y;
                split_index(i, w, x, y);
                const float pi = p[i];
                const float pl = x > 0 ? p[i - 1] : pi, pr = x + 1 < w ? p[i + 1] : pi;
                const float pu = y > 0 ? p[i - w] : pi, pd = y + 1 < h ? p[i + w] : pi;
                const float dl = x > 0 ? L.dx[i - 1] : 0.0f, du = y > 0 ? L.dy[i - w] : 0.0f;
                const float dr = L.dx[i], dd = L.dy[i], c = L.c[i];
                const bool m = L.mask[i];
                float a = c * pi;
                a += dl * (pi - pl);
                a += dr * (pi - pr);
                a += du * (pi - pu);
                a += dd * (pi - pd);
                pv[u] = pi;
                v[u] = m ? a : 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < ILP; u++) {
            const size_t i = base + u * stride;
            if (i < n) {
                q[i] = v[u];
                acc += (double)pv[u] * v[u];
            }
        }
    }
    grid_sum_last1(acc, R.part, R.counter, R.out);
}

// e += α p, r -= α q (α = <r,z>/<p,q> from the device scalars), partials of <r, r>.
__global__ void pcg_update_kernel(size_t n, const double* __restrict__ scal, int rz_slot, const float* __restrict__ p,
                                  const float* __restrict__ q, float* __restrict__ e, float* __restrict__ r, Red R) {
    const float alpha = (float)(scal[rz_slot] / scal[S_PQ]);
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    double acc = 0.0;
    for (size_t base = (size_t)blockIdx.x * blockDim.x + threadIdx.x; base < n; base += ILP * stride) {
        float pv[ILP], qv[ILP], ev[ILP], rv[ILP];
#pragma unroll
        for (int u = 0; u < ILP; u++) {
            const size_t i = base + u * stride;
            if (i < n) {
                pv[u] = p[i];
                qv[u] = q[i];
                ev[u] = e[i];
                rv[u] = r[i];
            }
        }
#pragma unroll
        for (int u = 0; u < ILP; u++) {
            const size_t i = base + u * stride;
            if (i < n) {
                e[i] = ev[u] + alpha * pv[u];
                const float ri = rv[u] - alpha * qv[u];
                r[i] = ri;
                acc += (double)ri * ri;
            }
        }
    }
    grid_sum_last1(acc, R.part, R.counter, R.out);
}

// p = z + β p (β = <r,z>_new / <r,z>_old); the first direction (old slot < 0) is p = z.
__global__ void pcg_direction_kernel(size_t n, const double* __restrict__ scal, int old_slot, int new_slot,
                                     const float* __restrict__ z, float* __restrict__ p) {
    const float beta = old_slot < 0 ? 0.0f : (float)(scal[new_slot] / scal[old_slot]);
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t base = (size_t)blockIdx.x * blockDim.x + threadIdx.x; base < n; base += ILP * stride) {
        float zv[ILP], pv[ILP];
#pragma unroll
        for (int u = 0; u < ILP; u++) {
            const size_t i = base + u * stride;
            if (i < n) {
                zv[u] = z[i];
                pv[u] = old_slot < 0 ? 0.0f : p[i];
            }
        }
#pragma unroll
        for (int u = 0; u < ILP; u++) {
            const size_t i = base + u * stride;
            if (i < n) p[i] = old_slot < 0 ? zv[u] : zv[u] + beta * pv[u];
        }
    }
}

// The block's Σ acc into part[blockIdx.x], in a fixed order.
__device__ __forceinline__ void block_partial(double acc, double* part) {
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
        part[blockIdx.x] = t;
    }
}

// Σ v[0..n) by the block, in an order that depends on n and the block's size alone; valid in thread 0.
__device__ __forceinline__ double block_sum_ordered(const double* v, int n) {
    __shared__ double red[32];
    double x = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) x += v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    return t;
}

__global__ void sum_parts_kernel(const double* v, int n, double* out) {
    const double t = block_sum_ordered(v, n);
    if (threadIdx.x == 0) *out = t;
}

// After a (non-flexible) round's preconditioner: the search direction p_new = z + β p (β = <r,z> / <r,z>_prev, or
// p_new = z while the S_BETA flag is 0: the first round) and q = A p_new in difference form, with partials of
// <p_new, q>, left for pcg_update4_kernel to sum. The neighbours' p_new are formed from their z and old p, so p_new goes
// to the other of the two direction buffers (S_PAR says which holds the old one).
// <r, z> comes as the preconditioner's `parts` partials, which every CTA sums for itself in the same order (0: it is in
// S_RZN already); the first CTA leaves it there.
// A thread takes four consecutive columns (W is a multiple of 8) of `rows` rows and walks down them: the row above and
// its own stay in registers, its side neighbours come from the next lanes, so a row costs one 16-byte load of each plane
// (a thread a row: three of z and of p, two of dy, and six words at its sides; 2048²: 28.0 -> 20.2 us; 512²: 6.2 -> 4.4). `rows` is what
// puts all threads on the GPU at once (1 up to some 600,000 cells); the next row's operands are in flight behind this
// row's arithmetic.
__global__ void __launch_bounds__(RED_THREADS, 3)
    spmv_dir_kernel(MgLevel L, int rows, double* scal, const float* z, float* pa, float* pb, float* __restrict__ q,
                    double* pq_part, const double* rz_part, int parts) {
    __shared__ double s_rz;
    pdl_launch();
    const int w = L.w, h = L.h, w4 = w / 4, lane = threadIdx.x & 31;
    const int t = blockIdx.x * RED_THREADS + threadIdx.x, bands = (h + rows - 1) / rows;
    const bool live = t < w4 * bands;
    const int band = live ? t / w4 : 0, x = 4 * (live ? t - band * w4 : 0), y0 = band * rows;
    struct Op {
        float4 c, dx, dy;
        float dl;  // the coupling to the left of lane 0's columns
        uchar4 m;
    };
    auto op_at = [&](int y) {
        const size_t i = (size_t)y * w + x;
        Op o;
        o.c = *reinterpret_cast<const float4*>(L.c + i);
        o.dx = *reinterpret_cast<const float4*>(L.dx + i);
        o.dy = *reinterpret_cast<const float4*>(L.dy + i);
        o.dl = lane == 0 && x > 0 ? L.dx[i - 1] : 0.0f;
        o.m = *reinterpret_cast<const uchar4*>(L.mask + i);
        return o;
    };
    Op o = op_at(y0);
    float4 dyu = y0 > 0 ? *reinterpret_cast<const float4*>(L.dy + (size_t)(y0 - 1) * w + x) : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();
    if (parts > 0) {
        const double v = block_sum_ordered(rz_part, parts);
        if (threadIdx.x == 0) {
            s_rz = v;
            if (blockIdx.x == 0) scal[S_RZN] = v;
        }
    } else if (threadIdx.x == 0) {
        s_rz = scal[S_RZN];
    }
    __syncthreads();
    const bool first = scal[S_BETA] == 0.0;  // p = z: the old direction is not read (it may hold anything)
    const float beta = first ? 0.0f : (float)(s_rz / scal[S_RZP]);
    const bool par = scal[S_PAR] != 0.0;
    const float* __restrict__ p = par ? pb : pa;
    float* __restrict__ pnew = par ? pa : pb;
    struct Raw {
        float4 z, p;
        float ze, pe;  // the column beside the warp's, lane 0's left and lane 31's right
    };
    const int side = lane == 0 ? (x > 0 ? -1 : 0) : (lane == 31 && x + 4 < w ? 4 : 0);
    auto raw_at = [&](int y) {
        const size_t i = (size_t)y * w + x;
        Raw a;
        a.z = *reinterpret_cast<const float4*>(z + i);
        a.ze = side ? z[i + side] : 0.0f;
        a.p = make_float4(0.f, 0.f, 0.f, 0.f);
        a.pe = 0.0f;
        if (!first) {
            a.p = *reinterpret_cast<const float4*>(p + i);
            a.pe = side ? p[i + side] : 0.0f;
        }
        return a;
    };
    auto dir4 = [&](const Raw& a) {
        if (first) return a.z;
        return make_float4(a.z.x + beta * a.p.x, a.z.y + beta * a.p.y, a.z.z + beta * a.p.z, a.z.w + beta * a.p.w);
    };
    auto dir_side = [&](const Raw& a) { return first ? a.ze : a.ze + beta * a.pe; };
    Raw ra = raw_at(max(y0 - 1, 0)), rc = raw_at(y0), rd = raw_at(min(y0 + 1, h - 1));
    float4 pu = dir4(ra), pc = dir4(rc);
    float pe = dir_side(rc);
    double acc = 0.0;
    for (int r = 0; r < rows; r++) {
        const int y = y0 + r;
        const float4 pd = dir4(rd);
        const float pde = dir_side(rd);
        Op on = o;
        if (r + 1 < rows) {  // rows past the last are the last again, and leave nothing
            on = op_at(min(y + 1, h - 1));
            rd = raw_at(min(y + 2, h - 1));
        }
        float pl = __shfl_up_sync(0xffffffffu, pc.w, 1), pr = __shfl_down_sync(0xffffffffu, pc.x, 1);
        float dl = __shfl_up_sync(0xffffffffu, o.dx.w, 1);
        if (lane == 0) {
            pl = pe;
            dl = o.dl;
        }
        if (lane == 31) pr = pe;
        if (x == 0) {
            pl = pc.x;
            dl = 0.0f;
        }
        if (x + 4 >= w) pr = pc.w;
        const float4 up = y > 0 ? pu : pc, dn = y + 1 < h ? pd : pc;
        const float P[6] = {pl, pc.x, pc.y, pc.z, pc.w, pr};
        const float U[4] = {up.x, up.y, up.z, up.w}, D[4] = {dn.x, dn.y, dn.z, dn.w};
        const float CC[4] = {o.c.x, o.c.y, o.c.z, o.c.w}, DXs[5] = {dl, o.dx.x, o.dx.y, o.dx.z, o.dx.w};
        const float DYu[4] = {dyu.x, dyu.y, dyu.z, dyu.w}, DYd[4] = {o.dy.x, o.dy.y, o.dy.z, o.dy.w};
        const unsigned char M[4] = {o.m.x, o.m.y, o.m.z, o.m.w};
        float out[4];
        const bool on_row = live && y < h;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float pi = P[k + 1];
            float a = CC[k] * pi;
            a += DXs[k] * (pi - P[k]);
            a += DXs[k + 1] * (pi - P[k + 2]);
            a += DYu[k] * (pi - U[k]);
            a += DYd[k] * (pi - D[k]);
            out[k] = M[k] ? a : 0.0f;
            if (on_row) acc += (double)pi * out[k];
        }
        if (on_row) {
            const size_t i = (size_t)y * w + x;
            *reinterpret_cast<float4*>(pnew + i) = pc;
            *reinterpret_cast<float4*>(q + i) = make_float4(out[0], out[1], out[2], out[3]);
        }
        dyu = o.dy;
        pu = pc;
        pc = pd;
        pe = pde;
        o = on;
    }
    block_partial(acc, pq_part);
}

// e += α p, r -= α q with 16-byte accesses (four cells per thread), p the round's new direction; partials of <r, r>.
// <p, q> comes as `parts` partials, which every CTA sums in the same order; the first CTA leaves it in S_PQ.
__global__ void pcg_update4_kernel(size_t n, double* scal, const double* pq_part, int parts, const float* pa,
                                   const float* pb, const float* q, float* __restrict__ e, float* __restrict__ r, Red R,
                                   const __grid_constant__ Ctl ctl) {
    __shared__ double s_pq;
    pdl_wait();
    const double pq = block_sum_ordered(pq_part, parts);
    if (threadIdx.x == 0) {
        s_pq = pq;
        if (blockIdx.x == 0) scal[S_PQ] = pq;
    }
    __syncthreads();
    const float alpha = (float)(scal[S_RZN] / s_pq);
    const float* p = scal[S_PAR] != 0.0 ? pa : pb;
    const size_t n4 = n / 4, stride = (size_t)gridDim.x * blockDim.x;
    double acc = 0.0;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n4; t += stride) {
        const float4 pv = reinterpret_cast<const float4*>(p)[t], qv = reinterpret_cast<const float4*>(q)[t];
        float4 ev = reinterpret_cast<float4*>(e)[t], rv = reinterpret_cast<float4*>(r)[t];
        ev.x += alpha * pv.x; ev.y += alpha * pv.y; ev.z += alpha * pv.z; ev.w += alpha * pv.w;
        rv.x -= alpha * qv.x; rv.y -= alpha * qv.y; rv.z -= alpha * qv.z; rv.w -= alpha * qv.w;
        reinterpret_cast<float4*>(e)[t] = ev;
        reinterpret_cast<float4*>(r)[t] = rv;
        acc += (double)rv.x * rv.x + (double)rv.y * rv.y + (double)rv.z * rv.z + (double)rv.w * rv.w;
    }
    const bool last = grid_sum_last1(acc, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_RRI, C_ROUND);
}

// Flexible CG (the learned preconditioner is not a fixed linear operator): the update keeps the residual it replaces,
// <z, r_old> is formed after the preconditioner, and β = (<z, r> - <z, r_old>) / <z_old, r_old> (Polak-Ribière).
__global__ void pcg_update_flex_kernel(size_t n, const double* __restrict__ scal, int rz_slot,
                                       const float* __restrict__ p, const float* __restrict__ q, float* e, float* r,
                                       float* r_old, Red R) {
    const float alpha = (float)(scal[rz_slot] / scal[S_PQ]);
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        e[i] += alpha * p[i];
        const float ro = r[i];
        const float ri = ro - alpha * q[i];
        r_old[i] = ro;
        r[i] = ri;
        acc += (double)ri * ri;
    }
    grid_sum_last1(acc, R.part, R.counter, R.out);
}

__global__ void dot_kernel(size_t n, const float* __restrict__ a, const float* __restrict__ b, Red R) {
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        acc += (double)a[i] * b[i];
    grid_sum_last1(acc, R.part, R.counter, R.out);
}

__global__ void pcg_direction_flex_kernel(size_t n, const double* __restrict__ scal, int old_slot, int new_slot,
                                          const float* __restrict__ z, float* p) {
    const float beta = (float)((scal[new_slot] - scal[S_ZRO]) / scal[old_slot]);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        p[i] = z[i] + beta * p[i];
}

// The residual a V-cycle leaves, r1 = r − A z (gas cells; 0 elsewhere), and optionally ez = e + z.
__global__ void vcycle_residual_kernel(MgLevel L, const float* __restrict__ r, const float* __restrict__ z,
                                       const float* __restrict__ e, float* r1, float* ez) {
    const int w = L.w, h = L.h;
    const size_t n = (size_t)w * h;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        int x, y;
        split_index(i, w, x, y);
        float v = 0.0f;
        const float zi = z[i];
        if (L.mask[i]) {
            float az = L.c[i] * zi;
            if (x > 0) az += L.dx[i - 1] * (zi - z[i - 1]);
            if (x + 1 < w) az += L.dx[i] * (zi - z[i + 1]);
            if (y > 0) az += L.dy[i - w] * (zi - z[i - w]);
            if (y + 1 < h) az += L.dy[i] * (zi - z[i + w]);
            v = r[i] - az;
        }
        r1[i] = v;
        if (ez) ez[i] = e[i] + zi;
    }
}

// z = r / diag (Jacobi), partials of <r, z>.
__global__ void jacobi_kernel(MgLevel L, const float* __restrict__ r, float* z, Red R) {
    const int w = L.w, h = L.h;
    const size_t n = (size_t)w * h;
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        int x, y;
        split_index(i, w, x, y);
        const float dl = x > 0 ? L.dx[i - 1] : 0.0f, du = y > 0 ? L.dy[i - w] : 0.0f;
        const float zi = L.mask[i] ? r[i] / (L.c[i] + dl + L.dx[i] + du + L.dy[i]) : 0.0f;
        z[i] = zi;
        acc += (double)r[i] * zi;
    }
    grid_sum_last1(acc, R.part, R.counter, R.out);
}

// z += v, and <r, z>.
__global__ void add_dot_kernel(size_t n, const float* __restrict__ r, const float* __restrict__ v, float* z, Red R) {
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float zi = z[i] + v[i];
        z[i] = zi;
        acc += (double)r[i] * zi;
    }
    grid_sum_last1(acc, R.part, R.counter, R.out);
}

__global__ void correction_kernel(size_t n, const uint8_t* __restrict__ gas, const float* __restrict__ e,
                                  const double* __restrict__ scal, double* x) {
    const double scale = scal[S_SCALE];
    if (scale == 0.0) return;  // no inner solve, or one that broke down
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (gas[i]) x[i] += scale * (double)e[i];
}

// The pass's update (heat.rs:494-509: u >= u_vac, T within a factor 2) and the next pass's system at the new iterate
// (as heat_system_kernel builds it) in one sweep over the cells; partials of Σ C|ΔT|, the cells moved by more than
// newton_cell of their T, Σ c_i u² and Σ (C/Δt) T² (four consecutive slots from S_MOVED). When the passes end here
// the system goes unused.
__global__ void newton_system_kernel(HeatConst K, double cell_tol, const double* __restrict__ scal,
                                     const uint8_t* __restrict__ gas,
                                     const double* __restrict__ C, const double* __restrict__ kvac, double* t, double* x,
                                     float* c0, Red R, const __grid_constant__ Ctl ctl) {
    if (ctl.c && !ctl.c->newton) return;
    const size_t n = (size_t)K.w * K.h, stride = (size_t)gridDim.x * blockDim.x;
    const double u_vac = u_of(K, K.t_floor);
    const double dt = scal[S_DT];
    double moved = 0.0, viol = 0.0, ub = 0.0, tb = 0.0;
    // two cells a grid stride apart per iteration, all loads issued before the arithmetic
    for (size_t base = (size_t)blockIdx.x * blockDim.x + threadIdx.x; base < n; base += 2 * stride) {
        const size_t i2 = base + stride;
        const bool g1 = gas[base], g2 = i2 < n && gas[i2];
        double tv[2], xv[2], Cv[2], kv[2];
        tv[0] = t[base];
        xv[0] = x[base];
        Cv[0] = C[base];
        kv[0] = kvac[base];
        if (i2 < n) {
            tv[1] = t[i2];
            xv[1] = x[i2];
            Cv[1] = C[i2];
            kv[1] = kvac[i2];
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const size_t i = e ? i2 : base;
            if (!(e ? g2 : g1)) continue;  // the system's masked rows (c = 1, x = 0) are already in place
            const double ti = tv[e];
            double nx = t_of(K, fmax(xv[e], u_vac));
            nx = fmin(fmax(nx, 0.5 * ti), 2.0 * ti);
            const double d = fabs(nx - ti);
            moved += Cv[e] * d;
            if (!(d <= cell_tol * ti)) viol += 1.0;
            const double un = u_of(K, nx);
            t[i] = nx;
            const double heat = Cv[e] / dt;
            const double ci = heat * dt_du(K, nx);
            c0[i] = (float)(ci + kv[e]);
            x[i] = un;
            ub += ci * un * un;
            tb += heat * nx * nx;
        }
    }
    const double v[4] = {moved, viol, ub, tb};
    const bool last = grid_sum_last<4>(v, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_MOVED, C_NEWTON);
}

// F = -k (v_b - v_a) at every face (heat.rs:338-361), v = u(T) on gas cells, u_vac elsewhere; FP32 out.
__device__ __forceinline__ double face_flux(const HeatConst& K, const uint8_t* gas, const double* t, double k,
                                            long a, long b, double u_vac) {
    if (k == 0.0) return 0.0;
    const double va = (a >= 0 && gas[a]) ? u_of(K, t[a]) : u_vac;
    const double vb = (b >= 0 && gas[b]) ? u_of(K, t[b]) : u_vac;
    return -k * (vb - va);
}

__global__ void heat_flux_kernel(HeatConst K, const uint8_t* __restrict__ gas, const double* __restrict__ kx,
                                 const double* __restrict__ ky, const double* __restrict__ t,
                                 const double* __restrict__ scale, float* fx, float* fy) {
    const int w = K.w, h = K.h;
    const size_t nx = (size_t)(w + 1) * h, ny = (size_t)w * (h + 1);
    const double u_vac = u_of(K, K.t_floor);
    for (size_t f = (size_t)blockIdx.x * blockDim.x + threadIdx.x; f < nx + ny; f += (size_t)gridDim.x * blockDim.x) {
        long a, b;
        double k;
        if (f < nx) {
            int x, y;
            split_index(f, (w + 1), x, y);
            a = x > 0 ? (long)y * w + x - 1 : -1;
            b = x < w ? (long)y * w + x : -1;
            k = kx[f];
        } else {
            const size_t g = f - nx;
            int x, y;
            split_index(g, w, x, y);
            a = y > 0 ? (long)(y - 1) * w + x : -1;
            b = y < h ? (long)y * w + x : -1;
            k = ky[g];
        }
        double F = face_flux(K, gas, t, k, a, b, u_vac);
        if (scale) {
            const long from = F > 0.0 ? a : b;
            F *= from >= 0 ? scale[from] : 1.0;
        }
        if (f < nx) fx[f] = (float)F;
        else fy[f - nx] = (float)F;
    }
}

// The commit's sums (heat.rs:521-531): radiated, gained and held.
__global__ void commit_sums_kernel(HeatConst K, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                                   const double* __restrict__ C, const double* __restrict__ t,
                                   const double* __restrict__ t0, const double* __restrict__ kvac, Red R, const __grid_constant__ Ctl ctl) {
    const size_t n = (size_t)K.w * K.h;
    const double u_vac = u_of(K, K.t_floor);
    const double dt = scal[S_DT];
    double rad = 0.0, gain = 0.0, held = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!gas[i]) continue;
        rad += dt * kvac[i] * (u_of(K, t[i]) - u_vac);
        gain += C[i] * (t[i] - t0[i]);
        held += C[i] * t[i];
    }
    const double v[3] = {rad, gain, held};
    const bool last = grid_sum_last<3>(v, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_RAD, C_DELTA);
}

// E_i += C_i ((1 + δ) T_i - T_i⁰) (heat.rs:532-535), and the cell's rate (T - T⁰)/Δt kept for the next step's first
// iterate (heat.wgsl:1139-1155).
__global__ void commit_apply_kernel(HeatConst K, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                                    const double* __restrict__ C, const double* __restrict__ t,
                                    const double* __restrict__ t0, float* U, double* rate) {
    const size_t n = (size_t)K.w * K.h;
    const double delta = scal[S_DELTA], dt = scal[S_DT];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (gas[i]) U[3 * n + i] = (float)((double)U[3 * n + i] + C[i] * ((1.0 + delta) * t[i] - t0[i]));
        rate[i] = gas[i] ? (t[i] - t0[i]) / dt : 0.0;
    }
}

// The first iterate on the V-cycle (heat.wgsl:710-722): T⁰ + the last step's rate × Δt, T⁰ where that is off by more
// than a factor 2 or not finite, floored at T_floor.
__global__ void warm_start_kernel(HeatConst K, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                                  const double* __restrict__ t0, const double* __restrict__ rate, double* t) {
    const size_t n = (size_t)K.w * K.h;
    const double dt = scal[S_DT];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!gas[i]) continue;
        double tg = t0[i] + rate[i] * dt;
        if (!(tg >= 0.5 * t0[i] && tg <= 2.0 * t0[i])) tg = t0[i];
        tg = fmax(tg, K.t_floor);
        t[i] = tg;
    }
}

// Past the ceiling (heat.rs:545-564): each gas cell's outflow scaled to the heat it holds above its floor.
__global__ void limited_scale_kernel(HeatConst K, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                                     const double* __restrict__ kx, const double* __restrict__ ky,
                                     const double* __restrict__ t, const double* __restrict__ C,
                                     const double* __restrict__ t0, double* scale) {
    const int w = K.w, h = K.h;
    const size_t n = (size_t)w * h;
    const double u_vac = u_of(K, K.t_floor);
    const double dt = scal[S_DT];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!gas[i]) {
            scale[i] = 1.0;
            continue;
        }
        int x, y;
        split_index(i, w, x, y);
        const long L = x > 0 ? (long)i - 1 : -1, R = x + 1 < w ? (long)i + 1 : -1;
        const long Uu = y > 0 ? (long)i - w : -1, D = y + 1 < h ? (long)i + w : -1;
        const double lv[4] = {-face_flux(K, gas, t, kx[(size_t)y * (w + 1) + x], L, (long)i, u_vac),
                              face_flux(K, gas, t, kx[(size_t)y * (w + 1) + x + 1], (long)i, R, u_vac),
                              -face_flux(K, gas, t, ky[(size_t)y * w + x], Uu, (long)i, u_vac),
                              face_flux(K, gas, t, ky[(size_t)(y + 1) * w + x], (long)i, D, u_vac)};
        double out = 0.0;
        for (int f = 0; f < 4; f++) out += fmax(lv[f], 0.0);
        out *= dt;
        const double held = C[i] * fmax(t0[i] - K.t_floor, 0.0);
        scale[i] = out > held ? held / out : 1.0;
    }
}

// E -= Δt Σ_f F_f with every face's F at the scale of the cell it leaves (heat.rs:565-592); partials of radiated.
__global__ void limited_apply_kernel(HeatConst K, const double* __restrict__ scal, const uint8_t* __restrict__ gas,
                                     const double* __restrict__ kx, const double* __restrict__ ky,
                                     const double* __restrict__ t, const double* __restrict__ scale, float* U,
                                     Red R, const __grid_constant__ Ctl ctl) {
    const int w = K.w, h = K.h;
    const size_t n = (size_t)w * h;
    const double u_vac = u_of(K, K.t_floor);
    const double dt = scal[S_DT];
    double rad = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!gas[i]) continue;
        int x, y;
        split_index(i, w, x, y);
        const long nb[4] = {x > 0 ? (long)i - 1 : -1, x + 1 < w ? (long)i + 1 : -1, y > 0 ? (long)i - w : -1,
                            y + 1 < h ? (long)i + w : -1};
        double F[4] = {face_flux(K, gas, t, kx[(size_t)y * (w + 1) + x], nb[0], (long)i, u_vac),
                       face_flux(K, gas, t, kx[(size_t)y * (w + 1) + x + 1], (long)i, nb[1], u_vac),
                       face_flux(K, gas, t, ky[(size_t)y * w + x], nb[2], (long)i, u_vac),
                       face_flux(K, gas, t, ky[(size_t)(y + 1) * w + x], (long)i, nb[3], u_vac)};
        // the low cell of faces 0 and 2 is the neighbour, of faces 1 and 3 this cell
        const long low[4] = {nb[0], (long)i, nb[2], (long)i}, high[4] = {(long)i, nb[1], (long)i, nb[3]};
        double out[4];
        for (int f = 0; f < 4; f++) {
            const long from = F[f] > 0.0 ? low[f] : high[f];
            F[f] *= from >= 0 ? scale[from] : 1.0;
        }
        out[0] = -F[0];
        out[1] = F[1];
        out[2] = -F[2];
        out[3] = F[3];
        for (int f = 0; f < 4; f++)
            if (!(nb[f] >= 0 && gas[nb[f]])) rad += dt * out[f];
        U[3 * n + i] = (float)((double)U[3 * n + i] - dt * (((out[0] + out[1]) + out[2]) + out[3]));
    }
    const bool last = grid_sum_last1(rad, R.part, R.counter, R.out);
    if (last && threadIdx.x == 0 && ctl.c) ctl_run(ctl, R.out - S_RAD, C_LIMITED);
}

__global__ void zero_kernel(double* a, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) a[i] = 0.0;
}

__global__ void f64_to_f32_kernel(float* dst, const double* __restrict__ src, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}

__global__ void f32_to_f64_kernel(double* dst, const float* __restrict__ src, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

// One device scalar set by the host's launch (a value captured at launch time, so no staging buffer is reused).
__global__ void set_scalar_kernel(double* scal, int slot, double value) {
    if (threadIdx.x == 0 && blockIdx.x == 0) scal[slot] = value;
}

// A fused PCG solve's start: the first direction is z, the direction buffers start at pa.
__global__ void pcg_start_kernel(double* scal) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    scal[S_BETA] = 0.0;
    scal[S_PAR] = 0.0;
}

// A fused PCG round's end: its <r, z> becomes the last one, later directions take β, the new direction buffer is the old.
__global__ void pcg_rotate_kernel(double* scal) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    scal[S_RZP] = scal[S_RZN];
    scal[S_BETA] = 1.0;
    scal[S_PAR] = scal[S_PAR] != 0.0 ? 0.0 : 1.0;
}

int grid_for(size_t n) {
    size_t b = (n + RED_THREADS - 1) / RED_THREADS;
    return (int)(b < 1 ? 1 : (b > (size_t)MAX_PART ? (size_t)MAX_PART : b));
}

// CTAs for `turns` turns of RED_THREADS threads, at most one wave of them.
template <class F>
int whole_waves(F kernel, size_t turns) {
    int per_sm = 0, dev = 0, sms = 0;
    SR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, RED_THREADS, 0));
    SR_CUDA_TRY(cudaGetDevice(&dev));
    SR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::max(1, std::min(grid_for(turns), per_sm * sms));
}

}  // namespace

struct RoundGraph {
    cudaGraphExec_t exec = nullptr;
    long long launches = 0;  // kernel nodes in the graph
};

struct HeatSolver {
    sr_config cfg{};
    HeatConst K{};
    HeatRef ref{};
    int w = 0, h = 0;
    size_t n = 0;
    int grid = 0;  // CTAs of the grid-stride kernels
    // of the solve's heaviest, by the cells a thread takes a turn (two, two, four and four) and by what fits the GPU at
    // once: a CTA without a turn still takes a sum's ticket (512²: the SpMV 256 CTAs instead of 1,024), and a wave that
    // does not fill costs a whole one
    int grid_residual = 0, grid_newton = 0, grid_spmv = 0, grid_update = 0;
    int spmv_rows = 1, residual_rows = 1;
    uint32_t precond = SR_PRECOND_MG;
    uint32_t max_passes = 128, max_rounds = 4096;
    double inner_floor = 1e-5;  // the smallest residual reduction asked of one inner FP32 solve
    bool use_graphs = true;
    uint8_t* gas = nullptr;
    double *t0 = nullptr, *C = nullptr, *t = nullptr, *kx = nullptr, *ky = nullptr;
    double *kvac = nullptr, *x = nullptr, *r64 = nullptr;
    double* lscale = nullptr;
    double* rate = nullptr;      // each cell's P5 rate (T - T⁰)/Δt in the last step, for the next first iterate
    float *kap = nullptr, *sig = nullptr;
    float *r32 = nullptr, *e32 = nullptr, *p32 = nullptr, *q32 = nullptr, *z32 = nullptr;
    float* p2 = nullptr;  // the fused rounds' second direction buffer (rounds alternate p32 -> p2 -> p32)
    float *fx = nullptr, *fy = nullptr;
    double* part = nullptr;      // grid-sum partials: 4 x PART_CAP
    double *rz_part = nullptr, *pq_part = nullptr;  // the preconditioner's partials of <r, z>, the SpMV's of <p, q>
    unsigned* counter = nullptr;  // grid-sum ticket
    double* scal = nullptr;       // S_COUNT device scalars
    double* hscal = nullptr;      // pinned host copy
    Multigrid mg;
    int n_gas = 0;
    RoundGraph graphs[3][2];      // one PCG round per preconditioner and <r,z> slot parity
    Learner* learner = nullptr;   // the learned preconditioner, when attached
    LearnedApply* lapply = nullptr;
    float* r_old = nullptr;       // flexible CG's previous residual
    float* ez = nullptr;          // sample collection: the iterate after each round's V-cycle
    float* vz = nullptr;          // the learned preconditioner's second V-cycle
    void* flush = nullptr;        // timing hook: a buffer larger than L2
    // the device-controlled step: its control block, the captured graphs (one per state buffer the step updates),
    // the extra streams its nested bodies are captured on, and each body's kernel count
    HeatCtl* ctl = nullptr;
    HeatCtl* hctl = nullptr;      // pinned host copy
    std::map<const float*, cudaGraphExec_t> step_graphs;
    cudaStream_t cap[6] = {};  // [5]: the captured pass's branch
    cudaEvent_t fork[2] = {};  // its start and its end
    long long body_launches[B_COUNT + 1] = {};  // [B_COUNT]: the graph's own top-level kernels
    bool report_pending = false;  // the last step ran as a graph: its report is in ctl
    cudaStream_t stream = nullptr;  // the owning context's stream
    sr_heat_report report{};

    Red red(int slot) { return Red{part, counter, scal + slot}; }

    // Reads device scalars [first, first + count) into hscal (synchronises the stream).
    void read(int first, int count, cudaStream_t s) {
        SR_CUDA_TRY(cudaMemcpyAsync(hscal + first, scal + first, sizeof(double) * count, cudaMemcpyDeviceToHost, s));
        SR_CUDA_TRY(cudaStreamSynchronize(s));
    }
};

namespace {

void set_scalar(HeatSolver* H, int slot, double value, cudaStream_t s) {
    set_scalar_kernel<<<1, 32, 0, s>>>(H->scal, slot, value);
    sr_note_launch();
}

void setup_step(HeatSolver* H, const float* U, const float* kappa, cudaStream_t s, const Ctl& ctl = Ctl{}) {
    const HeatConst& K = H->K;
    heat_cells_kernel<<<H->grid, RED_THREADS, 0, s>>>(K, H->ref, U, kappa, H->gas, H->t0, H->C, H->kap, H->sig, H->t,
                                                      H->red(S_HEAT0), ctl);
    sr_note_launch();
    const size_t nf = (size_t)(H->w + 1) * H->h + (size_t)H->w * (H->h + 1);
    heat_faces_kernel<<<grid_for(nf), RED_THREADS, 0, s>>>(K, H->gas, H->t0, H->kap, H->sig, H->C, H->kx, H->ky);
    sr_note_launch();
    heat_ksum_kernel<<<H->grid, RED_THREADS, 0, s>>>(K, H->gas, H->kx, H->ky, H->kvac);
    sr_note_launch();
    H->mg.set_couplings(H->kx, H->ky, H->gas, s);
}

// `overlap`: multigrid's launches start while the one before still runs, which takes the launch gaps out of the host's
// rounds (learned preconditioner at 512²: 6.84 -> 6.54 ms a step) and of the captured step of a world alone (with the
// SpMV's and the update's; 512² reference mode, four steps: 39.98 -> 38.60 ms; 2048², three: 29.87 -> 29.75). Not of a
// batch's step: its other worlds want the SMs that an early kernel waits on (10 % slower).
// z = M r, and <r, z> into scalar `rz_slot` (into S_RZN, multigrid's: as partials, for spmv_dir_kernel to sum).
void precondition(HeatSolver* H, uint32_t precond, int rz_slot, bool overlap, cudaStream_t s) {
    if (precond == SR_PRECOND_JACOBI) {
        jacobi_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->mg.L[0], H->r32, H->z32, H->red(rz_slot));
        sr_note_launch();
    } else if (precond == SR_PRECOND_LEARNED) {
        // V-cycle, network, V-cycle: z1 = M r; z2 = z1 + N(r − A z1); z = z2 + M (r − A z2). The network predicts the
        // smooth error the first cycle leaves; the second cycle removes the rounding noise of its BF16 output (high
        // frequencies, which the smoothers take out) and what remains of the smooth error.
        const MgLevel& L0 = H->mg.L[0];
        H->mg.apply(H->r32, H->z32, nullptr, overlap, s);
        vcycle_residual_kernel<<<H->grid, RED_THREADS, 0, s>>>(L0, H->r32, H->z32, nullptr, H->q32, nullptr);
        sr_note_launch();
        learned_apply(H->lapply, L0, H->q32, H->z32, H->r32, H->z32, H->part, H->counter, H->scal + S_MGRZ, s);
        vcycle_residual_kernel<<<H->grid, RED_THREADS, 0, s>>>(L0, H->r32, H->z32, nullptr, H->q32, nullptr);
        sr_note_launch();
        H->mg.apply(H->q32, H->vz, nullptr, overlap, s);
        add_dot_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->r32, H->vz, H->z32, H->red(rz_slot));
        sr_note_launch();
    } else {
        H->mg.apply(H->r32, H->z32, H->rz_part, overlap, s);
        if (rz_slot != S_RZN) {  // a round outside the fused loop: its kernels read the sum
            sum_parts_kernel<<<1, RED_THREADS, 0, s>>>(H->rz_part, H->mg.parts(), H->scal + rz_slot);
            sr_note_launch();
        }
    }
}

// One PCG round. MG and Jacobi: z = M r, β, p = z + β p, q = A p, α, e += α p, r -= α q — a round opens with its
// preconditioner, so the solve's last round ends on the residual it tests and applies none in vain (a V-cycle less per
// inner solve: 17 of 140 over three 2048² steps of the full world). Flexible CG: q = A p, α, e, r, z = M r, β, p;
// `parity` picks its <r,z> slots.
void round_launches(HeatSolver* H, uint32_t precond, int parity, cudaStream_t s) {
    const int rz_old = parity ? S_RZ1 : S_RZ0, rz_new = parity ? S_RZ0 : S_RZ1;
    if (precond == SR_PRECOND_LEARNED) {
        spmv_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->mg.L[0], H->p32, H->q32, H->red(S_PQ));
        sr_note_launch();
        pcg_update_flex_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->scal, rz_old, H->p32, H->q32, H->e32, H->r32,
                                                               H->r_old, H->red(S_RRI));
        sr_note_launch();
        precondition(H, precond, rz_new, true, s);
        dot_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->z32, H->r_old, H->red(S_ZRO));
        sr_note_launch();
        pcg_direction_flex_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->scal, rz_old, rz_new, H->z32, H->p32);
        sr_note_launch();
        return;
    }
    // the fused round: the state (<r, z> slots, which direction buffer is current) lives in the device scalars, so
    // one captured graph serves every round
    (void)rz_old;
    (void)rz_new;
    precondition(H, precond, S_RZN, true, s);
    spmv_dir_kernel<<<H->grid_spmv, RED_THREADS, 0, s>>>(H->mg.L[0], H->spmv_rows, H->scal, H->z32, H->p32, H->p2, H->q32,
                                                    H->pq_part, H->rz_part,
                                                    precond == SR_PRECOND_MG ? H->mg.parts() : 0);
    sr_note_launch();
    pcg_update4_kernel<<<H->grid_update, RED_THREADS, 0, s>>>(H->n, H->scal, H->pq_part, H->grid_spmv, H->p32, H->p2, H->q32, H->e32, H->r32,
                                                       H->red(S_RRI), Ctl{});
    sr_note_launch();
    pcg_rotate_kernel<<<1, 32, 0, s>>>(H->scal);
    sr_note_launch();
}

// A round as one CUDA graph launch (captured once per preconditioner and parity; every pointer it reads is fixed).
void run_round(HeatSolver* H, uint32_t precond, int parity, cudaStream_t s) {
    if (!H->use_graphs) {
        round_launches(H, precond, parity, s);
        return;
    }
    RoundGraph& g = H->graphs[precond][precond == SR_PRECOND_LEARNED ? parity : 0];
    if (!g.exec) {
        const long long before = (long long)sr_launches();
        cudaGraph_t graph;
        SR_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        round_launches(H, precond, parity, s);
        SR_CUDA_TRY(cudaStreamEndCapture(s, &graph));
        cudaError_t e = cudaGraphInstantiate(&g.exec, graph, 0);
        cudaGraphDestroy(graph);
        SR_CUDA_TRY(e);
        g.launches = (long long)sr_launches() - before;
        sr_note_launches(-g.launches);  // captured, not launched
    }
    SR_CUDA_TRY(cudaGraphLaunch(g.exec, s));
    sr_note_launches(g.launches);
}

struct SolveResult {
    int rounds = 0;
    int refinements = 0;
    double rel = 0.0;
    bool ok = true;
    bool fallback = false;  // the learned preconditioner stalled and MG-PCG finished
};

constexpr int kStallRounds = 24;  // learned: rounds after which a solve that has not gained 100x falls back

// PCG on A32 e = r32 from e = 0 to a residual reduction `eta` or `max_it` rounds. Returns the rounds, -1 on a
// breakdown (a non-positive or non-finite curvature), or with the learned preconditioner -2 - rounds when it stalls
// (a breakdown, or less than a 100x reduction after kStallRounds): plain MG-PCG then takes over.
int inner_pcg(HeatSolver* H, uint32_t precond, double eta, int max_it, cudaStream_t s, bool* reached = nullptr) {
    if (reached) *reached = false;
    if (precond == SR_PRECOND_LEARNED) {  // flexible CG forms its direction at the end of a round
        precondition(H, precond, S_RZ0, true, s);
        pcg_direction_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->scal, -1, S_RZ0, H->z32, H->p32);
        sr_note_launch();
    } else {  // the first round's fused direction is p = z
        pcg_start_kernel<<<1, 32, 0, s>>>(H->scal);
        sr_note_launch();
    }
    H->read(S_R32, 1, s);  // <r, r> of the scaled residual (written by scale_kernel)
    const double rr0 = H->hscal[S_R32];
    if (!(rr0 > 0.0)) return 0;
    int it = 0;
    int next_check = 1;
    while (it < max_it) {
        run_round(H, precond, it & 1, s);
        it++;
        if (it == next_check || it == max_it) {
            H->read(S_PQ, 2, s);  // S_PQ, S_RRI
            const double pq = H->hscal[S_PQ], rr = H->hscal[S_RRI];
            if (!(pq > 0.0) || !isfinite(pq) || !isfinite(rr)) return precond == SR_PRECOND_LEARNED ? -2 - it : -1;
            if (rr <= eta * eta * rr0) {
                if (reached) *reached = true;
                break;
            }
            if (precond == SR_PRECOND_LEARNED && it >= kStallRounds && rr > 1e-4 * rr0) return -2 - it;
            // after the first three rounds, the next check one round before the rate seen so far (the geometric mean
            // per round) reaches the target: each check costs a host round trip, each round past convergence a V-cycle
            int more = 1;
            const double ratio = pow(rr / rr0, 1.0 / it);
            if (ratio > 0.0 && ratio < 1.0) more = (int)ceil(log(eta * eta * rr0 / rr) / log(ratio)) - 1;
            next_check = it < 3 ? it + 1 : it + std::max(1, std::min(more, 8));
        }
    }
    return it;
}

// The pass's system by FP64 refinement around FP32 PCG, x starting at the iterate, until the plain relative residual
// ||b - A x|| / ||b|| and the reference's two measures (rᵀD⁻¹r against Σ c_i u², the heat measure against
// Σ (C/Δt) T², heat.rs:480-487 and 422-431) are all within `tol`; stops early when a refinement no longer halves the
// worst of the three ratios, or past `max_rounds`.
SolveResult solve_pass(HeatSolver* H, uint32_t precond, double tol, int max_rounds, double dt, cudaStream_t s) {
    SolveResult R;
    const HeatConst& K = H->K;
    double prev = INFINITY;
    const double ub = H->hscal[S_UB], tb = H->hscal[S_TB];
    for (int ref = 0; ref < 16; ref++) {
        heat_residual64_kernel<<<H->grid_residual, RED_THREADS, 0, s>>>(K, H->residual_rows, H->scal, H->gas, H->kvac, H->kx, H->ky, H->C,
                                                               H->t, H->t0, H->x, H->r64, H->red(S_RR), Ctl{});
        sr_note_launch();
        H->read(S_RR, 4, s);
        const double rr = H->hscal[S_RR], bb = H->hscal[S_BB], gam = H->hscal[S_GAM], hm = H->hscal[S_HM];
        if (!isfinite(rr) || !isfinite(bb) || !isfinite(gam) || !isfinite(hm)) {
            R.ok = false;
            return R;
        }
        R.rel = bb > 0.0 ? sqrt(rr / bb) : 0.0;
        double worst = R.rel / tol;
        if (ub > 0.0) worst = std::max(worst, sqrt(gam / ub) / tol);
        if (tb > 0.0) worst = std::max(worst, sqrt(hm / tb) / tol);
        if (worst <= 1.0 || rr == 0.0) return R;
        if (worst > 0.5 * prev || R.rounds >= max_rounds) return R;  // stagnating, or out of rounds
        prev = worst;
        const double scale = sqrt(rr / (double)std::max(1, H->n_gas));
        set_scalar(H, S_SCALE, scale, s);
        set_scalar(H, S_ISCALE, 1.0 / scale, s);
        scale_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->r64, H->scal, H->r32, H->e32, H->red(S_R32), Ctl{});
        sr_note_launch();
        const double eta = std::min(0.5, std::max(H->inner_floor, 0.5 / worst));
        bool reached = false;
        int it = inner_pcg(H, precond, eta, max_rounds - R.rounds, s, &reached);
        if (it <= -2) {  // the learned preconditioner stalled: its inner solve is dropped, MG-PCG restarts from x
            R.rounds += -2 - it;
            R.fallback = true;
            precond = SR_PRECOND_MG;
            prev = INFINITY;
            continue;
        }
        if (it < 0) {
            R.ok = false;
            return R;
        }
        R.rounds += it;
        R.refinements++;
        correction_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->gas, H->e32, H->scal, H->x);
        sr_note_launch();
        // an intermediate Newton pass (its tolerance far above the FP32 solve's floor) trusts the FP32 solve that
        // reached its reduction: the next pass starts from a fresh residual anyway; the final pass is always verified
        if (reached && tol >= kTrustedPassTol) {
            R.rel *= eta;
            return R;
        }
    }
    return R;
}

// A pass's system and its measures' bounds (read to the host), then every coarse level and the coarsest inverse.
void build_system(HeatSolver* H, double dt, cudaStream_t s) {
    set_scalar(H, S_DT, dt, s);
    heat_system_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->K, H->scal, H->gas, H->C, H->t, H->kvac,
                                                       H->mg.L[0].c, H->x, H->red(S_UB), Ctl{});
    sr_note_launch();
    H->mg.coarsen(s);
    H->read(S_UB, 2, s);
}

// Appends a conditional node of `type` steered by `h` after everything captured so far on `s` (which is capturing),
// makes the stream's later work follow it, and returns its body graph.
cudaGraph_t capture_conditional(cudaStream_t s, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type) {
    cudaStreamCaptureStatus st;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    SR_CUDA_TRY(cudaStreamGetCaptureInfo(s, &st, nullptr, &g, &deps, &nd));
    SR_REQUIRE(st == cudaStreamCaptureStatusActive, "a conditional node outside a stream capture");
    cudaGraphNodeParams p{};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = type;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    SR_CUDA_TRY(cudaGraphAddNode(&node, g, deps, nd, &p));
    SR_CUDA_TRY(cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies));
    return p.conditional.phGraph_out[0];
}

// Captures `body(stream)` into the body graph `g` on stream `cs`; returns the kernels it launched.
template <class F>
long long capture_body(cudaGraph_t g, cudaStream_t cs, F body) {
    const long long before = (long long)sr_launches();
    SR_CUDA_TRY(cudaStreamBeginCaptureToGraph(cs, g, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    body(cs);
    cudaGraph_t out;
    SR_CUDA_TRY(cudaStreamEndCapture(cs, &out));
    const long long n = (long long)sr_launches() - before;
    sr_note_launches(-n);  // captured, not launched
    return n;
}

// The whole implicit step (MG or Jacobi preconditioner) appended to the capture in progress on `s`, whose root graph
// is `root` (the conditional handles belong to it): set-up, Δt from the device record, the device-controlled Newton
// passes, refinements and PCG rounds, and the commit. The state buffer `U` and the opacity plane are fixed in it.
void capture_heat_step(HeatSolver* H, float* U, const float* kappa, const double* dt_dev, cudaStream_t s,
                       cudaGraph_t root, bool alone) {
    Ctl ctl{H->ctl, dt_dev, {}};
    const CtlHandles& hd = ctl.hd;
    for (int b = 0; b < B_COUNT; b++) SR_CUDA_TRY(cudaGraphConditionalHandleCreate(&ctl.hd.h[b], root, 0, 0));
    const uint32_t precond = H->precond;
    const size_t nf = (size_t)(H->w + 1) * H->h + (size_t)H->w * (H->h + 1);
    long long* nb = H->body_launches;
    const long long top0 = (long long)sr_launches();
    setup_step(H, U, kappa, s, ctl);
    const long long top1 = (long long)sr_launches();
    nb[B_MAIN] = capture_body(capture_conditional(s, hd.h[B_MAIN], cudaGraphCondTypeIf), H->cap[0], [&](cudaStream_t s0) {
        if (precond != SR_PRECOND_JACOBI) {
            warm_start_kernel<<<H->grid, RED_THREADS, 0, s0>>>(H->K, H->scal, H->gas, H->t0, H->rate, H->t);
            sr_note_launch();
        }
        heat_system_kernel<<<H->grid, RED_THREADS, 0, s0>>>(H->K, H->scal, H->gas, H->C, H->t, H->kvac,
                                                            H->mg.L[0].c, H->x, H->red(S_UB), ctl);
        sr_note_launch();
        nb[B_LOOP] = capture_body(capture_conditional(s0, hd.h[B_LOOP], cudaGraphCondTypeWhile), H->cap[1],
                                  [&](cudaStream_t s1) {
            // a new system's coarse levels beside its first FP64 residual: a chain of small kernels (39 us of latency at
            // 512², 95 at 2048²) and one that takes the whole GPU, neither of which the other needs
            SR_CUDA_TRY(cudaEventRecord(H->fork[0], s1));
            SR_CUDA_TRY(cudaStreamWaitEvent(H->cap[5], H->fork[0], 0));
            nb[B_COARSEN] = capture_body(capture_conditional(H->cap[5], hd.h[B_COARSEN], cudaGraphCondTypeIf),
                                         H->cap[2], [&](cudaStream_t s2) { H->mg.coarsen(s2); });
            SR_CUDA_TRY(cudaEventRecord(H->fork[1], H->cap[5]));
            heat_residual64_kernel<<<H->grid_residual, RED_THREADS, 0, s1>>>(
                H->K, H->residual_rows, H->scal, H->gas, H->kvac, H->kx, H->ky, H->C, H->t, H->t0, H->x, H->r64,
                H->red(S_RR), ctl);
            sr_note_launch();
            SR_CUDA_TRY(cudaStreamWaitEvent(s1, H->fork[1], 0));
            scale_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->n, H->r64, H->scal, H->r32, H->e32, H->red(S_R32), ctl);
            sr_note_launch();
            nb[B_ROUND] = capture_body(capture_conditional(s1, hd.h[B_ROUND], cudaGraphCondTypeWhile), H->cap[2],
                                       [&](cudaStream_t s2) {
                precondition(H, precond, S_RZN, alone, s2);
                launch_kernel(alone && precond == SR_PRECOND_MG, spmv_dir_kernel, dim3(H->grid_spmv), dim3(RED_THREADS), 0,
                              s2, H->mg.L[0], H->spmv_rows, H->scal, H->z32, H->p32, H->p2, H->q32, H->pq_part,
                              H->rz_part, precond == SR_PRECOND_MG ? H->mg.parts() : 0);
                sr_note_launch();
                launch_kernel(alone, pcg_update4_kernel, dim3(H->grid_update), dim3(RED_THREADS), 0, s2, H->n, H->scal,
                              H->pq_part, H->grid_spmv, H->p32, H->p2, H->q32, H->e32, H->r32, H->red(S_RRI), ctl);
                sr_note_launch();
            });
            correction_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->n, H->gas, H->e32, H->scal, H->x);
            sr_note_launch();
            newton_system_kernel<<<H->grid_newton, RED_THREADS, 0, s1>>>(H->K, H->cfg.newton_cell, H->scal, H->gas, H->C,
                                                                        H->kvac, H->t, H->x, H->mg.L[0].c,
                                                                        H->red(S_MOVED), ctl);
            sr_note_launch();
        });
        nb[B_CONV] = capture_body(capture_conditional(s0, hd.h[B_CONV], cudaGraphCondTypeIf), H->cap[1],
                                  [&](cudaStream_t s1) {
            heat_flux_kernel<<<grid_for(nf), RED_THREADS, 0, s1>>>(H->K, H->gas, H->kx, H->ky, H->t, nullptr, H->fx,
                                                                   H->fy);
            sr_note_launch();
            commit_sums_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->K, H->scal, H->gas, H->C, H->t, H->t0,
                                                                H->kvac, H->red(S_RAD), ctl);
            sr_note_launch();
            commit_apply_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->K, H->scal, H->gas, H->C, H->t, H->t0, U, H->rate);
            sr_note_launch();
        });
        nb[B_LIM] = capture_body(capture_conditional(s0, hd.h[B_LIM], cudaGraphCondTypeIf), H->cap[1],
                                 [&](cudaStream_t s1) {
            limited_scale_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->K, H->scal, H->gas, H->kx, H->ky, H->t, H->C,
                                                                  H->t0, H->lscale);
            sr_note_launch();
            heat_flux_kernel<<<grid_for(nf), RED_THREADS, 0, s1>>>(H->K, H->gas, H->kx, H->ky, H->t, H->lscale, H->fx,
                                                                   H->fy);
            sr_note_launch();
            limited_apply_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->K, H->scal, H->gas, H->kx, H->ky, H->t,
                                                                  H->lscale, U, H->red(S_RAD), ctl);
            sr_note_launch();
            zero_kernel<<<H->grid, RED_THREADS, 0, s1>>>(H->rate, H->n);
            sr_note_launch();
        });
    });
    nb[B_SKIP] = capture_body(capture_conditional(s, hd.h[B_SKIP], cudaGraphCondTypeIf), H->cap[0],
                              [&](cudaStream_t s0) {
        heat_flux_kernel<<<grid_for(nf), RED_THREADS, 0, s0>>>(H->K, H->gas, H->kx, H->ky, H->t, nullptr, H->fx, H->fy);
        sr_note_launch();
    });
    nb[B_COUNT] = top1 - top0;
    sr_note_launches(-(top1 - top0));  // captured, not launched
}

// The control block's configuration for the next steps.
void ctl_configure(HeatSolver* H, cudaStream_t s) {
    HeatCtl c{};
    c.tol = H->cfg.solve_tol;
    c.nheat = H->cfg.newton_heat;
    c.ncell = H->cfg.newton_cell;
    c.inner_floor = H->inner_floor;
    c.max_passes = (int)H->max_passes;
    c.max_rounds = (int)H->max_rounds;
    c.pin = H->cfg.pin_temperature ? 1 : 0;
    *H->hctl = c;
    SR_CUDA_TRY(cudaMemcpyAsync(H->ctl, H->hctl, sizeof(HeatCtl), cudaMemcpyHostToDevice, s));
    SR_CUDA_TRY(cudaStreamSynchronize(s));
}

void drop_step_graphs(HeatSolver* H) {
    if (!H->step_graphs.empty() && H->stream) cudaStreamSynchronize(H->stream);  // none of them still running
    for (auto& kv : H->step_graphs) cudaGraphExecDestroy(kv.second);
    H->step_graphs.clear();
}

}  // namespace

HeatSolver* heat_create(const sr_config& cfg, cudaStream_t s) {
    HeatSolver* H = new HeatSolver();
    try {
        H->cfg = cfg;
        H->w = (int)cfg.width;
        H->h = (int)cfg.height;
        H->n = (size_t)H->w * H->h;
        SR_REQUIRE(cfg.precond != SR_PRECOND_LEARNED, "the learned preconditioner is loaded after creation");
        H->stream = s;
        H->precond = cfg.precond;
        H->max_passes = cfg.max_passes ? cfg.max_passes : 128;
        H->max_rounds = cfg.max_rounds ? cfg.max_rounds : 4096;
        HeatConst& K = H->K;
        K.w = H->w;
        K.h = H->h;
        K.gm1 = cfg.gamma - 1.0;
        K.mu = cfg.mu;
        K.t_floor = cfg.t_floor;
        K.sigma_vac = cfg.sigma_vac;
        K.sigma_floor = cfg.sigma_floor;
        K.a_r = cfg.a_r;
        K.c_sb = cfg.c_sb;
        K.kappa0 = cfg.kappa0;
        K.k_cond = cfg.k_cond;
        K.chi = cfg.chi;
        K.limiter_on = cfg.flux_limiter != 0;
        H->grid = grid_for(H->n);
        H->grid_newton = whole_waves(newton_system_kernel, H->n / 2);
        // rows a thread of the kernels that walk: as few as leave their threads room on the GPU all at once
        auto walk = [&](auto kernel, int columns, int& rows, int& grid) {
            const int bands = std::max(1, whole_waves(kernel, H->n) * RED_THREADS / columns);
            rows = (H->h + bands - 1) / bands;
            grid = grid_for((size_t)columns * ((H->h + rows - 1) / rows));
        };
        walk(spmv_dir_kernel, H->w / 4, H->spmv_rows, H->grid_spmv);
        walk(heat_residual64_kernel, H->w, H->residual_rows, H->grid_residual);
        H->grid_update = whole_waves(pcg_update4_kernel, H->n / 4);
        const size_t n = H->n, nx = (size_t)(H->w + 1) * H->h, ny = (size_t)H->w * (H->h + 1);
        SR_CUDA_TRY(cudaMalloc(&H->gas, n));
        double** d64[] = {&H->t0, &H->C, &H->t, &H->kvac, &H->x, &H->r64,
                          &H->lscale, &H->rate};
        for (double** p : d64) SR_CUDA_TRY(cudaMalloc(p, sizeof(double) * n));
        SR_CUDA_TRY(cudaMemset(H->rate, 0, sizeof(double) * n));
        SR_CUDA_TRY(cudaMalloc(&H->kx, sizeof(double) * nx));
        SR_CUDA_TRY(cudaMalloc(&H->ky, sizeof(double) * ny));
        float** d32[] = {&H->kap, &H->sig, &H->r32, &H->e32, &H->p32, &H->q32, &H->z32, &H->p2};
        for (float** p : d32) SR_CUDA_TRY(cudaMalloc(p, sizeof(float) * n));
        SR_CUDA_TRY(cudaMalloc(&H->fx, sizeof(float) * nx));
        SR_CUDA_TRY(cudaMalloc(&H->fy, sizeof(float) * ny));
        SR_CUDA_TRY(cudaMemset(H->fx, 0, sizeof(float) * nx));
        SR_CUDA_TRY(cudaMemset(H->fy, 0, sizeof(float) * ny));
        SR_CUDA_TRY(cudaMalloc(&H->part, sizeof(double) * 4 * PART_CAP));
        SR_CUDA_TRY(cudaMalloc(&H->rz_part, sizeof(double) * kMgMaxParts));
        SR_CUDA_TRY(cudaMalloc(&H->pq_part, sizeof(double) * MAX_PART));
        SR_CUDA_TRY(cudaMalloc(&H->counter, sizeof(unsigned)));
        SR_CUDA_TRY(cudaMemset(H->counter, 0, sizeof(unsigned)));
        SR_CUDA_TRY(cudaMalloc(&H->scal, sizeof(double) * S_COUNT));
        SR_CUDA_TRY(cudaMemset(H->scal, 0, sizeof(double) * S_COUNT));
        SR_CUDA_TRY(cudaMallocHost(&H->hscal, sizeof(double) * S_COUNT));
        SR_CUDA_TRY(cudaMalloc(&H->ctl, sizeof(HeatCtl)));
        SR_CUDA_TRY(cudaMemset(H->ctl, 0, sizeof(HeatCtl)));
        SR_CUDA_TRY(cudaMallocHost(&H->hctl, sizeof(HeatCtl)));
        for (cudaStream_t& c : H->cap) SR_CUDA_TRY(cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
        for (cudaEvent_t& e : H->fork) SR_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        H->mg.create(H->w, H->h, (int)cfg.mg_pre, (int)cfg.mg_post);
        H->mg.omega = cfg.mg_omega > 0.0 ? (float)cfg.mg_omega : 1.0f;
        H->inner_floor = cfg.inner_tol > 0.0 ? cfg.inner_tol : 1e-5;
        (void)s;
    } catch (...) {
        heat_destroy(H);
        throw;
    }
    return H;
}

void heat_destroy(HeatSolver* H) {
    if (!H) return;
    for (auto& row : H->graphs)
        for (auto& g : row)
            if (g.exec) cudaGraphExecDestroy(g.exec);
    drop_step_graphs(H);
    cudaFree(H->ctl);
    if (H->hctl) cudaFreeHost(H->hctl);
    for (cudaEvent_t e : H->fork)
        if (e) cudaEventDestroy(e);
    for (cudaStream_t c : H->cap)
        if (c) cudaStreamDestroy(c);
    cudaFree(H->gas);
    double* d64[] = {H->t0, H->C, H->t, H->kvac, H->x, H->r64, H->lscale, H->rate,
                     H->kx, H->ky};
    for (double* p : d64) cudaFree(p);
    float* d32[] = {H->kap, H->sig, H->r32, H->e32, H->p32, H->q32, H->z32, H->fx, H->fy, H->p2};
    for (float* p : d32) cudaFree(p);
    cudaFree(H->part);
    cudaFree(H->rz_part);
    cudaFree(H->pq_part);
    cudaFree(H->counter);
    cudaFree(H->scal);
    cudaFree(H->r_old);
    cudaFree(H->ez);
    cudaFree(H->vz);
    cudaFree(H->flush);
    learned_apply_destroy(H->lapply);
    if (H->hscal) cudaFreeHost(H->hscal);
    H->mg.destroy();
    delete H;
}

void heat_set_precond(HeatSolver* H, uint32_t precond) {
    if (precond == SR_PRECOND_LEARNED && !H->lapply)
        throw SrError{SR_E_UNSUPPORTED, "the learned preconditioner is not attached (sr_attach_learner)"};
    if (precond != H->precond) drop_step_graphs(H);  // a captured step holds its preconditioner
    H->precond = precond;
}

void heat_attach_learned(HeatSolver* H, Learner* L) {
    for (auto& g : H->graphs[SR_PRECOND_LEARNED])
        if (g.exec) {
            cudaGraphExecDestroy(g.exec);
            g.exec = nullptr;
        }
    learned_apply_destroy(H->lapply);
    H->lapply = nullptr;
    H->learner = L;
    if (!L) {
        if (H->precond == SR_PRECOND_LEARNED) H->precond = SR_PRECOND_MG;
        return;
    }
    if (!H->r_old) SR_CUDA_TRY(cudaMalloc(&H->r_old, sizeof(float) * H->n));
    if (!H->vz) SR_CUDA_TRY(cudaMalloc(&H->vz, sizeof(float) * H->n));
    H->lapply = learned_apply_create(L, H->w, H->h);
}

int heat_collect(HeatSolver* H, Learner* L, const float* U, const float* kappa, double dt, int crops, uint64_t seed,
                 cudaStream_t s) {
    setup_step(H, U, kappa, s);
    H->read(S_HEAT0, 2, s);
    H->n_gas = (int)H->hscal[S_NGAS];
    build_system(H, dt, s);
    heat_residual64_kernel<<<H->grid_residual, RED_THREADS, 0, s>>>(H->K, H->residual_rows, H->scal, H->gas, H->kvac, H->kx, H->ky, H->C,
                                                           H->t, H->t0, H->x, H->r64, H->red(S_RR), Ctl{});
    sr_note_launch();
    H->read(S_RR, 1, s);
    const double rr = H->hscal[S_RR];
    if (!(rr > 0.0) || !isfinite(rr)) return 0;
    const double scale = sqrt(rr / (double)std::max(1, H->n_gas));
    set_scalar(H, S_SCALE, scale, s);
    set_scalar(H, S_ISCALE, 1.0 / scale, s);
    scale_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->r64, H->scal, H->r32, H->e32, H->red(S_R32), Ctl{});
    sr_note_launch();
    if (!H->ez) SR_CUDA_TRY(cudaMalloc(&H->ez, sizeof(float) * H->n));
    // after each V-cycle z_k = M_mg r_k: the sample (r_k − A z_k, e_k + z_k); q32 is free until the next round's SpMV
    auto snapshot = [&] {
        vcycle_residual_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->mg.L[0], H->r32, H->z32, H->e32, H->q32, H->ez);
        sr_note_launch();
        learned_snapshot(L, H->mg.L[0], H->q32, H->ez, s);
    };
    const int before = learned_samples(L);
    learned_begin_collect(L, H->w, H->h, crops, seed);
    precondition(H, SR_PRECOND_MG, S_RZ0, true, s);
    snapshot();
    pcg_direction_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->scal, -1, S_RZ0, H->z32, H->p32);
    sr_note_launch();
    H->read(S_R32, 1, s);
    const double rr0 = H->hscal[S_R32];
    for (int it = 0; it < 200; it++) {
        const int rz_old = (it & 1) ? S_RZ1 : S_RZ0, rz_new = (it & 1) ? S_RZ0 : S_RZ1;
        spmv_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->mg.L[0], H->p32, H->q32, H->red(S_PQ));
        sr_note_launch();
        pcg_update_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->scal, rz_old, H->p32, H->q32, H->e32, H->r32,
                                                          H->red(S_RRI));
        sr_note_launch();
        H->read(S_PQ, 2, s);
        // solve on to a 1e-6 residual reduction; samples only while the remaining error is large against that
        if (!(H->hscal[S_PQ] > 0.0) || H->hscal[S_RRI] <= 1e-12 * rr0) break;
        precondition(H, SR_PRECOND_MG, rz_new, true, s);
        if (H->hscal[S_RRI] > 1e-8 * rr0) snapshot();
        pcg_direction_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->n, H->scal, rz_old, rz_new, H->z32, H->p32);
        sr_note_launch();
    }
    learned_end_collect(L, H->mg.L[0], H->e32, s);
    return learned_samples(L) - before;
}

void heat_reset(HeatSolver* H, cudaStream_t s) { SR_CUDA_TRY(cudaMemsetAsync(H->rate, 0, sizeof(double) * H->n, s)); }

void heat_rate_to_f32(HeatSolver* H, float* dst, cudaStream_t s) {
    f64_to_f32_kernel<<<H->grid, RED_THREADS, 0, s>>>(dst, H->rate, H->n);
    sr_note_launch();
    SR_CUDA_TRY(cudaGetLastError());
}

void heat_rate_from_f32(HeatSolver* H, const float* src, cudaStream_t s) {
    if (!src) {
        heat_reset(H, s);
        return;
    }
    f32_to_f64_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->rate, src, H->n);
    sr_note_launch();
    SR_CUDA_TRY(cudaGetLastError());
}

void heat_set_reference(HeatSolver* H, const HeatRef& R) {
    H->ref = R;
    H->K.ref = R.on;
    drop_step_graphs(H);
}

void heat_flux_planes(const HeatSolver* H, const float** fx, const float** fy) {
    *fx = H->fx;
    *fy = H->fy;
}

double* heat_rate_plane(HeatSolver* H) { return H->rate; }

bool heat_wait_error(HeatSolver* H, cudaStream_t s) { return H->mg.error(s); }

void heat_set_limits(HeatSolver* H, uint32_t max_passes, uint32_t max_rounds) {
    H->max_passes = max_passes;
    H->max_rounds = max_rounds;
    drop_step_graphs(H);  // the next step captures again, with the new limits in its control block
}

void heat_read_flux(HeatSolver* H, float* fx, float* fy) {
    const size_t nx = (size_t)(H->w + 1) * H->h, ny = (size_t)H->w * (H->h + 1);
    if (fx) SR_CUDA_TRY(cudaMemcpy(fx, H->fx, sizeof(float) * nx, cudaMemcpyDeviceToHost));
    if (fy) SR_CUDA_TRY(cudaMemcpy(fy, H->fy, sizeof(float) * ny, cudaMemcpyDeviceToHost));
}

// Reads the device-controlled steps' control block: the last step's report, and the kernels its bodies launched since
// the last read (added to the library's launch count).
void heat_sync_report(HeatSolver* H, cudaStream_t s) {
    if (!H->report_pending) return;
    SR_CUDA_TRY(cudaMemcpyAsync(H->hctl, H->ctl, sizeof(HeatCtl), cudaMemcpyDeviceToHost, s));
    SR_CUDA_TRY(cudaMemsetAsync(H->ctl->runs, 0, sizeof(H->ctl->runs), s));
    SR_CUDA_TRY(cudaStreamSynchronize(s));
    const HeatCtl& c = *H->hctl;
    long long n = 0;
    for (int b = 0; b < B_COUNT; b++) n += (long long)c.runs[b] * H->body_launches[b];
    sr_note_launches(n);
    sr_heat_report R{};
    R.precond = H->precond;
    R.dt = c.dt;
    R.passes = (uint32_t)c.passes;
    R.rounds = (uint32_t)c.rounds;
    R.refinements = (uint32_t)c.refinements;
    R.converged = (uint32_t)c.converged;
    R.delta = c.delta;
    R.radiated = c.radiated;
    R.rel_residual = c.rel;
    H->report = R;
    H->report_pending = false;
}

void heat_step(HeatSolver* H, float* U, const float* kappa, const double* dt_dev, cudaStream_t s,
               sr_heat_report* rep) {
    if (H->precond != SR_PRECOND_LEARNED && H->use_graphs) {
        // the device-controlled step: captured once per state buffer, then replayed with no host round trip
        auto it = H->step_graphs.find(U);
        if (it == H->step_graphs.end()) {
            heat_sync_report(H, s);
            ctl_configure(H, s);
            cudaGraph_t g;
            SR_CUDA_TRY(cudaGraphCreate(&g, 0));
            SR_CUDA_TRY(cudaStreamBeginCaptureToGraph(s, g, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
            try {
                capture_heat_step(H, U, kappa, dt_dev, s, g, true);
            } catch (...) {
                cudaGraph_t dead;
                cudaStreamEndCapture(s, &dead);
                cudaGraphDestroy(g);
                throw;
            }
            cudaGraph_t out;
            SR_CUDA_TRY(cudaStreamEndCapture(s, &out));
            cudaGraphExec_t exec;
            const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
            cudaGraphDestroy(g);
            SR_CUDA_TRY(e);
            it = H->step_graphs.emplace(U, exec).first;
        }
        SR_CUDA_TRY(cudaGraphLaunch(it->second, s));
        sr_note_launches(H->body_launches[B_COUNT]);
        H->report_pending = true;
        (void)rep;
        return;
    }
    heat_sync_report(H, s);
    sr_heat_report R{};
    R.precond = H->precond;
    setup_step(H, U, kappa, s);
    SR_CUDA_TRY(cudaMemcpyAsync(H->scal + S_DT, dt_dev, sizeof(double), cudaMemcpyDeviceToDevice, s));
    H->read(S_HEAT0, 3, s);  // Σ C T⁰, gas cells, Δt
    H->n_gas = (int)H->hscal[S_NGAS];
    const double dt = H->hscal[S_DT];
    const double heat0 = H->hscal[S_HEAT0];
    const size_t nf = (size_t)(H->w + 1) * H->h + (size_t)H->w * (H->h + 1);
    if (H->cfg.pin_temperature || H->n_gas == 0 || !(dt > 0.0)) {
        heat_flux_kernel<<<grid_for(nf), RED_THREADS, 0, s>>>(H->K, H->gas, H->kx, H->ky, H->t, nullptr, H->fx,
                                                               H->fy);
        sr_note_launch();
        R.converged = 1;
        H->report = R;
        *rep = R;
        return;
    }
    R.dt = dt;
    if (H->precond != SR_PRECOND_JACOBI) {
        warm_start_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->K, H->scal, H->gas, H->t0, H->rate, H->t);
        sr_note_launch();
    }
    uint32_t passes = 0, rounds = 0;
    bool converged = false;
    // Inexact Newton: a pass's solve is asked for the last pass's relative heat moved (the first pass for
    // kFirstPassTol), never more than kFirstPassTol nor less than solve_tol; the passes end only on a pass solved to
    // solve_tol. Loose early passes cost fewer rounds in all than accurate ones: each pass's system is rebuilt at the
    // new iterate anyway, and the last pass meets the same tolerances.
    const double tol = H->cfg.solve_tol;
    double pass_tol = std::max(tol, kFirstPassTol);
    const double nheat = H->cfg.newton_heat, ncell = H->cfg.newton_cell;
    double moved_prev = 0.0;
    build_system(H, dt, s);
    while (passes < H->max_passes && rounds < H->max_rounds) {
        passes++;
        SolveResult S = solve_pass(H, H->precond, pass_tol, (int)(H->max_rounds - rounds), dt, s);
        rounds += (uint32_t)S.rounds;
        R.refinements += (uint32_t)S.refinements;
        R.rel_residual = S.rel;
        if (S.fallback) R.fallback_used = 1;
        if (!S.ok) break;
        newton_system_kernel<<<H->grid_newton, RED_THREADS, 0, s>>>(H->K, ncell, H->scal, H->gas, H->C, H->kvac, H->t, H->x, H->mg.L[0].c, H->red(S_MOVED), Ctl{});
        sr_note_launch();
        H->read(S_MOVED, 4, s);  // moved, violations, and the next system's two bounds
        const double rel_moved = heat0 > 0.0 ? H->hscal[S_MOVED] / heat0 : 0.0;
        if (rel_moved <= nheat && H->hscal[S_VIOL] == 0.0 && pass_tol <= tol) {
            converged = true;
            break;
        }
        // the next pass is solved to solve_tol once it is expected to move less than newton_heat (the passes' observed
        // contraction times this pass's move), since only a pass solved to solve_tol can end them
        const double ratio = moved_prev > 0.0 ? std::min(1.0, std::max(0.01, rel_moved / moved_prev)) : 0.1;
        moved_prev = rel_moved;
        pass_tol = std::max(tol, std::min(kFirstPassTol, rel_moved));
        if (ratio * rel_moved <= nheat) pass_tol = tol;
        H->mg.coarsen(s);  // the next pass's coarse levels (its level-0 c is in place)
    }
    R.passes = passes;
    R.rounds = rounds;
    if (converged) {
        heat_flux_kernel<<<grid_for(nf), RED_THREADS, 0, s>>>(H->K, H->gas, H->kx, H->ky, H->t, nullptr, H->fx, H->fy);
        sr_note_launch();
        commit_sums_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->K, H->scal, H->gas, H->C, H->t, H->t0, H->kvac,
                                                           H->red(S_RAD), Ctl{});
        sr_note_launch();
        H->read(S_RAD, 3, s);
        const double rad = H->hscal[S_RAD], gain = H->hscal[S_GAIN], held = H->hscal[S_HELD];
        const double delta = -(gain + rad) / held;
        set_scalar(H, S_DELTA, delta, s);
        commit_apply_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->K, H->scal, H->gas, H->C, H->t, H->t0, U, H->rate);
        sr_note_launch();
        R.converged = 1;
        R.delta = delta;
        R.radiated = rad;
    } else {
        limited_scale_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->K, H->scal, H->gas, H->kx, H->ky, H->t, H->C, H->t0,
                                                             H->lscale);
        sr_note_launch();
        heat_flux_kernel<<<grid_for(nf), RED_THREADS, 0, s>>>(H->K, H->gas, H->kx, H->ky, H->t, H->lscale, H->fx,
                                                               H->fy);
        sr_note_launch();
        limited_apply_kernel<<<H->grid, RED_THREADS, 0, s>>>(H->K, H->scal, H->gas, H->kx, H->ky, H->t, H->lscale, U,
                                                             H->red(S_RAD), Ctl{});
        sr_note_launch();
        SR_CUDA_TRY(cudaMemsetAsync(H->rate, 0, sizeof(double) * H->n, s));
        H->read(S_RAD, 1, s);
        R.converged = 0;
        R.delta = 0.0;
        R.radiated = H->hscal[S_RAD];
    }
    SR_CUDA_TRY(cudaGetLastError());
    H->report = R;
    *rep = R;
}

void heat_report(HeatSolver* H, cudaStream_t s, sr_heat_report* rep) {
    heat_sync_report(H, s);
    *rep = H->report;
}

void heat_account_launches(HeatSolver* H, cudaStream_t s) { heat_sync_report(H, s); }

bool heat_capturable(const HeatSolver* H) {
    return H->precond != SR_PRECOND_LEARNED && H->use_graphs;
}

void heat_prepare_capture(HeatSolver* H, cudaStream_t s) {
    heat_sync_report(H, s);
    ctl_configure(H, s);
}

long long heat_capture_step(HeatSolver* H, float* U, const float* kappa, const double* dt_dev, cudaStream_t s,
                            cudaGraph_t root, bool alone) {
    capture_heat_step(H, U, kappa, dt_dev, s, root, alone);
    return H->body_launches[B_COUNT];
}

void heat_graph_launched(HeatSolver* H) { H->report_pending = true; }

void heat_first_solve(HeatSolver* H, const float* U, const float* kappa, double dt, uint32_t precond, cudaStream_t s,
                      double* ms, uint32_t* rounds, double* rel_residual, double* x, uint32_t* fallback) {
    if (precond == SR_PRECOND_LEARNED && !H->lapply)
        throw SrError{SR_E_UNSUPPORTED, "the learned preconditioner is not attached (sr_attach_learner)"};
    setup_step(H, U, kappa, s);
    H->read(S_HEAT0, 2, s);
    H->n_gas = (int)H->hscal[S_NGAS];
    build_system(H, dt, s);
    cudaEvent_t a, b;
    SR_CUDA_TRY(cudaEventCreate(&a));
    SR_CUDA_TRY(cudaEventCreate(&b));
    SR_CUDA_TRY(cudaEventRecord(a, s));
    SolveResult S = solve_pass(H, precond, H->cfg.solve_tol, (int)H->max_rounds, dt, s);
    SR_CUDA_TRY(cudaEventRecord(b, s));
    SR_CUDA_TRY(cudaEventSynchronize(b));
    float t = 0.0f;
    SR_CUDA_TRY(cudaEventElapsedTime(&t, a, b));
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (ms) *ms = t;
    if (rounds) *rounds = (uint32_t)S.rounds;
    if (rel_residual) *rel_residual = S.rel;
    if (fallback) *fallback = S.fallback ? 1u : 0u;
    if (x) SR_CUDA_TRY(cudaMemcpy(x, H->x, sizeof(double) * H->n, cudaMemcpyDeviceToHost));
    SR_CUDA_TRY(cudaGetLastError());
}

void heat_time_smoother(HeatSolver* H, int reps, cudaStream_t s, double* pre_ms, double* post_ms) {
    constexpr size_t kFlush = (size_t)256 << 20;  // twice the L2
    if (!H->flush) SR_CUDA_TRY(cudaMalloc(&H->flush, kFlush));
    H->mg.time_level0(reps, H->flush, kFlush, s, pre_ms, post_ms);
}
