// hydro.cu — P4, the MUSCL-Hancock/HLL gas step, as one tiled stencil kernel per pass (sm_100a, FP32).
//
// One CTA owns a tile of output cells; the tile grown by two cells (the reconstruction's reach) arrives in shared
// memory by one TMA box, the world's ghosts are formed there, every lane runs the Hancock predictor for one cell (the
// tile's and the one-cell ring around it), the faces meet for the HLL fluxes by warp shuffles (x) and shared memory
// (y), and the per-cell epilogue of the pass finishes:
//   - kHydroStep:       U' = U - Δt ΔF, then P8's floors and P9's Δt on U' (no gravity, no heat: the whole step);
//   - kHydroUpdate:     U' = U - Δt ΔF (no gravity; heat follows, or the passes are timed one by one);
//   - kHydroPredict:    with gravity: U - Δt ΔF, the half step's source ½(Σⁿ + Σⁿ⁺¹), masked (reference
//                       hydro.rs:815-836), and what gravity's work reads — the half-step (Σ, Σu, Σv) and the faces'
//                       mass fluxes. Once φ_mid is solved, hydro_gravity_kernel adds the half-step kick and the faces'
//                       work across it (hydro.rs:871-947) and takes the net kick back from the densest cell.
// The predictor runs once a step: it is what the step costs (FP32 issue), and a second run of it after the solve, to
// recompute fluxes that 20 B a cell can carry over, took 172 + 331 us at 2048² where predict and gravity take 208 + 89.
// The scheme follows crates/sr-physics/src/reference/hydro.rs (step_held without held cells, sinks or radiation).
#include "hydro.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <tuple>

#include "tma.cuh"

namespace {

__device__ __forceinline__ float lim_mc(float l, float c, float r) {
    float a = c - l, b = r - c;
    if (a * b <= 0.0f) return 0.0f;
    return copysignf(fminf(fminf(fabsf(0.5f * (a + b)), 2.0f * fabsf(a)), 2.0f * fabsf(b)), a);
}

__device__ __forceinline__ float lim_minmod(float l, float c, float r) {
    float a = c - l, b = r - c;
    if (a * b <= 0.0f) return 0.0f;
    return copysignf(fminf(fabsf(a), fabsf(b)), a);
}

template <int LIM>
__device__ __forceinline__ float lim(float l, float c, float r) {
    return LIM == SR_LIMITER_MINMOD ? lim_minmod(l, c, r) : lim_mc(l, c, r);
}

// Limited slopes of (Σ, u, v, Π) along one axis; Σ and Π flat where the thermal bracket refuses a face
// (hydro.rs:293-331, HOT_FACE = 2). The limiter and the bracket are the kernel's template parameters.
template <int LIM, bool BRACKET>
__device__ __forceinline__ Prim slope(const Prim& l, const Prim& c, const Prim& r, float ql, float qc, float qr) {
    Prim s;
    s.s = lim<LIM>(l.s, c.s, r.s);
    s.u = lim<LIM>(l.u, c.u, r.u);
    s.v = lim<LIM>(l.v, c.v, r.v);
    s.p = lim<LIM>(l.p, c.p, r.p);
    if (BRACKET) {
        float hottest = fmaxf(fmaxf(ql, qc), qr);  // Π/Σ of the three cells, staged once per cell
        float plo = c.p - 0.5f * s.p, blo = 2.0f * hottest * (c.s - 0.5f * s.s);
        float phi = c.p + 0.5f * s.p, bhi = 2.0f * hottest * (c.s + 0.5f * s.s);
        if (!(plo <= blo) || !(phi <= bhi)) {
            s.s = 0.0f;
            s.p = 0.0f;
        }
    }
    return s;
}

__device__ __forceinline__ Prim offset(const Prim& c, const Prim& s, float f) {
    Prim o;
    o.s = c.s + f * s.s;
    o.u = c.u + f * s.u;
    o.v = c.v + f * s.v;
    o.p = c.p + f * s.p;
    return o;
}

// Gravity's source at one face over the step (hydro.rs:1042-1067): [impulse to the low cell, low energy, high energy].
__device__ __forceinline__ void face_work(float q, float sl, float sh, float pl, float ph, float d, float dt, float* o) {
    float a = fmaxf(sl, 0.0f), b = fmaxf(sh, 0.0f);
    float w = a + b > 0.0f ? sr_div(a, a + b) : 0.5f;
    float extra = dt * (q - 0.5f * (pl + ph)) * d;
    float c = 0.0f, kick = 0.0f, el = 0.0f, eh = 0.0f;
    if (extra < 0.0f && a > 0.0f && b > 0.0f) {
        float ul = sr_div(pl, a), uh = sr_div(ph, b);
        float du = ul - uh;
        float inv = sr_div(1.0f, a) + sr_div(1.0f, b);
        c = fminf(-extra, sr_div(0.25f * du * du, inv));
        if (c > 0.0f) {
            float disc = sr_sqrt(du * du - 2.0f * inv * c);
            kick = sr_div(-2.0f * c, du + copysignf(1.0f, du) * disc);
            el = ul * kick + sr_div(0.5f * kick * kick, a);
            eh = -uh * kick + sr_div(0.5f * kick * kick, b);
        }
    }
    float rest = extra + c;
    o[0] = kick;
    o[1] = 0.5f * dt * pl * d + w * rest + el;
    o[2] = 0.5f * dt * ph * d + (1.0f - w) * rest + eh;
}

// ---- the band kernel: one warp per row of the tile, one lane per cell
//
// A CTA covers HB_TX x HB_TY output cells with HB_W = HB_TY + 2 warps of 32 lanes: warp r is the row y0 - 1 + r and
// lane l the column x0 - 1 + l, so the ring of cells around the tile (whose faces toward the tile the fluxes need) is
// computed by the same straight-line code as the tile itself: lanes 0 and 31 and warps 0 and HB_W - 1 predict but
// write nothing. The four planes of the tile grown by two cells (the reconstruction's reach) arrive in one TMA box;
// the world's ghosts (hydro.rs:686-709) are formed from it in shared memory. Each lane predicts its cell's four faces
// (hydro.rs:587-614); the x faces meet by warp shuffles (a lane's x+ face against the next lane's x- face), the y faces
// through shared memory (a row's y+ faces against the next row's y- faces); the fluxes go back the same ways. The kernel
// is persistent, two CTAs per SM walking the tiles: a tile's box lands while the one before is worked on, and the grid's
// sum takes one ticket a CTA (a CTA per tile held its SM for the box's and the ticket's latency: gas alone at 512²,
// 23.6 -> 19.6 us a step).
constexpr int HB_TX = 30, HB_TY = 14, HB_W = HB_TY + 2, HB_NT = 32 * HB_W;
constexpr int HB_SX = HB_TX + 4, HB_SY = HB_TY + 4;  // the staged region: the tile grown by 2
constexpr int HB_BX = 40, HB_BY = HB_SY;             // the TMA box: from a 16-byte aligned column, wide enough
constexpr uint32_t kHydroWaitPolls = 1u << 24;       // an mbarrier wait gives up after this many polls

// A predicted face: its conserved vector and the primitives it stands for (Σ is U0).
struct FaceS {
    float U0, U1, U2, U3, u, v, P;
};

// What the CTAs sum: gravity's net kick (FP64) and the densest cell (the lowest index on a tie), or the largest wave
// rate and the first non-finite value (cell * 4 + channel).
struct KickPart {
    double kx, ky;
    float best;
    int idx;
    __device__ __forceinline__ static KickPart none() { return KickPart{0.0, 0.0, 0.0f, -1}; }
    __device__ __forceinline__ void merge(const KickPart& o) {
        kx += o.kx;
        ky += o.ky;
        if (o.idx >= 0 && (idx < 0 || o.best > best || (o.best == best && o.idx < idx))) {
            best = o.best;
            idx = o.idx;
        }
    }
    __device__ __forceinline__ KickPart down(int o) const {
        return KickPart{__shfl_down_sync(0xffffffffu, kx, o), __shfl_down_sync(0xffffffffu, ky, o),
                        __shfl_down_sync(0xffffffffu, best, o), __shfl_down_sync(0xffffffffu, idx, o)};
    }
};
struct RatePart {
    long long nf;
    float rate;
    __device__ __forceinline__ static RatePart none() { return RatePart{LLONG_MAX, 0.0f}; }
    __device__ __forceinline__ void merge(const RatePart& o) {
        nf = o.nf < nf ? o.nf : nf;
        rate = fmaxf(rate, o.rate);
    }
    __device__ __forceinline__ RatePart down(int o) const {
        return RatePart{__shfl_down_sync(0xffffffffu, nf, o), __shfl_down_sync(0xffffffffu, rate, o)};
    }
};
static_assert(sizeof(KickPart) == kHydroPartBytes && sizeof(RatePart) <= kHydroPartBytes, "a partial's slot");

template <class P>
__device__ __forceinline__ P warp_merge(P v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v.merge(v.down(o));
    return v;
}

// The grid's total of the CTAs' partials `v` (lane 0's), by warp 0 of every CTA: the last CTA of a grid row to arrive
// merges the row's partials and the last row to arrive the rows', each in a fixed order (two short tickets instead of
// one CTA walking all partials: at 2048² 10,143 of them took a kernel of their own 52 us). True, with the total in
// lane 0, in the one warp that arrives last; the tickets are left at 0 for the next launch.
template <class P>
__device__ __forceinline__ bool grid_total(P& v, void* parts, unsigned* tickets) {
    P* part = reinterpret_cast<P*>(parts);
    P* rows = part + (size_t)gridDim.x * gridDim.y;
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int level = 0; level < (gridDim.y > 1 ? 2 : 1); level++) {
        P* slot = level ? rows + blockIdx.y : part + (size_t)blockIdx.y * gridDim.x + blockIdx.x;
        unsigned* ticket = tickets + (level ? gridDim.y : blockIdx.y);
        const unsigned count = level ? gridDim.y : gridDim.x;
        const P* from = level ? rows : part + (size_t)blockIdx.y * gridDim.x;
        bool last = false;
        if (lane == 0) {
            *slot = v;
            __threadfence();
            last = atomicAdd(ticket, 1u) == count - 1;
            if (last) *ticket = 0u;
            __threadfence();
        }
        if (!__shfl_sync(0xffffffffu, last, 0)) return false;
        P t = P::none();
        for (unsigned k = lane; k < count; k += 32) {
            P o;
            const double* src = reinterpret_cast<const double*>(from + k);
#pragma unroll
            for (int q = 0; q < (int)(sizeof(P) / sizeof(double)); q++) reinterpret_cast<double*>(&o)[q] = __ldcg(src + q);
            t.merge(o);
        }
        v = warp_merge(t);
    }
    return true;
}

struct __align__(128) BandShared {
    float raw2[2][4][HB_BY][HB_BX];  // the TMA boxes of Σ, Σu, Σv, E, this tile's and the next's (128-byte aligned)
    float4 P[HB_SY][HB_SX];      // primitives (Σ, u, v, Π) of the staged region, ghosts included
    float Q[HB_SY][HB_SX];       // Π/Σ (the thermal bracket's temperatures)
    float S[HB_SY][HB_SX];       // raw Σ (out of the world: -1, read as vacuum)
    float M[3][HB_W][32];        // half-step (Σ, Σu, Σv) of each lane's cell
    float YF[7][HB_W][32];       // each lane's y+ face
    float FY[4][HB_W][32];       // the flux through each lane's top face
    RatePart red[HB_W];          // the rows' partials
    uint64_t mbar[2];
};
static_assert(sizeof(float) * 4 * HB_BY * HB_BX % 128 == 0, "the second box is 128-byte aligned");

__device__ __forceinline__ Prim prim_at(const BandShared& sh, int y, int x) {
    const float4 q = sh.P[y][x];
    Prim p;
    p.s = q.x; p.u = q.y; p.v = q.z; p.p = q.w;
    return p;
}

// The Euler flux of the unevolved face c + f s normal to `dir` (the Hancock increment's terms).
__device__ __forceinline__ void face_flux(const HydroConst& H, const Prim& c, const Prim& s, float f, int dir,
                                          float* out) {
    const Prim wf = offset(c, s, f);
    float uf[4];
    eos_cons(H, wf, uf);
    euler_flux(wf, uf[3], dir, out);
}

// The face c + f s advanced by the Hancock increment and gravity's half-kick, or unevolved when the advanced one is no
// state (hydro.rs:501-513, 587-614).
__device__ __forceinline__ FaceS face_state(const HydroConst& H, const Prim& c, const Prim& s, float f,
                                            const float* delta, float half, bool grav, float gx, float gy) {
    const Prim wf = offset(c, s, f);
    float uf[4];
    eos_cons(H, wf, uf);
    float d[4] = {delta[0], delta[1], delta[2], delta[3]};
    if (grav) {
        d[1] += half * wf.s * gx;
        d[2] += half * wf.s * gy;
        d[3] += half * wf.s * ((wf.u + 0.5f * half * gx) * gx + (wf.v + 0.5f * half * gy) * gy);
    }
    const float U[4] = {uf[0] + d[0], uf[1] + d[1], uf[2] + d[2], uf[3] + d[3]};
    Prim p;
    FaceS F;
    if (eos_prim(H, U, p)) {
        F.U0 = U[0]; F.U1 = U[1]; F.U2 = U[2]; F.U3 = U[3];
        F.u = p.u; F.v = p.v; F.P = p.p;
    } else {
        F.U0 = uf[0]; F.U1 = uf[1]; F.U2 = uf[2]; F.U3 = uf[3];
        F.u = wf.u; F.v = wf.v; F.P = wf.p;
    }
    return F;
}

__device__ __forceinline__ FaceS shfl_face_down(const FaceS& F) {
    FaceS R;
    R.U0 = __shfl_down_sync(0xffffffffu, F.U0, 1);
    R.U1 = __shfl_down_sync(0xffffffffu, F.U1, 1);
    R.U2 = __shfl_down_sync(0xffffffffu, F.U2, 1);
    R.U3 = __shfl_down_sync(0xffffffffu, F.U3, 1);
    R.u = __shfl_down_sync(0xffffffffu, F.u, 1);
    R.v = __shfl_down_sync(0xffffffffu, F.v, 1);
    R.P = __shfl_down_sync(0xffffffffu, F.P, 1);
    return R;
}

__device__ __forceinline__ void flux_of(const FaceS& F, int dir, float* f) {
    Prim p;
    p.s = F.U0; p.u = F.u; p.v = F.v; p.p = F.P;
    euler_flux(p, F.U3, dir, f);
}

// HLL with Davis speeds across a face normal to `dir` (hydro.rs:516-540).
__device__ __forceinline__ void hll_s(const HydroConst& H, const FaceS& l, const FaceS& r, int dir, float* f) {
    const float unl = dir == 0 ? l.u : l.v, unr = dir == 0 ? r.u : r.v;
    const float cl = sr_sqrt(H.gamma * sr_div(l.P, l.U0)), cr = sr_sqrt(H.gamma * sr_div(r.P, r.U0));
    const float s_l = fminf(unl - cl, unr - cr);
    const float s_r = fmaxf(unl + cl, unr + cr);
    float fl[4], fr[4];
    flux_of(l, dir, fl);
    flux_of(r, dir, fr);
    if (s_l >= 0.0f) {
#pragma unroll
        for (int k = 0; k < 4; k++) f[k] = fl[k];
    } else if (s_r <= 0.0f) {
#pragma unroll
        for (int k = 0; k < 4; k++) f[k] = fr[k];
    } else {
        const float inv = sr_div(1.0f, s_r - s_l);
        const float dU[4] = {r.U0 - l.U0, r.U1 - l.U1, r.U2 - l.U2, r.U3 - l.U3};
#pragma unroll
        for (int k = 0; k < 4; k++) f[k] = (s_r * fl[k] - s_l * fr[k] + s_l * s_r * dU[k]) * inv;
    }
}

__device__ __forceinline__ void wall_s(const FaceS& own, int dir, float* f) {  // hydro.rs:556-562
    f[0] = 0.0f; f[1] = 0.0f; f[2] = 0.0f; f[3] = 0.0f;
    f[1 + dir] = own.P;
}

// The flux through face `at` (along `dir`) of the world (0 and `edge` are its walls; hydro.rs:564-582, 744-775),
// between the faces L and R; zero for a face outside the world (`inside` false).
__device__ __forceinline__ void face_flux_at(const HydroConst& H, const FaceS& L, const FaceS& R, int dir, int at,
                                             int edge, bool inside, float* f) {
    if (!inside || at < 0 || at > edge) {
        f[0] = f[1] = f[2] = f[3] = 0.0f;
    } else if (at == 0) {
        if (H.edge == SR_EDGE_BOUNCE) {
            wall_s(R, dir, f);
        } else {
            hll_s(H, L, R, dir, f);
            if (f[0] > 0.0f) wall_s(R, dir, f);
        }
    } else if (at == edge) {
        if (H.edge == SR_EDGE_BOUNCE) {
            wall_s(L, dir, f);
        } else {
            hll_s(H, L, R, dir, f);
            if (f[0] < 0.0f) wall_s(L, dir, f);
        }
    } else {
        hll_s(H, L, R, dir, f);
    }
}

// P8 on one cell: the vacuum reset and the thermal floor (reference/floors.rs:124-196, Σ_vac and Σ_floor as the planes'
// f32); returns which values changed (1: E alone, 2: all).
__device__ __forceinline__ int floor_cell(const HydroConst& H, float& s, float& mx, float& my, float& e) {
    if (s < H.sigma_vac) {
        s = H.sigma_floor;
        mx = 0.0f;
        my = 0.0f;
        e = H.sigma_floor * H.eps_floor;
        return 2;
    }
    const float kinetic = 0.5f * (mx * mx + my * my) / (s * s);
    const float raw = e / s - kinetic;
    if (raw < H.eps_floor) {
        e = e + s * (H.eps_floor - raw);
        return 1;
    }
    return 0;
}

// P9's terms of one floored cell: its wave rate (|u|+c)+(|v|+c) (hydro.rs:618-634) and the non-finite guard's code.
__device__ __forceinline__ void rate_cell(const HydroConst& H, float s, float mx, float my, float e, size_t i,
                                          float& rate, long long& nf) {
    if (!(isfinite(s) && isfinite(mx) && isfinite(my) && isfinite(e))) {
        const int c = !isfinite(s) ? 0 : (!isfinite(mx) ? 1 : (!isfinite(my) ? 2 : 3));
        const long long code = (long long)i * 4 + c;
        nf = code < nf ? code : nf;
    }
    const Prim p = eos_read(H, s, mx, my, e);
    const float c = eos_sound(H, p);
    rate = fmaxf(rate, (fabsf(p.u) + c) + (fabsf(p.v) + c));
}

// Δt_{n+1} = min(C / max rate, η_g / sqrt(max |g|)) (hydro.rs:618-634), the configured fixed Δt or cap, and the guard;
// with `advance` the step that ends here is booked first (P1: it ran on Δt_n = the last Δt_{n+1}, f64 sim time).
__device__ void dt_close(const DtRule& R, float rate, float gmax, long long nf, int channels) {
    DtRecord* rec = R.rec;
    if (R.advance) {
        rec->dt = rec->dt_next;
        rec->sim_time += rec->dt;
        rec->steps += 1;
    }
    double dt = R.cfl / (double)rate;
    if (gmax > 0.0f) dt = fmin(dt, R.eta_g / sqrt((double)gmax));
    if (R.dt_fixed > 0.0) dt = R.dt_fixed;
    if (R.dt_cap > 0.0) dt = fmin(dt, R.dt_cap);
    rec->dt_next = dt;
    if (nf != LLONG_MAX && !rec->non_finite) {
        rec->non_finite = 1;
        rec->nf_cell = nf / channels;
        rec->nf_channel = (int)(nf % channels);
        rec->nf_step = rec->steps;
    }
}

// The CTA's last word on gravity's kick: its warps' partials merged, then the grid's; the warp that arrives last takes
// the net kick on the gas's own field back from the densest cell (hydro.rs:1004-1012).
template <int WARPS>
__device__ __forceinline__ void take_back(KickPart kp, KickPart* red, const HydroArgs& A) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t n = (size_t)A.H.w * A.H.h;
    kp = warp_merge(kp);
    if (lane == 0) red[warp] = kp;
    __syncthreads();
    if (warp > 0) return;
    kp = warp_merge(lane < WARPS ? red[lane] : KickPart::none());
    if (grid_total(kp, A.part, A.tickets) && lane == 0 && kp.idx >= 0) {
        A.Uout[n + kp.idx] = __ldcg(A.Uout + n + kp.idx) - (float)kp.kx;
        A.Uout[2 * n + kp.idx] = __ldcg(A.Uout + 2 * n + kp.idx) - (float)kp.ky;
    }
}

// Gravity's part of the step, after the half step's solve: each cell's kick Δt Σ_src g_mid and its four faces' work.
// A thread takes four neighbouring columns (16-byte accesses: the world's width is a multiple of 8) of HG_R rows,
// works out the faces to the right of and below each of its cells once, and hands the right one to the next lane; a
// cell with no gas around it (its source stored as -0) takes nothing but lends its faces. Bound by latency: 60 B a cell at
// 2.8 TB/s (2048²: 89 us, DRAM at 32 %, issue 42 %) with the 16 warps an SM that 125 registers leave, each waiting on its
// row's loads and on the faces' divisions and square roots in turn.
constexpr int HG_R = 4, HG_WARPS = 4, HG_COLS = 128;

__global__ void __launch_bounds__(32 * HG_WARPS, 4) hydro_gravity_kernel(HydroArgs A) {
    __shared__ KickPart red[HG_WARPS];
    const int w = A.H.w, h = A.H.h;
    const size_t n = (size_t)w * h;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * HG_COLS + 4 * lane, y0 = (blockIdx.y * HG_WARPS + warp) * HG_R;
    const float dt = (float)(*A.dt);
    const bool on = x < w;
    struct Row {
        float m[3][4], p[4];
    };
    // what this kernel does not write, as read-only loads: the stores of one row hold back no load of the next
    auto load4 = [&](const float* a, size_t i, float* v) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(a + i));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    };
    auto load_row = [&](int y, Row& r) {
        const bool ok = on && y >= 0 && y < h;
        const size_t i = ok ? (size_t)y * w + x : 0;
#pragma unroll
        for (int k = 0; k < 3; k++) load4(A.mid + k * n, i, r.m[k]);
        load4(A.phim, i, r.p);
    };
    KickPart kp = KickPart::none();
    Row c, d;
    float upk[4], upe[4];  // the face above each cell: impulse to the cell above, energy to this one
    load_row(y0, c);
    {
        Row a;
        float f[4];
        load_row(y0 - 1, a);
        const bool ok = on && y0 > 0 && y0 < h;
        load4(A.mfy, ok ? (size_t)(y0 - 1) * w + x : 0, f);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float o[3] = {0.0f, 0.0f, 0.0f};
            if (ok) face_work(f[k], a.m[0][k], c.m[0][k], a.m[2][k], c.m[2][k], a.p[k] - c.p[k], dt, o);
            upk[k] = o[0];
            upe[k] = o[2];
        }
    }
#pragma unroll
    for (int r = 0; r < HG_R; r++) {
        const int y = y0 + r;
        const bool row = y < h;
        const bool ok = on && row;
        const size_t i = ok ? (size_t)y * w + x : 0;
        load_row(y + 1, d);
        float fx[4], fy[4], src[4], gx[4], gy[4], u1[4], u2[4], u3[4];
        load4(A.mfx, i, fx);
        load4(A.mfy, i, fy);
        load4(A.src, i, src);
        load4(A.gxm, i, gx);
        load4(A.gym, i, gy);
        auto load_own = [&](const float* a, float* v) {
            const float4 q = *reinterpret_cast<const float4*>(a + i);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        };
        load_own(A.Uout + n, u1);
        load_own(A.Uout + 2 * n, u2);
        load_own(A.Uout + 3 * n, u3);
        // the next column's mids and potential
        float mn[2], pn;
        mn[0] = __shfl_down_sync(0xffffffffu, c.m[0][0], 1);
        mn[1] = __shfl_down_sync(0xffffffffu, c.m[1][0], 1);
        pn = __shfl_down_sync(0xffffffffu, c.p[0], 1);
        const bool has_right = ok && x + 4 < w;
        if (lane == 31 && has_right) {
            mn[0] = A.mid[i + 4];
            mn[1] = A.mid[n + i + 4];
            pn = A.phim[i + 4];
        }
        float rk[4], rl[4], rh[4];  // the face right of each cell: impulse and energy to the cell, energy to the next
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float o[3] = {0.0f, 0.0f, 0.0f};
            if (k < 3 ? ok : has_right)
                face_work(fx[k], c.m[0][k], k < 3 ? c.m[0][k < 3 ? k + 1 : 3] : mn[0], c.m[1][k],
                          k < 3 ? c.m[1][k < 3 ? k + 1 : 3] : mn[1], c.p[k] - (k < 3 ? c.p[k < 3 ? k + 1 : 3] : pn), dt, o);
            rk[k] = o[0];
            rl[k] = o[1];
            rh[k] = o[2];
        }
        float lk = __shfl_up_sync(0xffffffffu, rk[3], 1), lh = __shfl_up_sync(0xffffffffu, rh[3], 1);
        if (lane == 0) {
            float o[3] = {0.0f, 0.0f, 0.0f};
            if (ok && x > 0)
                face_work(A.mfx[i - 1], A.mid[i - 1], c.m[0][0], A.mid[n + i - 1], c.m[1][0], A.phim[i - 1] - c.p[0], dt, o);
            lk = o[0];
            lh = o[2];
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float o[3] = {0.0f, 0.0f, 0.0f};
            if (ok && y + 1 < h)
                face_work(fy[k], c.m[0][k], d.m[0][k], c.m[2][k], d.m[2][k], c.p[k] - d.p[k], dt, o);
            const bool empty = src[k] == 0.0f && signbit(src[k]);
            if (ok && !empty) {
                float kick[2] = {dt * src[k] * gx[k], dt * src[k] * gy[k]};
                KickPart one{(double)kick[0], (double)kick[1], 0.0f, -1};
                if (src[k] > 0.0f) {
                    one.best = src[k];
                    one.idx = (int)i + k;
                }
                kp.merge(one);
                kick[0] += rk[k] - (k ? rk[k ? k - 1 : 0] : lk);
                kick[1] += o[0] - upk[k];
                u1[k] += kick[0];
                u2[k] += kick[1];
                u3[k] += rl[k] + (k ? rh[k ? k - 1 : 0] : lh) + o[1] + upe[k];
            }
            upk[k] = o[0];
            upe[k] = o[2];
        }
        if (ok) {
            *reinterpret_cast<float4*>(A.Uout + n + i) = make_float4(u1[0], u1[1], u1[2], u1[3]);
            *reinterpret_cast<float4*>(A.Uout + 2 * n + i) = make_float4(u2[0], u2[1], u2[2], u2[3]);
            *reinterpret_cast<float4*>(A.Uout + 3 * n + i) = make_float4(u3[0], u3[1], u3[2], u3[3]);
        }
        c = d;
    }
    take_back<HG_WARPS>(kp, red, A);
}

template <int MODE, int LIM, bool BRACKET>
__global__ void __launch_bounds__(HB_NT, 2) hydro_band_kernel(const __grid_constant__ CUtensorMap map, HydroArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    BandShared& sh = *reinterpret_cast<BandShared*>(smem_raw);
    const HydroConst H = A.H;
    const int w = H.w, h = H.h;
    const size_t n = (size_t)w * h;
    const int tid = threadIdx.x, lane = tid & 31, row = tid >> 5;
    const bool grav = A.gx != nullptr;
    const int ntx = (w + HB_TX - 1) / HB_TX, tiles = ntx * ((h + HB_TY - 1) / HB_TY);

    // ---- the four planes of a tile's staged region by one TMA box (x on a 16-byte boundary); every wait is bounded
    if (tid == 0) {
        tc::mbar_init(&sh.mbar[0], 1);
        tc::mbar_init(&sh.mbar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_launch();
    __syncthreads();
    pdl_wait();
    const float dt = (float)(*A.dt);
    const float half = 0.5f * dt;
    auto request = [&](int tile, int buf) {
        const int ty = tile / ntx, tx = tile - ty * ntx;
        tma::expect_tx(&sh.mbar[buf], (uint32_t)sizeof(sh.raw2[0]));
        tma::load_3d(&sh.raw2[buf][0][0][0], &map, (tx * HB_TX - 2) & ~3, ty * HB_TY - 2, 0, &sh.mbar[buf]);
    };
    if (tid == 0 && (int)blockIdx.x < tiles) request(blockIdx.x, 0);
    RatePart rp = RatePart::none();
    int it = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, it++) {
        const int buf = it & 1, next = tile + (int)gridDim.x;
        const int x0 = (tile % ntx) * HB_TX, y0 = (tile / ntx) * HB_TY;
        const int xs = (x0 - 2) & ~3, ys = y0 - 2;
        float(&raw)[4][HB_BY][HB_BX] = sh.raw2[buf];
        if (it > 0) __syncthreads();  // the tile before is done with the shared planes and with the other box
        if (tid == 0 && next < tiles) request(next, 1 - buf);
        const bool landed = tc::mbar_wait(&sh.mbar[buf], (it >> 1) & 1, kHydroWaitPolls);
        if (__syncthreads_or(!landed)) {
            if (tid == 0) atomicOr(A.err, 1);
            tc::mbar_wait(&sh.mbar[buf], (it >> 1) & 1, kHydroWaitPolls);  // the copies still in flight land before the
            if (next < tiles) tc::mbar_wait(&sh.mbar[1 - buf], ((it + 1) >> 1) & 1, kHydroWaitPolls);  // CTA leaves
            break;  // its share of the grid's sum is still due
        }

        // ---- primitives of the staged region: world cells, or ghosts past the edges (bounce mirrors the cells beyond
        // with the normal velocity negated, leave copies the edge cell with it clamped outward)
        for (int k = tid; k < HB_SY * HB_SX; k += HB_NT) {
            const int ly = k / HB_SX, lx = k - ly * HB_SX;
            const int x = x0 - 2 + lx, y = y0 - 2 + ly;
            Prim p;
            float solid = -1.0f;
            if (x >= -2 && x <= w + 1 && y >= -2 && y <= h + 1) {
                const bool xo = x < 0 || x >= w, yo = y < 0 || y >= h;
                int cx, cy;
                if (H.edge == SR_EDGE_BOUNCE) {
                    cx = x < 0 ? -x - 1 : (x >= w ? 2 * w - 1 - x : x);
                    cy = y < 0 ? -y - 1 : (y >= h ? 2 * h - 1 - y : y);
                } else {
                    cx = min(max(x, 0), w - 1);
                    cy = min(max(y, 0), h - 1);
                }
                const int bx = cx - xs, by = cy - ys;
                const float s = raw[0][by][bx];
                p = eos_read(H, s, raw[1][by][bx], raw[2][by][bx], raw[3][by][bx]);
                solid = (xo || yo) ? -1.0f : s;
                if (H.edge == SR_EDGE_BOUNCE) {
                    if (xo) p.u = -p.u;
                    if (yo) p.v = -p.v;
                } else {
                    if (x < 0) p.u = fminf(p.u, 0.0f);
                    if (x >= w) p.u = fmaxf(p.u, 0.0f);
                    if (y < 0) p.v = fminf(p.v, 0.0f);
                    if (y >= h) p.v = fmaxf(p.v, 0.0f);
                }
            } else {
                p.s = 1.0f; p.u = 0.0f; p.v = 0.0f; p.p = 1.0f;  // past every ghost: never reaches a kept cell
            }
            sh.P[ly][lx] = make_float4(p.s, p.u, p.v, p.p);
            sh.Q[ly][lx] = sr_div(p.p, p.s);
            sh.S[ly][lx] = solid;
        }
        __syncthreads();

        // ---- this lane's cell: slopes, the Hancock increment and the half-step centre (hydro.rs:587-614)
        const int sx = lane + 1, sy = row + 1;  // the cell in the staged region
        const int X = x0 - 1 + lane, Y = y0 - 1 + row;
        const Prim c = prim_at(sh, sy, sx);
        const Prim slx = slope<LIM, BRACKET>(prim_at(sh, sy, sx - 1), c, prim_at(sh, sy, sx + 1), sh.Q[sy][sx - 1],
                                             sh.Q[sy][sx], sh.Q[sy][sx + 1]);
        const Prim sly = slope<LIM, BRACKET>(prim_at(sh, sy - 1, sx), c, prim_at(sh, sy + 1, sx), sh.Q[sy - 1][sx],
                                             sh.Q[sy][sx], sh.Q[sy + 1][sx]);
        float gxv = 0.0f, gyv = 0.0f;
        if (grav) {  // a ghost takes its edge cell's g
            const size_t gi = (size_t)min(max(Y, 0), h - 1) * w + min(max(X, 0), w - 1);
            gxv = A.gx[gi];
            gyv = A.gy[gi];
        }
        float delta[4];
        {
            float a[4], b[4], dxs[4];
            face_flux(H, c, slx, -0.5f, 0, a);
            face_flux(H, c, slx, 0.5f, 0, b);
#pragma unroll
            for (int k = 0; k < 4; k++) dxs[k] = a[k] - b[k];
            face_flux(H, c, sly, -0.5f, 1, a);
            face_flux(H, c, sly, 0.5f, 1, b);
#pragma unroll
            for (int k = 0; k < 4; k++) delta[k] = half * (dxs[k] + (a[k] - b[k]));
        }
        {
            float m1 = c.s * c.u + delta[1], m2 = c.s * c.v + delta[2];
            if (grav) {
                m1 += half * c.s * gxv;
                m2 += half * c.s * gyv;
            }
            sh.M[0][row][lane] = c.s + delta[0];
            sh.M[1][row][lane] = m1;
            sh.M[2][row][lane] = m2;
        }

        // ---- x faces: this lane's x+ face against the next lane's x- face; the left face's flux from the lane before
        float fr[4], fl[4];
        {
            const FaceS R = shfl_face_down(face_state(H, c, slx, -0.5f, delta, half, grav, gxv, gyv));
            const FaceS L = face_state(H, c, slx, 0.5f, delta, half, grav, gxv, gyv);
            face_flux_at(H, L, R, 0, X + 1, w, Y >= 0 && Y < h, fr);
#pragma unroll
            for (int k = 0; k < 4; k++) fl[k] = __shfl_up_sync(0xffffffffu, fr[k], 1);
        }
        // ---- y faces: the row above's y+ faces against this row's y- faces, through shared memory
        {
            const FaceS T = face_state(H, c, sly, 0.5f, delta, half, grav, gxv, gyv);
            sh.YF[0][row][lane] = T.U0;
            sh.YF[1][row][lane] = T.U1;
            sh.YF[2][row][lane] = T.U2;
            sh.YF[3][row][lane] = T.U3;
            sh.YF[4][row][lane] = T.u;
            sh.YF[5][row][lane] = T.v;
            sh.YF[6][row][lane] = T.P;
        }
        const FaceS B = face_state(H, c, sly, -0.5f, delta, half, grav, gxv, gyv);
        __syncthreads();
        if (row >= 1) {
            FaceS L;
            L.U0 = sh.YF[0][row - 1][lane];
            L.U1 = sh.YF[1][row - 1][lane];
            L.U2 = sh.YF[2][row - 1][lane];
            L.U3 = sh.YF[3][row - 1][lane];
            L.u = sh.YF[4][row - 1][lane];
            L.v = sh.YF[5][row - 1][lane];
            L.P = sh.YF[6][row - 1][lane];
            float ft[4];
            face_flux_at(H, L, B, 1, Y, h, X >= 0 && X < w, ft);
#pragma unroll
            for (int k = 0; k < 4; k++) sh.FY[k][row][lane] = ft[k];
        }
        __syncthreads();

        // ---- epilogue: the tile's cells
        const bool inside = lane >= 1 && lane <= HB_TX && row >= 1 && row <= HB_TY && X < w && Y < h;
        const size_t i = inside ? (size_t)Y * w + X : 0;
        float fu[4], fd[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            fu[k] = row >= 1 ? sh.FY[k][row][lane] : 0.0f;
            fd[k] = row + 1 < HB_W ? sh.FY[k][row + 1][lane] : 0.0f;
        }
        // a cell with no gas around it stays empty (hydro.rs:733-742); out-of-world neighbours read as vacuum
        const float sv = H.sigma_vac;
        const bool vac = sh.S[sy][sx] < sv;
        const bool empty = vac && sh.S[sy][sx - 1] < sv && sh.S[sy][sx + 1] < sv && sh.S[sy - 1][sx] < sv &&
                           sh.S[sy + 1][sx] < sv;

        if (inside) {
            const int bx = X - xs, by = Y - ys;
            float u[4];
            if (empty || !vac) {
                u[0] = raw[0][by][bx]; u[1] = raw[1][by][bx]; u[2] = raw[2][by][bx]; u[3] = raw[3][by][bx];
            } else {
                eos_cons(H, c, u);
            }
            if (!empty) {
#pragma unroll
                for (int q = 0; q < 4; q++) u[q] -= dt * ((fr[q] - fl[q]) + (fd[q] - fu[q]));
            }
            if (MODE == kHydroPredict) {
                // what follows the half step's solve: an empty cell's source is -0 (gravity leaves the cell as it is)
                float src = -0.0f;
                if (!empty) {
                    const float start = vac ? sh.P[sy][sx].x : sh.S[sy][sx];
                    const float div = (fr[0] - fl[0]) + (fd[0] - fu[0]);
                    src = 0.5f * (sh.S[sy][sx] + (start - dt * div));
                    src = src >= sv ? src : 0.0f;
                }
                A.src[i] = src;
                A.mid[i] = sh.M[0][row][lane];
                A.mid[n + i] = sh.M[1][row][lane];
                A.mid[2 * n + i] = sh.M[2][row][lane];
                A.mfx[i] = fr[0];
                A.mfy[i] = fd[0];
            }
            if (MODE == kHydroStep) {
                floor_cell(H, u[0], u[1], u[2], u[3]);
                rate_cell(H, u[0], u[1], u[2], u[3], i, rp.rate, rp.nf);
            }
            A.Uout[i] = u[0];
            A.Uout[n + i] = u[1];
            A.Uout[2 * n + i] = u[2];
            A.Uout[3 * n + i] = u[3];
        }

    }
    // ---- the grid's sums, in a fixed order: a thread's tiles, the CTA's rows, the CTAs
    if (MODE != kHydroStep) return;
    rp = warp_merge(rp);
    if (lane == 0) sh.red[row] = rp;
    __syncthreads();
    if (row > 0) return;
    rp = warp_merge(lane < HB_W ? sh.red[lane] : RatePart::none());
    if (grid_total(rp, A.part, A.tickets) && lane == 0) dt_close(A.rule, rp.rate, 0.0f, rp.nf, 4);
}

}  // namespace


size_t hydro_smem_bytes() { return sizeof(BandShared); }

size_t hydro_part_count(int w, int h) {
    return std::max((size_t)2 * 148, (size_t)(div_up(w, HG_COLS) + 1) * div_up(h, HG_WARPS * HG_R));
}

size_t hydro_ticket_count(int h) { return (size_t)div_up(h, HG_WARPS * HG_R) + 1; }

void tma_encode_planes(CUtensorMap* map, const float* base, int w, int h, int planes, int bx, int by) {
    // encoded maps are kept by their arguments: a launch on the same planes (every launch of a step, every smoother
    // launch of a level) copies its map instead of paying the driver call before the launch
    static std::mutex mu;
    static std::map<std::tuple<const float*, int, int, int, int, int>, CUtensorMap> cache;
    const auto key = std::make_tuple(base, w, h, planes, bx, by);
    {
        std::lock_guard<std::mutex> lock(mu);
        const auto it = cache.find(key);
        if (it != cache.end()) {
            *map = it->second;
            return;
        }
    }
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        SR_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        SR_REQUIRE(q == cudaDriverEntryPointSuccess && fn, "the driver has no cuTensorMapEncodeTiled");
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    SR_REQUIRE(w % 4 == 0 && ((uintptr_t)base & 15) == 0, "a TMA plane needs 16-byte rows and a 16-byte base");
    const cuuint64_t dims[3] = {(cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)w * sizeof(float), (cuuint64_t)w * h * sizeof(float)};
    const cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)planes};
    const cuuint32_t unit[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box,
                              unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw SrError{SR_E_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r)};
    std::lock_guard<std::mutex> lock(mu);
    if (cache.size() > 4096) cache.clear();
    cache[key] = *map;
}

template <int MODE, int LIM, bool BRACKET>
void hydro_launch_t(const CUtensorMap& map, const HydroArgs& A, cudaStream_t s) {
    static bool attr = false;  // the attribute of this instance, once per process
    if (!attr) {
        SR_CUDA_TRY(cudaFuncSetAttribute(hydro_band_kernel<MODE, LIM, BRACKET>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BandShared)));
        attr = true;
    }
    const unsigned grid = std::min(div_up(A.H.w, HB_TX) * div_up(A.H.h, HB_TY), 2u * 148u);
    launch_kernel(MODE == kHydroStep, hydro_band_kernel<MODE, LIM, BRACKET>, dim3(grid), dim3(HB_NT), sizeof(BandShared), s, map, A);
    sr_note_launch();
}

template <int MODE>
void hydro_launch_m(const CUtensorMap& map, const HydroArgs& A, cudaStream_t s) {
    const bool mc = A.H.limiter != SR_LIMITER_MINMOD, br = A.H.bracket != 0;
    if (mc && br) hydro_launch_t<MODE, SR_LIMITER_MC, true>(map, A, s);
    else if (mc) hydro_launch_t<MODE, SR_LIMITER_MC, false>(map, A, s);
    else if (br) hydro_launch_t<MODE, SR_LIMITER_MINMOD, true>(map, A, s);
    else hydro_launch_t<MODE, SR_LIMITER_MINMOD, false>(map, A, s);
}

void hydro_launch(int mode, const HydroArgs& A, cudaStream_t s) {
    CUtensorMap map;
    tma_encode_planes(&map, A.U, A.H.w, A.H.h, 4, HB_BX, HB_BY);
    if (mode == kHydroStep) hydro_launch_m<kHydroStep>(map, A, s);
    else if (mode == kHydroUpdate) hydro_launch_m<kHydroUpdate>(map, A, s);
    else hydro_launch_m<kHydroPredict>(map, A, s);
}

void hydro_gravity_launch(const HydroArgs& A, cudaStream_t s) {
    const dim3 grid(div_up(A.H.w, HG_COLS), div_up(A.H.h, HG_WARPS * HG_R));
    hydro_gravity_kernel<<<grid, 32 * HG_WARPS, 0, s>>>(A);
    sr_note_launch();
}

// ------------------------------------------------------------------------------------------------ P8 + P9
// P8's floors, then P9's per-cell Δt terms of the floored state and |g| of the step's P2 field; per-CTA partials, the
// last CTA to arrive (a ticket) reduces them (max and min are exact in any order) and closes the step's Δt record. Four CTAs
// an SM (63 registers), as many as the grid has for each: with three the grid was a wave and a third (1024²: 13.8 -> 11.9
// us).
__global__ void __launch_bounds__(256, 4)
    floors_dt_kernel(HydroConst H, float* __restrict__ U, const float* __restrict__ gx, const float* __restrict__ gy,
                     int do_floors, float* part_rate, float* part_g, long long* part_nf, unsigned* ticket, DtRule rule) {
    const size_t n = (size_t)H.w * H.h, n4 = n / 4;  // the world's axes are multiples of 8
    float rate = 0.0f, gmax = 0.0f;
    double g2 = 0.0;  // |g|²: no square of an f32 leaves f64's range
    long long nf = LLONG_MAX;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (size_t)gridDim.x * blockDim.x) {
        float4 p[4];
#pragma unroll
        for (int k = 0; k < 4; k++) p[k] = reinterpret_cast<const float4*>(U + k * n)[q];
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (gx) {
            a = reinterpret_cast<const float4*>(gx)[q];
            b = reinterpret_cast<const float4*>(gy)[q];
        }
        float s[4] = {p[0].x, p[0].y, p[0].z, p[0].w}, mx[4] = {p[1].x, p[1].y, p[1].z, p[1].w};
        float my[4] = {p[2].x, p[2].y, p[2].z, p[2].w}, e[4] = {p[3].x, p[3].y, p[3].z, p[3].w};
        int changed = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (do_floors) changed = max(changed, floor_cell(H, s[k], mx[k], my[k], e[k]));
            rate_cell(H, s[k], mx[k], my[k], e[k], 4 * q + k, rate, nf);
        }
        if (changed == 2) {
            reinterpret_cast<float4*>(U)[q] = make_float4(s[0], s[1], s[2], s[3]);
            reinterpret_cast<float4*>(U + n)[q] = make_float4(mx[0], mx[1], mx[2], mx[3]);
            reinterpret_cast<float4*>(U + 2 * n)[q] = make_float4(my[0], my[1], my[2], my[3]);
        }
        if (changed) reinterpret_cast<float4*>(U + 3 * n)[q] = make_float4(e[0], e[1], e[2], e[3]);
        const float ga[4] = {a.x, a.y, a.z, a.w}, gb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 4; k++) g2 = fmax(g2, (double)ga[k] * ga[k] + (double)gb[k] * gb[k]);
    }
    gmax = (float)sqrt(g2);
    __shared__ float sr[32], sg[32];
    __shared__ long long sn[32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x / 32;
    for (int level = 0; level < 2; level++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            rate = fmaxf(rate, __shfl_down_sync(0xffffffffu, rate, o));
            gmax = fmaxf(gmax, __shfl_down_sync(0xffffffffu, gmax, o));
            const long long on = __shfl_down_sync(0xffffffffu, nf, o);
            nf = on < nf ? on : nf;
        }
        if (lane == 0) {
            sr[warp] = rate;
            sg[warp] = gmax;
            sn[warp] = nf;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < warps; k++) {
                rate = fmaxf(rate, sr[k]);
                gmax = fmaxf(gmax, sg[k]);
                nf = sn[k] < nf ? sn[k] : nf;
            }
            if (level == 0) {
                part_rate[blockIdx.x] = rate;
                part_g[blockIdx.x] = gmax;
                part_nf[blockIdx.x] = nf;
                __threadfence();
                last = atomicAdd(ticket, 1u) == gridDim.x - 1;
                if (last) *ticket = 0u;
                __threadfence();
            } else {
                dt_close(rule, rate, gmax, nf, 4);
            }
        }
        __syncthreads();
        if (level == 1 || !last) return;
        rate = gmax = 0.0f;
        nf = LLONG_MAX;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
            rate = fmaxf(rate, __ldcg(part_rate + b));
            gmax = fmaxf(gmax, __ldcg(part_g + b));
            const long long o = __ldcg(part_nf + b);
            nf = o < nf ? o : nf;
        }
    }
}

// The same from partials another kernel left. One CTA: each thread takes a strided share of them, then a shuffle and
// shared-memory tree.
__global__ void dt_finalize_kernel(int nblocks, int channels, const float* part_rate, const float* part_g,
                                   const long long* part_nf, DtRule rule) {
    float rate = 0.0f, gmax = 0.0f;
    long long nf = LLONG_MAX;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        rate = fmaxf(rate, part_rate[b]);
        gmax = fmaxf(gmax, part_g[b]);
        nf = part_nf[b] < nf ? part_nf[b] : nf;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rate = fmaxf(rate, __shfl_down_sync(0xffffffffu, rate, o));
        gmax = fmaxf(gmax, __shfl_down_sync(0xffffffffu, gmax, o));
        const long long on = __shfl_down_sync(0xffffffffu, nf, o);
        nf = on < nf ? on : nf;
    }
    __shared__ float sr[32], sg[32];
    __shared__ long long sn[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sr[warp] = rate;
        sg[warp] = gmax;
        sn[warp] = nf;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int k = 1; k < (int)(blockDim.x / 32); k++) {
        rate = fmaxf(rate, sr[k]);
        gmax = fmaxf(gmax, sg[k]);
        nf = sn[k] < nf ? sn[k] : nf;
    }
    dt_close(rule, rate, gmax, nf, channels);
}

int floors_dt_blocks(int w, int h) {
    size_t n = (size_t)w * h;
    int b = (int)div_up((unsigned)(n / 4), 256u);
    return b < 1 ? 1 : (b > 148 * 4 ? 148 * 4 : b);
}

void floors_dt_launch(const HydroConst& H, float* U, const float* gx, const float* gy, int do_floors, float* part_rate,
                      float* part_g, long long* part_nf, unsigned* ticket, const DtRule& rule, cudaStream_t s) {
    floors_dt_kernel<<<floors_dt_blocks(H.w, H.h), 256, 0, s>>>(H, U, gx, gy, do_floors, part_rate, part_g, part_nf,
                                                                ticket, rule);
    sr_note_launch();
}

void dt_finalize_launch(int nblocks, int channels, const float* part_rate, const float* part_g,
                        const long long* part_nf, const DtRule& rule, cudaStream_t s) {
    dt_finalize_kernel<<<1, 256, 0, s>>>(nblocks, channels, part_rate, part_g, part_nf, rule);
    sr_note_launch();
}
