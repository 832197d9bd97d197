// mg.cu — the multigrid V-cycle (FP32) of the implicit FLD solve; see mg.cuh for the scheme.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

#include "mg.cuh"
#include "reduce.cuh"
#include "tma.cuh"

namespace {

// Smoother tiles (outputs; even, so a tile's 2x2 aggregates stay inside it): 64 x 32 with 512 threads on big levels,
// 32 x 16 with 256 threads where the big tile leaves fewer than 2 CTAs per SM (a quarter of the work per CTA: the
// small levels are bound by one CTA's latency).
constexpr int BIG_SX = 64, BIG_SY = 32, BIG_NT = 512;
constexpr int SMALL_SX = 32, SMALL_SY = 16, SMALL_NT = 256;
constexpr int TAIL_THREADS = 512;

// A tail level's arrays as offsets (floats) into the tail's image, rows padded to an even pitch p and height hp.
struct TailLevel {
    int w, h, p, hp;
    int dx, dy, inv, t, c, b, x;  // inv: the inverse diagonal (0 on masked cells); t: the weights towards the next
                                  // coarser level; b and x: the lower levels' right-hand side and iterate
};

constexpr int kTailLevels = 5;  // 64 x 64 down to 4 x 4
struct TailArgs {
    int nl, pre, post;        // nl: the tail's levels
    float omega;
    int sinv;                 // offset of the coarsest level's inverse (nc x nc)
    int img_f4;               // the lower levels' part of the image in 16-byte words
    const float* img;
    const float* b;           // the top level's right-hand side and result
    float* x2;
    double* out;              // non-null when the tail's top level is level 0: <b, x2> written here
    TailLevel T[kTailLevels];  // the top first
};

// Level 0's couplings to the +x / +y neighbours from the f64 faces, zero unless both cells are gas.
__global__ void mg_couplings0_kernel(MgLevel L, const double* __restrict__ kx, const double* __restrict__ ky,
                                     const uint8_t* __restrict__ gas) {
    const int w = L.w, h = L.h;
    const size_t n = (size_t)w * h;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        int x, y;
        split_index(i, w, x, y);
        const bool g = gas[i];
        L.mask[i] = g;
        L.dx[i] = (g && x + 1 < w && gas[i + 1]) ? (float)kx[(size_t)y * (w + 1) + x + 1] : 0.0f;
        L.dy[i] = (g && y + 1 < h && gas[i + w]) ? (float)ky[(size_t)(y + 1) * w + x] : 0.0f;
    }
}

// Level 1 from level 0: Galerkin aggregation of 2x2 cells with constant weights (mg.cuh). The mass term c sums over
// the aggregate's system cells; a coarse coupling sums the two fine couplings across the aggregates' shared side.
__global__ void mg_aggregate_kernel(MgLevel F, MgLevel C) {
    const int wc = C.w, hc = C.h, wf = F.w, hf = F.h;
    const size_t nc = (size_t)wc * hc;
    for (size_t I = (size_t)blockIdx.x * blockDim.x + threadIdx.x; I < nc; I += (size_t)gridDim.x * blockDim.x) {
        const int X = (int)(I % wc), Y = (int)(I / wc);
        const int fx0 = 2 * X, fy0 = 2 * Y;
        const bool has_x1 = fx0 + 1 < wf, has_y1 = fy0 + 1 < hf;
        float c = 0.0f;
        bool any = false;
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int a = 0; a < 2; a++) {
                if ((a && !has_x1) || (b && !has_y1)) continue;
                size_t j = (size_t)(fy0 + b) * wf + fx0 + a;
                if (F.mask[j]) {
                    c += F.c[j];
                    any = true;
                }
            }
        float dxc = 0.0f, dyc = 0.0f;
        if (X + 1 < wc) {
            dxc = F.dx[(size_t)fy0 * wf + fx0 + 1];
            if (has_y1) dxc += F.dx[(size_t)(fy0 + 1) * wf + fx0 + 1];
        }
        if (Y + 1 < hc) {
            dyc = F.dy[(size_t)(fy0 + 1) * wf + fx0];
            if (has_x1) dyc += F.dy[(size_t)(fy0 + 1) * wf + fx0 + 1];
        }
        C.c[I] = any ? c : 1.0f;
        C.dx[I] = dxc;
        C.dy[I] = dyc;
        C.mask[I] = any;
    }
}

// Level l+1 from level l >= 1 (mg.cuh): each 2x2 aggregate's basis function is the fine weight vector t restricted to
// the aggregate, t from two red-black Gauss-Seidel sweeps on A t = 0 from t = 1 (masked cells 0), scaled so that its
// largest value in the aggregate is 1; the coarse operator is the Galerkin product, still 5-point:
//   coarse coupling to +x  = sum over the two fine couplings crossing the shared side of t_j t_k d_jk,
//   coarse c (diagonal less couplings) = sum_j t_j (A t)_j over the aggregate = (P^T A t)_I,
// with (A t)_j = c_j t_j + sum_k d_jk (t_j - t_k) in difference form, summed in f64 from the f32 weights the
// restriction and prolongation use. One tile of CO_S x CO_S fine cells per CTA, all four half-sweeps in shared
// memory: the tile's halo is as deep as the half-sweeps plus the two rings whose aggregates' scale the Galerkin sums
// read (t of the cells next to the tile's aggregates).
constexpr int CO_S = 32, CO_H = 6, CO_R = CO_S + 2 * CO_H, CO_N = CO_R * CO_R, CO_NT = 512;

__global__ void __launch_bounds__(CO_NT) mg_coarsen_kernel(MgLevel F, MgLevel C) {
    __shared__ float sc[CO_N], sdx[CO_N], sdy[CO_N], st[CO_N];
    __shared__ uint8_t sm[CO_N];
    const int wf = F.w, hf = F.h;
    const int X0 = blockIdx.x * CO_S - CO_H, Y0 = blockIdx.y * CO_S - CO_H;  // even: local parity = global parity
    // all of a thread's loads in flight together: the launch is one CTA's latency on the coarse levels (11.2 -> 6.7 us)
    constexpr int PER = (CO_N + CO_NT - 1) / CO_NT;
    float lc[PER], ldx[PER], ldy[PER];
    uint8_t lm[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int k = threadIdx.x + u * CO_NT, gx = X0 + k % CO_R, gy = Y0 + k / CO_R;
        lc[u] = 1.0f;
        ldx[u] = ldy[u] = 0.0f;
        lm[u] = 0;
        if (k < CO_N && gx >= 0 && gx < wf && gy >= 0 && gy < hf) {
            const int i = gy * wf + gx;
            lc[u] = F.c[i];
            ldx[u] = F.dx[i];
            ldy[u] = F.dy[i];
            lm[u] = F.mask[i];
        }
    }
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int k = threadIdx.x + u * CO_NT;
        if (k >= CO_N) break;
        sm[k] = lm[u];
        sc[k] = lc[u];
        sdx[k] = ldx[u];
        sdy[k] = ldy[u];
        st[k] = lm[u] ? 1.0f : 0.0f;
    }
    __syncthreads();
    // four half-sweeps, colour 0 first, over the region less its outermost ring (a cell's value is exact once it
    // lies as many rings inside as half-sweeps were taken)
    for (int sweep = 0; sweep < 4; sweep++) {
        const int col = sweep & 1;
        for (int k = threadIdx.x; k < CO_N / 2; k += CO_NT) {
            const int ly = k / (CO_R / 2), lx = 2 * (k - ly * (CO_R / 2)) + ((ly + col) & 1);
            if (lx < 1 || lx > CO_R - 2 || ly < 1 || ly > CO_R - 2) continue;
            const int q = ly * CO_R + lx;
            // a masked or outside cell has c = 1 and no couplings (nor do its neighbours towards it): it stays 0
            const float dl = sdx[q - 1], dr = sdx[q], du = sdy[q - CO_R], dd = sdy[q];
            const float num = dl * st[q - 1] + dr * st[q + 1] + du * st[q - CO_R] + dd * st[q + CO_R];
            st[q] = num / (sc[q] + dl + dr + du + dd);
        }
        __syncthreads();
    }
    // each aggregate of the tile and of the two rings around it, scaled to a largest weight of 1 (an aggregate whose
    // weights all vanished takes 1 on its system cells, as plain aggregation would)
    constexpr int AG = (CO_S + 4) / 2;
    for (int k = threadIdx.x; k < AG * AG; k += CO_NT) {
        const int ay = k / AG, ax = k - ay * AG;
        const int lx = CO_H - 2 + 2 * ax, ly = CO_H - 2 + 2 * ay;
        const int q = ly * CO_R + lx;
        const float m = fmaxf(fmaxf(st[q], st[q + 1]), fmaxf(st[q + CO_R], st[q + CO_R + 1]));
        const int offs[4] = {0, 1, CO_R, CO_R + 1};
        for (int e = 0; e < 4; e++) {
            const int j = q + offs[e];
            st[j] = !sm[j] ? 0.0f : (m > 1e-30f ? st[j] / m : 1.0f);  // outside the level: mask 0
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < CO_S * CO_S; k += CO_NT) {
        const int gx = X0 + CO_H + k % CO_S, gy = Y0 + CO_H + k / CO_S;
        if (gx < wf && gy < hf) F.t[gy * wf + gx] = st[(k / CO_S + CO_H) * CO_R + k % CO_S + CO_H];
    }
    const int wc = C.w, hc = C.h;
    for (int k = threadIdx.x; k < (CO_S / 2) * (CO_S / 2); k += CO_NT) {
        const int cy = k / (CO_S / 2), cx = k - cy * (CO_S / 2);
        const int X = blockIdx.x * (CO_S / 2) + cx, Y = blockIdx.y * (CO_S / 2) + cy;
        if (X >= wc || Y >= hc) continue;
        const int lx0 = CO_H + 2 * cx, ly0 = CO_H + 2 * cy;
        double csum = 0.0;
        bool any = false;
        for (int b = 0; b < 2; b++)
            for (int a = 0; a < 2; a++) {
                const int q = (ly0 + b) * CO_R + lx0 + a;
                if (!sm[q]) continue;
                any = true;
                const double tj = st[q];
                const double at = (double)sc[q] * tj + (double)sdx[q - 1] * (tj - st[q - 1]) +
                                  (double)sdx[q] * (tj - st[q + 1]) + (double)sdy[q - CO_R] * (tj - st[q - CO_R]) +
                                  (double)sdy[q] * (tj - st[q + CO_R]);
                csum += tj * at;
            }
        double dxc = 0.0, dyc = 0.0;
        if (X + 1 < wc)
            for (int b = 0; b < 2; b++) {
                const int q = (ly0 + b) * CO_R + lx0 + 1;
                dxc += (double)st[q] * st[q + 1] * sdx[q];
            }
        if (Y + 1 < hc)
            for (int a = 0; a < 2; a++) {
                const int q = (ly0 + 1) * CO_R + lx0 + a;
                dyc += (double)st[q] * st[q + CO_R] * sdy[q];
            }
        const size_t I = (size_t)Y * wc + X;
        C.c[I] = any ? (float)csum : 1.0f;
        C.dx[I] = any ? (float)dxc : 0.0f;
        C.dy[I] = any ? (float)dyc : 0.0f;
        C.mask[I] = any;
    }
}

// One smoother on a big level, all NS half-sweeps of a tile in shared memory (the tile's halo as deep as the
// half-sweeps, so the tile's result is exactly the global red-black sweeps'). PRE: from x = 0, red first, into L.x,
// then the residual summed over each 2x2 aggregate into the coarse level's b (one more halo ring keeps the residual's
// neighbours exact). POST: from x = L.x + ω P xc, black first, into L.x2.
//
// The tile is stored split by colour (cell (lx, ly) of colour (lx + ly) & 1 at ly * HX + lx / 2 of its colour's
// arrays), so that a half-sweep's consecutive threads update consecutive cells of one colour and read their
// neighbours, all of the other colour, at consecutive addresses: no bank conflicts. Per cell: x, b, the inverse
// diagonal, the couplings to +x and +y, and for PRE the mass term c (the residual is taken in difference form,
// c x + Σ d (x − x_j), which keeps its FP32 accuracy when c is far below the couplings). The mask is not read: a
// masked cell has b = 0, c = 1 and no couplings (nor do its neighbours towards it), so its update is 0 and it
// influences nobody; the cells outside the world get the same values. Each thread's cells of a half-sweep are the
// same in every half-sweep of a colour: their indices and validity are computed once.
constexpr int A_X = 0, A_B = 1, A_INV = 2, A_DX = 3, A_DY = 4, A_C = 5;

template <int NS, bool PRE, int SX, int SY>
constexpr size_t smooth_smem() {
    constexpr int H = PRE ? NS + 1 : NS;
    constexpr int RN = (SX + 2 * H) * (SY + 2 * H);
    return (size_t)RN * (PRE ? 6 : 5) * sizeof(float);
}

template <int NS, bool PRE, int SX, int SY, int NT>
__global__ void __launch_bounds__(NT) mg_smooth_kernel(MgLevel L, MgLevel C, const float* __restrict__ xc,
                                                                    float omega) {
    constexpr int H = PRE ? NS + 1 : NS;
    constexpr int RX = SX + 2 * H, RY = SY + 2 * H, RN = RX * RY, HX = RX / 2, HN = HX * RY;
    static_assert(RX % 2 == 0, "the tile's rows split evenly by colour");
    extern __shared__ __align__(16) float smem_f[];
    auto arr = [&](int a, int k) { return smem_f + (2 * a + k) * HN; };
    const int w = L.w, h = L.h;
    const int X0 = blockIdx.x * SX - H, Y0 = blockIdx.y * SY - H;  // X0 + Y0 even: local colour = global colour
    const int tid = threadIdx.x;
    constexpr int NLOAD = (RN + NT - 1) / NT;
#pragma unroll
    for (int it = 0; it < NLOAD; it++) {
        const int k = tid + it * NT;
        if (k >= RN) break;
        const int lx = k % RX, ly = k / RX;
        const int gx = X0 + lx, gy = Y0 + ly;
        float b = 0.0f, c = 1.0f, dx = 0.0f, dy = 0.0f, x = 0.0f, inv = 0.0f;
        if (gx >= 0 && gx < w && gy >= 0 && gy < h) {
            const int i = gy * w + gx;  // a level holds fewer than 2^31 cells
            b = L.b[i];
            c = L.c[i];
            dx = L.dx[i];
            dy = L.dy[i];
            const float dxl = gx > 0 ? L.dx[i - 1] : 0.0f, dyu = gy > 0 ? L.dy[i - w] : 0.0f;
            if (!PRE) x = L.x[i] + omega * L.t[i] * xc[(size_t)(gy >> 1) * C.w + (gx >> 1)];
            inv = __fdividef(1.0f, c + dx + dxl + dy + dyu);  // the smoother's diagonal: an approximate reciprocal
        }
        const int col = (lx + ly) & 1, q = ly * HX + (lx >> 1);
        arr(A_X, col)[q] = x;
        arr(A_B, col)[q] = b;
        arr(A_INV, col)[q] = inv;
        arr(A_DX, col)[q] = dx;
        arr(A_DY, col)[q] = dy;
        if (PRE) arr(A_C, col)[q] = c;
    }
    __syncthreads();
    constexpr int NSWEEP = (HN + NT - 1) / NT;
    int qinfo[NSWEEP];  // per cell slot: q | o of colour 0 << 28 | updatable in colour 0 << 29 | in colour 1 << 30
#pragma unroll
    for (int it = 0; it < NSWEEP; it++) {
        const int q = tid + it * NT;
        int info = -1;
        if (q < HN) {
            const int ly = q / HX, j = q - ly * HX;
            const bool yok = ly >= 1 && ly <= RY - 2;
            const int o0 = ly & 1, lx0 = 2 * j + o0, lx1 = 2 * j + 1 - o0;
            const int ok0 = yok && lx0 >= 1 && lx0 <= RX - 2, ok1 = yok && lx1 >= 1 && lx1 <= RX - 2;
            info = q | (o0 << 28) | (ok0 << 29) | (ok1 << 30);
        }
        qinfo[it] = info;
    }
#pragma unroll 1
    for (int s = 0; s < NS; s++) {
        const int col = PRE ? (s & 1) : 1 - (s & 1), oth = 1 - col;
        float* x = arr(A_X, col);
        const float* b = arr(A_B, col);
        const float* inv = arr(A_INV, col);
        const float* dx = arr(A_DX, col);
        const float* dy = arr(A_DY, col);
        const float* xo = arr(A_X, oth);
        const float* dxo = arr(A_DX, oth);
        const float* dyo = arr(A_DY, oth);
#pragma unroll
        for (int it = 0; it < NSWEEP; it++) {
            const int info = qinfo[it];
            if (info < 0 || !((info >> (29 + col)) & 1)) continue;
            const int q = info & 0x0FFFFFFF, o = ((info >> 28) & 1) ^ col;
            const int left = q - 1 + o, right = q + o;  // the other colour's cells at lx - 1 and lx + 1
            x[q] = (b[q] + dxo[left] * xo[left] + dx[q] * xo[right] + dyo[q - HX] * xo[q - HX] + dy[q] * xo[q + HX]) *
                   inv[q];
        }
        __syncthreads();
    }
    float* dst = PRE ? L.x : L.x2;
    for (int k = tid; k < SX * SY; k += NT) {
        const int ox = k % SX, oy = k / SX;
        const int gx = X0 + H + ox, gy = Y0 + H + oy;
        if (gx < w && gy < h) {
            const int lx = ox + H, ly = oy + H, col = (lx + ly) & 1, q = ly * HX + (lx >> 1);
            const float xv = arr(A_X, col)[q];
            dst[(size_t)gy * w + gx] = xv;
        }
    }
    if (PRE) {
        // the coarse right-hand side: the residual, in difference form, weighted by t and summed over each aggregate of
        // the tile
        for (int k = tid; k < (SX / 2) * (SY / 2); k += NT) {
            const int cxl = k % (SX / 2), cyl = k / (SX / 2);
            const int X = (X0 + H) / 2 + cxl, Y = (Y0 + H) / 2 + cyl;
            if (X >= C.w || Y >= C.h) continue;
            float sum = 0.0f;
#pragma unroll
            for (int bb = 0; bb < 2; bb++)
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    const int lx = 2 * cxl + a + H, ly = 2 * cyl + bb + H;
                    const int col = (lx + ly) & 1, oth = 1 - col, q = ly * HX + (lx >> 1);
                    const int o = (col + ly) & 1, left = q - 1 + o, right = q + o;
                    const float xj = arr(A_X, col)[q];
                    const float* xo = arr(A_X, oth);
                    float ax = arr(A_C, col)[q] * xj;
                    ax += arr(A_DX, oth)[left] * (xj - xo[left]);
                    ax += arr(A_DX, col)[q] * (xj - xo[right]);
                    ax += arr(A_DY, oth)[q - HX] * (xj - xo[q - HX]);
                    ax += arr(A_DY, col)[q] * (xj - xo[q + HX]);
                    const int gx = X0 + lx, gy = Y0 + ly;
                    sum += (gx < w && gy < h ? L.t[gy * w + gx] : 0.0f) * (arr(A_B, col)[q] - ax);
                }
            C.b[(size_t)Y * C.w + X] = C.mask[(size_t)Y * C.w + X] ? sum : 0.0f;
        }
    }
}

// The row-band smoother of the big levels of even width: the same smoother as mg_smooth_kernel (NS red-black
// half-sweeps of a tile whose halo is as deep as the half-sweeps, then the restriction or <b, x2>), with every cell's
// coefficients and iterate held in registers. A CTA covers a 64 x 64 region (RB_RX x RB_RY): warp w owns rows
// 4w .. 4w+3 (a band), lane j owns the cell pair (2j, 2j+1) of each of its rows. In a half-sweep a cell's horizontal
// neighbours are its pair partner (a register) and one cell of the next lane's pair (a shuffle), its vertical
// neighbours the same lane's rows above and below (registers), except across a band edge, whose rows go through shared
// memory once per half-sweep (double-buffered: one barrier per half-sweep). Which cell of a pair a colour updates is
// fixed by the row's parity (the region starts on an even column and row, so local parity = global parity), so the
// sweeps unroll into straight-line code. The halo is NS for both: the post-smoother's first half-sweep reads
// neighbours and its last result none beyond; the pre-smoother's first half-sweep starts from x = 0 and reads none, and
// the residual after the last one reads them. (NS + 2 for the pre-smoother, as if its first half-sweep read
// neighbours, took 19 % more CTAs under V(4,4).) An even halo keeps pairs on 8-byte words inside one aggregate. Cells
// outside the level: b = 0, c = 1, no couplings, inverse diagonal 0.
constexpr int RB_R = 4, RB_WARPS = 16, RB_NT = 32 * RB_WARPS, RB_RX = 64, RB_RY = RB_R * RB_WARPS;

template <int NS, bool PRE>
constexpr int rb_halo() { return NS; }

// The CTA's share of <b, x2>, left for the kernel that reads it to sum (Multigrid::apply). A ticket and a last CTA here
// would hold every CTA's registers and shared memory for an atomic's round trip at its end.
__device__ __forceinline__ void cta_partial(double acc, double* part) {
    __shared__ double red[RB_WARPS];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < RB_WARPS; q++) t += red[q];
        part[blockIdx.x] = t;
    }
}

template <int NS, bool PRE, bool WT>
__global__ void __launch_bounds__(RB_NT, 2) mg_rowband_kernel(MgLevel L, MgLevel C, const float* __restrict__ xc,
                                                            float omega) {
    constexpr int H = rb_halo<NS, PRE>(), SX = RB_RX - 2 * H, SY = RB_RY - 2 * H;
    static_assert(H % 2 == 0 && NS % 2 == 0, "the region starts on an even column and row");
    __shared__ float2 edge[2][2][RB_WARPS][32];  // [buffer][top row / bottom row][warp][lane]: (x of 2j, x of 2j+1)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = L.w, h = L.h;
    const int X0 = blockIdx.x * SX - H, Y0 = blockIdx.y * SY - H;
    const int gx = X0 + 2 * lane;             // the pair's first column (even)
    const bool xin = gx >= 0 && gx < w;        // w is even: both cells of the pair lie inside, or neither
    const int gy0 = Y0 + RB_R * warp;          // the band's first row (even)

    float bA[RB_R], bB[RB_R], iA[RB_R], iB[RB_R], dl[RB_R], dm[RB_R], dr[RB_R], dA[RB_R], dB[RB_R];
    float xA[RB_R], xB[RB_R], cA[RB_R], cB[RB_R];
    float uA = 0.0f, uB = 0.0f;  // the couplings of row 0 to the row above
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        const int gy = gy0 + r;
        const bool in = xin && gy >= 0 && gy < h;
        const size_t i = (size_t)gy * w + gx;
        float2 b2 = make_float2(0.f, 0.f), c2 = make_float2(1.f, 1.f), dx2 = b2, dy2 = b2;
        if (in) {
            b2 = *reinterpret_cast<const float2*>(L.b + i);
            c2 = *reinterpret_cast<const float2*>(L.c + i);
            dx2 = *reinterpret_cast<const float2*>(L.dx + i);
            dy2 = *reinterpret_cast<const float2*>(L.dy + i);
            if (r == 0 && gy > 0) {
                const float2 u2 = *reinterpret_cast<const float2*>(L.dy + i - w);
                uA = u2.x;
                uB = u2.y;
            }
        }
        bA[r] = b2.x;
        bB[r] = b2.y;
        cA[r] = c2.x;
        cB[r] = c2.y;
        dm[r] = dx2.x;
        dr[r] = dx2.y;
        dA[r] = dy2.x;
        dB[r] = dy2.y;
        // the coupling of cell 2j to 2j - 1 is the previous pair's right coupling (0 from a pair outside the level)
        dl[r] = __shfl_up_sync(0xffffffffu, dx2.y, 1);
        if (lane == 0) dl[r] = (in && gx > 0) ? L.dx[i - 1] : 0.0f;
        const float upA = r ? dA[r - 1] : uA, upB = r ? dB[r - 1] : uB;
        iA[r] = in ? __fdividef(1.0f, c2.x + dl[r] + dx2.x + upA + dy2.x) : 0.0f;
        iB[r] = in ? __fdividef(1.0f, c2.y + dx2.x + dx2.y + upB + dy2.y) : 0.0f;
        float x0 = 0.0f, x1 = 0.0f;
        if (!PRE && in) {
            const float2 xv = *reinterpret_cast<const float2*>(L.x + i);
            const float corr = omega * xc[(size_t)(gy >> 1) * C.w + (gx >> 1)];
            if constexpr (WT) {
                const float2 t2 = *reinterpret_cast<const float2*>(L.t + i);
                x0 = xv.x + corr * t2.x;
                x1 = xv.y + corr * t2.y;
            } else {
                x0 = xv.x + corr;
                x1 = xv.y + corr;
            }
        }
        xA[r] = x0;
        xB[r] = x1;
    }
    edge[0][0][warp][lane] = make_float2(xA[0], xB[0]);
    edge[0][1][warp][lane] = make_float2(xA[RB_R - 1], xB[RB_R - 1]);
    __syncthreads();
    const int wu = warp > 0 ? warp - 1 : warp, wd = warp + 1 < RB_WARPS ? warp + 1 : warp;
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const int col = PRE ? (s & 1) : 1 - (s & 1);
        const int rd = s & 1, wr = (s + 1) & 1;
        const float2 above = edge[rd][1][wu][lane], below = edge[rd][0][wd][lane];
#pragma unroll
        for (int r = 0; r < RB_R; r++) {
            if ((r & 1) == col) {  // the pair's first cell has this colour
                const float left = __shfl_up_sync(0xffffffffu, xB[r], 1);
                const float up = r ? xA[r - 1] : above.x, down = r + 1 < RB_R ? xA[r + 1] : below.x;
                const float cu = r ? dA[r - 1] : uA;
                xA[r] = (bA[r] + dl[r] * left + dm[r] * xB[r] + cu * up + dA[r] * down) * iA[r];
            } else {
                const float right = __shfl_down_sync(0xffffffffu, xA[r], 1);
                const float up = r ? xB[r - 1] : above.y, down = r + 1 < RB_R ? xB[r + 1] : below.y;
                const float cu = r ? dB[r - 1] : uB;
                xB[r] = (bB[r] + dm[r] * xA[r] + dr[r] * right + cu * up + dB[r] * down) * iB[r];
            }
        }
        edge[wr][0][warp][lane] = make_float2(xA[0], xB[0]);
        edge[wr][1][warp][lane] = make_float2(xA[RB_R - 1], xB[RB_R - 1]);
        __syncthreads();
    }
    const bool xout = xin && 2 * lane >= H && 2 * lane < RB_RX - H;
    if constexpr (PRE) {
        const float2 above = edge[NS & 1][1][wu][lane], below = edge[NS & 1][0][wd][lane];
        float ragg[RB_R / 2] = {};
#pragma unroll
        for (int r = 0; r < RB_R; r++) {
            const int gy = gy0 + r, ly = RB_R * warp + r;
            const bool o = xout && ly >= H && ly < RB_RY - H && gy < h;
            const size_t i = (size_t)gy * w + gx;
            if (o) *reinterpret_cast<float2*>(L.x + i) = make_float2(xA[r], xB[r]);
            // the residual in difference form, c x + Σ d (x - x_nb), for both cells
            const float left = __shfl_up_sync(0xffffffffu, xB[r], 1);
            const float right = __shfl_down_sync(0xffffffffu, xA[r], 1);
            const float upA = r ? xA[r - 1] : above.x, dnA = r + 1 < RB_R ? xA[r + 1] : below.x;
            const float upB = r ? xB[r - 1] : above.y, dnB = r + 1 < RB_R ? xB[r + 1] : below.y;
            const float cuA = r ? dA[r - 1] : uA, cuB = r ? dB[r - 1] : uB;
            float axA = cA[r] * xA[r];
            axA += dl[r] * (xA[r] - left);
            axA += dm[r] * (xA[r] - xB[r]);
            axA += cuA * (xA[r] - upA);
            axA += dA[r] * (xA[r] - dnA);
            float axB = cB[r] * xB[r];
            axB += dm[r] * (xB[r] - xA[r]);
            axB += dr[r] * (xB[r] - right);
            axB += cuB * (xB[r] - upB);
            axB += dB[r] * (xB[r] - dnB);
            float rA = bA[r] - axA, rB = bB[r] - axB;
            if constexpr (WT) {
                if (o) {
                    const float2 t2 = *reinterpret_cast<const float2*>(L.t + i);
                    rA *= t2.x;
                    rB *= t2.y;
                }
            }
            ragg[r >> 1] += rA + rB;
        }
#pragma unroll
        for (int k = 0; k < RB_R / 2; k++) {
            const int ly = RB_R * warp + 2 * k;
            const int X = gx >> 1, Y = (gy0 + 2 * k) >> 1;
            if (xout && ly >= H && ly < RB_RY - H && X < C.w && Y < C.h && gy0 + 2 * k >= 0) {
                const size_t I = (size_t)Y * C.w + X;
                C.b[I] = C.mask[I] ? ragg[k] : 0.0f;
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < RB_R; r++) {
            const int gy = gy0 + r, ly = RB_R * warp + r;
            if (xout && ly >= H && ly < RB_RY - H && gy < h) {
                const size_t i = (size_t)gy * w + gx;
                *reinterpret_cast<float2*>(L.x2 + i) = make_float2(xA[r], xB[r]);
            }
        }
    }
    (void)SX;
    (void)SY;
}

// The row-band smoother with its regions staged by TMA: the same smoother as mg_rowband_kernel, its coefficients (b, c,
// dx, dy), after the coarse correction the iterate x, and before the restriction of a weighted level the weights read
// from shared memory where one thread's bulk tensor copies put them: the region's 64 rows and the row above it, 68
// columns from a 16-byte boundary left of the region (the pair's left coupling included), zero past the level's edges.
// A CTA walks over regions: once a region's coefficients are in registers its boxes are free, and the next region's
// land behind this one's sweeps. (A region a CTA, two CTAs an SM: the loads of a pair of CTAs, 3.8 us of the memory's
// rate, and their sweeps came one after the other, 6.7 us a wave at 2048².) Level 0 at 2048² under V(4,4): pre-smoother
// 35.3 -> 31.7 us, post-smoother 37.9 -> 32.2. The pre-smoother reads c again for the residual, so its c alternates between
// two boxes; a weighted level has no room for that and asks for c and the weights once its residual is done. Every
// wait is bounded: a wait that gives up sets the level's error flag and the CTA leaves without its stores.
constexpr int RB_TMA_X = 68, RB_TMA_Y = RB_RY + 1;
constexpr uint32_t kMgWaitPolls = 1u << 24;
// b, dx, dy, c, then x (post), the other c (pre) or the weights (pre of a weighted level); the post-smoother of a
// weighted level reads its weights while the boxes land
constexpr int RB_BOXES = 5;
constexpr size_t kRbBox = ((size_t)RB_TMA_X * RB_TMA_Y * sizeof(float) + 127) / 128 * 128;
constexpr size_t kRbEdges = sizeof(float2) * 2 * 2 * RB_WARPS * 32, kRbCoarse = sizeof(float) * RB_NT * (RB_R / 2);
constexpr size_t kRbSmem = RB_BOXES * kRbBox + kRbEdges + kRbCoarse + 16;
// two CTAs an SM and no more than there are regions
inline unsigned rb_regions(const MgLevel& L, int halo) { return div_up(L.w, RB_RX - 2 * halo) * div_up(L.h, RB_RY - 2 * halo); }
inline unsigned rb_grid(const MgLevel& L, int halo) { return std::min(rb_regions(L, halo), (unsigned)kMgMaxParts); }

template <int NS, bool PRE, bool WT>
__global__ void __launch_bounds__(RB_NT, 2)
    mg_rowband_tma_kernel(const __grid_constant__ CUtensorMap mb, const __grid_constant__ CUtensorMap mc,
                          const __grid_constant__ CUtensorMap mdx, const __grid_constant__ CUtensorMap mdy,
                          const __grid_constant__ CUtensorMap mx, MgLevel L, MgLevel C, const float* xc, float omega,
                          double* part) {
    constexpr int H = rb_halo<NS, PRE>(), SX = RB_RX - 2 * H, SY = RB_RY - 2 * H;
    constexpr int XO = (H % 4 == 2) ? 2 : 4;  // the region's first column within the box (X0 - XO on a 16-byte boundary)
    constexpr bool TWO_C = PRE && !WT, LATE = PRE && WT;
    constexpr size_t AB = kRbBox / sizeof(float);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* sarr = reinterpret_cast<float*>(smem_raw);
    float2(*edge)[2][RB_WARPS][32] = reinterpret_cast<float2(*)[2][RB_WARPS][32]>(smem_raw + RB_BOXES * kRbBox);
    float* sxc = reinterpret_cast<float*>(smem_raw + RB_BOXES * kRbBox + kRbEdges);
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + RB_BOXES * kRbBox + kRbEdges + kRbCoarse);
    const float* sb = sarr;
    const float* sdx = sarr + AB;
    const float* sdy = sarr + 2 * AB;
    const float* sx = sarr + 4 * AB;  // post: the iterate; pre of a weighted level: the weights
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int w = L.w, h = L.h;
    const int nx = (w + SX - 1) / SX, regions = nx * ((h + SY - 1) / SY);
    if (tid == 0) {
        tc::mbar_init(mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch();
    auto arm = [&] { tma::expect_tx(mbar, (uint32_t)((PRE && !WT ? 4 : 5) * RB_TMA_X * RB_TMA_Y * sizeof(float))); };
    // (x, y): a region's corner on the level
    auto request_couplings = [&](int x, int y) {
        tma::load_3d(sarr + AB, &mdx, x - XO, y - 1, 0, mbar);
        tma::load_3d(sarr + 2 * AB, &mdy, x - XO, y - 1, 0, mbar);
    };
    auto request_c = [&](int x, int y, int it) {  // c, and what a weighted level's restriction takes
        tma::load_3d(sarr + (TWO_C ? 3 + (it & 1) : 3) * AB, &mc, x - XO, y - 1, 0, mbar);
        if constexpr (PRE && WT) tma::load_3d(sarr + 4 * AB, &mx, x - XO, y - 1, 0, mbar);
    };
    auto request_iterate = [&](int x, int y) {
        tma::load_3d(sarr, &mb, x - XO, y - 1, 0, mbar);
        if constexpr (!PRE) tma::load_3d(sarr + 4 * AB, &mx, x - XO, y - 1, 0, mbar);
    };
    // the post-smoother's coarse values, one per aggregate of the thread's rows, by a copy that only the thread reads
    auto request_coarse = [&](int x, int y) {
        if constexpr (!PRE) {
            const int X = (x + 2 * lane) >> 1, Y = (y + RB_R * warp) >> 1;
#pragma unroll
            for (int k = 0; k < RB_R / 2; k++) {
                const bool in = X >= 0 && X < C.w && Y + k >= 0 && Y + k < C.h;
                const float* src = in ? xc + (size_t)(Y + k) * C.w + X : xc;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc::smem_addr(sxc + k * RB_NT + tid)), "l"(src),
                             "r"(in ? 4 : 0) : "memory");
            }
        }
    };
    int yt = blockIdx.x / nx, xt = blockIdx.x - yt * nx;  // the region
    int X0 = xt * SX - H, Y0 = yt * SY - H;
    // the operator's boxes (fixed over a solve) while the kernel before still runs, the iterates' after it
    if (tid == 0) {
        arm();
        request_couplings(X0, Y0);
        request_c(X0, Y0, 0);
    }
    pdl_wait();
    if (tid == 0) request_iterate(X0, Y0);
    request_coarse(X0, Y0);
    double acc = 0.0;
    int it = 0;
    for (int t = blockIdx.x; t < regions; t += gridDim.x, it++) {
        const int next = t + (int)gridDim.x;
        int Xn = 0, Yn = 0;  // the next region's corner
        const int gx = X0 + 2 * lane;
        const bool xin = gx >= 0 && gx < w;
        const int gy0 = Y0 + RB_R * warp;
        // read while the boxes land: a weighted level's prolongation weights, the pre-smoother's coarse mask
        float2 t2[RB_R];
        uint8_t cmask[RB_R / 2];
        if constexpr (WT && !PRE) {
#pragma unroll
            for (int r = 0; r < RB_R; r++) {
                const int gy = gy0 + r;
                t2[r] = xin && gy >= 0 && gy < h ? *reinterpret_cast<const float2*>(L.t + (size_t)gy * w + gx) : make_float2(0.f, 0.f);
            }
        }
#pragma unroll
        for (int k = 0; k < RB_R / 2; k++) {
            const int X = gx >> 1, Y = (gy0 + 2 * k) >> 1;
            cmask[k] = (PRE && xin && gy0 + 2 * k >= 0 && X < C.w && Y < C.h) ? C.mask[(size_t)Y * C.w + X] : 0;
        }
        const bool landed = tc::mbar_wait(mbar, it & 1, kMgWaitPolls);
        if (__syncthreads_or(!landed)) {
            if (tid == 0 && L.err) atomicOr(L.err, 1);
            tc::mbar_wait(mbar, it & 1, kMgWaitPolls);  // copies still in flight land before the CTA leaves
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
        }
        const float* sc = sarr + (TWO_C ? 3 + (it & 1) : 3) * AB;
        if constexpr (!PRE) asm volatile("cp.async.wait_all;" ::: "memory");
        float bA[RB_R], bB[RB_R], iA[RB_R], iB[RB_R], dl[RB_R], dm[RB_R], dr[RB_R], dA[RB_R], dB[RB_R];
        float xA[RB_R], xB[RB_R];
        float uA = 0.0f, uB = 0.0f;
        const int col0 = XO + 2 * lane;  // the pair's first column within the box
#pragma unroll
        for (int r = 0; r < RB_R; r++) {
            const int gy = gy0 + r;
            const bool in = xin && gy >= 0 && gy < h;
            const int q = (RB_R * warp + r + 1) * RB_TMA_X + col0;  // the box's row 0 is the region's row -1
            float2 b2 = make_float2(0.f, 0.f), c2 = make_float2(1.f, 1.f), dx2 = b2, dy2 = b2;
            float left = 0.0f;
            if (in) {
                b2 = *reinterpret_cast<const float2*>(sb + q);
                c2 = *reinterpret_cast<const float2*>(sc + q);
                dx2 = *reinterpret_cast<const float2*>(sdx + q);
                dy2 = *reinterpret_cast<const float2*>(sdy + q);
                left = sdx[q - 1];  // zero past the level's left edge
                if (r == 0) {
                    const float2 u2 = *reinterpret_cast<const float2*>(sdy + q - RB_TMA_X);  // zero above row 0
                    uA = u2.x;
                    uB = u2.y;
                }
            }
            bA[r] = b2.x;
            bB[r] = b2.y;
            dm[r] = dx2.x;
            dr[r] = dx2.y;
            dA[r] = dy2.x;
            dB[r] = dy2.y;
            dl[r] = left;
            const float upA = r ? dA[r - 1] : uA, upB = r ? dB[r - 1] : uB;
            iA[r] = in ? __fdividef(1.0f, c2.x + dl[r] + dx2.x + upA + dy2.x) : 0.0f;
            iB[r] = in ? __fdividef(1.0f, c2.y + dx2.x + dx2.y + upB + dy2.y) : 0.0f;
            float x0 = 0.0f, x1 = 0.0f;
            if (!PRE && in) {
                const float2 xv = *reinterpret_cast<const float2*>(sx + q);
                const float corr = omega * sxc[(r >> 1) * RB_NT + tid];
                if constexpr (WT) {
                    x0 = xv.x + corr * t2[r].x;
                    x1 = xv.y + corr * t2[r].y;
                } else {
                    x0 = xv.x + corr;
                    x1 = xv.y + corr;
                }
            }
            xA[r] = x0;
            xB[r] = x1;
        }
        edge[0][0][warp][lane] = make_float2(xA[0], xB[0]);
        edge[0][1][warp][lane] = make_float2(xA[RB_R - 1], xB[RB_R - 1]);
        __syncthreads();
        if (next < regions) {  // this region's boxes are read
            yt = next / nx;
            xt = next - yt * nx;
            Xn = xt * SX - H;
            Yn = yt * SY - H;
            if (tid == 0) {
                arm();
                request_couplings(Xn, Yn);
                if constexpr (!LATE) request_c(Xn, Yn, it + 1);
                request_iterate(Xn, Yn);
            }
            request_coarse(Xn, Yn);
        }
        const int wu = warp > 0 ? warp - 1 : warp, wd = warp + 1 < RB_WARPS ? warp + 1 : warp;
#pragma unroll
        for (int s = 0; s < NS; s++) {
            const int col = PRE ? (s & 1) : 1 - (s & 1);
            const int rd = s & 1, wr = (s + 1) & 1;
            const float2 above = edge[rd][1][wu][lane], below = edge[rd][0][wd][lane];
#pragma unroll
            for (int r = 0; r < RB_R; r++) {
                if (PRE && s == 0) {  // the pre-smoother starts from x = 0: its first half-sweep is b times the inverse
                    if ((r & 1) == col) xA[r] = bA[r] * iA[r];
                    else xB[r] = bB[r] * iB[r];
                    continue;
                }
                if ((r & 1) == col) {
                    const float left = __shfl_up_sync(0xffffffffu, xB[r], 1);
                    const float up = r ? xA[r - 1] : above.x, down = r + 1 < RB_R ? xA[r + 1] : below.x;
                    const float cu = r ? dA[r - 1] : uA;
                    xA[r] = (bA[r] + dl[r] * left + dm[r] * xB[r] + cu * up + dA[r] * down) * iA[r];
                } else {
                    const float right = __shfl_down_sync(0xffffffffu, xA[r], 1);
                    const float up = r ? xB[r - 1] : above.y, down = r + 1 < RB_R ? xB[r + 1] : below.y;
                    const float cu = r ? dB[r - 1] : uB;
                    xB[r] = (bB[r] + dm[r] * xA[r] + dr[r] * right + cu * up + dB[r] * down) * iB[r];
                }
            }
            edge[wr][0][warp][lane] = make_float2(xA[0], xB[0]);
            edge[wr][1][warp][lane] = make_float2(xA[RB_R - 1], xB[RB_R - 1]);
            __syncthreads();
        }
        const bool xout = xin && 2 * lane >= H && 2 * lane < RB_RX - H;
        if constexpr (PRE) {
            const float2 above = edge[NS & 1][1][wu][lane], below = edge[NS & 1][0][wd][lane];
            float ragg[RB_R / 2] = {};
#pragma unroll
            for (int r = 0; r < RB_R; r++) {
                const int gy = gy0 + r, ly = RB_R * warp + r;
                const bool o = xout && ly >= H && ly < RB_RY - H && gy < h;
                const size_t i = (size_t)gy * w + gx;
                if (o) *reinterpret_cast<float2*>(L.x + i) = make_float2(xA[r], xB[r]);
                const float left = __shfl_up_sync(0xffffffffu, xB[r], 1);
                const float right = __shfl_down_sync(0xffffffffu, xA[r], 1);
                const float upA = r ? xA[r - 1] : above.x, dnA = r + 1 < RB_R ? xA[r + 1] : below.x;
                const float upB = r ? xB[r - 1] : above.y, dnB = r + 1 < RB_R ? xB[r + 1] : below.y;
                const float cuA = r ? dA[r - 1] : uA, cuB = r ? dB[r - 1] : uB;
                const float2 c2 = *reinterpret_cast<const float2*>(sc + (RB_R * warp + r + 1) * RB_TMA_X + col0);
                float axA = c2.x * xA[r];
                axA += dl[r] * (xA[r] - left);
                axA += dm[r] * (xA[r] - xB[r]);
                axA += cuA * (xA[r] - upA);
                axA += dA[r] * (xA[r] - dnA);
                float axB = c2.y * xB[r];
                axB += dm[r] * (xB[r] - xA[r]);
                axB += dr[r] * (xB[r] - right);
                axB += cuB * (xB[r] - upB);
                axB += dB[r] * (xB[r] - dnB);
                float rA = bA[r] - axA, rB = bB[r] - axB;
                if constexpr (WT) {  // the restriction's weights, zero past the level (the box's fill)
                    const float2 wt = *reinterpret_cast<const float2*>(sx + (RB_R * warp + r + 1) * RB_TMA_X + col0);
                    rA *= wt.x;
                    rB *= wt.y;
                }
                ragg[r >> 1] += rA + rB;
            }
#pragma unroll
            for (int k = 0; k < RB_R / 2; k++) {
                const int ly = RB_R * warp + 2 * k;
                const int X = gx >> 1, Y = (gy0 + 2 * k) >> 1;
                if (xout && ly >= H && ly < RB_RY - H && X < C.w && Y < C.h && gy0 + 2 * k >= 0)
                    C.b[(size_t)Y * C.w + X] = cmask[k] ? ragg[k] : 0.0f;
            }
            if constexpr (LATE) {
                if (next < regions) {
                    __syncthreads();
                    if (tid == 0) request_c(Xn, Yn, it + 1);
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < RB_R; r++) {
                const int gy = gy0 + r, ly = RB_R * warp + r;
                if (xout && ly >= H && ly < RB_RY - H && gy < h) {
                    const size_t i = (size_t)gy * w + gx;
                    *reinterpret_cast<float2*>(L.x2 + i) = make_float2(xA[r], xB[r]);
                    if (part) acc += (double)bA[r] * (double)xA[r] + (double)bB[r] * (double)xB[r];
                }
            }
        }
        X0 = Xn;
        Y0 = Yn;
    }
    if (!PRE && part) cta_partial(acc, part);
}

// ---- the coarse tail: every level of at most 64 x 64 cells, inside one CTA
//
// What bounds it is latency: sixteen dependent half-sweeps a level under V(4,4), a few hundred cells each. So a level
// is held in registers by no more warps than it fills, each thread a band of 4 rows of one column pair (as in the
// row-band smoother), and synchronises only those: the top level by up to 16 warps, lanes = 32 column pairs, band edges
// through shared memory; the next level (at most 32 x 32) by up to 4 warps of two 16-pair row groups; every level of at
// most 16 x 16 by warp 0 alone, 8 pairs x 4 row groups, neighbours by shuffles and no barrier at all. The top level's
// coefficients stay in registers from its pre- to its post-smoother; the lower levels are read from the image
// mg_tail_setup_kernel writes once per Newton pass, whose rows are padded to even pitches and heights so that no access
// has an edge case. 64 x 64 top under V(4,4): 27 -> 15.5 us a V-cycle against the whole CTA of 1,024 threads meeting at
// every half-sweep of every level.
extern __shared__ __align__(16) unsigned char tail_smem_raw[];

struct TailBand {
    float bA[RB_R], bB[RB_R], iA[RB_R], iB[RB_R], dl[RB_R], dm[RB_R], dr[RB_R], dA[RB_R], dB[RB_R], xA[RB_R], xB[RB_R];
    float uA, uB;  // the couplings of row 0 to the row above
};

using TailEdge = float2[2][RB_WARPS][32];  // [top row / bottom row][warp][lane]: (x of 2j, x of 2j + 1)

__device__ __forceinline__ void tail_bar(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The band's coefficients from arrays of pitch p and hp rows (both even): column pair j of LC, rows row0 .. row0 + 3.
template <int LC>
__device__ __forceinline__ void tail_load(TailBand& B, const float* inv, const float* dx, const float* dy, int p, int hp,
                                          int j, int row0) {
    const bool in = 2 * j < p;
    const float2 z = make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        const int row = row0 + r, q = row * p + 2 * j;
        const bool ok = in && row < hp;
        const float2 i2 = ok ? *reinterpret_cast<const float2*>(inv + q) : z;
        const float2 x2 = ok ? *reinterpret_cast<const float2*>(dx + q) : z;
        const float2 y2 = ok ? *reinterpret_cast<const float2*>(dy + q) : z;
        B.iA[r] = i2.x;
        B.iB[r] = i2.y;
        B.dm[r] = x2.x;
        B.dr[r] = x2.y;
        B.dA[r] = y2.x;
        B.dB[r] = y2.y;
        const float l = __shfl_up_sync(0xffffffffu, x2.y, 1);
        B.dl[r] = j ? l : 0.0f;
    }
    const float2 u2 = in && row0 > 0 && row0 - 1 < hp ? *reinterpret_cast<const float2*>(dy + (row0 - 1) * p + 2 * j) : z;
    B.uA = u2.x;
    B.uB = u2.y;
}

// The rows above and below the band, as the last half-sweep left them.
template <int LC>
__device__ __forceinline__ void tail_rows(const TailBand& B, const TailEdge& e, int warp, int lane, float2& above,
                                          float2& below) {
    if constexpr (LC == 32) {
        above = e[1][warp > 0 ? warp - 1 : 0][lane];
        below = e[0][warp + 1 < RB_WARPS ? warp + 1 : warp][lane];
    } else {
        above = make_float2(__shfl_up_sync(0xffffffffu, B.xA[RB_R - 1], LC), __shfl_up_sync(0xffffffffu, B.xB[RB_R - 1], LC));
        below = make_float2(__shfl_down_sync(0xffffffffu, B.xA[0], LC), __shfl_down_sync(0xffffffffu, B.xB[0], LC));
        if constexpr (LC == 16) {  // two row groups a warp: the outer rows belong to the next warps
            const int j = lane & 15;
            if (lane < 16) above = e[1][warp > 0 ? warp - 1 : 0][j];
            else below = e[0][warp + 1 < RB_WARPS ? warp + 1 : warp][j];
        }
    }
}

template <int LC>
__device__ __forceinline__ void tail_post_edges(const TailBand& B, TailEdge& e, int warp, int lane) {
    if constexpr (LC == 32) {
        e[0][warp][lane] = make_float2(B.xA[0], B.xB[0]);
        e[1][warp][lane] = make_float2(B.xA[RB_R - 1], B.xB[RB_R - 1]);
    } else if constexpr (LC == 16) {
        if (lane < 16) e[0][warp][lane] = make_float2(B.xA[0], B.xB[0]);
        else e[1][warp][lane - 16] = make_float2(B.xA[RB_R - 1], B.xB[RB_R - 1]);
    }
}

template <int LC, int COL>
__device__ __forceinline__ void tail_half_sweep(TailBand& B, const TailEdge& e, int warp, int lane) {
    float2 above, below;
    tail_rows<LC>(B, e, warp, lane, above, below);
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        if ((r & 1) == COL) {
            const float left = __shfl_up_sync(0xffffffffu, B.xB[r], 1);
            const float up = r ? B.xA[r - 1] : above.x, down = r + 1 < RB_R ? B.xA[r + 1] : below.x;
            const float cu = r ? B.dA[r - 1] : B.uA;
            B.xA[r] = (B.bA[r] + B.dl[r] * left + B.dm[r] * B.xB[r] + cu * up + B.dA[r] * down) * B.iA[r];
        } else {
            const float right = __shfl_down_sync(0xffffffffu, B.xA[r], 1);
            const float up = r ? B.xB[r - 1] : above.y, down = r + 1 < RB_R ? B.xB[r + 1] : below.y;
            const float cu = r ? B.dB[r - 1] : B.uB;
            B.xB[r] = (B.bB[r] + B.dm[r] * B.xA[r] + B.dr[r] * right + cu * up + B.dB[r] * down) * B.iB[r];
        }
    }
}

// `sweeps` sweeps, colour FIRST before the other; the edges in e[0] on entry and on return.
template <int LC, int FIRST>
__device__ __forceinline__ void tail_sweeps(TailBand& B, TailEdge* e, int sweeps, int warp, int lane, int bar,
                                            int threads) {
    for (int s = 0; s < sweeps; s++) {
        tail_half_sweep<LC, FIRST>(B, e[0], warp, lane);
        if constexpr (LC > 8) {
            tail_post_edges<LC>(B, e[1], warp, lane);
            tail_bar(bar, threads);
        }
        tail_half_sweep<LC, 1 - FIRST>(B, e[1], warp, lane);
        if constexpr (LC > 8) {
            tail_post_edges<LC>(B, e[0], warp, lane);
            tail_bar(bar, threads);
        }
    }
}

// One array's cells of the band (0 outside).
__device__ __forceinline__ void tail_cells(float2 (&v)[RB_R], const float* a, int p, int hp, int j, int row0) {
#pragma unroll
    for (int r = 0; r < RB_R; r++)
        v[r] = 2 * j < p && row0 + r < hp ? *reinterpret_cast<const float2*>(a + (row0 + r) * p + 2 * j)
                                          : make_float2(0.f, 0.f);
}

// The residual in difference form, weighted and summed over each 2 x 2 aggregate, into the next level's b.
template <int LC>
__device__ __forceinline__ void tail_restrict(const TailBand& B, const TailEdge* e, const float2 (&cc)[RB_R],
                                              const float2 (&tt)[RB_R], int j, int row0, int warp, int lane, float* cb,
                                              int cp, int cw, int ch) {
    float2 above, below;
    tail_rows<LC>(B, e[0], warp, lane, above, below);
    float ragg[RB_R / 2] = {};
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        const float2 c2 = cc[r], t2 = tt[r];
        const float left = __shfl_up_sync(0xffffffffu, B.xB[r], 1);
        const float right = __shfl_down_sync(0xffffffffu, B.xA[r], 1);
        const float upA = r ? B.xA[r - 1] : above.x, dnA = r + 1 < RB_R ? B.xA[r + 1] : below.x;
        const float upB = r ? B.xB[r - 1] : above.y, dnB = r + 1 < RB_R ? B.xB[r + 1] : below.y;
        const float cuA = r ? B.dA[r - 1] : B.uA, cuB = r ? B.dB[r - 1] : B.uB;
        float axA = c2.x * B.xA[r];
        axA += B.dl[r] * (B.xA[r] - left);
        axA += B.dm[r] * (B.xA[r] - B.xB[r]);
        axA += cuA * (B.xA[r] - upA);
        axA += B.dA[r] * (B.xA[r] - dnA);
        float axB = c2.y * B.xB[r];
        axB += B.dm[r] * (B.xB[r] - B.xA[r]);
        axB += B.dr[r] * (B.xB[r] - right);
        axB += cuB * (B.xB[r] - upB);
        axB += B.dB[r] * (B.xB[r] - dnB);
        // masked and padding cells: b = 0, x = 0 and no couplings, so their residual is 0
        ragg[r >> 1] += t2.x * (B.bA[r] - axA) + t2.y * (B.bB[r] - axB);
    }
#pragma unroll
    for (int k = 0; k < RB_R / 2; k++) {
        const int Y = (row0 >> 1) + k;
        if (j < cw && Y < ch) cb[Y * cp + j] = ragg[k];
    }
}

// x += ω t x_c
__device__ __forceinline__ void tail_correct(TailBand& B, const float2 (&tt)[RB_R], int j, int row0, float omega,
                                             const float* cx, int cp, int cw, int ch) {
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        const int Y = (row0 + r) >> 1;
        if (j < cw && Y < ch) {
            const float v = omega * cx[Y * cp + j];
            B.xA[r] += v * tt[r].x;
            B.xB[r] += v * tt[r].y;
        }
    }
}

// A lower level's pre-smoother from x = 0, its restriction, and its iterate left in shared memory.
template <int LC>
__device__ __forceinline__ void tail_down(const TailLevel& T, const TailLevel& C, float* f, TailEdge* e, int pre,
                                          int warp, int lane, int bar, int threads) {
    const int j = lane & (LC - 1), row0 = RB_R * ((32 / LC) * warp + lane / LC);
    TailBand B;
    tail_load<LC>(B, f + T.inv, f + T.dx, f + T.dy, T.p, T.hp, j, row0);
    const bool in = 2 * j < T.p;
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        const bool ok = in && row0 + r < T.hp;
        const float2 b2 = ok ? *reinterpret_cast<const float2*>(f + T.b + (row0 + r) * T.p + 2 * j) : make_float2(0.f, 0.f);
        B.bA[r] = b2.x;
        B.bB[r] = b2.y;
        B.xA[r] = B.xB[r] = 0.0f;
    }
    if constexpr (LC > 8) {
        tail_post_edges<LC>(B, e[0], warp, lane);
        tail_bar(bar, threads);
    }
    tail_sweeps<LC, 0>(B, e, pre, warp, lane, bar, threads);
    float2 c2[RB_R], t2[RB_R];
    tail_cells(c2, f + T.c, T.p, T.hp, j, row0);
    tail_cells(t2, f + T.t, T.p, T.hp, j, row0);
    tail_restrict<LC>(B, e, c2, t2, j, row0, warp, lane, f + C.b, C.p, C.w, C.h);
#pragma unroll
    for (int r = 0; r < RB_R; r++)
        if (in && row0 + r < T.hp)
            *reinterpret_cast<float2*>(f + T.x + (row0 + r) * T.p + 2 * j) = make_float2(B.xA[r], B.xB[r]);
}

// A lower level's coarse correction and post-smoother, its result left in shared memory.
template <int LC>
__device__ __forceinline__ void tail_up(const TailLevel& T, const TailLevel& C, float* f, TailEdge* e, int post,
                                        float omega, int warp, int lane, int bar, int threads) {
    const int j = lane & (LC - 1), row0 = RB_R * ((32 / LC) * warp + lane / LC);
    TailBand B;
    tail_load<LC>(B, f + T.inv, f + T.dx, f + T.dy, T.p, T.hp, j, row0);
    const bool in = 2 * j < T.p;
#pragma unroll
    for (int r = 0; r < RB_R; r++) {
        const int q = (row0 + r) * T.p + 2 * j;
        const bool ok = in && row0 + r < T.hp;
        const float2 z = make_float2(0.f, 0.f);
        const float2 b2 = ok ? *reinterpret_cast<const float2*>(f + T.b + q) : z;
        const float2 x2 = ok ? *reinterpret_cast<const float2*>(f + T.x + q) : z;
        B.bA[r] = b2.x;
        B.bB[r] = b2.y;
        B.xA[r] = x2.x;
        B.xB[r] = x2.y;
    }
    float2 t2[RB_R];
    tail_cells(t2, f + T.t, T.p, T.hp, j, row0);
    tail_correct(B, t2, j, row0, omega, f + C.x, C.p, C.w, C.h);
    if constexpr (LC > 8) {
        tail_post_edges<LC>(B, e[0], warp, lane);
        tail_bar(bar, threads);
    }
    tail_sweeps<LC, 1>(B, e, post, warp, lane, bar, threads);
#pragma unroll
    for (int r = 0; r < RB_R; r++)
        if (in && row0 + r < T.hp)
            *reinterpret_cast<float2*>(f + T.x + (row0 + r) * T.p + 2 * j) = make_float2(B.xA[r], B.xB[r]);
}

// The coarsest level exactly, by warp 0: x = A⁻¹ b with the inverse built once per Newton pass (at most 4 x 4 cells).
__device__ __forceinline__ void tail_coarsest(const TailLevel& T, float* f, const float* sinv, int lane) {
    const int nc = T.w * T.h;
    if (lane < nc) {
        float s = 0.0f;
        for (int y = 0, k = 0; y < T.h; y++)
            for (int x = 0; x < T.w; x++, k++) s += sinv[lane * nc + k] * f[T.b + y * T.p + x];
        f[T.x + (lane / T.w) * T.p + lane % T.w] = s;  // a masked cell: an identity row and b = 0
    }
    __syncwarp();
}

__global__ void __launch_bounds__(TAIL_THREADS, 1) mg_tail_kernel(const __grid_constant__ TailArgs A) {
    float* f = reinterpret_cast<float*>(tail_smem_raw + 2 * sizeof(TailEdge));
    TailEdge* e = reinterpret_cast<TailEdge*>(tail_smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_launch();
    pdl_wait();
    // the level table, read by run-time index below, out of the constant bank once; the lower levels' image (b and x 0)
    // into shared memory while the top level's loads are in flight
    __shared__ TailLevel sT[kTailLevels];
    if (threadIdx.x < kTailLevels * (int)(sizeof(TailLevel) / 4))
        reinterpret_cast<int*>(sT)[threadIdx.x] = reinterpret_cast<const int*>(A.T)[threadIdx.x];
    for (int q = threadIdx.x; q < A.img_f4; q += TAIL_THREADS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_addr(f + 4 * q)), "l"(A.img + 4 * q) : "memory");
    const TailLevel& T = A.T[0];
    const TailLevel& T1 = sT[1];
    const int nw = (T.h + RB_R - 1) / RB_R, nw1 = (A.T[1].h + 2 * RB_R - 1) / (2 * RB_R);
    const int row0 = RB_R * warp;
    TailBand B;
    float2 c2[RB_R], t2[RB_R];
    tail_load<32>(B, A.img + T.inv, A.img + T.dx, A.img + T.dy, T.p, T.hp, lane, row0);
    {
        const float* b = A.b;
        const bool two = 2 * lane + 1 < T.w;
#pragma unroll
        for (int r = 0; r < RB_R; r++) {
            const bool ok = 2 * lane < T.w && row0 + r < T.h;
            const int q = (row0 + r) * T.w + 2 * lane;
            B.bA[r] = ok ? b[q] : 0.0f;
            B.bB[r] = ok && two ? b[q + 1] : 0.0f;
            B.xA[r] = B.xB[r] = 0.0f;
        }
    }
    tail_cells(c2, A.img + T.c, T.p, T.hp, lane, row0);
    tail_cells(t2, A.img + T.t, T.p, T.hp, lane, row0);
    // every warp's rows in both edge buffers: a band past the level's last row reads 0 (times no coupling)
    tail_post_edges<32>(B, e[0], warp, lane);
    tail_post_edges<32>(B, e[1], warp, lane);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (warp < nw) {
        tail_sweeps<32, 0>(B, e, A.pre, warp, lane, 1, 32 * nw);
        tail_restrict<32>(B, e, c2, t2, lane, row0, warp, lane, f + T1.b, T1.p, T1.w, T1.h);
    }
    __syncthreads();
    if (warp < nw1) {
        tail_down<16>(T1, sT[2], f, e, A.pre, warp, lane, 2, 32 * nw1);
        tail_bar(2, 32 * nw1);
        if (warp == 0) {
            for (int l = 2; l < A.nl - 1; l++) {
                tail_down<8>(sT[l], sT[l + 1], f, e, A.pre, 0, lane, 0, 0);
                __syncwarp();
            }
            tail_coarsest(sT[A.nl - 1], f, f + A.sinv, lane);
            for (int l = A.nl - 2; l >= 2; l--) {
                tail_up<8>(sT[l], sT[l + 1], f, e, A.post, A.omega, 0, lane, 0, 0);
                __syncwarp();
            }
        }
        tail_bar(2, 32 * nw1);
        tail_up<16>(T1, sT[2], f, e, A.post, A.omega, warp, lane, 2, 32 * nw1);
    }
    __syncthreads();
    double acc = 0.0;
    tail_correct(B, t2, lane, row0, A.omega, f + T1.x, T1.p, T1.w, T1.h);
    tail_post_edges<32>(B, e[0], warp, lane);
    __syncthreads();
    if (warp < nw) {
        tail_sweeps<32, 1>(B, e, A.post, warp, lane, 1, 32 * nw);
        const bool two = 2 * lane + 1 < T.w;
#pragma unroll
        for (int r = 0; r < RB_R; r++) {
            if (!(2 * lane < T.w && row0 + r < T.h)) continue;
            const int q = (row0 + r) * T.w + 2 * lane;
            A.x2[q] = B.xA[r];
            if (two) A.x2[q + 1] = B.xB[r];
            acc += (double)B.bA[r] * (double)B.xA[r] + (double)B.bB[r] * (double)B.xB[r];
        }
    }
    if (A.out) {
        __shared__ double red[RB_WARPS];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (lane == 0) red[warp] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int q = 0; q < RB_WARPS; q++) t += red[q];
            *A.out = t;
        }
    }
}

// The image's layout, in floats: the lower levels' seven arrays and the coarsest inverse (the part the tail copies to
// shared memory, a multiple of 16 bytes), then the top level's five coefficient arrays. Every array has an even pitch
// and an even number of rows. Fills A.T, A.sinv and A.img_f4; returns the image's size in floats.
int tail_layout(const Multigrid& M, TailArgs& A) {
    int off = 0;
    const int nl = M.nlevels - M.tail;
    for (int q = 1; q <= nl; q++) {
        const int k = q % nl, l = M.tail + k;  // the top level last
        if (k == 0) {
            const int nc = M.L[M.nlevels - 1].w * M.L[M.nlevels - 1].h;
            A.sinv = off;
            off = (off + nc * nc + 3) & ~3;
            A.img_f4 = off / 4;
        }
        TailLevel& T = A.T[k];
        T.w = M.L[l].w;
        T.h = M.L[l].h;
        T.p = (T.w + 1) & ~1;
        T.hp = (T.h + 1) & ~1;
        const int n = T.p * T.hp;
        T.dx = off;
        T.dy = off + n;
        T.inv = off + 2 * n;
        T.t = off + 3 * n;
        T.c = off + 4 * n;
        T.b = off + 5 * n;
        T.x = off + 6 * n;
        off += (k == 0 ? 5 : 7) * n;
    }
    return off;
}

// The tail's shared memory at most: 32 x 32, 16 x 16, 8 x 8 and 4 x 4 levels of seven arrays, a 16 x 16 inverse, edges.
constexpr size_t kTailSmem = 2 * sizeof(TailEdge) + (7 * (1024 + 256 + 64 + 16) + 256) * sizeof(float);

// Everything the tail kernel and its packing need but the output slot; returns the launch's shared memory.
size_t tail_args(const Multigrid& M, TailArgs& T) {
    tail_layout(M, T);
    T.nl = M.nlevels - M.tail;
    T.pre = M.pre;
    T.post = M.post;
    T.omega = M.omega;
    T.img = M.tail_img;
    T.out = nullptr;
    T.b = M.L[M.tail].b;
    T.x2 = M.L[M.tail].x2;
    return 2 * sizeof(TailEdge) + (size_t)T.img_f4 * 16;
}

// The tail's levels below its top, and its image for the next V-cycles, once per Newton pass: level by level in shared
// memory, the weights (mg_coarsen_kernel's four half-sweeps and scaling; level 0 takes none), the Galerkin operator
// (f64 sums) and the level's part of the image — couplings, inverse diagonal, weights and c, 0 (c: 1) on the padding, b
// and x at 0 — then the coarsest operator's inverse. One CTA: the levels are a serial chain of a few thousand cells at
// most, so launches and their ramps were what it cost (a coarsening a level, the inverse and the packing: 53 us for a
// 64 x 64 top, in six launches; now one of 23 us). Every level has the top's pitch, so that a thread's cell is its
// index's bits and not a division, and the column before and the row above a level (couplings 0) are never written.
constexpr int TS_NT = 1024, TS_P = kMgTailSide + 2, TS_N = TS_P * TS_P;  // a level with a rim of one cell around it

struct TailSetupShared {
    float c[2][TS_N], dx[2][TS_N], dy[2][TS_N], t[TS_N];  // this level and the next
    uint8_t m[2][TS_N];
    double aug[2][16 * 32];
    double rpiv[2];
};

// The coarsest operator's inverse by Gauss-Jordan elimination in f64 (SPD: no pivoting; masked cells are identity rows),
// one thread per element of [A | I]; the thread that writes the next pivot leaves its reciprocal. Stored f32.
__device__ __forceinline__ void tail_inverse(TailSetupShared& S, int k, int w, int h, float* inv, int room) {
    constexpr int p = TS_P;
    const int n = w * h, i = threadIdx.x >> 5, j = threadIdx.x & 31;
    if (i < n && j < 2 * n) {
        double v = 0.0;
        if (j >= n) {
            v = j - n == i ? 1.0 : 0.0;
        } else {
            const int xi = i % w, yi = i / w, q = (yi + 1) * p + xi + 1;
            if (!S.m[k][q]) {
                v = i == j ? 1.0 : 0.0;
            } else {
                const double dl = S.dx[k][q - 1], dr = S.dx[k][q], du = S.dy[k][q - p], dd = S.dy[k][q];
                if (j == i) v = (double)S.c[k][q] + dl + dr + du + dd;
                else if (xi > 0 && j == i - 1) v = -dl;
                else if (xi + 1 < w && j == i + 1) v = -dr;
                else if (yi > 0 && j == i - w) v = -du;
                else if (yi + 1 < h && j == i + w) v = -dd;
            }
        }
        S.aug[0][i * 32 + j] = v;
        if (i == 0 && j == 0) S.rpiv[0] = 1.0 / v;
    }
    __syncthreads();
    for (int s = 0; s < n; s++) {
        if (i < n && j < 2 * n) {
            const double* src = S.aug[s & 1];
            const double pj = src[s * 32 + j] * S.rpiv[s & 1];
            const double v = i == s ? pj : src[i * 32 + j] - src[i * 32 + s] * pj;
            S.aug[(s + 1) & 1][i * 32 + j] = v;
            if (i == s + 1 && j == s + 1) S.rpiv[(s + 1) & 1] = 1.0 / v;
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < room; e += TS_NT) inv[e] = e < n * n ? (float)S.aug[n & 1][(e / n) * 32 + n + e % n] : 0.0f;
}

__global__ void __launch_bounds__(TS_NT) mg_tail_setup_kernel(const __grid_constant__ TailArgs A, MgLevel top, bool level0,
                                                              float* img) {
    extern __shared__ __align__(16) unsigned char setup_smem[];
    TailSetupShared& S = *reinterpret_cast<TailSetupShared*>(setup_smem);
    constexpr int p = TS_P;
    // cells by 64 columns x 16 rows of threads, aggregates and a sweep's pairs by 32 x 32
    const int tid = threadIdx.x, x64 = tid & 63, y64 = tid >> 6, x32 = tid & 31, y32 = tid >> 5;
    {
        float lc[4], ldx[4], ldy[4];
        uint8_t lm[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int y = y64 + 16 * u, i = y * top.w + x64;
            const bool in = x64 < top.w && y < top.h;
            lc[u] = in ? top.c[i] : 1.0f;
            ldx[u] = in ? top.dx[i] : 0.0f;
            ldy[u] = in ? top.dy[i] : 0.0f;
            lm[u] = in ? top.mask[i] : 0;
        }
        for (int q = tid; q < TS_N; q += TS_NT) S.t[q] = 0.0f;
        if (tid < TS_P) {
            S.dx[0][tid * p] = S.dx[1][tid * p] = 0.0f;
            S.dy[0][tid] = S.dy[1][tid] = 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int q = (y64 + 16 * u + 1) * p + x64 + 1;
            S.c[0][q] = lc[u];
            S.dx[0][q] = ldx[u];
            S.dy[0][q] = ldy[u];
            S.m[0][q] = lm[u];
        }
    }
    for (int l = 0; l < A.nl; l++) {
        const TailLevel& T = A.T[l];
        const int k = l & 1, w = T.w, h = T.h;
        const float *c = S.c[k], *dx = S.dx[k], *dy = S.dy[k];
        const uint8_t* m = S.m[k];
        float* t = S.t;
        const bool coarsest = l + 1 == A.nl;
        __syncthreads();
        if (!coarsest) {
            if (x64 < w)
                for (int y = y64; y < h; y += 16) {
                    const int q = (y + 1) * p + x64 + 1;
                    t[q] = m[q] ? 1.0f : 0.0f;
                }
            __syncthreads();
            if (l > 0 || !level0) {
                for (int sweep = 0; sweep < 4; sweep++) {
                    for (int y = y32; y < h; y += 32) {
                        const int x = 2 * x32 + ((y + sweep) & 1);
                        if (x >= w) continue;
                        // a masked cell has c = 1 and no couplings (nor do its neighbours towards it): it stays 0
                        const int q = (y + 1) * p + x + 1;
                        const float dl = dx[q - 1], dr = dx[q], du = dy[q - p], dd = dy[q];
                        const float num = dl * t[q - 1] + dr * t[q + 1] + du * t[q - p] + dd * t[q + p];
                        t[q] = num / (c[q] + dl + dr + du + dd);
                    }
                    __syncthreads();
                }
            }
            // each aggregate scaled to a largest weight of 1 (1 on its system cells where all weights vanished), then
            // the Galerkin operator, whose couplings read the neighbouring aggregates' scaled weights
            const int cw = A.T[l + 1].w, ch = A.T[l + 1].h;
            const int X = x32, Y = y32;
            const bool agg = X < cw && Y < ch;
            const int q = (2 * Y + 1) * p + 2 * X + 1;
            const bool x1 = 2 * X + 1 < w, y1 = 2 * Y + 1 < h;
            const bool has[4] = {agg, agg && x1, agg && y1, agg && x1 && y1};
            const int at[4] = {q, q + 1, q + p, q + p + 1};
            if (agg) {
                float big = 0.0f;
#pragma unroll
                for (int a = 0; a < 4; a++)
                    if (has[a]) big = fmaxf(big, t[at[a]]);
#pragma unroll
                for (int a = 0; a < 4; a++)
                    if (has[a]) t[at[a]] = !m[at[a]] ? 0.0f : (big > 1e-30f ? t[at[a]] / big : 1.0f);
            }
            __syncthreads();
            if (agg) {
                double csum = 0.0, sx = 0.0, sy = 0.0;
                bool any = false;
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    const int j = at[a];
                    if (!has[a] || !m[j]) continue;
                    any = true;
                    const double tj = t[j];
                    csum += tj * ((double)c[j] * tj + (double)dx[j - 1] * (tj - t[j - 1]) + (double)dx[j] * (tj - t[j + 1]) +
                                  (double)dy[j - p] * (tj - t[j - p]) + (double)dy[j] * (tj - t[j + p]));
                    if (a & 1) sx += tj * t[j + 1] * dx[j];
                    if (a & 2) sy += tj * t[j + p] * dy[j];
                }
                const int o = (Y + 1) * p + X + 1;
                S.c[1 - k][o] = any ? (float)csum : 1.0f;
                S.dx[1 - k][o] = any ? (float)sx : 0.0f;
                S.dy[1 - k][o] = any ? (float)sy : 0.0f;
                S.m[1 - k][o] = any;
            }
        }
        if (x64 < T.p)
            for (int y = y64; y < T.hp; y += 16) {
                const int q = y * T.p + x64, j = (y + 1) * p + x64 + 1;
                const bool ok = x64 < w && y < h;
                img[T.dx + q] = ok ? dx[j] : 0.0f;
                img[T.dy + q] = ok ? dy[j] : 0.0f;
                img[T.inv + q] = ok && m[j] ? 1.0f / (c[j] + dx[j] + dy[j] + dx[j - 1] + dy[j - p]) : 0.0f;
                img[T.t + q] = ok && !coarsest ? t[j] : 0.0f;
                img[T.c + q] = ok ? c[j] : 1.0f;
                if (l > 0) {
                    img[T.b + q] = 0.0f;
                    img[T.x + q] = 0.0f;
                }
            }
        if (coarsest) tail_inverse(S, k, w, h, img + A.sinv, 4 * A.img_f4 - A.sinv);
    }
}

// Level 0's width is even, so every level that comes here has weights.
template <int NS, bool PRE, int SX, int SY, int NT>
void launch_smooth_t(const MgLevel& L, const MgLevel& C, const float* xc, float omega, cudaStream_t s) {
    const dim3 grid(div_up(L.w, SX), div_up(L.h, SY));
    mg_smooth_kernel<NS, PRE, SX, SY, NT><<<grid, NT, smooth_smem<NS, PRE, SX, SY>(), s>>>(L, C, xc, omega);
    sr_note_launch();
}

bool small_tiles(const MgLevel& L) { return (size_t)div_up(L.w, BIG_SX) * div_up(L.h, BIG_SY) < 2 * 148; }

// A smoother's tile height: of the even heights from SY_MAX down to SY_MAX - 6, the one with the most output cells per
// sweep slot (a half-sweep gives each thread ceil(cells of one colour in the halo'd tile / NT) slots; the last slot
// round should be nearly full, or most threads wait at its barrier).
template <int NS, bool PRE, int SX, int SY_MAX, int NT>
constexpr int tile_sy() {
    constexpr int H = PRE ? NS + 1 : NS;
    int best = SY_MAX;
    double best_rate = 0.0;
    for (int sy = SY_MAX; sy >= SY_MAX - 6; sy -= 2) {
        const int hn = (SX + 2 * H) / 2 * (sy + 2 * H);
        const int slots = (hn + NT - 1) / NT;
        const double rate = (double)(SX * sy) / slots;
        if (rate > best_rate) {
            best_rate = rate;
            best = sy;
        }
    }
    return best;
}

template <int NS, bool PRE>
void launch_rowband(const MgLevel& L, const MgLevel& C, const float* xc, float omega, double* part, bool overlap,
                    cudaStream_t s) {
    constexpr int H = rb_halo<NS, PRE>();
    // Level 0 (a world's axes are multiples of 8, its planes allocations of their own) and every other level with
    // rows of 16 bytes and 16-byte bases: the region staged by TMA
    auto aligned = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    if (L.w % 4 == 0 && aligned(L.b) && aligned(L.c) && aligned(L.dx) && aligned(L.dy) && aligned(L.x) &&
        (!L.t || aligned(L.t))) {
        CUtensorMap mb, mc, mdx, mdy, mx;
        tma_encode_planes(&mb, L.b, L.w, L.h, 1, RB_TMA_X, RB_TMA_Y);
        tma_encode_planes(&mc, L.c, L.w, L.h, 1, RB_TMA_X, RB_TMA_Y);
        tma_encode_planes(&mdx, L.dx, L.w, L.h, 1, RB_TMA_X, RB_TMA_Y);
        tma_encode_planes(&mdy, L.dy, L.w, L.h, 1, RB_TMA_X, RB_TMA_Y);
        if (!PRE) tma_encode_planes(&mx, L.x, L.w, L.h, 1, RB_TMA_X, RB_TMA_Y);
        else if (L.t) tma_encode_planes(&mx, L.t, L.w, L.h, 1, RB_TMA_X, RB_TMA_Y);
        else mx = mb;
        auto go = [&](auto kernel, bool& attr) {
            if (!attr) {  // the instance's shared-memory attribute, once per process
                SR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRbSmem));
                attr = true;
            }
            launch_kernel(overlap, kernel, dim3(rb_grid(L, H)), dim3(RB_NT), kRbSmem, s, mb, mc, mdx, mdy, mx, L, C, xc, omega, part);
        };
        static bool attr_w = false, attr_u = false;
        if (L.t) go(mg_rowband_tma_kernel<NS, PRE, true>, attr_w);
        else go(mg_rowband_tma_kernel<NS, PRE, false>, attr_u);
        sr_note_launch();
        return;
    }
    if (part) throw SrError{SR_E_CUDA, "multigrid: level 0 is not laid out in 16-byte rows"};
    const dim3 grid(div_up(L.w, RB_RX - 2 * H), div_up(L.h, RB_RY - 2 * H));
    if (L.t) mg_rowband_kernel<NS, PRE, true><<<grid, RB_NT, 0, s>>>(L, C, xc, omega);
    else mg_rowband_kernel<NS, PRE, false><<<grid, RB_NT, 0, s>>>(L, C, xc, omega);
    sr_note_launch();
}

// The row-band kernel wherever the level's width is even (it loads cell pairs as 8-byte words): its registers beat the
// shared-memory tiles at every size (level 0 of a 512² world under V(4,4): pre 11.9 -> 4.7 us, post 12.5 -> 7.0). Levels
// of odd width take the shared-memory tiles, the small one where the big one leaves fewer than 2 CTAs per SM.
template <int NS, bool PRE>
void launch_smooth(const MgLevel& L, const MgLevel& C, const float* xc, float omega, double* part, bool overlap,
                   cudaStream_t s) {
    if (L.w % 2 == 0)
        launch_rowband<NS, PRE>(L, C, xc, omega, part, overlap, s);
    else if (small_tiles(L))
        launch_smooth_t<NS, PRE, SMALL_SX, tile_sy<NS, PRE, SMALL_SX, SMALL_SY, SMALL_NT>(), SMALL_NT>(
            L, C, xc, omega, s);
    else
        launch_smooth_t<NS, PRE, BIG_SX, tile_sy<NS, PRE, BIG_SX, BIG_SY, BIG_NT>(), BIG_NT>(L, C, xc, omega, s);
}

// `overlap`: the launch before on the stream is a kernel of the same V-cycle.
void smooth(int nu, bool pre, const MgLevel& L, const MgLevel& C, const float* xc, float omega, double* part,
            bool overlap, cudaStream_t s) {
    if (pre) {
        if (nu == 1) launch_smooth<2, true>(L, C, xc, omega, part, overlap, s);
        else if (nu == 2) launch_smooth<4, true>(L, C, xc, omega, part, overlap, s);
        else if (nu == 3) launch_smooth<6, true>(L, C, xc, omega, part, overlap, s);
        else launch_smooth<8, true>(L, C, xc, omega, part, overlap, s);
    } else {
        if (nu == 1) launch_smooth<2, false>(L, C, xc, omega, part, overlap, s);
        else if (nu == 2) launch_smooth<4, false>(L, C, xc, omega, part, overlap, s);
        else if (nu == 3) launch_smooth<6, false>(L, C, xc, omega, part, overlap, s);
        else launch_smooth<8, false>(L, C, xc, omega, part, overlap, s);
    }
}

template <int NS, bool PRE, int SX, int SY, int NT>
void set_attribute_one() {
    SR_CUDA_TRY(cudaFuncSetAttribute(mg_smooth_kernel<NS, PRE, SX, SY, NT>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smooth_smem<NS, PRE, SX, SY>()));
}

template <int NS, int SX, int SY, int NT>
void set_attributes_tile() {
    constexpr int PSY = tile_sy<NS, true, SX, SY, NT>(), QSY = tile_sy<NS, false, SX, SY, NT>();
    set_attribute_one<NS, true, SX, PSY, NT>();
    set_attribute_one<NS, false, SX, QSY, NT>();
}

template <int NS>
void set_attributes_ns() {
    set_attributes_tile<NS, BIG_SX, BIG_SY, BIG_NT>();
    set_attributes_tile<NS, SMALL_SX, SMALL_SY, SMALL_NT>();
}

int grid_for(size_t n) {
    size_t b = (n + 255) / 256;
    return (int)(b < 1 ? 1 : (b > 148 * 16 ? 148 * 16 : b));
}

}  // namespace

void Multigrid::create(int w, int h, int pre_, int post_) {
    SR_REQUIRE(pre_ >= 1 && pre_ <= 4 && post_ >= 1 && post_ <= 4, "V-cycle sweeps must be 1..4");
    pre = pre_;
    post = post_;
    nlevels = 0;
    int lw = w, lh = h;
    for (;;) {
        MgLevel& L = this->L[nlevels];
        L.w = lw;
        L.h = lh;
        nlevels++;
        if ((lw <= 4 && lh <= 4) || nlevels == kMgMaxLevels) break;
        lw = (lw + 1) / 2;
        lh = (lh + 1) / 2;
    }
    tail = 0;
    while (L[tail].w > kMgTailSide || L[tail].h > kMgTailSide) tail++;
    SR_REQUIRE(nlevels - tail >= 3 && nlevels - tail <= kTailLevels && (size_t)L[nlevels - 1].w * L[nlevels - 1].h <= 16, "the coarse tail's levels");
    // the levels down to the tail's top; those below it live in the tail's image
    for (int l = 0; l <= tail; l++) {
        MgLevel& L = this->L[l];
        const size_t n = (size_t)L.w * L.h;
        SR_CUDA_TRY(cudaMalloc(&L.c, n * sizeof(float)));
        SR_CUDA_TRY(cudaMalloc(&L.dx, n * sizeof(float)));
        SR_CUDA_TRY(cudaMalloc(&L.dy, n * sizeof(float)));
        SR_CUDA_TRY(cudaMalloc(&L.mask, n));
        SR_CUDA_TRY(cudaMalloc(&L.x, n * sizeof(float)));
        if (l > 0) {
            SR_CUDA_TRY(cudaMalloc(&L.t, n * sizeof(float)));
            SR_CUDA_TRY(cudaMalloc(&L.b, n * sizeof(float)));
            SR_CUDA_TRY(cudaMalloc(&L.x2, n * sizeof(float)));
        }
    }
    TailArgs layout;
    SR_CUDA_TRY(cudaMalloc(&tail_img, (size_t)tail_layout(*this, layout) * sizeof(float)));
    SR_CUDA_TRY(cudaMalloc(&err, sizeof(int)));
    SR_CUDA_TRY(cudaMemset(err, 0, sizeof(int)));
    for (int l = 0; l < nlevels; l++) L[l].err = err;
    // the same for every world: a world's creation leaves the launches of the others' tails as they were
    SR_CUDA_TRY(cudaFuncSetAttribute(mg_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem));
    SR_CUDA_TRY(cudaFuncSetAttribute(mg_tail_setup_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(TailSetupShared)));
    set_attributes_ns<2>();
    set_attributes_ns<4>();
    set_attributes_ns<6>();
    set_attributes_ns<8>();
}

void Multigrid::destroy() {
    for (int l = 0; l < nlevels; l++) {
        cudaFree(L[l].c);
        cudaFree(L[l].dx);
        cudaFree(L[l].dy);
        cudaFree(L[l].mask);
        cudaFree(L[l].x);
        if (l > 0) {
            cudaFree(L[l].t);
            cudaFree(L[l].b);
            cudaFree(L[l].x2);
        }
        L[l] = MgLevel();
    }
    cudaFree(tail_img);
    tail_img = nullptr;
    cudaFree(err);
    err = nullptr;
    nlevels = 0;
}

bool Multigrid::error(cudaStream_t s) {
    if (!err) return false;
    int v = 0;
    SR_CUDA_TRY(cudaMemcpyAsync(&v, err, sizeof v, cudaMemcpyDeviceToHost, s));
    SR_CUDA_TRY(cudaStreamSynchronize(s));
    if (v) SR_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), s));
    return v != 0;
}

size_t Multigrid::bytes() const {
    size_t s = 0;
    for (int l = 0; l <= tail; l++)
        s += (size_t)L[l].w * L[l].h * (l ? 7 * sizeof(float) + 1 : 4 * sizeof(float) + 1);
    return s;
}

void Multigrid::set_couplings(const double* kx, const double* ky, const uint8_t* gas, cudaStream_t s) {
    mg_couplings0_kernel<<<grid_for((size_t)L[0].w * L[0].h), 256, 0, s>>>(L[0], kx, ky, gas);
    sr_note_launch();
}

void Multigrid::coarsen(cudaStream_t s) {
    for (int l = 1; l <= tail; l++) {
        if (l == 1) {
            mg_aggregate_kernel<<<grid_for((size_t)L[1].w * L[1].h), 256, 0, s>>>(L[0], L[1]);
        } else {
            const dim3 grid(div_up(L[l - 1].w, CO_S), div_up(L[l - 1].h, CO_S));
            mg_coarsen_kernel<<<grid, CO_NT, 0, s>>>(L[l - 1], L[l]);
        }
        sr_note_launch();
    }
    TailArgs T;
    tail_args(*this, T);
    mg_tail_setup_kernel<<<1, TS_NT, sizeof(TailSetupShared), s>>>(T, L[tail], tail == 0, tail_img);
    sr_note_launch();
}

int Multigrid::parts() const {
    if (tail == 0) return 1;
    return (int)rb_grid(L[0], 2 * post);  // the post-smoother's halo is its half-sweeps
}

void Multigrid::apply(const float* r, float* z, double* rz_part, bool overlap, cudaStream_t s) {
    L[0].b = const_cast<float*>(r);
    L[0].x2 = z;
    for (int l = 0; l < tail; l++) smooth(pre, true, L[l], L[l + 1], nullptr, omega, nullptr, overlap && l > 0, s);
    TailArgs T;
    const size_t ts = tail_args(*this, T);
    T.out = tail == 0 ? rz_part : nullptr;
    launch_kernel(overlap && tail > 0, mg_tail_kernel, dim3(1), dim3(TAIL_THREADS), ts, s, T);
    sr_note_launch();
    for (int l = tail - 1; l >= 0; l--)
        smooth(post, false, L[l], L[l + 1], L[l + 1].x2, omega, l == 0 ? rz_part : nullptr, overlap, s);
}

void Multigrid::time_level0(int reps, void* flush, size_t flush_bytes, cudaStream_t s, double* pre_ms,
                            double* post_ms) {
    *pre_ms = *post_ms = 0.0;
    if (tail == 0 || !L[0].b || !L[0].x2 || reps < 1) return;
    cudaEvent_t a, b;
    SR_CUDA_TRY(cudaEventCreate(&a));
    SR_CUDA_TRY(cudaEventCreate(&b));
    for (int which = 0; which < 2; which++) {
        double total = 0.0;
        for (int k = 0; k < reps; k++) {
            SR_CUDA_TRY(cudaMemsetAsync(flush, k & 0xff, flush_bytes, s));
            SR_CUDA_TRY(cudaEventRecord(a, s));
            if (which == 0)
                smooth(pre, true, L[0], L[1], nullptr, omega, nullptr, false, s);
            else
                smooth(post, false, L[0], L[1], L[1].x2, omega, nullptr, false, s);
            SR_CUDA_TRY(cudaEventRecord(b, s));
            SR_CUDA_TRY(cudaEventSynchronize(b));
            float t = 0.0f;
            SR_CUDA_TRY(cudaEventElapsedTime(&t, a, b));
            total += t;
        }
        (which ? *post_ms : *pre_ms) = total / reps;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
}
