// grav.cu — P2, self-gravity by zero-padded FFT convolution (Hockney–Eastwood), FP32 on sm_100a.
//
// φ = K ∗ Σ_src over the w x h world padded to px x py (px the smallest power of two >= 2w, >= 32), then
// g = -∇φ by central differences, the outer ring reading the free-space φ one cell past the world
// (crates/sr-physics/src/reference/grav.rs, reference/fft.rs:238-282). Three FFT passes and a gradient pass:
//   1. rows: two real rows packed as one complex row, a px-point FFT in shared memory, unpacked to the half spectrum
//      kx = 0..px/2, written column-major (each spectrum column kx contiguous in y);
//   2. columns: each kx column zero-padded to py, forward FFT, times the kernel's real-even spectrum K̂ (the quarter
//      table, 1/(px py) folded in), inverse FFT, the world's rows and the two ring rows kept, in place;
//   3. inverse rows: two output rows packed through Hermitian symmetry into one complex inverse FFT, the world's
//      columns and the ring columns kept; up to 1,024 points the CTA's eight rows give φ and g = -∇φ of the six between
//      them right away;
//   4. longer rows: φ and g from the ringed potential, in a kernel of its own.
// The FFT is a Stockham autosort over radix-16 stages and one radix-2/4/8 stage when log2 N is not a multiple of 4 (last
// in a forward transform, first in an inverse one), each thread holding 16 points in registers. A transform's first
// stage takes its points straight from global memory and its last leaves them in natural order in registers, so the
// column pass multiplies by K̂ between the forward's last and the inverse's first stage without leaving registers, and
// shared memory only carries the exchanges between stages: 4 of them for a 4096-point column, where staging every
// stage through shared memory took 16 passes over it. Stage twiddles come from a table built in f64 on the host, laid
// out so that neighbouring threads read neighbouring entries.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <tuple>
#include <vector>

#include "grav.cuh"

namespace {

// Shared-memory FFT buffers hold one float2 of padding after every 16 points: the radix-16 stages' scattered writes
// (stride Ns·16 elements in the first stage) and strided reads then fall on different banks.
__device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }
template <int N>
constexpr int fft_len() {
    return N + N / 16;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// e^{-2πi m/16} for 0 < m < 8, m != 4
__host__ __device__ constexpr float cos16(int m) {
    return m == 1 ? 9.238795325e-01f : m == 2 ? 7.071067812e-01f : m == 3 ? 3.826834324e-01f
         : m == 5 ? -3.826834324e-01f : m == 6 ? -7.071067812e-01f : -9.238795325e-01f;
}
__host__ __device__ constexpr float sin16(int m) {
    return m == 1 || m == 7 ? 3.826834324e-01f : m == 2 || m == 6 ? 7.071067812e-01f : 9.238795325e-01f;
}

// In-register DFT of R (<= 16) points, natural order in and out, by recursive decimation in time. Forward uses
// e^{-2πik/R}; inverse its conjugate (unscaled).
template <int R, bool INV>
struct Dft {
    __device__ __forceinline__ static void run(float2* v) {
        float2 e[R / 2], o[R / 2];
#pragma unroll
        for (int k = 0; k < R / 2; k++) {
            e[k] = v[2 * k];
            o[k] = v[2 * k + 1];
        }
        Dft<R / 2, INV>::run(e);
        Dft<R / 2, INV>::run(o);
#pragma unroll
        for (int k = 0; k < R / 2; k++) {
            const int m = k * (16 / R);
            float2 t;
            if (m == 0) t = o[k];
            else if (m == 4) t = INV ? make_float2(-o[k].y, o[k].x) : make_float2(o[k].y, -o[k].x);
            else t = cmul(o[k], make_float2(cos16(m), INV ? sin16(m) : -sin16(m)));
            v[k] = make_float2(e[k].x + t.x, e[k].y + t.y);
            v[k + R / 2] = make_float2(e[k].x - t.x, e[k].y - t.y);
        }
    }
};
template <bool INV>
struct Dft<1, INV> {
    __device__ __forceinline__ static void run(float2*) {}
};

// The stages of an N-point transform: their radices, the product Ns of the radices before each, and where each one's
// twiddles (R x Ns entries, e^{-2πi r k/(Ns R)} at r Ns + k) begin in the axis's table, the forward's before the
// inverse's. Evaluated by the kernels at compile time and by the host when it builds the table.
struct FftPlan {
    int full, rest, stages;
    __host__ __device__ constexpr explicit FftPlan(int n) : full(0), rest(1), stages(0) {
        int l = 0;
        while ((1 << l) < n) l++;
        full = l / 4;
        rest = 1 << (l % 4);
        stages = full + (rest > 1 ? 1 : 0);
    }
    __host__ __device__ constexpr int radix(bool inv, int s) const {
        return rest == 1 ? 16 : (s == (inv ? 0 : full) ? rest : 16);
    }
    __host__ __device__ constexpr int ns(bool inv, int s) const {
        int p = 1;
        for (int q = 0; q < s; q++) p *= radix(inv, q);
        return p;
    }
    __host__ __device__ constexpr int offset(bool inv, int s) const {
        int o = 0;
        for (int q = 1; q < (inv ? stages : s); q++) o += radix(false, q) * ns(false, q);
        if (inv)
            for (int q = 1; q < s; q++) o += radix(true, q) * ns(true, q);
        return o;
    }
    __host__ __device__ constexpr int entries() const { return offset(true, stages); }
};

template <int N>
constexpr int fft_threads() {
    return N / 16;
}

// A barrier of one transform's threads: a warp's (or less) in lockstep, or `N / 16` threads on barrier `bar`.
template <int N>
__device__ __forceinline__ void fft_sync(int bar) {
    if constexpr (N / 16 <= 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(N / 16) : "memory");
}

// The points of stage S's butterflies of thread t: v[b R + r] = x[j + r N/R], j = t + b N/16.
template <int N, bool INV, int S>
__device__ __forceinline__ void fft_gather(float2 (&v)[16], const float2* buf, int t) {
    constexpr int R = FftPlan(N).radix(INV, S);
#pragma unroll
    for (int b = 0; b < 16 / R; b++)
#pragma unroll
        for (int r = 0; r < R; r++) v[b * R + r] = buf[fpad(t + b * (N / 16) + r * (N / R))];
}

// Stages S and on of an N-point transform by its N/16 threads, `v` gathered for stage S on entry; on return v holds
// the last stage's outputs, X[j + r N/R] at b R + r, in natural order. `buf` is free to be written on entry.
template <int N, bool INV, int S>
__device__ __forceinline__ void fft_stages(float2 (&v)[16], float2* buf, const float2* __restrict__ tw, int t, int bar) {
    constexpr FftPlan P(N);
    constexpr int R = P.radix(INV, S), Ns = P.ns(INV, S);
    if constexpr (S > 0) {
        constexpr int OFF = P.offset(INV, S);
        const float2* w = tw + OFF;
#pragma unroll
        for (int b = 0; b < 16 / R; b++) {
            const int k = (t + b * (N / 16)) & (Ns - 1);
#pragma unroll
            for (int r = 1; r < R; r++) {
                float2 wv = __ldg(w + r * Ns + k);
                if (INV) wv.y = -wv.y;
                v[b * R + r] = cmul(v[b * R + r], wv);
            }
        }
    }
#pragma unroll
    for (int b = 0; b < 16 / R; b++) Dft<R, INV>::run(v + b * R);
    if constexpr (S + 1 < P.stages) {
#pragma unroll
        for (int b = 0; b < 16 / R; b++) {
            const int j = t + b * (N / 16), k = j & (Ns - 1), base = (j - k) * R + k;
#pragma unroll
            for (int r = 0; r < R; r++) buf[fpad(base + r * Ns)] = v[b * R + r];
        }
        fft_sync<N>(bar);
        fft_gather<N, INV, S + 1>(v, buf, t);
        fft_sync<N>(bar);
        fft_stages<N, INV, S + 1>(v, buf, tw, t, bar);
    }
}

// ---- pass 1: two real rows per complex FFT, two FFTs per CTA (four rows: 32-byte runs of the column-major spectrum),
// or as many as fill a warp
template <int N>
constexpr int rows_group() {
    return fft_threads<N>() < 16 ? 32 / fft_threads<N>() : 2;
}

template <int N>
__global__ void __launch_bounds__(rows_group<N>() * fft_threads<N>()) grav_rows_kernel(GravArgs A) {
    extern __shared__ float2 sm[];
    constexpr int T = fft_threads<N>(), G = rows_group<N>();
    const int f = threadIdx.x / T, t = threadIdx.x % T;
    const int w = A.w, h = A.h, y0 = blockIdx.x * 2 * G;
    const float sv = A.sigma_vac;
    float2* buf = sm + f * fft_len<N>();
    pdl_launch();
    {
        const int ya = y0 + 2 * f;
        const float* ra = A.src + (size_t)ya * w;
        float2 v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int x = t + r * T;
            float a = 0.0f, b = 0.0f;
            if (x < w) {
                if (ya < h) a = ra[x];
                if (ya + 1 < h) b = ra[w + x];
            }
            v[r] = make_float2(a >= sv ? a : 0.0f, b >= sv ? b : 0.0f);
        }
        fft_stages<N, false, 0>(v, buf, A.tw_x, t, 1 + f);
        constexpr int R = FftPlan(N).radix(false, FftPlan(N).stages - 1);
#pragma unroll
        for (int b = 0; b < 16 / R; b++)
#pragma unroll
            for (int r = 0; r < R; r++) buf[fpad(t + b * T + r * (N / R))] = v[b * R + r];
    }
    __syncthreads();
    // unpack: X_a[k] = (Z[k] + conj Z[N-k]) / 2, X_b[k] = (Z[k] - conj Z[N-k]) / 2i, k = 0..N/2; column-major out, the
    // CTA's rows of a column by neighbouring threads
    const size_t ld = A.ld;
    for (int e = threadIdx.x; e < 2 * G * (N / 2 + 1); e += G * T) {
        const int q = e % (2 * G), k = e / (2 * G);
        if (y0 + q >= h) continue;
        const float2* bq = sm + (q >> 1) * fft_len<N>();
        const float2 z = bq[fpad(k)], zc = bq[fpad((N - k) & (N - 1))];
        A.spec[(size_t)k * ld + y0 + q] = q & 1 ? make_float2(0.5f * (z.y + zc.y), 0.5f * (zc.x - z.x))
                                                : make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
    }
}

// ---- pass 2: spectrum columns, one per N/16 threads: forward, × K̂, inverse, rows -1..h kept
template <int N>
constexpr int column_group() {
    return fft_threads<N>() < 32 ? 32 / fft_threads<N>() : 1;
}

template <int N>
__global__ void __launch_bounds__(column_group<N>() * fft_threads<N>(), N == 4096 ? 3 : 1) grav_columns_kernel(GravArgs A) {
    extern __shared__ float2 sm[];
    constexpr int T = fft_threads<N>(), G = column_group<N>();
    constexpr FftPlan P(N);
    constexpr int R = P.radix(true, 0);
    const int f = threadIdx.x / T, t = threadIdx.x % T;
    const int kx = blockIdx.x * G + f;
    const bool on = G == 1 || kx <= A.px / 2;
    const int h = A.h;
    float2* buf = sm + f * fft_len<N>();
    float2* col = A.spec + (size_t)(on ? kx : 0) * A.ld;
    float2 v[16];
    pdl_launch();
    pdl_wait();
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int y = t + r * T;
        v[r] = on && y < h ? col[y] : make_float2(0.0f, 0.0f);
    }
    fft_stages<N, false, 0>(v, buf, A.tw_y, t, 0);
    const float* kq = A.khat + (size_t)(on ? kx : 0) * (N / 2 + 1);
#pragma unroll
    for (int b = 0; b < 16 / R; b++)
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int ky = t + b * T + r * (N / R);
            const float k = kq[ky <= N / 2 ? ky : N - ky];
            v[b * R + r].x *= k;
            v[b * R + r].y *= k;
        }
    fft_stages<N, true, 0>(v, buf, A.tw_y, t, 0);
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int row = (t + r * T + 1) & (N - 1);  // the world's row y at y + 1, row -1 (the last point) at 0
        if (on && row < h + 2) col[row] = v[r];
    }
}

// ---- pass 3: two output rows per complex inverse FFT. FUSED (rows of up to 1,024 points): a CTA's 2G rows overlap the
// next CTA's by two, and it writes φ and g of the rows between its first and last; the third more transforms cost less
// than the ring's round trip and a launch while the launch is latency (256²: 5.9 + 2.0 us and a launch -> 4.4), and more
// once it is work (2,048 points, 1024²: 7.8 + 3.7 -> 14.6, so those keep the two kernels). Not FUSED: columns -1..w kept
// into φ_ring.
template <int N>
constexpr bool inverse_fused() { return N <= kRingless; }
template <int N>
constexpr int inverse_group() {
    return !inverse_fused<N>() ? 2 : (fft_threads<N>() < 8 ? 32 / fft_threads<N>() : 4);
}

// VEC: φ and g begin on 16 bytes and are stored so; sr_gravity_solve_static's may not, and are then stored float by float
// (as an instance of its own: the choice in the store cost 136 x 104 worlds 0.2 of 10.6 us).
template <int N, bool VEC>
__global__ void __launch_bounds__(inverse_group<N>() * fft_threads<N>()) grav_rows_inverse_kernel(GravArgs A) {
    extern __shared__ float2 sm[];
    constexpr int T = fft_threads<N>(), G = inverse_group<N>(), NT = G * T;
    constexpr bool FUSED = inverse_fused<N>();
    const int rows = A.h + 2, r0 = blockIdx.x * (FUSED ? 2 * G - 2 : 2 * G);  // rows is even (the world's height is)
    const size_t ld = A.ld;
    auto place = [&](int f, int k, const float4& x) {
        // Z[k] = X_a[k] + i X_b[k]; Z[N-k] = conj X_a[k] + i conj X_b[k]
        float2* buf = sm + f * fft_len<N>();
        buf[fpad(k)] = make_float2(x.x - x.w, x.y + x.z);
        if (k > 0 && k < N / 2) buf[fpad(N - k)] = make_float2(x.x + x.w, x.z - x.y);
    };
    auto load = [&](int f, int k) {
        const int ra = r0 + 2 * f;
        return ra < rows ? *reinterpret_cast<const float4*>(A.spec + (size_t)k * ld + ra) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    pdl_launch();
    pdl_wait();
    if constexpr (!FUSED) {  // many CTAs per SM hide each other's loads
        for (int e = threadIdx.x; e < G * (N / 2 + 1); e += NT) place(e % G, e / G, load(e % G, e / G));
    } else {
        float4 x[8];  // X_a[k], X_b[k] of k = 0..N/2-1, all loads in flight together
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = load((threadIdx.x + u * NT) % G, (threadIdx.x + u * NT) / G);
#pragma unroll
        for (int u = 0; u < 8; u++) place((threadIdx.x + u * NT) % G, (threadIdx.x + u * NT) / G, x[u]);
        if (threadIdx.x < G) place(threadIdx.x, N / 2, load(threadIdx.x, N / 2));
    }
    __syncthreads();
    const int f = threadIdx.x / T, t = threadIdx.x % T;
    float2* buf = sm + f * fft_len<N>();
    float2 v[16];
    fft_gather<N, true, 0>(v, buf, t);
    fft_sync<N>(1 + f);
    fft_stages<N, true, 0>(v, buf, A.tw_x, t, 1 + f);
    const int w = A.w, rw = w + 2;
    if constexpr (!FUSED) {
        const int ra = r0 + 2 * f;
        if (ra >= rows) return;
        float* ring = A.phi_ring + (size_t)ra * A.rp + kRingPad;
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int c = (t + r * T + 1) & (N - 1);
            if (c < rw) {
                ring[c] = v[r].x;
                ring[A.rp + c] = v[r].y;
            }
        }
    } else {
        // the transform's two ring rows over its own buffer (free since its last gather): N/2 + 2 columns at most each
        constexpr int RP = fft_len<N>();
        float* own = reinterpret_cast<float*>(buf);
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int c = (t + r * T + 1) & (N - 1);
            if (c < rw) {
                own[c] = v[r].x;
                own[RP + c] = v[r].y;
            }
        }
        __syncthreads();
        const float* ring = reinterpret_cast<const float*>(sm);  // ring row r0 + i at i RP
        const int w4 = w / 4;
        for (int e = threadIdx.x; e < (2 * G - 2) * w4; e += NT) {
            const int i = e / w4, x = 4 * (e - i * w4), y = r0 + i;  // the world's row y is ring row y + 1
            if (y >= A.h) break;
            const float* c = ring + (i + 1) * RP + x;  // columns x - 1 on
            float4 p, gx, gy;
            p = make_float4(c[1], c[2], c[3], c[4]);
            gx = make_float4(-(c[2] - c[0]) / 2.0f, -(c[3] - c[1]) / 2.0f, -(c[4] - c[2]) / 2.0f, -(c[5] - c[3]) / 2.0f);
            const float *u = c - RP, *d = c + RP;
            gy = make_float4(-(d[1] - u[1]) / 2.0f, -(d[2] - u[2]) / 2.0f, -(d[3] - u[3]) / 2.0f, -(d[4] - u[4]) / 2.0f);
            const size_t o = (size_t)y * w + x;
            auto store = [&](float* a, const float4& v) {
                if constexpr (VEC) {
                    *reinterpret_cast<float4*>(a + o) = v;
                } else {
                    a[o] = v.x;
                    a[o + 1] = v.y;
                    a[o + 2] = v.z;
                    a[o + 3] = v.w;
                }
            };
            store(A.phi, p);
            store(A.gx, gx);
            store(A.gy, gy);
        }
    }
}

// ---- pass 4 (rows past 1,024 points): φ and g = -∇φ by central differences over the ringed potential (grav.rs:55-70),
// four cells a thread (the world's width is a multiple of 8 and the ring's rows are padded so that its cells lie on
// 16-byte boundaries; a context's planes, the only ones that come here, are allocations of their own)
__global__ void grav_gradient_kernel(GravArgs A) {
    const int w = A.w, h = A.h, rp = A.rp;
    const int n4 = w * h / 4;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += gridDim.x * blockDim.x) {
        int x, y;
        split_index((size_t)q * 4, w, x, y);
        const float* r1 = A.phi_ring + (size_t)(y + 1) * rp + kRingPad + 1 + x;
        const float4 c = *reinterpret_cast<const float4*>(r1);
        const float l = r1[-1], r = r1[4];
        const float4 u = *reinterpret_cast<const float4*>(r1 - rp), d = *reinterpret_cast<const float4*>(r1 + rp);
        reinterpret_cast<float4*>(A.gx)[q] = make_float4(-(c.y - l) / 2.0f, -(c.z - c.x) / 2.0f, -(c.w - c.y) / 2.0f,
                                                         -(r - c.z) / 2.0f);
        reinterpret_cast<float4*>(A.gy)[q] = make_float4(-(d.x - u.x) / 2.0f, -(d.y - u.y) / 2.0f, -(d.z - u.z) / 2.0f,
                                                         -(d.w - u.w) / 2.0f);
        reinterpret_cast<float4*>(A.phi)[q] = c;
    }
}

// The opt-in past 48 KB of shared memory (per device, so with every launch that needs it: the longest transforms).
template <class K>
void allow_smem(K kernel, size_t smem) {
    if (smem > 48 * 1024)
        SR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
}

// Short transforms (the inverse takes the gradient too) overlap: their kernels are a fraction of a wave, and a launch is
// as long as they are (256², solve and read: 18.2 -> 12.3 us). Past that an early CTA takes a slot on whichever SM is
// free first, the next kernel's load is uneven, and a 1024² disk's step got 1.3 % slower.
template <int N>
void launch_rows(const GravArgs& A, cudaStream_t s) {
    constexpr size_t smem = rows_group<N>() * fft_len<N>() * sizeof(float2);
    allow_smem(grav_rows_kernel<N>, smem);
    grav_rows_kernel<N><<<div_up(A.h, 2 * rows_group<N>()), rows_group<N>() * fft_threads<N>(), smem, s>>>(A);
    sr_note_launch();
}

template <int N>
void launch_columns(const GravArgs& A, cudaStream_t s) {
    constexpr size_t smem = column_group<N>() * fft_len<N>() * sizeof(float2);
    allow_smem(grav_columns_kernel<N>, smem);
    launch_kernel(N <= kRingless, grav_columns_kernel<N>, dim3(div_up(A.px / 2 + 1, column_group<N>())),
                  dim3(column_group<N>() * fft_threads<N>()), smem, s, A);
    sr_note_launch();
}

template <int N>
void launch_rows_inverse(const GravArgs& A, cudaStream_t s) {
    constexpr int G = inverse_group<N>();
    constexpr size_t smem = G * fft_len<N>() * sizeof(float2);
    const unsigned grid = inverse_fused<N>() ? div_up(A.h, 2 * G - 2) : div_up(A.h + 2, 2 * G);
    auto go = [&](auto kernel) {
        allow_smem(kernel, smem);
        launch_kernel(N <= kRingless, kernel, dim3(grid), dim3(G * fft_threads<N>()), smem, s, A);
    };
    if constexpr (inverse_fused<N>()) {
        if ((((uintptr_t)A.phi | (uintptr_t)A.gx | (uintptr_t)A.gy) & 15) != 0) go(grav_rows_inverse_kernel<N, false>);
        else go(grav_rows_inverse_kernel<N, true>);
    } else {
        go(grav_rows_inverse_kernel<N, true>);
    }
    sr_note_launch();
    if (inverse_fused<N>()) return;
    const int nb = std::min<int>(div_up((unsigned)((size_t)A.w * A.h / 4), 256u), 148 * 8);
    grav_gradient_kernel<<<nb, 256, 0, s>>>(A);
    sr_note_launch();
}

#define SR_FFT_SIZES(X) X(32) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096) X(8192)

void dispatch_rows(int n, const GravArgs& A, cudaStream_t s) {
    switch (n) {
#define X(N) case N: launch_rows<N>(A, s); break;
        SR_FFT_SIZES(X)
#undef X
    }
}
void dispatch_columns(int n, const GravArgs& A, cudaStream_t s) {
    switch (n) {
#define X(N) case N: launch_columns<N>(A, s); break;
        SR_FFT_SIZES(X)
#undef X
    }
}
void dispatch_rows_inverse(int n, const GravArgs& A, cudaStream_t s) {
    switch (n) {
#define X(N) case N: launch_rows_inverse<N>(A, s); break;
        SR_FFT_SIZES(X)
#undef X
    }
}

// ------------------------------------------------------------------------------------------------ host: K̂ in f64
// A radix-2 complex FFT in f64 (forward, unnormalised), for the kernel's spectrum built once per padded size.
void fft_f64(std::vector<double>& re, std::vector<double>& im, size_t off, size_t stride, int n,
             const std::vector<double>& c, const std::vector<double>& s) {
    int bits = 0;
    while ((1 << bits) < n) bits++;
    for (int i = 0; i < n; i++) {
        int j = 0;
        for (int b = 0; b < bits; b++)
            if (i & (1 << b)) j |= 1 << (bits - 1 - b);
        if (i < j) {
            std::swap(re[off + i * stride], re[off + j * stride]);
            std::swap(im[off + i * stride], im[off + j * stride]);
        }
    }
    for (int half = 1; half < n; half *= 2) {
        int step = n / (2 * half);
        for (int start = 0; start < n; start += 2 * half)
            for (int k = 0; k < half; k++) {
                double wr = c[k * step], wi = s[k * step];
                size_t a = off + (start + k) * stride, b = off + (start + k + half) * stride;
                double br = re[b] * wr - im[b] * wi, bi = re[b] * wi + im[b] * wr;
                double ar = re[a], ai = im[a];
                re[a] = ar + br; im[a] = ai + bi;
                re[b] = ar - br; im[b] = ai - bi;
            }
    }
}

void parallel_for(int n, const std::function<void(int, int)>& body) {
    int nt = (int)std::thread::hardware_concurrency();
    if (nt < 1) nt = 1;
    if (nt > 32) nt = 32;
    std::vector<std::thread> th;
    for (int t = 0; t < nt; t++) {
        int a = (int)((long long)n * t / nt), b = (int)((long long)n * (t + 1) / nt);
        th.emplace_back([=, &body] { body(a, b); });
    }
    for (auto& x : th) x.join();
}

// K(dx, dy): the reference's exact self cell (grav.rs:25-34) or the softened kernel.
double kernel_value(int kind, double G, double eps, long dx, long dy) {
    double r2 = (double)(dx * dx + dy * dy);
    if (kind == SR_KERNEL_SOFTENED) return -G / sqrt(r2 + eps * eps);
    if (dx == 0 && dy == 0) return -G * 3.525494348078172;
    return -G / sqrt(r2);
}

std::mutex g_khat_mutex;
std::map<std::tuple<int, int, int, double, double>, std::vector<float>> g_khat_cache;

// The quarter (px/2+1) x (py/2+1) of K's real-even spectrum, in f64, scaled by 1/(px py) and stored f32
// (crates/sr-engine/src/step/grav.rs:76-130 builds the same quarter).
const std::vector<float>& khat_quarter(int px, int py, int kind, double G, double eps) {
    std::lock_guard<std::mutex> lock(g_khat_mutex);
    auto key = std::make_tuple(px, py, kind, G, eps);
    auto it = g_khat_cache.find(key);
    if (it != g_khat_cache.end()) return it->second;
    std::vector<double> re((size_t)px * py), im((size_t)px * py, 0.0);
    for (int j = 0; j < py; j++)
        for (int i = 0; i < px; i++) {
            long dx = i < px / 2 ? i : i - px, dy = j < py / 2 ? j : j - py;
            re[(size_t)j * px + i] = kernel_value(kind, G, eps, dx, dy);
        }
    auto twiddles = [](int n, std::vector<double>& c, std::vector<double>& s) {
        c.resize(n / 2 > 0 ? n / 2 : 1);
        s.resize(n / 2 > 0 ? n / 2 : 1);
        for (int k = 0; k < n / 2; k++) {
            double a = -2.0 * M_PI * (double)k / (double)n;
            c[k] = cos(a);
            s[k] = sin(a);
        }
    };
    std::vector<double> cx, sx, cy, sy;
    twiddles(px, cx, sx);
    twiddles(py, cy, sy);
    parallel_for(py, [&](int a, int b) {
        for (int j = a; j < b; j++) fft_f64(re, im, (size_t)j * px, 1, px, cx, sx);
    });
    parallel_for(px / 2 + 1, [&](int a, int b) {
        for (int i = a; i < b; i++) fft_f64(re, im, (size_t)i, (size_t)px, py, cy, sy);
    });
    std::vector<float> q((size_t)(px / 2 + 1) * (py / 2 + 1));
    const double scale = 1.0 / ((double)px * (double)py);
    for (int i = 0; i <= px / 2; i++)
        for (int j = 0; j <= py / 2; j++) q[(size_t)i * (py / 2 + 1) + j] = (float)(re[(size_t)j * px + i] * scale);
    return g_khat_cache.emplace(key, std::move(q)).first->second;
}

}  // namespace

int grav_padded_size(int len) {
    // reference/fft.rs:92-101 with the cap lifted to 8192
    if (len <= 0) return 0;
    int n = 1;
    while (n < 2 * len) n <<= 1;
    if (n < 32) n = 32;
    return n > 8192 ? 0 : n;
}

size_t grav_twiddle_count(int n) { return (size_t)FftPlan(n).entries(); }

void grav_twiddles(int n, float2* out) {
    const FftPlan P(n);
    for (int inv = 0; inv < 2; inv++)
        for (int s = 1; s < P.stages; s++) {
            const int R = P.radix(inv != 0, s), Ns = P.ns(inv != 0, s);
            for (int r = 0; r < R; r++)
                for (int k = 0; k < Ns; k++) {
                    const double a = -2.0 * M_PI * (double)r * (double)k / ((double)Ns * R);
                    out[P.offset(inv != 0, s) + r * Ns + k] = make_float2((float)cos(a), (float)sin(a));
                }
        }
}

void GravPlan::create(int w_, int h_, int kernel, double G, double eps, float sigma_vac_) {
    w = w_;
    h = h_;
    px = grav_padded_size(w);
    py = grav_padded_size(h);
    SR_REQUIRE(px && py, "a world axis pads past the FFT's 8192 points");
    sigma_vac = sigma_vac_;
    ld = grav_column_stride(h);
    SR_CUDA_TRY(cudaMalloc(&spec, sizeof(float2) * (size_t)(px / 2 + 1) * ld));
    if (px > kRingless) SR_CUDA_TRY(cudaMalloc(&phi_ring, sizeof(float) * (size_t)grav_ring_stride(w) * (h + 2)));
    const std::vector<float>& q = khat_quarter(px, py, kernel, G, eps);
    SR_CUDA_TRY(cudaMalloc(&khat, sizeof(float) * q.size()));
    SR_CUDA_TRY(cudaMemcpy(khat, q.data(), sizeof(float) * q.size(), cudaMemcpyHostToDevice));
    std::vector<float2> tx(grav_twiddle_count(px)), ty(grav_twiddle_count(py));
    grav_twiddles(px, tx.data());
    grav_twiddles(py, ty.data());
    SR_CUDA_TRY(cudaMalloc(&tw_x, sizeof(float2) * tx.size()));
    SR_CUDA_TRY(cudaMalloc(&tw_y, sizeof(float2) * ty.size()));
    SR_CUDA_TRY(cudaMemcpy(tw_x, tx.data(), sizeof(float2) * tx.size(), cudaMemcpyHostToDevice));
    SR_CUDA_TRY(cudaMemcpy(tw_y, ty.data(), sizeof(float2) * ty.size(), cudaMemcpyHostToDevice));
}

void GravPlan::destroy() {
    cudaFree(spec);
    cudaFree(phi_ring);
    cudaFree(khat);
    cudaFree(tw_x);
    cudaFree(tw_y);
    spec = nullptr;
    phi_ring = nullptr;
    khat = nullptr;
    tw_x = tw_y = nullptr;
}

size_t GravPlan::bytes() const {
    return sizeof(float2) * (size_t)(px / 2 + 1) * ld +
           (px > kRingless ? sizeof(float) * (size_t)grav_ring_stride(w) * (h + 2) : 0) +
           sizeof(float) * (size_t)(px / 2 + 1) * (py / 2 + 1) +
           sizeof(float2) * (grav_twiddle_count(px) + grav_twiddle_count(py));
}

void GravPlan::solve(const float* src, float* phi, float* gx, float* gy, cudaStream_t s) const {
    GravArgs A;
    A.w = w;
    A.h = h;
    A.px = px;
    A.py = py;
    A.ld = ld;
    A.rp = grav_ring_stride(w);
    A.sigma_vac = sigma_vac;
    A.src = src;
    A.spec = spec;
    A.khat = khat;
    A.tw_x = tw_x;
    A.tw_y = tw_y;
    A.phi_ring = phi_ring;
    A.phi = phi;
    A.gx = gx;
    A.gy = gy;
    dispatch_rows(px, A, s);
    dispatch_columns(py, A, s);
    dispatch_rows_inverse(px, A, s);
}
