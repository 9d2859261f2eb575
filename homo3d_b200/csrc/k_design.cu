// k_design.cu -- density input, OC update, sensitivity filter, symmetrisation.
//
// Reference behaviour restated (homo3d):
//   update_rho_kernel (grid.cu:4025-4064): pitched lexicographic density in.
//   OCOptimizer::update (OCOptimizer.cu:12-67): rho_new = clamp(rho *
//     max(-s/g, 0.01)^damp, rho +- step, [rho_min, 1]), 20 bisection steps on g
//     over [0, max|s|] until |vol - target| <= 1e-4.  Here the bisection state
//     lives on the device, so the update needs no host round trip per step.
//   OCOptimizer::filterSens (OCOptimizer.cu:76-152): s~_e = sum w rho s /
//     (sum w * rho_e), linear cone weight 1 - |d|/r on a (2*int(r+0.5)+1)^3
//     window, normalised by the full-window weight sum, optionally periodic.
//   symetrize_tensor_kernel (TensorExpression.cuh:72-): orbit averages with the
//     reference's FP32 summation order, so results are bit-identical.
#include "h3d_internal.cuh"

namespace h3d {

__global__ void k_density_in(int n0, int n1, int n2, const float *__restrict__ src, int pitch, float *dst) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long ne = (long long)n0 * n1 * n2;
    if (e >= ne) return;
    const int x = (int)(e % n0);
    const long long t = e / n0;
    const int y = (int)(t % n1), z = (int)(t / n1);
    dst[e] = src[x + ((long long)y + (long long)z * n1) * pitch];
}

// SIMP penalisation rho_phys = rho^p and its backward grad *= p rho^(p-1)
// (the reference builds these as the expression rho.pow(3), TensorExpression.h:517-531, 781-)
__global__ void k_penalize(long long n, const float *__restrict__ rho, float *out, float p, int backward) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float r = rho[i];
    if (backward) out[i] *= p * powf(r, p - 1.f);
    else out[i] = powf(r, p);
}

void launch_penalize(long long n, const float *rho, float *out, float p, int backward, cudaStream_t s) {
    k_penalize<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, rho, out, p, backward);
}

void launch_density_in(const int n[3], const float *src, int pitch, float *dst, cudaStream_t s) {
    const long long ne = (long long)n[0] * n[1] * n[2];
    k_density_in<<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(n[0], n[1], n[2], src, pitch, dst);
}

// ---- OC ----------------------------------------------------------------------
// scratch layout: [0] lo, [1] hi, [2] done, [3] arrival counter, [4..] partial sums.
// The CTA of a pass that arrives last combines the partials (in a fixed order) and
// takes the decision, so a bisection step is one launch; a second launch whose one
// thread added the 1184 partials took 15-18 us a step.
constexpr int OC_BS = 256;
constexpr int OC_NB = 1184;  // 8 blocks per SM on 148 SMs

// whether this CTA is the last of its launch to arrive (the others' writes are then
// visible); every thread must call it, and the counter is left at zero
__device__ __forceinline__ bool last_cta(double *st) {
    __shared__ bool last;
    unsigned *count = reinterpret_cast<unsigned *>(st + 3);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(count, 1u) == gridDim.x - 1;
        if (last) *count = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// the sum of the launch's partials st[4 ..], in thread 0 of an OC_BS-thread CTA
__device__ __forceinline__ double sum_partials(const double *st, int nb) {
    __shared__ double sm[OC_BS / 32];
    double s = 0;
    for (int b = threadIdx.x; b < nb; b += OC_BS) s += __ldcg(&st[4 + b]);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < OC_BS / 32; ++w) s += sm[w];
    return s;
}

__global__ void __launch_bounds__(OC_BS) k_oc_maxabs(const float *__restrict__ s, long long n, double *partial) {
    double m = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        m = fmax(m, (double)fabsf(s[i]));
    __shared__ double sm[32];
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) partial[4 + blockIdx.x] = m;
    }
    if (!last_cta(partial)) return;
    m = 0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) m = fmax(m, __ldcg(&partial[4 + b]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < OC_BS / 32; ++w) m = fmax(m, sm[w]);
        partial[0] = 0.0;
        partial[1] = (double)(float)m;
        partial[2] = 0.0;
    }
}

__global__ void __launch_bounds__(OC_BS) k_oc_step(const float *__restrict__ sens, const float *__restrict__ rho,
                                                   float *rho_new, long long n, float vol, float minrho, float step, float damp,
                                                   double *st) {
    if (st[2] != 0.0) return;  // converged in an earlier step: keep its densities
    const float g = ((float)st[1] + (float)st[0]) / 2;
    double s = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float r = rho[i];
        float B = -sens[i] / g;
        if (B < 0) B = 0.01f;
        float v = powf(B, damp) * r;
        if (v - r < -step) v = r - step;
        if (v - r > step) v = r + step;
        if (v < minrho) v = minrho;
        if (v > 1) v = 1;
        rho_new[i] = v;
        s += v;
    }
    double ss[1] = {s};
    block_reduce<1>(ss, st + 4, blockIdx.x);
    if (!last_cta(st)) return;
    s = sum_partials(st, gridDim.x);
    if (threadIdx.x == 0) {
        const float cur = (float)(s / (double)n);
        if (cur < vol - 0.0001f) st[1] = g;
        else if (cur > vol + 0.0001f) st[0] = g;
        else st[2] = 1.0;
    }
}

void launch_oc(const float *sens, float *rho, float *rho_new, long long n, float vol, float minrho, float step,
               float damp, double *scratch, cudaStream_t s) {
    cudaMemsetAsync(scratch, 0, 4 * sizeof(double), s);
    k_oc_maxabs<<<OC_NB, OC_BS, 0, s>>>(sens, n, scratch);
    for (int it = 0; it < 20; ++it)
        k_oc_step<<<OC_NB, OC_BS, 0, s>>>(sens, rho, rho_new, n, vol, minrho, step, damp, scratch);
    cudaMemcpyAsync(rho, rho_new, sizeof(float) * n, cudaMemcpyDeviceToDevice, s);
}

// ---- window sums: sensitivity filter and radial convolution -----------------------
// Both sum a window of (2 hw + 1)^3 cells around a cell, the weight a function of
// |o|^2 alone.  The weights are formed once per call (k_window_table, one per |o|^2, and
// their sum over the window in the order of the taps) and kept in shared memory; a cell
// whose window is inside the grid takes its norm from the table.  Rows of taps are
// contiguous, so a tap is a load (mostly L1), a weight and an FMA.  Bound by issue.
// Forming each weight (a division and a square root), the wrapped index and three
// integer divisions per tap took 1.54 ms per pass of 343 taps on 112^3 and 1.29 ms for
// the 125-tap filter on 128^3.
constexpr int WIN_X = 32, WIN_Y = 8;
constexpr int WIN_SMEM = 12000;  // largest table kept in shared memory (48 KB); wider windows read it from L1
enum WindowMode {
    WIN_CONV,    // out = sum w in / sum w
    WIN_DIV,     // out = in / sum w
    WIN_ADJ,     // out = sum w in, at p - o
    WIN_FILTER   // out = sum w in rho / (sum w * rho)
};

__device__ __forceinline__ float spline4_weight(int d2, float r) {
    const float q = (float)d2 / (r * r);
    const float rq = sqrtf(q);
    return q < 1.f ? 1.f - 6.f * q + 8.f * q * rq - 3.f * q * q : 0.f;
}

// tab[d2], d2 = 0 .. 3 hw^2: the spline weight, or (cone) the linear one over wtot;
// tab[3 hw^2 + 1]: their sum over the window
__global__ void __launch_bounds__(1024) k_window_table(float *tab, int hw, float r, float wtot, int cone) {
    extern __shared__ float sw[];
    const int m = 3 * hw * hw + 1;
    float *t = m + 1 <= WIN_SMEM ? sw : tab;
    for (int d2 = threadIdx.x; d2 < m; d2 += blockDim.x) {
        const float r2 = (float)d2 / (r * r);
        tab[d2] = t[d2] = cone ? (r2 < 1.f ? 1.f - sqrtf(r2) : 0.f) / wtot : spline4_weight(d2, r);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    float s = 0.f;
    for (int oz = -hw; oz <= hw; ++oz)
        for (int oy = -hw; oy <= hw; ++oy)
            for (int ox = -hw; ox <= hw; ++ox) s += t[ox * ox + oy * oy + oz * oz];
    tab[m] = s;
}

template <int MODE>
__global__ void __launch_bounds__(WIN_X *WIN_Y) k_window(int n0, int n1, int n2, int pitch, const float *__restrict__ in,
                                                        const float *__restrict__ rho, float *out,
                                                        const float *__restrict__ tab, int hw, int periodic) {
    extern __shared__ float sw[];
    const int m = 3 * hw * hw + 2;
    const float *tw = tab;
    if (m <= WIN_SMEM) {
        for (int i = threadIdx.y * WIN_X + threadIdx.x; i < m; i += WIN_X * WIN_Y) sw[i] = __ldg(tab + i);
        __syncthreads();
        tw = sw;
    }
    const int x = blockIdx.x * WIN_X + threadIdx.x;
    if (x >= n0) return;
    constexpr int sg = MODE == WIN_ADJ ? -1 : 1;
    const bool inx = x >= hw && x + hw < n0;
    for (int y = blockIdx.y * WIN_Y + threadIdx.y; y < n1; y += gridDim.y * WIN_Y)
        for (int z = blockIdx.z; z < n2; z += gridDim.z) {
            const long long me = x + ((long long)y + (long long)z * n1) * pitch;
            // every tap in the grid: the norm is the table's
            const bool whole = periodic ? hw <= n0 && hw <= n1 && hw <= n2 : (inx && y >= hw && y + hw < n1 && z >= hw && z + hw < n2);
            float sum = 0.f, ws = 0.f;
            if (MODE != WIN_DIV || !whole) {
                for (int oz = -hw; oz <= hw; ++oz) {
                    int pz = z + sg * oz;
                    if (pz < 0 || pz >= n2) {
                        if (!periodic) continue;
                        pz = (pz + n2) % n2;
                        if (pz < 0) continue;  // a window wider than the grid
                    }
                    for (int oy = -hw; oy <= hw; ++oy) {
                        int py = y + sg * oy;
                        if (py < 0 || py >= n1) {
                            if (!periodic) continue;
                            py = (py + n1) % n1;
                            if (py < 0) continue;
                        }
                        const long long ro = ((long long)py + (long long)pz * n1) * pitch;
                        const float *row = in + ro, *rrow = MODE == WIN_FILTER ? rho + ro : nullptr;
                        const float *wr = tw + (oy * oy + oz * oz);
                        if (inx) {
#pragma unroll 4
                            for (int ox = -hw; ox <= hw; ++ox) {
                                const float w = wr[ox * ox];
                                const int px = x + sg * ox;
                                if (MODE == WIN_FILTER) sum += __ldg(row + px) * __ldg(rrow + px) * w;
                                else if (MODE != WIN_DIV) sum += w * __ldg(row + px);
                                ws += w;
                            }
                        } else {
                            for (int ox = -hw; ox <= hw; ++ox) {
                                int px = x + sg * ox;
                                if (px < 0 || px >= n0) {
                                    if (!periodic) continue;
                                    px = (px + n0) % n0;
                                    if (px < 0) continue;
                                }
                                const float w = wr[ox * ox];
                                if (MODE == WIN_FILTER) sum += __ldg(row + px) * __ldg(rrow + px) * w;
                                else if (MODE != WIN_DIV) sum += w * __ldg(row + px);
                                ws += w;
                            }
                        }
                    }
                }
            }
            if (whole) ws = tw[m - 1];
            if (MODE == WIN_CONV) out[me] = sum / ws;
            else if (MODE == WIN_DIV) out[me] = __ldg(in + me) / ws;
            else if (MODE == WIN_ADJ) out[me] = sum;
            else out[me] = sum / (ws * __ldg(rho + me));
        }
}

static size_t window_smem(int hw) { return 3 * hw * hw + 2 <= WIN_SMEM ? sizeof(float) * (3 * hw * hw + 2) : 0; }

// The same sums for windows up to 9 cells wide that fit the grid: WIN_Z cells of a
// column per thread, so a value is loaded once for the WIN_Z windows that hold it and a
// weight serves them all: (WIN_Z + 2 HW + HW + 1) loads per column of taps and WIN_Z
// cells where one cell per thread takes 2 (2 HW + 1) for each.  The latter was bound by
// the load/store pipe: 0.70 ms per pass of 343 taps on 112^3, 0.10 ms here.
constexpr int WIN_Z = 4, WIN_HWMAX = 4;
template <int MODE, int HW>
__global__ void __launch_bounds__(WIN_X *WIN_Y) k_window_col(int n0, int n1, int n2, int pitch,
                                                            const float *__restrict__ in, const float *__restrict__ rho,
                                                            float *out, const float *__restrict__ tab, int periodic) {
    constexpr int T = WIN_Z + 2 * HW;
    __shared__ float tw[3 * HW * HW + 2];
    for (int i = threadIdx.y * WIN_X + threadIdx.x; i < 3 * HW * HW + 2; i += WIN_X * WIN_Y) tw[i] = __ldg(tab + i);
    __syncthreads();
    const int x = blockIdx.x * WIN_X + threadIdx.x, y = blockIdx.y * WIN_Y + threadIdx.y, z0 = blockIdx.z * WIN_Z;
    if (x >= n0 || y >= n1) return;
    const long long plane = (long long)n1 * pitch;
    long long zo[T];    // plane offsets of the column's values
    unsigned zin = 0;   // those that count
#pragma unroll
    for (int t = 0; t < T; ++t) {
        int pz = z0 + t - HW;
        bool ok = pz >= 0 && pz < n2;
        if (!ok && periodic) {
            pz = pz < 0 ? pz + n2 : pz - n2;
            ok = pz < n2;  // past the last cell of a partial column: unused
        }
        zo[t] = ok ? plane * pz : 0;
        zin |= (unsigned)ok << t;
    }
    const bool inxy = periodic || (x >= HW && x + HW < n0 && y >= HW && y + HW < n1);
    float sum[WIN_Z], ws[WIN_Z];
#pragma unroll
    for (int k = 0; k < WIN_Z; ++k) sum[k] = ws[k] = 0.f;
    for (int oy = -HW; oy <= HW; ++oy) {
        int py = y + oy;
        if (py < 0 || py >= n1) {
            if (!periodic) continue;
            py = py < 0 ? py + n1 : py - n1;
        }
        for (int ox = -HW; ox <= HW; ++ox) {
            int px = x + ox;
            if (px < 0 || px >= n0) {
                if (!periodic) continue;
                px = px < 0 ? px + n0 : px - n0;
            }
            const long long o = (long long)py * pitch + px;
            const float *wr = tw + (ox * ox + oy * oy);
            float w[HW + 1], v[T];
#pragma unroll
            for (int q = 0; q <= HW; ++q) w[q] = wr[q * q];
#pragma unroll
            for (int t = 0; t < T; ++t) {
                v[t] = __ldg(in + o + zo[t]);
                if (MODE == WIN_FILTER) v[t] *= __ldg(rho + o + zo[t]);
            }
            if (zin == (1u << T) - 1u) {
#pragma unroll
                for (int k = 0; k < WIN_Z; ++k)
#pragma unroll
                    for (int q = -HW; q <= HW; ++q) sum[k] = fmaf(w[q < 0 ? -q : q], v[k + HW + q], sum[k]);
            } else {
#pragma unroll
                for (int k = 0; k < WIN_Z; ++k)
#pragma unroll
                    for (int q = -HW; q <= HW; ++q)
                        if ((zin >> (k + HW + q)) & 1u) sum[k] = fmaf(w[q < 0 ? -q : q], v[k + HW + q], sum[k]);
            }
            if (MODE != WIN_ADJ && !(periodic || (inxy && zin == (1u << T) - 1u)))
#pragma unroll
                for (int k = 0; k < WIN_Z; ++k)
#pragma unroll
                    for (int q = -HW; q <= HW; ++q)
                        if ((zin >> (k + HW + q)) & 1u) ws[k] += w[q < 0 ? -q : q];
        }
    }
    const bool table = periodic || (inxy && zin == (1u << T) - 1u);
#pragma unroll
    for (int k = 0; k < WIN_Z; ++k) {
        if (z0 + k >= n2) break;
        const long long me = x + (long long)y * pitch + plane * (z0 + k);
        const float n = table ? tw[3 * HW * HW + 1] : ws[k];
        if (MODE == WIN_CONV) out[me] = sum[k] / n;
        else if (MODE == WIN_ADJ) out[me] = sum[k];
        else out[me] = sum[k] / (n * __ldg(rho + me));
    }
}

// whether k_window_col takes the call: window half width 1 to 4, inside the grid
static bool window_col_fits(const int n[3], int hw) {
    return hw >= 1 && hw <= WIN_HWMAX && hw <= n[0] && hw <= n[1] && hw <= n[2] && n[1] <= 65535 * WIN_Y &&
           n[2] <= 65535 * WIN_Z;
}

template <int MODE>
static void window_col_pass(const int n[3], int pitch, const float *in, const float *rho, float *out, const float *tab,
                            int hw, int periodic, cudaStream_t s) {
    const dim3 grid((unsigned)((n[0] + WIN_X - 1) / WIN_X), (unsigned)((n[1] + WIN_Y - 1) / WIN_Y),
                    (unsigned)((n[2] + WIN_Z - 1) / WIN_Z)), block(WIN_X, WIN_Y);
    switch (hw) {
    case 1: k_window_col<MODE, 1><<<grid, block, 0, s>>>(n[0], n[1], n[2], pitch, in, rho, out, tab, periodic); break;
    case 2: k_window_col<MODE, 2><<<grid, block, 0, s>>>(n[0], n[1], n[2], pitch, in, rho, out, tab, periodic); break;
    case 3: k_window_col<MODE, 3><<<grid, block, 0, s>>>(n[0], n[1], n[2], pitch, in, rho, out, tab, periodic); break;
    default: k_window_col<MODE, 4><<<grid, block, 0, s>>>(n[0], n[1], n[2], pitch, in, rho, out, tab, periodic); break;
    }
}

template <int MODE>
static void window_pass(const int n[3], int pitch, const float *in, const float *rho, float *out, const float *tab,
                        int hw, int periodic, cudaStream_t s) {
    if constexpr (MODE != WIN_DIV) {
        if (window_col_fits(n, hw)) {
            window_col_pass<MODE>(n, pitch, in, rho, out, tab, hw, periodic, s);
            return;
        }
    }
    const unsigned gy = (unsigned)((n[1] + WIN_Y - 1) / WIN_Y), gz = (unsigned)n[2];
    const dim3 grid((unsigned)((n[0] + WIN_X - 1) / WIN_X), gy < 65535u ? gy : 65535u, gz < 65535u ? gz : 65535u);
    k_window<MODE><<<grid, dim3(WIN_X, WIN_Y), window_smem(hw), s>>>(n[0], n[1], n[2], pitch, in, rho,
                                                                                      out, tab, hw, periodic);
}

int window_table_floats(float radius) {
    const int hw = (int)(radius + 0.5f);
    return 3 * hw * hw + 2;
}

void launch_filter(const int n[3], int pitch, const float *sens, const float *rho, float *out, float radius,
                   int periodic, float *tab, cudaStream_t s) {
    const int hw = (int)(radius + 0.5f);
    float wtot = 0.f;
    const int side = 2 * hw + 1;
    for (int id = 0; id < side * side * side; ++id) {
        const int ox = id % side - hw, oy = id / side % side - hw, oz = id / (side * side) - hw;
        const float r2 = (float)(ox * ox + oy * oy + oz * oz) / (radius * radius);
        wtot += r2 < 1.f ? 1.f - sqrtf(r2) : 0.f;
    }
    k_window_table<<<1, 1024, window_smem(hw), s>>>(tab, hw, radius, wtot, 1);
    window_pass<WIN_FILTER>(n, pitch, sens, rho, out, tab, hw, periodic, s);
}

// ---- symmetrisation ------------------------------------------------------------
__device__ __forceinline__ long long lid(const int n[3], int a, int b, int c) {
    return a + (long long)n[0] * (b + (long long)n[1] * c);
}

__global__ void k_sym_reflect3(int n0, int n1, int n2, float *v) {
    const int n[3] = {n0, n1, n2}, h[3] = {n0 / 2, n1 / 2, n2 / 2};
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)h[0] * h[1] * h[2]) return;
    const int rp[3] = {(int)(t % h[0]), (int)(t / h[0] % h[1]), (int)(t / ((long long)h[0] * h[1]))};
    int orb[8][3];
    for (int i = 0; i < 8; i++)
        for (int j = 0; j < 3; j++) orb[i][j] = ((i >> j) & 1) ? n[j] - 1 - rp[j] : rp[j];
    float val = v[lid(n, orb[0][0], orb[0][1], orb[0][2])];
    for (int i = 1; i < 8; i++) val += v[lid(n, orb[i][0], orb[i][1], orb[i][2])];
    val /= 8;
    for (int i = 0; i < 8; i++) v[lid(n, orb[i][0], orb[i][1], orb[i][2])] = val;
}

__global__ void k_sym_reflect6(int n0, int h, float *v, long long nrep) {
    const int n[3] = {n0, n0, n0};
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nrep) return;
    // representative x <= y <= z < h, enumerated tetrahedrally
    int z = (int)cbrtf(6.f * (float)t);
    while (z > 0 && (long long)z * (z + 1) * (z + 2) / 6 > t) z--;
    while ((long long)(z + 1) * (z + 2) * (z + 3) / 6 <= t) z++;
    long long rem = t - (long long)z * (z + 1) * (z + 2) / 6;
    int y = (int)sqrtf(2.f * (float)rem);
    while (y > 0 && (long long)y * (y + 1) / 2 > rem) y--;
    while ((long long)(y + 1) * (y + 2) / 2 <= rem) y++;
    const int x = (int)(rem - (long long)y * (y + 1) / 2);
    const int rp[3] = {x, y, z};
    float s = 0;
    for (int i = 0; i < 8; i++) {
        int o[3];
        for (int j = 0; j < 3; j++) o[j] = ((i >> j) & 1) ? n[j] - 1 - rp[j] : rp[j];
        s += v[lid(n, o[0], o[1], o[2])];
        s += v[lid(n, o[0], o[2], o[1])];
        s += v[lid(n, o[2], o[0], o[1])];
        s += v[lid(n, o[2], o[1], o[0])];
        s += v[lid(n, o[1], o[0], o[2])];
        s += v[lid(n, o[1], o[2], o[0])];
    }
    s /= 48;
    for (int i = 0; i < 8; i++) {
        int o[3];
        for (int j = 0; j < 3; j++) o[j] = ((i >> j) & 1) ? n[j] - 1 - rp[j] : rp[j];
        v[lid(n, o[0], o[1], o[2])] = s;
        v[lid(n, o[0], o[2], o[1])] = s;
        v[lid(n, o[2], o[0], o[1])] = s;
        v[lid(n, o[2], o[1], o[0])] = s;
        v[lid(n, o[1], o[0], o[2])] = s;
        v[lid(n, o[1], o[2], o[0])] = s;
    }
}

__global__ void k_sym_rotate3(int n0, int h, float *v, long long nrep) {
    const int n[3] = {n0, n0, n0};
    const int hh[3] = {h, h, h};
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nrep) return;
    // representative z in [0,h), x, y in [0, z]
    int z = (int)cbrtf(3.f * (float)t);
    while (z > 0 && (long long)z * (z + 1) * (2 * z + 1) / 6 > t) z--;
    while ((long long)(z + 1) * (z + 2) * (2 * z + 3) / 6 <= t) z++;
    const long long rem = t - (long long)z * (z + 1) * (2 * z + 1) / 6;
    const int y = (int)(rem / (z + 1)), x = (int)(rem % (z + 1));
    const int rp[3] = {x, y, z};
    const int perm[6][3] = {{0, 2, 1}, {2, 1, 0}, {1, 0, 2}, {2, 0, 1}, {1, 2, 0}, {0, 1, 2}};
    const int fo[4][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 1}};
    const int fe[4][3] = {{0, 0, 0}, {1, 1, 0}, {0, 1, 1}, {1, 0, 1}};
    // representatives with x, y <= z can share an orbit; the reference lets their
    // threads race, here each orbit is averaged once, by its first representative
    for (int i = 0; i < 6; i++) {
        const int o[3] = {rp[perm[i][0]], rp[perm[i][1]], rp[perm[i][2]]};
        for (int f = 0; f < 4; f++) {
            const int *fl = i < 3 ? fo[f] : fe[f];
            int q[3];
            for (int j = 0; j < 3; j++) q[j] = fl[j] ? -1 - o[j] : o[j];
            if (q[0] >= 0 && q[1] >= 0 && q[2] >= 0 && q[0] <= q[2] && q[1] <= q[2]) {
                const long long tq = (long long)q[2] * (q[2] + 1) * (2 * q[2] + 1) / 6 + (long long)q[1] * (q[2] + 1) + q[0];
                if (tq < t) return;
            }
        }
    }
    float s = 0;
    for (int i = 0; i < 6; i++) {
        const int o[3] = {rp[perm[i][0]], rp[perm[i][1]], rp[perm[i][2]]};
        for (int f = 0; f < 4; f++) {
            const int *fl = i < 3 ? fo[f] : fe[f];
            int p[3];
            for (int j = 0; j < 3; j++) p[j] = fl[j] ? hh[j] - 1 - o[j] : hh[j] + o[j];
            s += v[lid(n, p[0], p[1], p[2])];
        }
    }
    s /= 24;
    for (int i = 0; i < 6; i++) {
        const int o[3] = {rp[perm[i][0]], rp[perm[i][1]], rp[perm[i][2]]};
        for (int f = 0; f < 4; f++) {
            const int *fl = i < 3 ? fo[f] : fe[f];
            int p[3];
            for (int j = 0; j < 3; j++) p[j] = fl[j] ? hh[j] - 1 - o[j] : hh[j] + o[j];
            v[lid(n, p[0], p[1], p[2])] = s;
        }
    }
}

void launch_symmetrize(const int n[3], float *v, int sym, cudaStream_t s) {
    const int h = n[0] / 2;
    if (sym == 0) {
        const long long nr = (long long)(n[0] / 2) * (n[1] / 2) * (n[2] / 2);
        k_sym_reflect3<<<(unsigned)((nr + 255) / 256), 256, 0, s>>>(n[0], n[1], n[2], v);
    } else if (sym == 1) {
        const long long nr = (long long)h * (h + 1) * (h + 2) / 6;
        k_sym_reflect6<<<(unsigned)((nr + 255) / 256), 256, 0, s>>>(n[0], h, v, nr);
    } else if (sym == 2) {
        const long long nr = (long long)h * (h + 1) * (2 * h + 1) / 6;
        k_sym_rotate3<<<(unsigned)((nr + 255) / 256), 256, 0, s>>>(n[0], h, v, nr);
    }
}

// ---- the reference's trig-basis initial density -----------------------------------
// randTribase_sincos_kernel (Framework.cuh:106-222) and randTri (Framework.cuh:238-310):
// at voxel (x, y, z) with p = (x, y, z) / (dim - 1) (centred: p - 1/2 rotated by the
// unit quaternion of the four coefficients after the basis ones), with
// c[a][i] = cos(2 pi (i+1) p_a), s[a][i] = sin(2 pi (i+1) p_a), i < P:
//   first order,  6P terms:   coeff[i] c[i%3][i/3] for i < 3P, then
//                             coeff[i] s[j%3][j/3] with j = i - 3P;
//   second order, 36P^2 terms: coeff[6P + 6P j + k] v(j) v(k), j, k < 6P, where
//                             v(j) = c[j/P][j%P] for j < 3P, s[j/P-3][j%P] otherwise.
// One thread per voxel; its 6P basis values v(j) in shared memory (P <= 50).  The
// sum runs in FP64 and is rounded to FP32 (the reference sums eight FP32 partials of
// a warp-strided split).
struct TrigArgs {
    int n[3];
    int P;
    int centered;
    float rot[9];  // row-major rotation of the centred position
};

constexpr int TRIG_BS = 64;

__global__ void __launch_bounds__(TRIG_BS) k_trig_basis(TrigArgs a, const float *__restrict__ coeff, float *out) {
    extern __shared__ float tv[];  // [6P][TRIG_BS]
    const long long ne = (long long)a.n[0] * a.n[1] * a.n[2];
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int P = a.P, t = threadIdx.x;
    float p[3] = {0.f, 0.f, 0.f};
    if (e < ne) {
        const int x = (int)(e % a.n[0]);
        const long long tt = e / a.n[0];
        const int y = (int)(tt % a.n[1]), z = (int)(tt / a.n[1]);
        p[0] = (float)x / (float)(a.n[0] - 1);
        p[1] = (float)y / (float)(a.n[1] - 1);
        p[2] = (float)z / (float)(a.n[2] - 1);
        if (a.centered) {
            const float q[3] = {p[0] - 0.5f, p[1] - 0.5f, p[2] - 0.5f};
            for (int r = 0; r < 3; ++r) p[r] = a.rot[3 * r] * q[0] + a.rot[3 * r + 1] * q[1] + a.rot[3 * r + 2] * q[2];
        }
    }
    constexpr float pi2 = 3.1415926f * 2;  // the reference's constant (Framework.cuh:113)
    for (int j = 0; j < 3 * P; ++j) {
        const int ax = j / P, i = j % P;
        tv[j * TRIG_BS + t] = cosf(pi2 * (i + 1) * p[ax]);
        tv[(3 * P + j) * TRIG_BS + t] = sinf(pi2 * (i + 1) * p[ax]);
    }
    if (e >= ne) return;
    double sum = 0;
    for (int i = 0; i < 6 * P; ++i) {  // first order: component fastest
        const int j = i < 3 * P ? i : i - 3 * P;
        const int v = (j % 3) * P + j / 3 + (i < 3 * P ? 0 : 3 * P);
        sum += (double)coeff[i] * (double)tv[v * TRIG_BS + t];
    }
    const float *c2 = coeff + 6 * P;
    for (int j = 0; j < 6 * P; ++j) {
        const double vj = (double)tv[j * TRIG_BS + t];
        double inner = 0;
        for (int k = 0; k < 6 * P; ++k) inner += (double)c2[6 * P * j + k] * (double)tv[k * TRIG_BS + t];
        sum += vj * inner;
    }
    out[e] = (float)sum;
}

// level-set volume search of randTri: x = m + (M - m) / (1 + exp(-15 (v - t))),
// M = min(1.5 vol, 1), m = 0.001; t bisected on [-37 P^2, 37 P^2] for at most 60
// steps until the mean is within 1e-3 (relative) of vol.
// state: [0] t_l, [1] t_u, [2] done, [3] t, [4 ..] block partial sums
__device__ __forceinline__ float trig_level_map(float v, float t, float M) {
    const float sgm = 1.f / (1 + expf(-15.f * (v - t)));
    return sgm * (M - 0.001f) + 0.001f;
}

__global__ void k_level_init(double *st, float P) {
    if (threadIdx.x == 0) {
        const float tu = P * P * 37;
        st[0] = -tu;
        st[1] = tu;
        st[2] = 0.0;
        st[3] = 0.0;
    }
}

__global__ void __launch_bounds__(OC_BS) k_level_step(const float *__restrict__ v, long long n, float M, double *st) {
    if (st[2] != 0.0) return;
    const float t = ((float)st[1] + (float)st[0]) / 2;
    double s = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        s += trig_level_map(v[i], t, M);
    double ss[1] = {s};
    block_reduce<1>(ss, st + 4, blockIdx.x);
}

__global__ void __launch_bounds__(OC_BS) k_level_decide(double *st, int nb, long long n, float vol) {
    if (st[2] != 0.0) return;
    const double s = sum_partials(st, nb);
    if (threadIdx.x != 0) return;
    const float mean = (float)(s / (double)n);
    const float t = ((float)st[1] + (float)st[0]) / 2;
    st[3] = t;
    if (fabsf(mean - vol) / vol < 1e-3f) {
        st[2] = 1.0;
        return;
    }
    if (mean > vol) st[0] = t;
    if (mean < vol) st[1] = t;
}

__global__ void k_level_apply(float *v, long long n, float M, const double *st) {
    const float t = (float)st[3];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        v[i] = trig_level_map(v[i], t, M);
}

int launch_trig_init(const int n[3], int P, const float *coeff_dev, int centered, const float rot[9], float vol, int sym,
                     float *rho, double *scratch, cudaStream_t s) {
    TrigArgs a;
    for (int d = 0; d < 3; ++d) a.n[d] = n[d];
    a.P = P;
    a.centered = centered;
    for (int i = 0; i < 9; ++i) a.rot[i] = rot[i];
    const long long ne = (long long)n[0] * n[1] * n[2];
    const size_t smem = sizeof(float) * 6 * P * TRIG_BS;
    if (cudaFuncSetAttribute((const void *)k_trig_basis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return -1;
    k_trig_basis<<<(unsigned)((ne + TRIG_BS - 1) / TRIG_BS), TRIG_BS, smem, s>>>(a, coeff_dev, rho);
    if (sym >= 0) launch_symmetrize(n, rho, sym, s);
    const float M = fminf(vol * 1.5f, 1.f);
    k_level_init<<<1, 32, 0, s>>>(scratch, (float)P);
    for (int it = 0; it < 60; ++it) {
        k_level_step<<<OC_NB, OC_BS, 0, s>>>(rho, ne, M, scratch);
        k_level_decide<<<1, OC_BS, 0, s>>>(scratch, OC_NB, ne, vol);
    }
    k_level_apply<<<OC_NB, OC_BS, 0, s>>>(rho, ne, M, scratch);
    return 0;
}

// ---- radial convolution of the expression layer ---------------------------------
// rho.conv(radial_convker_t<Spline4>(r)) (TensorExpression.h:946-1131,
// TensorExpression.cuh:288-369): window offsets |o_a| <= (int)(r + 0.5), weight
// w(o) = 1 - 6 q + 8 q^1.5 - 3 q^2 for q = |o|^2 / r^2 < 1 (0 otherwise); out(p) =
// sum_o w(o) in(p + o) / ws(p) over the offsets inside the grid (periodic: all,
// wrapped), ws(p) the sum of those weights.  The adjoint (the backward of the
// expression) is g_in(p) = sum_o w(o) g_out(p - o) / ws(p - o).
void launch_conv_radial(const int n[3], const float *in, float *out, float *ws, float radius, int periodic,
                        int adjoint, float *tab, cudaStream_t s) {
    const int hw = (int)(radius + 0.5f);
    k_window_table<<<1, 1024, window_smem(hw), s>>>(tab, hw, radius, 1.f, 0);
    if (!adjoint) {
        window_pass<WIN_CONV>(n, n[0], in, nullptr, out, tab, hw, periodic, s);
    } else {
        window_pass<WIN_DIV>(n, n[0], in, nullptr, ws, tab, hw, periodic, s);
        window_pass<WIN_ADJ>(n, n[0], ws, nullptr, out, tab, hw, periodic, s);
    }
}

}  // namespace h3d
