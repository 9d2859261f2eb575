// k_galerkin.cu -- Galerkin coarse operators and the coarsest-grid dense solve.
//
// Reference behaviour restated (homo3d):
//   restrict_stencil_otf_aos_kernel_1 (grid_ex.cu:936-1060): level-1 stencils
//     R K(rho) P computed from the fine densities (rho^p, no 1e-9 floor) for the
//     lexicographic vertices 0..n_c per axis, elements clipped to the domain, the
//     self block's diagonal clamped to >= 1e-4, stored FP16; the periodic images
//     of a vertex on a min face are then summed in FP16 (grid.cu:2741-2772 ->
//     grid.cu:3103-3176).  On B200 the triple loop over fine elements is replaced
//     by the exact refactoring into coarse element matrices
//     K_E = sum_s rho_s P_s^T Ke P_s (Q_s = P_s^T Ke P_s precomputed), and the
//     images become the subsets of the 8 coarse elements around the vertex.
//   restrict_stencil_arround_dirichelt_boundary (grid.cpp:1184-1325): the 27
//     coarse vertices around the pinned fine origin use the pinned fine operator
//     (identity at the origin node, 1e-9 floor) in double precision.  With
//     pin_identity = 0 the identity is left out, which makes the coarse operator
//     the exact Galerkin product of the pinned fine operator.
//   restrict_stencil_aos_kernel_1 (grid_ex.cu:1065-1160): deeper levels R A P
//     from the FP16 finer stencil.
//   solveHostEquation / assembleHostMatrix (grid.cpp:349-424): coarsest level.
//     Replaced by a dense FP64 inverse built on the device (panel-wise Gauss-Jordan
//     with partial pivoting) and applied to the six load cases at once.
#include "h3d_internal.cuh"

namespace h3d {

__device__ __forceinline__ int modp(int a, int n) { return ((a % n) + n) % n; }

// ---- level 1 from densities ---------------------------------------------------
// R = 2 on every axis is compiled with the sub-element loop unrolled; R = 0 is
// the generic path for ratio 4 (or mixed ratios).
template <int R, bool F32>
__global__ void __launch_bounds__(128) k_galerkin_l1(Planes F, Planes C, int r0, int r1, int r2,
                                                     const float *__restrict__ rho, const float *__restrict__ q,
                                                     int nsub, uint4 *st) {
    extern __shared__ float sq[];
    for (int i = threadIdx.x; i < nsub * 576; i += blockDim.x) sq[i] = q[i];
    __syncthreads();
    const long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (v >= C.nv) return;
    if (R == 2) { r0 = r1 = r2 = 2; nsub = 8; }
    const int k = color_of_index(C, v);
    int X[3];
    vpos(C, k, v - C.base[k], X[0], X[1], X[2]);
    const int bmask = (X[0] == 0 ? 4 : 0) | (X[1] == 0 ? 2 : 0) | (X[2] == 0 ? 1 : 0);
    // lexicographic index of fine element (E*r + s) for the coarse element E = X - l
    long long ebase[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) {
        const int ex = wrap(X[0] - (l & 1), C.n[0]) * r0, ey = wrap(X[1] - ((l >> 1) & 1), C.n[1]) * r1,
                  ez = wrap(X[2] - (l >> 2), C.n[2]) * r2;
        ebase[l] = ex + (long long)F.n[0] * (ey + (long long)F.n[1] * ez);
    }
    uint32_t cbuf[4] = {0, 0, 0, 0};
#pragma unroll
    for (int d = 0; d < 27; ++d) {
        const int dx = d % 3 - 1, dy = d / 3 % 3 - 1, dz = d / 9 - 1;
        // the images are summed in the storage precision (FP16: grid.cu:3103-3176)
        float res[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) res[e] = 0.f;
        for (int img = 0; img < 8; ++img) {
            if (img & ~bmask) continue;
            float p[9];
#pragma unroll
            for (int e = 0; e < 9; ++e) p[e] = 0.f;
#pragma unroll
            for (int l = 0; l < 8; ++l) {
                const int lx = l & 1, ly = (l >> 1) & 1, lz = l >> 2;
                const int mx = lx + dx, my = ly + dy, mz = lz + dz;
                if (mx < 0 || mx > 1 || my < 0 || my > 1 || mz < 0 || mz > 1) continue;
                const int m = mx + 2 * my + 4 * mz;
                const int limg = ((lx << 2) | (ly << 1) | lz) & bmask;
                if (limg != img) continue;
                if (R == 2) {
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        const long long fe = ebase[l] + (s & 1) + (long long)F.n[0] * (((s >> 1) & 1) + (long long)F.n[1] * (s >> 2));
                        const float rp = __ldg(&rho[fe]);
                        const float *Q = sq + s * 576;
#pragma unroll
                        for (int i = 0; i < 3; ++i)
#pragma unroll
                            for (int j = 0; j < 3; ++j) p[3 * i + j] = fmaf(rp, Q[(3 * l + i) * 24 + 3 * m + j], p[3 * i + j]);
                    }
                } else {
                    for (int s = 0; s < nsub; ++s) {
                        const int sx = s % r0, sy = (s / r0) % r1, sz = s / (r0 * r1);
                        const long long fe = ebase[l] + sx + (long long)F.n[0] * (sy + (long long)F.n[1] * sz);
                        const float rp = __ldg(&rho[fe]);
                        const float *Q = sq + s * 576;
#pragma unroll
                        for (int i = 0; i < 3; ++i)
#pragma unroll
                            for (int j = 0; j < 3; ++j) p[3 * i + j] = fmaf(rp, Q[(3 * l + i) * 24 + 3 * m + j], p[3 * i + j]);
                    }
                }
            }
            if (d == 13) {
#pragma unroll
                for (int t = 0; t < 3; ++t)
                    if (fabsf(p[4 * t]) < 1e-4f) p[4 * t] = 1e-4f;
            }
#pragma unroll
            for (int e = 0; e < 9; ++e)
                res[e] = F32 ? res[e] + p[e] : __half2float(__hadd(__float2half_rn(res[e]), __float2half_rn(p[e])));
        }
        // stream the 9 entries into the packed chunks
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            const int g = 9 * d + e;
            if (F32) {
                cbuf[g & 3] = __float_as_uint(res[e]);
                if ((g & 3) == 3 || g == 242) {
                    if (g == 242) cbuf[3] = 0;  // entries 240..242 and the pad
                    st[(long long)(g >> 2) * C.nv + v] = make_uint4(cbuf[0], cbuf[1], cbuf[2], cbuf[3]);
                }
            } else {
                const uint32_t hv = (uint32_t)__half_as_ushort(__float2half_rn(res[e]));
                const int slot = (g & 7) >> 1;
                if (g & 1) cbuf[slot] |= hv << 16;
                else cbuf[slot] = hv;
                if ((g & 7) == 7 || g == 242) {
                    if (g == 242) { cbuf[1] &= 0xffffu; cbuf[2] = 0; cbuf[3] = 0; }
                    st[(long long)(g >> 3) * C.nv + v] = make_uint4(cbuf[0], cbuf[1], cbuf[2], cbuf[3]);
                }
            }
        }
    }
}

void launch_galerkin_l1(const Level &F, const Level &C, const float *rho, const float *q, int nsub, cudaStream_t s) {
    const int bs = 128;
    const unsigned nb = (unsigned)((C.P.nv + bs - 1) / bs);
    const size_t smem = (size_t)nsub * 576 * sizeof(float);
    if (C.ratio[0] == 2 && C.ratio[1] == 2 && C.ratio[2] == 2) {
        if (C.st32) k_galerkin_l1<2, true><<<nb, bs, smem, s>>>(F.P, C.P, 2, 2, 2, rho, q, nsub, C.st);
        else k_galerkin_l1<2, false><<<nb, bs, smem, s>>>(F.P, C.P, 2, 2, 2, rho, q, nsub, C.st);
    } else {
        static bool attr = false;
        if (!attr) {
            cudaFuncSetAttribute(k_galerkin_l1<0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            cudaFuncSetAttribute(k_galerkin_l1<0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            attr = true;
        }
        if (C.st32)
            k_galerkin_l1<0, true><<<nb, bs, smem, s>>>(F.P, C.P, C.ratio[0], C.ratio[1], C.ratio[2], rho, q, nsub, C.st);
        else
            k_galerkin_l1<0, false><<<nb, bs, smem, s>>>(F.P, C.P, C.ratio[0], C.ratio[1], C.ratio[2], rho, q, nsub,
                                                         C.st);
    }
}

// ---- the 27 coarse vertices around the pinned fine origin -----------------------
__device__ __forceinline__ double hat_w(int ox, int oy, int oz, int r0, int r1, int r2) {
    ox = abs(ox); oy = abs(oy); oz = abs(oz);
    if (ox >= r0 || oy >= r1 || oz >= r2) return 0.0;
    return (double)((r0 - ox) * (r1 - oy) * (r2 - oz)) / (double)(r0 * r1 * r2);
}

// one CTA per (coarse vertex offset vi in {-1,0,1}^3, neighbour d); its threads
// share the fine elements of the (2r)^3 box around the neighbour (one each for
// ratio 2 and 4, a fixed strided set above that) and the contributions are summed
// in a fixed tree order
constexpr int PATCH_MAX_THREADS = 512;
template <bool F32>
__global__ void __launch_bounds__(PATCH_MAX_THREADS) k_dirichlet_patch(Planes F, Planes C, int r0, int r1, int r2,
                                                                       const float *__restrict__ rho,
                                                                       const double *__restrict__ ked, int pin_identity,
                                                                       uint4 *st) {
    __shared__ double red[PATCH_MAX_THREADS][9];
    const int vi = blockIdx.x / 27, d = blockIdx.x % 27;
    const int vio[3] = {(vi % 3 - 1), (vi / 3 % 3 - 1), (vi / 9 - 1)};
    const int pi[3] = {vio[0] * r0, vio[1] * r1, vio[2] * r2};
    const int pj[3] = {pi[0] + (d % 3 - 1) * r0, pi[1] + (d / 3 % 3 - 1) * r1, pi[2] + (d / 9 - 1) * r2};
    const int tid = threadIdx.x;
    double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int e = tid; e < 8 * r0 * r1 * r2; e += blockDim.x) {  // this thread's elements, in order
    const int ex = e % (2 * r0) - r0, ey = (e / (2 * r0)) % (2 * r1) - r1, ez = e / (4 * r0 * r1) - r2;
    const int ep[3] = {pj[0] + ex, pj[1] + ey, pj[2] + ez};
    const int eo[3] = {ep[0] - pi[0], ep[1] - pi[1], ep[2] - pi[2]};
    if (!(eo[0] >= r0 || eo[0] < -r0 || eo[1] >= r1 || eo[1] < -r1 || eo[2] >= r2 || eo[2] < -r2)) {
        const long long fe =
            modp(ep[0], F.n[0]) + (long long)F.n[0] * (modp(ep[1], F.n[1]) + (long long)F.n[1] * modp(ep[2], F.n[2]));
        const double rp = 1e-9 + (double)rho[fe];
        for (int a = 0; a < 8; a++) {
            const int ap[3] = {ep[0] + (a & 1), ep[1] + ((a >> 1) & 1), ep[2] + (a >> 2)};
            const double wi = hat_w(ap[0] - pi[0], ap[1] - pi[1], ap[2] - pi[2], r0, r1, r2);
            if (wi == 0) continue;
            const bool ad = ap[0] == 0 && ap[1] == 0 && ap[2] == 0;
            for (int b = 0; b < 8; b++) {
                const int bp[3] = {ep[0] + (b & 1), ep[1] + ((b >> 1) & 1), ep[2] + (b >> 2)};
                const double wj = hat_w(bp[0] - pj[0], bp[1] - pj[1], bp[2] - pj[2], r0, r1, r2);
                if (wj == 0) continue;
                const bool bd = bp[0] == 0 && bp[1] == 0 && bp[2] == 0;
                if (ad || bd) {
                    if (a == b && pin_identity)
                        for (int i = 0; i < 3; i++) s[4 * i] += wi * wj;
                } else {
                    for (int i = 0; i < 3; i++)
                        for (int j = 0; j < 3; j++) s[3 * i + j] += wi * wj * rp * ked[(3 * a + i) * 24 + 3 * b + j];
                }
            }
        }
    }
    }
#pragma unroll
    for (int k = 0; k < 9; k++) red[tid][k] = s[k];
    __syncthreads();
    for (int half = blockDim.x / 2; half > 0; half /= 2) {  // blockDim.x is a power of two
        if (tid < half)
#pragma unroll
            for (int k = 0; k < 9; k++) red[tid][k] += red[tid + half][k];
        __syncthreads();
    }
    if (tid != 0) return;
    double t[9];
#pragma unroll
    for (int k = 0; k < 9; k++) t[k] = red[0][k];
    if (d == 13)
        for (int i = 0; i < 3; i++)
            if (fabs(t[4 * i]) < 1e-4) t[4 * i] = 1e-4;
    const long long v = vidx(C, modp(vio[0], C.n[0]), modp(vio[1], C.n[1]), modp(vio[2], C.n[2]));
    for (int e = 0; e < 9; e++) StencilStore<F32>::putd(st, C.nv, v, 9 * d + e, t[e]);
}

void launch_dirichlet_patch(const Level &F, const Level &C, const float *rho, const double *ked, int pin_identity,
                            cudaStream_t s) {
    int nt = 8 * C.ratio[0] * C.ratio[1] * C.ratio[2];  // (2r)^3 elements, a power of two
    if (nt > PATCH_MAX_THREADS) nt = PATCH_MAX_THREADS;
    if (C.st32)
        k_dirichlet_patch<true><<<27 * 27, nt, 0, s>>>(F.P, C.P, C.ratio[0], C.ratio[1], C.ratio[2], rho, ked,
                                                       pin_identity, C.st);
    else
        k_dirichlet_patch<false><<<27 * 27, nt, 0, s>>>(F.P, C.P, C.ratio[0], C.ratio[1], C.ratio[2], rho, ked,
                                                        pin_identity, C.st);
}

// ---- deeper levels: R A P from the finer stencil -----------------------------------
// the 9 entries of block J of fine vertex fv (compile-time J: fixed chunk slots)
template <int J, bool F32>
__device__ __forceinline__ void fine_block(const uint4 *__restrict__ st, long long nv, long long fv, float b[9]) {
    using S = StencilStore<F32>;
    constexpr int e0 = 9 * J, q0 = e0 / S::PER, q1 = (e0 + 8) / S::PER;
    float v[3 * S::PER];
#pragma unroll
    for (int q = q0; q <= q1; ++q) S::unpack(__ldg(st + q * nv + fv), v + (q - q0) * S::PER);
#pragma unroll
    for (int k = 0; k < 9; ++k) b[k] = v[e0 + k - S::PER * q0];
}

// One thread per (coarse vertex, coarse neighbour d): block d of the coarse
// stencil is sum over fine i in the support of the vertex and fine j in the
// support of neighbour d of w_i w_j A_ij.  The fine offsets are visited in the
// order x, y, z (z fastest) and the fine neighbours j in ascending order.  With
// dminor, d is the block index modulo 27, so the 27 CTAs of one block of coarse
// vertices run together and read the same fine stencil rows while they are in
// L2: for a finer stencil far larger than L2 (128^3 vertices, 1 GB) that is 9 %
// faster than d as the second grid dimension, which streams the finer stencil
// once per d; for smaller ones, where the stencil nearly fits in L2, it is slower
// (the 27 d of a vertex block have very different loop lengths).
template <bool F32>
__global__ void __launch_bounds__(128) k_galerkin(Planes F, Planes C, int r0, int r1, int r2,
                                                  const uint4 *__restrict__ fst, uint4 *cst, int dminor) {
    const int d = dminor ? (int)(blockIdx.x % 27u) : (int)blockIdx.y;
    const long long v = (dminor ? blockIdx.x / 27u : blockIdx.x) * (long long)blockDim.x + threadIdx.x;
    if (v >= C.nv) return;
    const int k = color_of_index(C, v);
    int X[3];
    vpos(C, k, v - C.base[k], X[0], X[1], X[2]);
    const float pr = (float)(r0 * r1 * r2);
    const int dj0 = r0 * (d % 3 - 1), dj1 = r1 * (d / 3 % 3 - 1), dj2 = r2 * (d / 9 - 1);
    float s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    // fine offsets oi from the coarse vertex with |oi| < r and |oi - dj| <= r
    const int a0 = max(-r0 + 1, dj0 - r0), b0 = min(r0 - 1, dj0 + r0);
    const int a1 = max(-r1 + 1, dj1 - r1), b1 = min(r1 - 1, dj1 + r1);
    const int a2 = max(-r2 + 1, dj2 - r2), b2 = min(r2 - 1, dj2 + r2);
    for (int o0 = a0; o0 <= b0; o0++)
        for (int o1 = a1; o1 <= b1; o1++)
            for (int o2 = a2; o2 <= b2; o2++) {
                const long long fv = vidx(F, modp(X[0] * r0 + o0, F.n[0]), modp(X[1] * r1 + o1, F.n[1]),
                                          modp(X[2] * r2 + o2, F.n[2]));
                const float wi = (float)((r0 - abs(o0)) * (r1 - abs(o1)) * (r2 - abs(o2))) / pr;
#pragma unroll
                for (int j = 0; j < 27; j++) {
                    const int q0 = abs(o0 + j % 3 - 1 - dj0), q1 = abs(o1 + j / 3 % 3 - 1 - dj1),
                              q2 = abs(o2 + j / 9 - 1 - dj2);
                    if (q0 >= r0 || q1 >= r1 || q2 >= r2) continue;
                    const float wj = (float)((r0 - q0) * (r1 - q1) * (r2 - q2)) / pr;
                    const float ww = wi * wj;
                    float bl[9];
                    switch (j) {  // compile-time block index for the chunk arithmetic
#define H3D_FB(J) case J: fine_block<J, F32>(fst, F.nv, fv, bl); break;
                        H3D_FB(0) H3D_FB(1) H3D_FB(2) H3D_FB(3) H3D_FB(4) H3D_FB(5) H3D_FB(6) H3D_FB(7) H3D_FB(8)
                        H3D_FB(9) H3D_FB(10) H3D_FB(11) H3D_FB(12) H3D_FB(13) H3D_FB(14) H3D_FB(15) H3D_FB(16)
                        H3D_FB(17) H3D_FB(18) H3D_FB(19) H3D_FB(20) H3D_FB(21) H3D_FB(22) H3D_FB(23) H3D_FB(24)
                        H3D_FB(25) H3D_FB(26)
#undef H3D_FB
                    }
#pragma unroll
                    for (int e = 0; e < 9; e++) s[e] = fmaf(ww, bl[e], s[e]);
                }
            }
    if (d == 13)
        for (int t = 0; t < 3; t++)
            if (fabsf(s[4 * t]) < 1e-4f) s[4 * t] = 1e-4f;
    for (int e = 0; e < 9; e++) StencilStore<F32>::put(cst, C.nv, v, 9 * d + e, s[e]);
}

void launch_galerkin(const Level &F, const Level &C, cudaStream_t s) {
    const int bs = 128;
    const unsigned nb = (unsigned)((C.P.nv + bs - 1) / bs);
    const int dminor = F.P.nv >= (1LL << 21);
    const dim3 grid = dminor ? dim3(nb * 27u, 1) : dim3(nb, 27);
    if (C.st32) k_galerkin<true><<<grid, bs, 0, s>>>(F.P, C.P, C.ratio[0], C.ratio[1], C.ratio[2], F.st, C.st, dminor);
    else k_galerkin<false><<<grid, bs, 0, s>>>(F.P, C.P, C.ratio[0], C.ratio[1], C.ratio[2], F.st, C.st, dminor);
}

// ---- coarsest level ---------------------------------------------------------------
// Coarsest matrix K over the unique DOFs (3*lexid + comp), n x n row-major.  One
// thread per (row, column vertex) adds the row vertex's neighbour blocks that fall
// on the column vertex, in neighbour order d = 0..26 (several do only on grids of
// two or three cells per axis), so the matrix is the same from run to run and is
// written once, coalesced, without a clearing pass.
template <bool F32>
__global__ void __launch_bounds__(256) k_coarse_assemble(Planes C, const uint4 *__restrict__ st, double *a, int n) {
    const int nv = n / 3;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)n * nv) return;
    const int w = (int)(t % nv), row = (int)(t / nv), i = row % 3, lex = row / 3;
    const int n0 = C.n[0], n1 = C.n[1], n2 = C.n[2];
    const int x = lex % n0, y = lex / n0 % n1, z = lex / (n0 * n1);
    const int wx = w % n0, wy = w / n0 % n1, wz = w / (n0 * n1);
    const long long v = vidx(C, x, y, z);
    double s[3] = {0, 0, 0};
    for (int dz = -1; dz <= 1; dz++) {
        if (wrap(z + dz, n2) != wz) continue;
        for (int dy = -1; dy <= 1; dy++) {
            if (wrap(y + dy, n1) != wy) continue;
            for (int dx = -1; dx <= 1; dx++) {
                if (wrap(x + dx, n0) != wx) continue;
                const int d = 9 * (dz + 1) + 3 * (dy + 1) + dx + 1;
                for (int j = 0; j < 3; j++) s[j] += (double)StencilStore<F32>::get(st, C.nv, v, 9 * d + 3 * i + j);
            }
        }
    }
    double *o = a + (long long)row * n + 3 * w;
    for (int j = 0; j < 3; j++) o[j] = s[j];
}

// Coarsest inverse: in-place Gauss-Jordan elimination with partial pivoting in FP64
// (grid.cpp:385-424 inverts the same matrix on the host), NB pivot columns (a panel)
// per launch.  The elimination of a panel, row swaps included, is T = I outside the
// panel's columns and the n x NB matrix G in them, so every other column becomes
//   x_i <- (i in the panel's rows ? 0 : x_i) + sum_j G_ij x_{k+j}   (rows after the swaps)
// and the panel's own columns become G.  Launch k applies panel k to all columns
// (32 columns per warp, one per lane, the NB pivot-row values of a column in
// registers), while its first CTA applies it to panel k + 1's columns alone and
// factors that panel at once: one row per thread (R rows for the large sizes), the
// panel in registers, two barriers per pivot.  The matrix goes back and forth
// between two buffers, so the row swaps are an index map (srow) on the reads; the
// last launch also undoes them on the columns, which leaves K^-1.
// The factorisation is a serial chain of n pivot steps, bound by their latency: one
// launch per pivot column over [K | I] took 7.3 us a step (1.41 ms for 192 unknowns,
// 5.9 ms for 648); here a panel's steps stay inside one CTA.
// The pivot is the largest |a_ij| to 20 mantissa bits; of equals the lowest row with one
// row per thread, the one of the lowest thread with two.
constexpr int GJ_ROWS_PER_WARP = 4;  // rows of a tile per warp

struct GjArgs {
    const double *src;   // the matrix before panel k
    double *dst;         // after it
    const double *G;     // panel k's G (n x NB, rows after its swaps, zero padded)
    double *Gn;          // panel k + 1's
    const int *srow;     // row of src that holds row i after panel k's swaps
    int *srown;          // the same for panel k + 1
    const int *orow;     // row of K that row i holds after panel k's swaps
    int *orown;
    int *flag;
    int n, k, np;        // k = -1: factor panel 0 only; k = np - 1: apply the last panel
};

template <int NB, int R, int MAXT>
__global__ void __launch_bounds__(MAXT) k_gj_panel(GjArgs g) {
    const int n = g.n, k = g.k, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    const int c0 = k * NB, cn = c0 + NB;  // first column of panel k, of panel k + 1
    const bool has_next = k + 1 < g.np;
    if (!has_next || blockIdx.x > 0) {
        // apply panel k to a tile of 32 columns
        const int ncol = (n + 31) / 32, t = (int)blockIdx.x - (has_next ? 1 : 0);
        const int rb = GJ_ROWS_PER_WARP * nw, r0 = (t / ncol) * rb, r1 = min(n, r0 + rb);
        const int c = (t % ncol) * 32 + lane;
        const bool own = c >= c0 && c < cn, skip = c >= n || (has_next && c >= cn && c < cn + NB);
        double x[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j)
            x[j] = (skip || own || c0 + j >= n) ? 0.0 : __ldg(&g.src[(long long)__ldg(&g.srow[c0 + j]) * n + c]);
        const int cd = skip ? 0 : (has_next ? c : __ldg(&g.orow[c]));
        for (int i = r0 + wid; i < r1; i += nw) {
            const double *Gi = g.G + (long long)i * NB;
            double v = (skip || own || (i >= c0 && i < cn)) ? 0.0 : __ldg(&g.src[(long long)__ldg(&g.srow[i]) * n + c]);
#pragma unroll
            for (int j = 0; j < NB; ++j) v = fma(__ldg(Gi + j), x[j], v);
            if (own) v = __ldg(Gi + (c - c0));
            if (!skip) g.dst[(long long)i * n + cd] = v;
        }
        return;
    }
    // panel k + 1: apply panel k to its columns, then factor it
    extern __shared__ int srow_s[];  // n: rows of dst after this panel's swaps
    __shared__ double xs[NB][NB];
    __shared__ double rowp[2][NB], rowq[2][NB];
    __shared__ unsigned keys[2][32];
    __shared__ int krow[2][32];
    const int nbn = min(NB, n - cn);
    for (int i = tid; i < n; i += blockDim.x) srow_s[i] = i;
    double a[R][NB];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = tid + r * (int)blockDim.x;
        const bool in = i < n, pan = k >= 0 && i >= c0 && i < cn;
        const int si = in ? (k >= 0 ? __ldg(&g.srow[i]) : i) : 0;
#pragma unroll
        for (int c = 0; c < NB; ++c) a[r][c] = (in && !pan && c < nbn) ? __ldg(&g.src[(long long)si * n + cn + c]) : 0.0;
    }
    if (k >= 0) {
        for (int q = tid; q < NB * NB; q += blockDim.x) {
            const int j = q / NB, c = q % NB;
            xs[j][c] = c < nbn ? __ldg(&g.src[(long long)__ldg(&g.srow[c0 + j]) * n + cn + c]) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = tid + r * (int)blockDim.x;
            const double *Gi = g.G + (long long)(i < n ? i : 0) * NB;
#pragma unroll 4
            for (int j = 0; j < NB; ++j) {
                const double gj = __ldg(Gi + j);
#pragma unroll
                for (int c = 0; c < NB; ++c) a[r][c] = fma(gj, xs[j][c], a[r][c]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        if (j >= nbn) break;
        const int q = cn + j, b = j & 1;  // pivot row; buffer of this step
        unsigned key = 0;                 // 0: not a candidate
        int kr = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = tid + r * (int)blockDim.x;
            const unsigned kk = (i >= q && i < n) ? ((unsigned)__double2hiint(a[r][j]) & 0x7fffffffu) + 1u : 0u;
            if (kk > key) { key = kk; kr = i; }
        }
        const unsigned wm = __reduce_max_sync(0xffffffffu, key);
        const unsigned who = __ballot_sync(0xffffffffu, key == wm);
        if (lane == __ffs(who) - 1) { keys[b][wid] = wm; krow[b][wid] = kr; }
        __syncthreads();
        const unsigned wk = lane < nw ? keys[b][lane] : 0u;
        const unsigned bm = __reduce_max_sync(0xffffffffu, wk);
        const int p = krow[b][__ffs(__ballot_sync(0xffffffffu, wk == bm)) - 1];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = tid + r * (int)blockDim.x;
            if (i == p)
#pragma unroll
                for (int c = 0; c < NB; ++c) rowp[b][c] = a[r][c];
            if (i == q)
#pragma unroll
                for (int c = 0; c < NB; ++c) rowq[b][c] = a[r][c];
        }
        __syncthreads();
        const double piv = rowp[b][j], inv = 1.0 / piv;
        if (tid == 0) {
            if (!(fabs(piv) > 0.0)) *g.flag = 1;
            const int t = srow_s[p];
            srow_s[p] = srow_s[q];
            srow_s[q] = t;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = tid + r * (int)blockDim.x;
            if (i == p && p != q)  // the row swapped out of the pivot position
#pragma unroll
                for (int c = 0; c < NB; ++c) a[r][c] = rowq[b][c];
            if (i == q) {
#pragma unroll
                for (int c = 0; c < NB; ++c) a[r][c] = c == j ? inv : rowp[b][c] * inv;
            } else {
                const double f = -(a[r][j] * inv);
#pragma unroll
                for (int c = 0; c < NB; ++c) a[r][c] = c == j ? f : fma(f, rowp[b][c], a[r][c]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = tid + r * (int)blockDim.x;
        if (i >= n) continue;
        g.srown[i] = srow_s[i];
        g.orown[i] = k >= 0 ? __ldg(&g.orow[srow_s[i]]) : srow_s[i];
#pragma unroll
        for (int c = 0; c < NB; ++c) g.Gn[(long long)i * NB + c] = c < nbn ? a[r][c] : 0.0;
    }
}

// panel width, rows per thread and thread limit by size: a panel row is 2 NB
// registers, so 16 columns fit up to 1024 one-row threads (coarsest grids to 6 x 7 x 8
// vertices), and 8 columns with two rows per thread hold the rest (7^3: 1029 unknowns
// to 8^3: 1536)
static int gj_width(int n) { return n <= 1024 ? 16 : 8; }
static int gj_panels(int n) { return (n + gj_width(n) - 1) / gj_width(n); }

// [K^-1 | the other buffer | two G | two srow, two orow]
size_t gauss_jordan_doubles(int n) { return (size_t)n * n * 2 + (size_t)n * 16 * 2 + (size_t)n * 2 + 2; }

// K is assembled into the buffer from which the panels' alternation ends in the first
static double *gj_start(double *aug, int n) { return aug + (gj_panels(n) & 1 ? (size_t)n * n : 0); }

void launch_coarse_assemble(const Level &C, double *aug, cudaStream_t s) {
    const int n = (int)(3 * C.P.nv);
    const long long nt = (long long)n * C.P.nv;
    double *a = gj_start(aug, n);
    if (C.st32) k_coarse_assemble<true><<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(C.P, C.st, a, n);
    else k_coarse_assemble<false><<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(C.P, C.st, a, n);
}

template <int NB, int R, int MAXT>
static void gj_run(double *aug, int n, int *flag, cudaStream_t s) {
    const int np = gj_panels(n);
    const unsigned nt = (unsigned)(((n + R - 1) / R + 31) / 32 * 32);
    const unsigned rb = GJ_ROWS_PER_WARP * (nt / 32);
    const unsigned tiles = (unsigned)((n + 31) / 32) * ((n + rb - 1) / rb);
    double *buf[2] = {aug, aug + (size_t)n * n};
    double *G[2] = {buf[1] + (size_t)n * n, buf[1] + (size_t)n * n + (size_t)n * NB};
    int *idx = reinterpret_cast<int *>(buf[1] + (size_t)n * n + (size_t)n * 16 * 2);
    int *srow[2] = {idx, idx + n}, *orow[2] = {idx + 2 * n, idx + 3 * n};
    for (int k = -1; k < np; k++) {
        GjArgs g;
        const int from = (np + (k < 0 ? 0 : k)) & 1, cur = k & 1, next = (k + 1) & 1;
        g.src = buf[from];
        g.dst = buf[from ^ 1];
        g.G = G[cur];
        g.Gn = G[next];
        g.srow = srow[cur];
        g.srown = srow[next];
        g.orow = orow[cur];
        g.orown = orow[next];
        g.flag = flag;
        g.n = n;
        g.k = k;
        g.np = np;
        const unsigned nb = k < 0 ? 1u : tiles + (k + 1 < np ? 1u : 0u);
        k_gj_panel<NB, R, MAXT><<<nb, nt, sizeof(int) * (size_t)n, s>>>(g);
    }
}

void launch_gauss_jordan(double *aug, int n, int *flag, cudaStream_t s) {
    if (n <= 704) gj_run<16, 1, 704>(aug, n, flag, s);
    else if (n <= 1024) gj_run<16, 1, 1024>(aug, n, flag, s);
    else gj_run<8, 2, 768>(aug, n, flag, s);
}

// x = K^-1 b for the six load cases: one warp per row of K^-1 (coarsest_rows), all
// cases from one read of the row.  One thread per row and one CTA per load case read
// the rows with a stride of 2n doubles, six times: 23 us for 192 unknowns, 237 us for
// 648.
__global__ void __launch_bounds__(COARSEST_T) k_coarse_apply(Planes C, const double *__restrict__ inv, int n,
                                                             int project, const float *__restrict__ f, float *u) {
    extern __shared__ float b[];
    coarsest_rows<false>(C, inv, n, project, f, u, b, blockIdx.x, gridDim.x);
}

static unsigned coarsest_blocks(int n) { return (unsigned)((n + COARSEST_T / 32 - 1) / (COARSEST_T / 32)); }

void launch_coarse_apply(const Level &C, const double *aug, int project, cudaStream_t s) {
    const int n = (int)(3 * C.P.nv);
    k_coarse_apply<<<coarsest_blocks(n), COARSEST_T, coarsest_smem(n), s>>>(C.P, aug, n, project, C.f, C.u);
}

// lockstep batches: the coarsest solves of several designs in one launch, grid row y
// for slot y; a slot's CTAs are those of the design's own launch
struct CoarsestEnt {
    Planes C;
    const double *aug;
    const float *f;
    float *u;
    int n, design;
};
struct CoarsestBatchTab {
    int n;
    CoarsestEnt e[BATCH_MAX];
};

__global__ void __launch_bounds__(COARSEST_T) k_coarse_apply_batch(const CoarsestBatchTab *__restrict__ t,
                                                            const int *__restrict__ active, int project) {
    extern __shared__ float b[];
    __shared__ __align__(16) unsigned buf[sizeof(CoarsestEnt) / 4];
    const int i = blockIdx.y;
    if (!__ldg(&active[t->e[i].design])) return;
    const CoarsestEnt &e = stage_args(t->e[i], buf);
    const unsigned nb = (unsigned)((e.n + COARSEST_T / 32 - 1) / (COARSEST_T / 32));
    if (blockIdx.x < nb) coarsest_rows<false>(e.C, e.aug, e.n, project, e.f, e.u, b, blockIdx.x, nb);
}

int coarsest_batch_create(const Level *const *lv, const double *const *aug, const int *design, int n, BatchTab *out) {
    if (n < 1 || n > BATCH_MAX) return -1;
    CoarsestBatchTab *t = new CoarsestBatchTab();
    t->n = n;
    int nmax = 0;
    for (int i = 0; i < n; i++) {
        CoarsestEnt &e = t->e[i];
        e.C = lv[i]->P;
        e.aug = aug[i];
        e.f = lv[i]->f;
        e.u = lv[i]->u;
        e.n = (int)(3 * lv[i]->P.nv);
        e.design = design[i];
        nmax = e.n > nmax ? e.n : nmax;
    }
    void *d = nullptr;
    int rc = cudaMalloc(&d, sizeof(CoarsestBatchTab)) == cudaSuccess ? 0 : -2;
    if (rc == 0 && cudaMemcpy(d, t, sizeof(CoarsestBatchTab), cudaMemcpyHostToDevice) != cudaSuccess) rc = -2;
    if (rc == 0) {
        out->dev = d;
        out->n = n;
        out->grid[0] = coarsest_blocks(nmax);
        out->smem = coarsest_smem(nmax);
    } else if (d) {
        cudaFree(d);
    }
    delete t;
    return rc;
}

void launch_coarse_apply_batch(const BatchTab &t, const int *active, int project, cudaStream_t s) {
    k_coarse_apply_batch<<<dim3(t.grid[0], (unsigned)t.n), COARSEST_T, t.smem, s>>>(static_cast<const CoarsestBatchTab *>(t.dev), active,
                                                         project);
}

}  // namespace h3d
