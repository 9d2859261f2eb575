// k_homog.cu -- homogenized elastic tensor and sensitivities.
//
// Reference behaviour restated (homo3d homogenization.cu):
//   elasticMatrix_kernel_opt (homogenization.cu:208-346), elasticMatrix
//   (:464-575): C_ij = (1/|Y|) sum_e (1e-9 + rho_e) (chi0_i - chi_i)^T Ke
//   (chi0_j - chi_j); Sensitivity_kernel_opt_2 (:697-858): per element
//   sum_{i<=j} (dC_ij + [i!=j] dC_ji) (chi0_i - chi_i)^T Ke (chi0_j - chi_j) / |Y|.
//
// B200 design.  One thread per element.  The eight node values of a component are
// turned into the coefficients of the eight products of the signs +-1 of the three
// axes (a 2 x 2 x 2 Hadamard transform, 24 additions).  An isotropic Ke commutes with
// the three mirrors, so between coefficients it couples only those of equal parity:
// eight classes of at most three entries (ModeMat) in place of 24 x 24, with the rigid
// translations (zero rows) left out 21 coefficients per load case.  The 21 energies of
// an element then take about 780 FMAs after 430 additions, where Ke U for six cases
// alone is 3456.  On the tensor cores (TF32 hi + lo, three products) the dense
// contraction had to stage operands in shared memory and read the products back from
// TMEM with 8 warps per SM.  C at 256^3 / 128^3: 5.23 / 0.67 -> 2.18 / 0.29 ms; a
// sensitivity call at 256^3 / 128^3 / 64^3: 6.90 / 0.91 / 0.131 -> 2.13 / 0.30 / 0.065 ms.
// chi is FP64 and taken relative to the element's first node before it is rounded to
// FP32; C is 2.8e-8 from 64 bits where the split operands were 3.6e-7.  Bound by the 144
// gathered FP64 values: at 128^3 the L1 data pipe is 51 % busy, issue 43 %, DRAM 19 %,
// with 8 warps per SM (233 registers) waiting on loads.
#include <stdint.h>

#include "h3d_internal.cuh"

namespace h3d {

constexpr int EN_T = 128;  // threads per CTA

// the energy in coefficients: k[p][m][n] couples component m's coefficient of the sign
// product p ^ (1 << m) with component n's of p ^ (1 << n)
struct ModeMat { float k[8][3][3]; };

static ModeMat mode_matrix(const double *ked) {
    ModeMat M;
    for (int p = 0; p < 8; p++)
        for (int m = 0; m < 3; m++)
            for (int n = 0; n < 3; n++) {
                const int S = p ^ (1 << m), T = p ^ (1 << n);
                double v = 0;
                for (int a = 0; a < 8; a++)
                    for (int b = 0; b < 8; b++) {
                        // sign of node a in product S: minus once per axis of S where its bit is 0
                        const int sa = __builtin_popcount(S & ~a & 7) & 1, sb = __builtin_popcount(T & ~b & 7) & 1;
                        v += ((sa ^ sb) ? -1.0 : 1.0) * ked[(3 * a + m) * 24 + 3 * b + n];
                    }
                M.k[p][m][n] = (float)(v / 64.0);
            }
    return M;
}

// the coefficient of product S of component m of the unit macro-strain displacement of
// case c (homoCommon.cuh:455-519): linear fields, products of one axis only
__host__ __device__ constexpr float mode_macro(int c, int m, int S) {
    return c < 3 ? (m == c && S == (1 << c) ? 4.f : 0.f)
         : c == 3 ? ((m == 1 && S == 4) || (m == 2 && S == 2) ? 2.f : 0.f)
         : c == 4 ? ((m == 0 && S == 4) || (m == 2 && S == 1) ? 2.f : 0.f)
                  : ((m == 0 && S == 2) || (m == 1 && S == 1) ? 2.f : 0.f);
}

struct EnDc { float w[21]; };  // (dC_ij + [i!=j] dC_ji) / |Y| for the 21 pairs

// E[t], t = pairs (i <= j) in row order: the energies of element (x, y, z)
__device__ __forceinline__ void element_energies(const Planes &P, const ModeMat &M, const double *__restrict__ chi,
                                                 int x, int y, int z, float E[21]) {
    const double *np[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const int vx = (a & 1) ? (x + 1 == P.n[0] ? 0 : x + 1) : x;
        const int vy = ((a >> 1) & 1) ? (y + 1 == P.n[1] ? 0 : y + 1) : y;
        const int vz = (a >> 2) ? (z + 1 == P.n[2] ? 0 : z + 1) : z;
        np[a] = chi + fidx(0, vidx(P, vx, vy, vz));
    }
    // A[c][m][S], S = 1..7: coefficients of chi0_c - chi_c
    float A[NCASE][3][8];
#pragma unroll
    for (int c = 0; c < NCASE; ++c)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int q = (3 * c + m) * FVB;
            const double c0 = __ldg(np[0] + q);
            float d[8];
            d[0] = 0.f;
#pragma unroll
            for (int a = 1; a < 8; ++a) d[a] = (float)(__ldg(np[a] + q) - c0);
            // sums and differences along each axis in turn
#pragma unroll
            for (int s = 1; s < 8; s *= 2)
#pragma unroll
                for (int a = 0; a < 8; ++a)
                    if (!(a & s)) {
                        const float lo = d[a], hi = d[a | s];
                        d[a] = lo + hi;
                        d[a | s] = hi - lo;
                    }
#pragma unroll
            for (int S = 1; S < 8; ++S) A[c][m][S] = mode_macro(c, m, S) - d[S];
        }
#pragma unroll
    for (int t = 0; t < 21; ++t) E[t] = 0.f;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
#pragma unroll
        for (int j = 0; j < NCASE; ++j) {
            float ku[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                ku[m] = 0.f;
                if ((p ^ (1 << m)) == 0) continue;  // a rigid translation
#pragma unroll
                for (int n = 0; n < 3; ++n)
                    if ((p ^ (1 << n)) != 0) ku[m] = fmaf(M.k[p][m][n], A[j][n][p ^ (1 << n)], ku[m]);
            }
#pragma unroll
            for (int i = 0; i <= j; ++i)
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    if ((p ^ (1 << m)) != 0) {
                        const int t = i * 6 - i * (i - 1) / 2 + (j - i);
                        E[t] = fmaf(A[i][m][p ^ (1 << m)], ku[m], E[t]);
                    }
        }
    }
}

// SENS = false: per-CTA FP64 partial sums of (1e-9 + rho_e) E_ij (21 values);
// SENS = true: sens[x + (y + z*ny)*pitch] = sum_t dc_t E_t per element
// dcw (SENS only, may be null): the 21 weights read from device memory instead of dc
template <bool SENS, int MB>
__global__ void __launch_bounds__(EN_T, MB) k_energy(Planes P, FastDiv dn0, FastDiv dn1, const double *__restrict__ chi,
                                                     const float *__restrict__ rho, const __grid_constant__ ModeMat M,
                                                     double *partial, EnDc dc, const float *dcw, float *sens, int pitch) {
    __shared__ float dcs[21];
    if (SENS) {
        if (threadIdx.x < 21) dcs[threadIdx.x] = dcw ? dcw[threadIdx.x] : dc.w[threadIdx.x];
        __syncthreads();
    }
    double acc[21];
    if (!SENS) {
#pragma unroll
        for (int t = 0; t < 21; ++t) acc[t] = 0;
    }
    for (long long e = blockIdx.x * (long long)EN_T + threadIdx.x; e < P.nv; e += (long long)gridDim.x * EN_T) {
        const unsigned q = (unsigned)e, tq = dn0.div(q), zq = dn1.div(tq);
        const int x = (int)(q - tq * (unsigned)P.n[0]), y = (int)(tq - zq * (unsigned)P.n[1]), z = (int)zq;
        float E[21];
        element_energies(P, M, chi, x, y, z, E);
        if (SENS) {
            float s = 0.f;
#pragma unroll
            for (int t = 0; t < 21; ++t) s = fmaf(E[t], dcs[t], s);
            sens[x + ((long long)y + (long long)z * P.n[1]) * pitch] = s;
        } else {
            const double rp = (double)(RHO_PENAL_MIN + __ldg(rho + e));
#pragma unroll
            for (int t = 0; t < 21; ++t) acc[t] = fma(rp, (double)E[t], acc[t]);
        }
    }
    if (!SENS) block_reduce<21>(acc, partial, blockIdx.x);
}

// fixed-order sum of the per-CTA partials of C
template <int N>
__global__ void __launch_bounds__(256) k_finish_n(const double *__restrict__ partial, int nblk, double *out) {
    double s[N];
#pragma unroll
    for (int c = 0; c < N; ++c) s[c] = 0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x)
#pragma unroll
        for (int c = 0; c < N; ++c) s[c] += partial[(long long)b * N + c];
    block_reduce<N>(s, out, 0);
}

void launch_elastic_finish(const double *partial, int nblk, double *out21, cudaStream_t s) {
    k_finish_n<21><<<1, 256, 0, s>>>(partial, nblk, out21);
}

// CTAs of the C form: four waves of two per SM, or one per 128 elements
int energy_blocks(const Planes &P, int num_sms) {
    const long long ntile = (P.nv + EN_T - 1) / EN_T;
    const long long nb = 8ll * num_sms;
    return (int)(ntile < nb ? ntile : nb);
}

void launch_elastic(const Planes &P, const double *chi, const float *rho, const double *ked, double *partial, int nblk,
                    cudaStream_t s) {
    k_energy<false, 2><<<nblk, EN_T, 0, s>>>(P, FastDiv((unsigned)P.n[0]), FastDiv((unsigned)P.n[1]), chi, rho,
                                             mode_matrix(ked), partial, EnDc{}, nullptr, nullptr, 0);
}

// the 21 weights (dC_ij + [i != j] dC_ji) / |Y| of the sensitivity for dC[36]
void sensitivity_weights(const Planes &P, const float *dc36, float w21[21]) {
    const double vol = (double)P.nv;
    int t = 0;
    for (int i = 0; i < 6; i++)
        for (int j = i; j < 6; j++, t++) {
            const double w = dc36[i * 6 + j] + (i != j ? dc36[j * 6 + i] : 0.f);
            w21[t] = (float)(w / vol);
        }
}

static void sensitivity(const Planes &P, const double *chi, const double *ked, const EnDc &dc, const float *dcw,
                        float *sens, int pitch, cudaStream_t s) {
    const long long ntile = (P.nv + EN_T - 1) / EN_T;
    k_energy<true, 3><<<(unsigned)ntile, EN_T, 0, s>>>(P, FastDiv((unsigned)P.n[0]), FastDiv((unsigned)P.n[1]), chi,
                                                       nullptr, mode_matrix(ked), nullptr, dc, dcw, sens, pitch);
}

void launch_sensitivity(const Planes &P, const double *chi, const double *ked, const float *dc36, float *sens, int pitch,
                        cudaStream_t s) {
    EnDc dc{};
    sensitivity_weights(P, dc36, dc.w);
    sensitivity(P, chi, ked, dc, nullptr, sens, pitch, s);
}

void launch_sensitivity_dev(const Planes &P, const double *chi, const double *ked, const float *dcw, float *sens,
                            int pitch, cudaStream_t s) {
    sensitivity(P, chi, ked, EnDc{}, dcw, sens, pitch, s);
}

}  // namespace h3d
