// k_fine.cu -- matrix-free fine-level operator: Gauss-Seidel colour sweeps,
// residuals (FP32 with fused per-case norms, and the refined FP64-solution form),
// the unit macro-strain right-hand side, and FP64 helpers of the refined mode.
//
// Reference behaviour restated (homo3d grid.cu):
//   gs_relaxation_otf_kernel (grid.cu:323-551): for each vertex of one colour,
//     sum over its 8 elements of (1e-9 + rho_e) * Ke[own rows][other nodes] * u,
//     then a 3x3 block Gauss-Seidel step on the components (x, then y, then z);
//     neighbours at the pinned origin count as zero; the origin stays zero.
//   update_residual_otf_kernel_1 (grid.cu:1277-1461): r = f - K(rho) u, r = 0 at
//     the pinned origin.
//   enforce_unit_macro_strain_kernel (grid.cu:1818-1919): f_i = K(rho) chi0_i.
//
// B200 design.  The element loop is reorganised per neighbour: for each of the 26
// neighbours the 3x3 coupling block sum_e rho_e Ke[a_e][b_e] is formed once (Ke
// entries are compile-time offsets into the kernel-parameter bank) and applied to a
// thread's load cases.  A thread serves the two vertices x = 2i + 1 and x = 2i of a
// row, as the two lanes of packed FP32x2 values: the 27 neighbours of both lie in nine
// rows, and each row gives both from four values per plane instead of six.  A sweep's
// launch takes the rows of one (y, z) parity, i.e. two of the eight colours: the odd
// vertices are updated first, the even ones after a barrier (a CTA holds whole rows, so
// the periodic neighbour in x is in the CTA); see k_fine_gs.  The residual runs all
// rows in one launch.  The operator is applied in difference form,
// sum_{d != 0} A_d (u_{v+d} - u_v), and the Gauss-Seidel step as u += D^-1 r with
// the components in the reference's order: the same iteration in exact
// arithmetic, and in FP32 it keeps rigid translations exact (see pair_rows).
#include <type_traits>

#include "h3d_internal.cuh"

namespace h3d {

constexpr int CPT = 2;            // load cases per thread of the FP32 residual
constexpr int RES_MINB = 4;       // its CTAs of 128 threads per SM
// Row blocks between a CTA of the pair kernels and the one whose rows it brings into L2.
// Both kernels wait on loads with few warps (128 registers: 4 CTAs/SM), and more than
// half of their L1 misses went on to DRAM.  Sweep / residual in us without prefetch, and
// at distances of 5, 20, 60 and 200 for both:
//   256^3  2666 / 3009    2328 / 2367   2320 / 2369   2330 / 2387   2449 / 2591
//   192^3  1198 / 1362    1089 / 1097   1089 / 1097   1092 / 1098   1107 / 1116
//   128^3   366 /  381     334 /  303    333 /  300    337 /  301    352 /  322
//    96^3   185 /  179     173 /  144    173 /  145    175 /  146    179 /  152
//    64^3    59 /   43      58 /   43     58 /   43     58 /   43     58 /   43
// and no difference at 32^3, where the fields stay in L2.
constexpr unsigned GS_AHEAD = 20, RES_AHEAD = 10;
constexpr int CPT64 = 2;          // load cases per thread of the FP64-solution residual
constexpr int MINB64 = 4;         // its CTAs per SM
constexpr int FBS = 128;          // threads per CTA

struct FineArgs {
    const float *__restrict__ rho;
    float *u;
    const float *__restrict__ f;
    float *r;
    int n[3];
    int h[3];
    long long nv;  // vertices
    long long P;   // vertices per colour plane
    float w;
    FastDiv dh0, dh1;  // division by h[0], h[1]
    int rows;          // whole rows per CTA of the pair kernels (pair_shape)
};

__device__ __forceinline__ void axis_nbrs(int i, int p, int h, int &im, int &ip) {
    if (p) { im = i; ip = (i + 1 == h) ? 0 : i + 1; }
    else { im = (i == 0) ? h - 1 : i - 1; ip = i; }
}

// (i, j, l) of index p (< 2^32) of a colour plane
__device__ __forceinline__ void plane_coords(const FineArgs &a, long long p, int &i, int &j, int &l) {
    const unsigned q = (unsigned)p;
    const unsigned t = a.dh0.div(q);
    i = (int)(q - t * (unsigned)a.h[0]);
    const unsigned z = a.dh1.div(t);
    j = (int)(t - z * (unsigned)a.h[1]);
    l = (int)z;
}

// first element (bit pattern w = ex | ey<<1 | ez<<2 of the element's offset from
// the vertex) shared by the vertex and its neighbour d, -1 if none
__host__ __device__ constexpr int first_shared(int d) {
    for (int w = 0; w < 8; ++w) {
        const int bx = 1 - (w & 1) + d % 3 - 1, by = 1 - ((w >> 1) & 1) + d / 3 % 3 - 1, bz = 1 - (w >> 2) + d / 9 - 1;
        if (bx >= 0 && bx <= 1 && by >= 0 && by <= 1 && bz >= 0 && bz <= 1) return w;
    }
    return -1;
}

// one value, or the same quantity of the two vertices of a pair
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ void vzero(float &a) { a = 0.f; }
__device__ __forceinline__ void vzero(double &a) { a = 0.0; }
__device__ __forceinline__ void vzero(float2 &a) { a = make_float2(0.f, 0.f); }

// The signed sums cs[m] of the densities rw over the elements shared with neighbour
// (dx, dy, dz), folded one free axis at a time:
// element pairs along the first free axis (their sum and difference), then
// pairs of those along the next.  Along a free axis a the element with bit a
// set enters with a minus sign when a lies in the mask m, so the sign of an
// element is the parity of the mask axes on which it differs from w0.
// 0 / 2 / 8 / 16 additions for a corner / edge / face neighbour / the vertex
// itself, where the element-by-element sums took 4 / 8 / 16 / 32.
template <typename T>
__device__ __forceinline__ void fold_signed(const T rw[8], int dx, int dy, int dz, int w0, T cs[8]) {
    int fa[3], nf = 0;  // the free axes (offset 0), ascending
    if (dx == 0) fa[nf++] = 0;
    if (dy == 0) fa[nf++] = 1;
    if (dz == 0) fa[nf++] = 2;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        if (m != 0 && m != 3 && m != 5 && m != 6) { vzero(cs[m]); continue; }
        if (nf == 0) {
            cs[m] = rw[w0];
        } else {
            const int a = fa[0];
            // level 1: pairs (w, w | a) for the 2^(nf-1) settings of the other free axes
            T v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k >= (1 << (nf - 1))) continue;
                int w = w0;
                if (nf > 1 && (k & 1)) w |= 1 << fa[1];
                if (nf > 2 && (k & 2)) w |= 1 << fa[2];
                v[k] = ((m >> a) & 1) ? vsub(rw[w], rw[w | (1 << a)]) : vadd(rw[w], rw[w | (1 << a)]);
            }
            if (nf >= 2) {  // level 2: along fa[1]
                const bool mb = (m >> fa[1]) & 1;
                v[0] = mb ? vsub(v[0], v[1]) : vadd(v[0], v[1]);
                if (nf == 3) v[2] = mb ? vsub(v[2], v[3]) : vadd(v[2], v[3]);
            }
            if (nf == 3) {  // level 3: along fa[2]
                const bool mc = (m >> fa[2]) & 1;
                v[0] = mc ? vsub(v[0], v[2]) : vadd(v[0], v[2]);
            }
            cs[m] = v[0];
        }
    }
}

// geometry of one colour-K vertex: its element densities and the offsets of its
// neighbours inside a colour plane (32-bit: a field plane holds < 2^31 vertices)
template <int KC>
struct VertexGeo {
    const int K;  // the colour: KC, or the run-time colour kr when KC < 0
    float rw[8];
    unsigned X[3], Y[3], Z[3];  // plane offsets of the neighbour rows: i, h0*j, h0*h1*l
    __device__ __forceinline__ VertexGeo(const FineArgs &a, long long p, int kr = KC) : K(KC >= 0 ? KC : kr) {
        const int px = (K & 1) ^ 1, py = ((K >> 1) & 1) ^ 1, pz = ((K >> 2) & 1) ^ 1;
        int i, j, l;
        plane_coords(a, p, i, j, l);
        const int x = 2 * i + px, y = 2 * j + py, z = 2 * l + pz;
        const int xe0 = x == 0 ? a.n[0] - 1 : x - 1;
        const int ye0 = y == 0 ? a.n[1] - 1 : y - 1;
        const int ze0 = z == 0 ? a.n[2] - 1 : z - 1;
        const unsigned n0 = (unsigned)a.n[0], n01 = (unsigned)a.n[0] * (unsigned)a.n[1];
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const unsigned ex = (w & 1) ? x : xe0, ey = ((w >> 1) & 1) ? y : ye0, ez = (w >> 2) ? z : ze0;
            rw[w] = RHO_PENAL_MIN + __ldg(&a.rho[ex + n0 * ey + n01 * ez]);
        }
        int ii[3], jj[3], ll[3];
        axis_nbrs(i, px, a.h[0], ii[0], ii[2]);
        axis_nbrs(j, py, a.h[1], jj[0], jj[2]);
        axis_nbrs(l, pz, a.h[2], ll[0], ll[2]);
        ii[1] = i; jj[1] = j; ll[1] = l;
        const unsigned h0 = (unsigned)a.h[0], h01 = (unsigned)a.h[0] * (unsigned)a.h[1];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            X[t] = (unsigned)ii[t];
            Y[t] = h0 * (unsigned)jj[t];
            Z[t] = h01 * (unsigned)ll[t];
        }
    }
    // coupling block of neighbour d (compile-time d after unrolling):
    // sum over the shared elements e of rho_e Ke[a_e][b_e].  The shared elements
    // are mirror images of the first one across the axes where they differ, and
    // an isotropic Ke is invariant under the mirrors up to the sign of the
    // components mirrored, so entry (r,c) = Ke[a_0][b_0](r,c) * sum_e +-rho_e with
    // the sign set by whether r and c lie on the mirrored axes: four signed
    // density sums per block (signed_sums) instead of 9 FMAs per shared element.
    template <typename T>
    __device__ __forceinline__ void block_t(const T *kk, int d, T A[9]) const {
        const int dx = d % 3 - 1, dy = d / 3 % 3 - 1, dz = d / 9 - 1;
        const int w0 = first_shared(d);
        T cs[8];  // cs[m]: signed sum for the axis mask m = (1<<r) ^ (1<<c); m in {0, 3, 5, 6}
        signed_sums<T>(dx, dy, dz, w0, cs);
        const int an = 7 - w0;
        const int bn = (1 - (w0 & 1) + dx) + 2 * (1 - ((w0 >> 1) & 1) + dy) + 4 * (1 - (w0 >> 2) + dz);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) A[3 * r + c] = kk[(3 * an + r) * 24 + 3 * bn + c] * cs[(1 << r) ^ (1 << c)];
    }
    template <typename T>
    __device__ __forceinline__ void signed_sums(int dx, int dy, int dz, int w0, T cs[8]) const {
        T v[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) v[w] = (T)rw[w];
        fold_signed<T>(v, dx, dy, dz, w0, cs);
    }
    __device__ __forceinline__ void block(const KeMat &ke, int d, float A[9]) const { block_t<float>(ke.k, d, A); }
    // the coupling block in FP64 from an FP64 element matrix (the exact refinement
    // residual): the same signed sums with FP64 densities and products
    __device__ __forceinline__ void block64(const KeMat64 &ke, int d, double A[9]) const {
        block_t<double>(ke.k, d, A);
    }
    // index of neighbour d in its colour plane set, and whether it is the pinned origin
    __device__ __forceinline__ unsigned nbr(const FineArgs &a, int d, int &Kn, bool &pinned) const {
        const int dx = d % 3 - 1, dy = d / 3 % 3 - 1, dz = d / 9 - 1;
        Kn = K ^ ((dx & 1) | ((dy & 1) << 1) | ((dz & 1) << 2));
        const unsigned off = X[dx + 1] + Y[dy + 1] + Z[dz + 1];
        pinned = (Kn == 7) && (off == 0u);
        return (unsigned)Kn * (unsigned)a.P + off;
    }
};

// what a thread reads for a vertex whose values count as 0 (the pinned origin)
__device__ float zero_planes[NF * FVB];

// fidx(0, v) for v < 2^32
__device__ __forceinline__ size_t fpos(unsigned v) { return (size_t)v + (size_t)(v >> 7) * ((NF - 1) * FVB); }

// bring a vertex range of a field (72 bytes a vertex, all planes) into L2
__device__ __forceinline__ void prefetch_field(const float *f, unsigned long long v0, unsigned long long v1) {
    const unsigned long long b0 = v0 * (NF * 4) & ~15ull, b1 = v1 * (NF * 4) & ~15ull;
    if (b1 > b0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global((const char *)f + b0)),
                     "r"((unsigned)(b1 - b0)));
}

// ---- vertex pairs --------------------------------------------------------------
// A CTA holds whole rows of h0 pairs, `rows` of them, on rows * h0 of its threads (a
// multiple of 32), chosen to leave the fewest threads idle.
struct PairShape {
    int rows, threads;
};
static PairShape pair_shape(int h0) {
    PairShape best = {1, (h0 + 31) / 32 * 32};
    auto use = [&](const PairShape &s) { return (double)s.rows * h0 / s.threads; };
    // up to 128 threads; up to 256 where that leaves more than 1 in 8 idle
    for (int lim = 128; lim <= 256; lim *= 2) {
        for (int r = 1; r * h0 <= lim; ++r) {
            const PairShape s = {r, (r * h0 + 31) / 32 * 32};
            if (use(s) > use(best) + 1e-9 || (use(s) > use(best) - 1e-9 && s.threads > best.threads))
                best = s;
        }
        if (use(best) >= 0.875) break;
    }
    return best;
}

// The pair (x = 2i + 1, x = 2i) of row (j, l) of the rows with colours K0 (odd x) and
// K0 + 1 (even x); lane x of every packed value is the odd vertex.
struct PairGeo {
    int K0;              // 0, 2, 4 or 6: the row's parities
    float2 rw[8];        // element densities
    int i, im, ip;       // pair index and its neighbours (periodic)
    unsigned Y[3], Z[3]; // plane offsets of the neighbour rows
    __device__ __forceinline__ PairGeo(const FineArgs &a, int k0, int ii, int j, int l) : K0(k0), i(ii) {
        const int py = ((K0 >> 1) & 1) ^ 1, pz = ((K0 >> 2) & 1) ^ 1;
        im = i == 0 ? a.h[0] - 1 : i - 1;
        ip = i + 1 == a.h[0] ? 0 : i + 1;
        const int y = 2 * j + py, z = 2 * l + pz;
        const unsigned n0 = (unsigned)a.n[0], n01 = n0 * (unsigned)a.n[1];
        const unsigned ye0 = (unsigned)(y == 0 ? a.n[1] - 1 : y - 1), ze0 = (unsigned)(z == 0 ? a.n[2] - 1 : z - 1);
        const unsigned xe = 2u * (unsigned)i, xm = i == 0 ? n0 - 1 : xe - 1;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float *row = a.rho + (n0 * ((t & 1) ? (unsigned)y : ye0) + n01 * ((t >> 1) ? (unsigned)z : ze0));
            const float em = RHO_PENAL_MIN + __ldg(row + xm), e0 = RHO_PENAL_MIN + __ldg(row + xe),
                        e1 = RHO_PENAL_MIN + __ldg(row + xe + 1);
            rw[2 * t] = make_float2(e0, em);
            rw[2 * t + 1] = make_float2(e1, e0);
        }
        int jm, jp, lm, lp;
        axis_nbrs(j, py, a.h[1], jm, jp);
        axis_nbrs(l, pz, a.h[2], lm, lp);
        const unsigned h0 = (unsigned)a.h[0], h01 = h0 * (unsigned)a.h[1];
        Y[0] = h0 * (unsigned)jm; Y[1] = h0 * (unsigned)j; Y[2] = h0 * (unsigned)jp;
        Z[0] = h01 * (unsigned)lm; Z[1] = h01 * (unsigned)l; Z[2] = h01 * (unsigned)lp;
    }
    // coupling blocks of neighbour d of both vertices (VertexGeo::block_t)
    __device__ __forceinline__ void block(const KeMat &ke, int d, float2 A[9]) const {
        const int dx = d % 3 - 1, dy = d / 3 % 3 - 1, dz = d / 9 - 1;
        const int w0 = first_shared(d);
        float2 cs[8];
        fold_signed<float2>(rw, dx, dy, dz, w0, cs);
        const int an = 7 - w0;
        const int bn = (1 - (w0 & 1) + dx) + 2 * (1 - ((w0 >> 1) & 1) + dy) + 4 * (1 - (w0 >> 2) + dz);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float k = ke.k[(3 * an + r) * 24 + 3 * bn + c];
                const float2 v = cs[(1 << r) ^ (1 << c)];
                A[3 * r + c] = make_float2(k * v.x, k * v.y);
            }
    }
    // first index of row (dy, dz) in its odd vertices' colour plane (the even ones: + P);
    // its first even vertex is the pinned origin if `origin`
    __device__ __forceinline__ unsigned row(const FineArgs &a, int dy, int dz, bool &origin) const {
        const unsigned off = Y[dy + 1] + Z[dz + 1];
        const int Kn = K0 ^ (((dy & 1) << 1) | ((dz & 1) << 2));
        origin = Kn == 6 && off == 0u;
        return (unsigned)Kn * (unsigned)a.P + off;
    }
};

// acc += A dd for the block of one neighbour (both vertices)
__device__ __forceinline__ void pair_madd(const float2 A[9], const float2 dd[3], float2 acc[3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
        acc[r] = __ffma2_rn(A[3 * r], dd[0], __ffma2_rn(A[3 * r + 1], dd[1], __ffma2_rn(A[3 * r + 2], dd[2], acc[r])));
}

// acc[3c+r] (cases cb .. cb+C-1) += the part of (K u)_v, in difference form
// sum_d A_d (u_{v+d} - u_v), of the eight neighbour rows other than the pair's own,
// u at the pinned origin counted as 0.  Equal to sum_d A_d u_{v+d} in exact arithmetic
// (the blocks of a row sum to zero), and exact for rigid translations in FP32 too, so
// the FP32 operator agrees with the FP64 difference-form residual of the refined mode
// on the near-null translation mode of the pinned problem.  nuv: -u of the pair.
// r0 .. r1-1: the rows, (dy, dz) with dy fastest.
template <int C>
__device__ __forceinline__ void pair_rows(const FineArgs &a, const KeMat &ke, const PairGeo &g, int cb,
                                          const float2 nuv[3 * C], float2 acc[3 * C], int r0, int r1) {
#pragma unroll
    for (int r = r0; r < r1; ++r) {
        const int dy = r % 3 - 1, dz = r / 3 - 1;
        bool origin;
        const unsigned ro = g.row(a, dy, dz, origin);
        const unsigned ev = ro + (unsigned)a.P;
        const float *u = a.u + 3 * cb * FVB;
        const float *po = u + fpos(ro + (unsigned)g.i), *pe = u + fpos(ev + (unsigned)g.i);
        const float *pm = u + fpos(ro + (unsigned)g.im), *pp = u + fpos(ev + (unsigned)g.ip);
        if (origin && g.i == 0) pe = zero_planes;
        if (origin && g.ip == 0) pp = zero_planes;
        float e0[3 * C], o0[3 * C];
        float2 A[9];
        g.block(ke, 3 * r, A);  // dx = -1: the odd vertex's left neighbour is e0
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float2 dd[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int q = 3 * c + m;
                e0[q] = __ldg(pe + q * FVB);
                dd[m] = make_float2(__fadd_rn(e0[q], nuv[q].x), __fadd_rn(__ldg(pm + q * FVB), nuv[q].y));
            }
            pair_madd(A, dd, acc + 3 * c);
        }
        g.block(ke, 3 * r + 1, A);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float2 dd[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int q = 3 * c + m;
                o0[q] = __ldg(po + q * FVB);
                dd[m] = make_float2(__fadd_rn(o0[q], nuv[q].x), __fadd_rn(e0[q], nuv[q].y));
            }
            pair_madd(A, dd, acc + 3 * c);
        }
        g.block(ke, 3 * r + 2, A);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float2 dd[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int q = 3 * c + m;
                const float e1 = __ldg(pp + q * FVB);
                dd[m] = make_float2(__fadd_rn(e1, nuv[q].x), __fadd_rn(o0[q], nuv[q].y));
            }
            pair_madd(A, dd, acc + 3 * c);
        }
    }
}

// thread -> pair: row block rb of the CTA, row slot and pair index; false for threads
// without one
__device__ __forceinline__ bool pair_task(const FineArgs &a, unsigned rb, int &slot, int &i, unsigned &row, int &j,
                                          int &l) {
    slot = (int)a.dh0.div(threadIdx.x);
    i = (int)threadIdx.x - slot * a.h[0];
    row = rb * (unsigned)a.rows + (unsigned)slot;
    l = (int)a.dh1.div(row);
    j = (int)row - l * a.h[1];
    return slot < a.rows && row < (unsigned)(a.h[1] * a.h[2]);
}

// the reference's component-wise block Gauss-Seidel step (x, then y, then z,
// each with the relaxed values of the earlier components) written as an
// update of u by the residual r = f - K u; rk: the reciprocals of ks's diagonal.  The
// quotients are corrected by their remainder (Markstein, IBM J. Res. Dev. 34, 1990, 111),
// which gives the division's result; the bare product is 3 to 5 % further from 64 bits
// over a sweep.  Sweep at 256^3 / 128^3 / 64^3: 2.30 / 0.329 / 0.0590 ms with the product,
// 2.34 / 0.336 / 0.0612 here, 2.44 / 0.352 / 0.0648 with divisions.
__device__ __forceinline__ float quotient(float a, float b, float rb) {
    const float q = a * rb;
    return fmaf(fmaf(-b, q, a), rb, q);
}
__device__ __forceinline__ void gs_step(const float ks[9], const float rk[3], float w, float r0, float r1, float r2,
                                        float &u0, float &u1, float &u2) {
    const float d0 = quotient(w * r0, ks[0], rk[0]);
    const float d1 = quotient(w * (r1 - ks[3] * d0), ks[4], rk[1]);
    const float d2 = quotient(w * (r2 - ks[6] * d0 - ks[7] * d1), ks[8], rk[2]);
    u0 += d0;
    u1 += d1;
    u2 += d2;
}

// Two colours of the sweep: the rows of parity K0, their odd vertices (colour K0)
// first, then, after a barrier, the even ones (colour K0 + 1), whose neighbours in the
// own row are the new odd values (handed over in shared memory).  Rows of the same
// parity are never neighbours, so the launch is the two colours' exact Gauss-Seidel
// order.  The neighbour rows' part of both vertices is formed together.  One launch per
// colour streamed all of u eight times a sweep (12 GB of DRAM traffic at 256^3) and
// fetched 17 row halves per 128 vertices from L2; this reads u four times and 18 row
// halves per 256 vertices.  Bound by load latency and issue (54-58 % of issue slots,
// 15 warps per SM, DRAM 29 % at 128^3).  Sweep at 256^3 / 128^3 / 64^3: 2.82 / 0.42 / 0.082
// ms with one colour per launch, 2.34 / 0.34 / 0.061 ms now.
// bid: the CTA's index in the design's launch; sm: 3 C x TM floats
template <int K0, int C, int TM>
__device__ __forceinline__ void fine_gs_block(const FineArgs &a, const KeMat &ke, unsigned bid) {
    __shared__ float sm[3 * C][TM];
    constexpr int NG = NCASE / C;
    const int cb = (int)(bid % NG) * C;
    int slot, i, j, l;
    unsigned row;
    const bool on = pair_task(a, bid / NG, slot, i, row, j, l);
    if (bid % NG == 0 && threadIdx.x < 10) {  // u of all colours, f of the two swept
        const unsigned r0 = (bid / NG + GS_AHEAD) * (unsigned)a.rows, rows = (unsigned)(a.h[1] * a.h[2]);
        if (r0 < rows) {
            const unsigned r1 = min(rows, r0 + (unsigned)a.rows), t = threadIdx.x, k = t < 8 ? t : K0 + t - 8;
            const unsigned long long v0 = (unsigned long long)k * a.P + r0 * (unsigned)a.h[0];
            prefetch_field(t < 8 ? a.u : a.f, v0, v0 + (r1 - r0) * (unsigned)a.h[0]);
        }
    }
    const unsigned vo = (unsigned)K0 * (unsigned)a.P + row * (unsigned)a.h[0] + (unsigned)i;
    const size_t po = fpos(vo) + 3 * cb * FVB, pe = fpos(vo + (unsigned)a.P) + 3 * cb * FVB;
    float *uo = a.u + po, *ue = a.u + pe;
    const float *fo = a.f + po, *fe = a.f + pe;
    float2 nuv[3 * C], acc[3 * C], A[9];
    const PairGeo g(a, K0, on ? i : 0, on ? j : 0, on ? l : 0);
    bool origin;
    const unsigned ro = g.row(a, 0, 0, origin);
    if (on) {
#pragma unroll
        for (int q = 0; q < 3 * C; ++q) {
            // the pinned origin counts as 0
            nuv[q] = make_float2(-uo[q * FVB], origin && i == 0 ? -0.f : -ue[q * FVB]);
            acc[q] = make_float2(0.f, 0.f);
        }
        pair_rows<C>(a, ke, g, cb, nuv, acc, 0, 4);
        pair_rows<C>(a, ke, g, cb, nuv, acc, 5, 9);
        // own row, odd vertex: the even neighbours' old values
        {
            const float *pp = a.u + fidx(3 * cb, ro + (unsigned)a.P + (unsigned)g.ip);
            float2 B[9];
            g.block(ke, 12, A);
            g.block(ke, 14, B);
            const bool z1 = origin && g.ip == 0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                float dl[3], dr[3];
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    const int q = 3 * c + m;
                    dl[m] = nuv[q].x - nuv[q].y;
                    dr[m] = (z1 ? 0.f : pp[q * FVB]) + nuv[q].x;
                }
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    float v = acc[3 * c + r].x;
                    v = fmaf(A[3 * r].x, dl[0], fmaf(A[3 * r + 1].x, dl[1], fmaf(A[3 * r + 2].x, dl[2], v)));
                    acc[3 * c + r].x = fmaf(B[3 * r].x, dr[0], fmaf(B[3 * r + 1].x, dr[1], fmaf(B[3 * r + 2].x, dr[2], v)));
                }
            }
        }
        g.block(ke, 13, A);
        float ks[9], rk[3];
#pragma unroll
        for (int e = 0; e < 9; ++e) ks[e] = A[e].x;
#pragma unroll
        for (int m = 0; m < 3; ++m) rk[m] = 1.f / ks[4 * m];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float u0 = -nuv[3 * c].x, u1 = -nuv[3 * c + 1].x, u2 = -nuv[3 * c + 2].x;
            gs_step(ks, rk, a.w, fo[3 * c * FVB] - acc[3 * c].x, fo[(3 * c + 1) * FVB] - acc[3 * c + 1].x,
                    fo[(3 * c + 2) * FVB] - acc[3 * c + 2].x, u0, u1, u2);
            sm[3 * c][threadIdx.x] = u0;
            sm[3 * c + 1][threadIdx.x] = u1;
            sm[3 * c + 2][threadIdx.x] = u2;
        }
    }
    __syncthreads();
    if (!on) return;
    const int tm = (int)threadIdx.x - i + g.im;
    float2 B[9];
    g.block(ke, 14, B);
    float ks[9], rk[3];
#pragma unroll
    for (int e = 0; e < 9; ++e) ks[e] = A[e].y;
    g.block(ke, 12, A);
#pragma unroll
    for (int m = 0; m < 3; ++m) rk[m] = 1.f / ks[4 * m];
    const bool pinned = origin && i == 0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        float dl[3], dr[3], v[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const float un = sm[3 * c + m][threadIdx.x];
            uo[(3 * c + m) * FVB] = un;
            dl[m] = sm[3 * c + m][tm] + nuv[3 * c + m].y;
            dr[m] = un + nuv[3 * c + m].y;
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            v[r] = acc[3 * c + r].y;
            v[r] = fmaf(A[3 * r].y, dl[0], fmaf(A[3 * r + 1].y, dl[1], fmaf(A[3 * r + 2].y, dl[2], v[r])));
            v[r] = fmaf(B[3 * r].y, dr[0], fmaf(B[3 * r + 1].y, dr[1], fmaf(B[3 * r + 2].y, dr[2], v[r])));
        }
        float u0 = -nuv[3 * c].y, u1 = -nuv[3 * c + 1].y, u2 = -nuv[3 * c + 2].y;
        gs_step(ks, rk, a.w, fe[3 * c * FVB] - v[0], fe[(3 * c + 1) * FVB] - v[1], fe[(3 * c + 2) * FVB] - v[2], u0, u1, u2);
        // the pinned origin stays zero (grid.cu:445-447, 545)
        ue[3 * c * FVB] = pinned ? 0.f : u0;
        ue[(3 * c + 1) * FVB] = pinned ? 0.f : u1;
        ue[(3 * c + 2) * FVB] = pinned ? 0.f : u2;
    }
}

// TM: threads per CTA at most; MB: CTAs per SM
template <int K0, int C, int TM, int MB>
__global__ void __launch_bounds__(TM, MB) k_fine_gs(FineArgs a, const __grid_constant__ KeMat ke) {
    fine_gs_block<K0, C, TM>(a, ke, blockIdx.x);
}

// Residual of all rows in one launch (there is no order between colours), the row
// parity the block index modulo 4 and a run-time value of one code body: the CTAs of
// neighbouring rows run together and read each other's rows while they are in L2.
// 256^3: 3.48 ms with one vertex per thread (2.95 to 3.06 ms without the last colour,
// which the sweep then wrote), 2.37 ms now back to back and 2.59 ms with the norms and a
// cold cache; three cases per thread or other register budgets measured 2.73 to 3.26.
// norm partials: the six weighted squared norms of every row of vertices, row
// K0/2 * (rows of a parity) + row, summed in an order that depends on the row length
// alone (the same in any launch shape and in lockstep batches).
template <int C, int TM>
__device__ __forceinline__ void fine_residual_block(const FineArgs &a, const KeMat &ke, double *partial, unsigned bid) {
    constexpr int NG = NCASE / C;
    const int K0 = (int)(bid & 3u) * 2;
    const unsigned bx = bid >> 2;
    const int cb = (int)(bx % NG) * C;
    int slot, i, j, l;
    unsigned row;
    const bool on = pair_task(a, bx / NG, slot, i, row, j, l);
    if (bx % NG == 0 && threadIdx.x < 4) {  // u and f of the row parity's two colours
        const unsigned r0 = (bx / NG + RES_AHEAD) * (unsigned)a.rows, rows = (unsigned)(a.h[1] * a.h[2]);
        if (r0 < rows) {
            const unsigned r1 = min(rows, r0 + (unsigned)a.rows), t = threadIdx.x, k = (unsigned)K0 + (t & 1);
            const unsigned long long v0 = (unsigned long long)k * a.P + r0 * (unsigned)a.h[0];
            prefetch_field(t < 2 ? a.u : a.f, v0, v0 + (r1 - r0) * (unsigned)a.h[0]);
        }
    }
    double nrm[C];
#pragma unroll
    for (int c = 0; c < C; ++c) nrm[c] = 0;
    if (on) {
        const unsigned vo = (unsigned)K0 * (unsigned)a.P + row * (unsigned)a.h[0] + (unsigned)i;
        const size_t oo = fpos(vo) + 3 * cb * FVB, oe = fpos(vo + (unsigned)a.P) + 3 * cb * FVB;
        const float *uo = a.u + oo, *ue = a.u + oe;
        const PairGeo g(a, K0, i, j, l);
        bool origin;
        const unsigned ro = g.row(a, 0, 0, origin);
        const bool pinned = origin && i == 0;
        float2 nuv[3 * C], acc[3 * C];
#pragma unroll
        for (int q = 0; q < 3 * C; ++q) {
            nuv[q] = make_float2(-__ldg(uo + q * FVB), pinned ? -0.f : -__ldg(ue + q * FVB));
            acc[q] = make_float2(0.f, 0.f);
        }
        pair_rows<C>(a, ke, g, cb, nuv, acc, 0, 4);
        {
            const float *pm = a.u + fidx(3 * cb, ro + (unsigned)g.im);
            const float *pp = a.u + fidx(3 * cb, ro + (unsigned)a.P + (unsigned)g.ip);
            const bool z1 = origin && g.ip == 0;
            float2 A[9], B[9];
            g.block(ke, 12, A);
            g.block(ke, 14, B);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                float2 dl[3], dr[3];
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    const int q = 3 * c + m;
                    dl[m] = make_float2(nuv[q].x - nuv[q].y, __ldg(pm + q * FVB) + nuv[q].y);
                    dr[m] = make_float2((z1 ? 0.f : __ldg(pp + q * FVB)) + nuv[q].x, nuv[q].y - nuv[q].x);
                }
                pair_madd(A, dl, acc + 3 * c);
                pair_madd(B, dr, acc + 3 * c);
            }
        }
        pair_rows<C>(a, ke, g, cb, nuv, acc, 5, 9);
        const int my = axis_mult(2 * j + (((K0 >> 1) & 1) ^ 1), a.n[1]) * axis_mult(2 * l + (((K0 >> 2) & 1) ^ 1), a.n[2]);
        const double mo = (double)(my * axis_mult(2 * i + 1, a.n[0])), me = (double)(my * axis_mult(2 * i, a.n[0]));
#pragma unroll
        for (int c = 0; c < C; ++c) {
            double so = 0, se = 0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int q = 3 * c + m;
                const float ro_ = a.f[oo + q * FVB] - acc[q].x;
                const float re_ = pinned ? 0.f : a.f[oe + q * FVB] - acc[q].y;
                a.r[oo + q * FVB] = ro_;
                a.r[oe + q * FVB] = re_;
                so += (double)ro_ * ro_;
                se += (double)re_ * re_;
            }
            nrm[c] = mo * so + me * se;
        }
    }
    if (!partial) return;
    __shared__ double sm[C][TM];
#pragma unroll
    for (int c = 0; c < C; ++c) sm[c][threadIdx.x] = nrm[c];
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const unsigned rows = (unsigned)(a.h[1] * a.h[2]), first = bx / NG * (unsigned)a.rows;
    for (int t = threadIdx.x >> 5; t < a.rows * C; t += nw) {
        const int rr = t / C, c = t % C;
        if (first + (unsigned)rr >= rows) continue;
        double v = 0;
        for (int e = lane; e < a.h[0]; e += 32) v += sm[c][rr * a.h[0] + e];
        v = warp_sum(v);
        if (lane == 0) partial[((long long)(K0 / 2) * rows + first + rr) * NCASE + cb + c] = v;
    }
}

template <int C, int TM, int MB>
__global__ void __launch_bounds__(TM, MB) k_fine_residual(FineArgs a, const __grid_constant__ KeMat ke,
                                                          double *partial) {
    fine_residual_block<C, TM>(a, ke, partial, blockIdx.x);
}

// thread -> (colour, vertex p of its plane, first case) of the FP64-solution residual:
// the colour the block index modulo 8, so the CTAs of one vertex block read each
// other's rows while they are in L2
template <int C>
__device__ __forceinline__ void colour_task(long long &p, int &cb, int &K, unsigned bid) {
    constexpr int NG = NCASE / C;
    K = (int)(bid % 8);
    const unsigned bx = bid / 8;
    cb = (int)(bx % NG) * C;
    p = (long long)(bx / NG) * blockDim.x + threadIdx.x;
}

// ---- refined precision: residual of an FP64 solution ----------------------------
// K u at vertex v equals sum_{d != 0} A_d (u_{v+d} - u_v), because the assembled
// blocks of a row sum to zero (Ke annihilates rigid translations).  The
// differences are taken in FP64 and are O(1) where u itself is O(N), so the
// residual floor no longer grows with the grid size.  The pinned origin enters as
// an ordinary neighbour: its value is held fixed by the correction sweeps, so a
// nonzero value only translates the solution.  EXACT accumulates the products in
// FP64 too (the FP32-product form floors near 1e-6 of ||f||, independent of N).
template <int KC, bool EXACT, int C64 = CPT64>
__device__ __forceinline__ void fine_residual64_vertex(const FineArgs &a, const KeMat &ke, const KeMat64 &ke64,
                                                       const double *__restrict__ u64, long long p, int cb,
                                                       int kr = KC) {
    const int K = KC >= 0 ? KC : kr;
    const long long me = (long long)K * a.P + p;
    if (K == 7 && p == 0) {
#pragma unroll
        for (int q = 0; q < 3 * C64; ++q) a.r[fidx(3 * cb + q, me)] = 0.f;
        return;
    }
    const VertexGeo<KC> g(a, p, K);
    const double *uvp = u64 + fidx(3 * cb, me);
    double uv[3 * C64];
#pragma unroll
    for (int q = 0; q < 3 * C64; ++q) uv[q] = __ldg(uvp + q * FVB);
    using Acc = typename std::conditional<EXACT, double, float>::type;
    Acc acc[3 * C64];
#pragma unroll
    for (int q = 0; q < 3 * C64; ++q) acc[q] = 0;
#pragma unroll
    for (int d = 0; d < 27; ++d) {
        if (d == 13) continue;
        int Kn;
        bool pinned;
        const unsigned nid = g.nbr(a, d, Kn, pinned);
        // EXACT: the block in FP64 (FP64 element matrix and densities, FP64
        // products): no per-entry FP32-to-FP64 conversions, which run on the narrow
        // conversion pipe; otherwise the FP32 block of the V-cycle operator
        Acc A[9];
        if (EXACT) {
            double A64[9];
            g.block64(ke64, d, A64);
#pragma unroll
            for (int k = 0; k < 9; ++k) A[k] = (Acc)A64[k];
        } else {
            float A32[9];
            g.block(ke, d, A32);
#pragma unroll
            for (int k = 0; k < 9; ++k) A[k] = (Acc)A32[k];
        }
        const double *up = u64 + fidx(3 * cb, nid);  // planes 3cb.. of the neighbour, FVB apart
#pragma unroll
        for (int c = 0; c < C64; ++c) {
            const Acc d0 = (Acc)(__ldg(up + (3 * c) * FVB) - uv[3 * c]);
            const Acc d1 = (Acc)(__ldg(up + (3 * c + 1) * FVB) - uv[3 * c + 1]);
            const Acc d2 = (Acc)(__ldg(up + (3 * c + 2) * FVB) - uv[3 * c + 2]);
            acc[3 * c + 0] = fma(A[0], d0, fma(A[1], d1, fma(A[2], d2, acc[3 * c + 0])));
            acc[3 * c + 1] = fma(A[3], d0, fma(A[4], d1, fma(A[5], d2, acc[3 * c + 1])));
            acc[3 * c + 2] = fma(A[6], d0, fma(A[7], d1, fma(A[8], d2, acc[3 * c + 2])));
        }
    }
#pragma unroll
    for (int q = 0; q < 3 * C64; ++q) {
        const long long o = fidx(3 * cb + q, me);
        a.r[o] = (float)((Acc)a.f[o] - acc[q]);
    }
}

// C64 load cases per thread (NCASE / C64 threads per vertex), MB CTAs per SM
template <bool EXACT, int C64 = CPT64, int MB = MINB64>
__global__ void __launch_bounds__(FBS, MB) k_fine_residual64(FineArgs a, const __grid_constant__ KeMat ke,
                                                         const __grid_constant__ KeMat64 ke64,
                                                         const double *__restrict__ u64) {
    long long p;
    int cb, K;
    colour_task<C64>(p, cb, K, blockIdx.x);  // all colours in one launch, colour-minor
    if (p >= a.P) return;
    fine_residual64_vertex<-1, EXACT, C64>(a, ke, ke64, u64, p, cb, K);
}

// f(case c) = sum_w (1e-9 + rho_w) * (Ke chi0_c)[rows of the vertex's local node in element w]
__global__ void __launch_bounds__(256) k_rhs(Planes P, const float *__restrict__ rho, float *f,
                                             const __grid_constant__ RhsTab g) {
    const long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (v >= P.nv) return;
    const int k = color_of_index(P, v);
    int x, y, z;
    vpos(P, k, v - P.base[k], x, y, z);
    const int n0 = P.n[0], n1 = P.n[1], n2 = P.n[2];
    const int xe0 = x == 0 ? n0 - 1 : x - 1, ye0 = y == 0 ? n1 - 1 : y - 1, ze0 = z == 0 ? n2 - 1 : z - 1;
    float acc[NF];
#pragma unroll
    for (int q = 0; q < NF; ++q) acc[q] = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const int ex = (w & 1) ? x : xe0, ey = ((w >> 1) & 1) ? y : ye0, ez = (w >> 2) ? z : ze0;
        const float rp = RHO_PENAL_MIN + __ldg(&rho[ex + (long long)n0 * (ey + (long long)n1 * ez)]);
        const int an = 7 - w;
#pragma unroll
        for (int c = 0; c < NCASE; ++c)
#pragma unroll
            for (int m = 0; m < 3; ++m) acc[3 * c + m] = fmaf(rp, g.g[c][3 * an + m], acc[3 * c + m]);
    }
#pragma unroll
    for (int q = 0; q < NF; ++q) f[fidx(q, v)] = acc[q];
}

static FineArgs make_args(const Level &L, const float *rho) {
    FineArgs a;
    a.rho = rho;
    a.u = L.u;
    a.f = L.f;
    a.r = L.r;
    for (int d = 0; d < 3; ++d) { a.n[d] = L.P.n[d]; a.h[d] = L.P.n[d] / 2; }
    a.nv = L.P.nv;
    a.P = L.P.nv / 8;
    a.w = 1.f;
    a.dh0 = FastDiv((unsigned)a.h[0]);
    a.dh1 = FastDiv((unsigned)a.h[1]);
    a.rows = pair_shape(a.h[0]).rows;
    return a;
}

static unsigned task_blocks(const FineArgs &a, int cpt) { return (unsigned)(((a.P + FBS - 1) / FBS) * (NCASE / cpt)); }

// row blocks of a launch over the rows of one parity, for CTAs of a.rows rows
static unsigned pair_blocks(const FineArgs &a) { return (unsigned)((a.h[1] * a.h[2] + a.rows - 1) / a.rows); }

int fine_residual_blocks(const Level &L) { return L.P.n[1] * L.P.n[2]; }

// The colour sweep in launch shape v: load cases per thread and CTAs of 128 threads
// per SM; all give the same result to the last bit (256^3 / 64^3: shape 0 2.34 / 0.061,
// 1 2.65 / 0.058, 2 2.63 / 0.067, 3 2.55 / 0.066 ms)
template <int C, int TM, int MB>
static void fine_gs_sweep(const FineArgs &a, const KeMat &ke, unsigned nt, cudaStream_t s) {
    const unsigned nb = pair_blocks(a) * (NCASE / C);
    k_fine_gs<0, C, TM, MB><<<nb, nt, 0, s>>>(a, ke);
    k_fine_gs<2, C, TM, MB><<<nb, nt, 0, s>>>(a, ke);
    k_fine_gs<4, C, TM, MB><<<nb, nt, 0, s>>>(a, ke);
    k_fine_gs<6, C, TM, MB><<<nb, nt, 0, s>>>(a, ke);
}

// CTAs of up to 128, 256 or 512 threads (pair_shape): MB, half of it (rounded down) or
// one per SM; the register budgets of longer rows differ from the shape's own
template <int C, int MB>
static void fine_gs_shape(const FineArgs &a, const KeMat &ke, cudaStream_t s) {
    const unsigned nt = (unsigned)pair_shape(a.h[0]).threads;
    if (nt <= 128) fine_gs_sweep<C, 128, MB>(a, ke, nt, s);
    else if (nt <= 256) fine_gs_sweep<C, 256, MB / 2>(a, ke, nt, s);
    else fine_gs_sweep<C, 512, 1>(a, ke, nt, s);
}

void launch_fine_gs(const Level &L, const float *rho, const KeMat &ke, float w, cudaStream_t s) {
    FineArgs a = make_args(L, rho);
    a.w = w;
    switch (L.gs_shape) {
    case 1: fine_gs_shape<6, 2>(a, ke, s); break;
    case 2: fine_gs_shape<2, 5>(a, ke, s); break;
    case 3: fine_gs_shape<3, 3>(a, ke, s); break;
    default: fine_gs_shape<3, 4>(a, ke, s); break;
    }
}

void launch_fine_gs_residual(const Level &L, const float *rho, const KeMat &ke, float w, double *norm_partial,
                             cudaStream_t s) {
    launch_fine_gs(L, rho, ke, w, s);
    launch_fine_residual(L, rho, ke, norm_partial, s);
}

void launch_fine_residual(const Level &L, const float *rho, const KeMat &ke, double *norm_partial, cudaStream_t s) {
    const FineArgs a = make_args(L, rho);
    const unsigned nb = pair_blocks(a) * (NCASE / CPT) * 4, nt = (unsigned)pair_shape(a.h[0]).threads;
    if (nt <= 128) k_fine_residual<CPT, 128, RES_MINB><<<nb, nt, 0, s>>>(a, ke, norm_partial);
    else if (nt <= 256) k_fine_residual<CPT, 256, RES_MINB / 2><<<nb, nt, 0, s>>>(a, ke, norm_partial);
    else k_fine_residual<CPT, 512, 1><<<nb, nt, 0, s>>>(a, ke, norm_partial);
}

void launch_fine_residual64(const Level &L, const float *rho, const KeMat &ke, const KeMat64 &ke64, const float *f,
                            const double *u64,
                            float *r, bool exact, cudaStream_t s) {
    FineArgs a = make_args(L, rho);
    a.f = f;
    a.r = r;
    if (exact) k_fine_residual64<true><<<task_blocks(a, CPT64) * 8, FBS, 0, s>>>(a, ke, ke64, u64);
    else k_fine_residual64<false><<<task_blocks(a, CPT64) * 8, FBS, 0, s>>>(a, ke, ke64, u64);
}

void launch_rhs(const Level &L, const float *rho, const RhsTab &g, float *f, cudaStream_t s) {
    const int bs = 256;
    k_rhs<<<(unsigned)((L.P.nv + bs - 1) / bs), bs, 0, s>>>(L.P, rho, f, g);
}

// ---- FP64 helpers of the refined mode ---------------------------------------------
// u64 += e + T (T: the pending rigid translation of each of the 18 planes, see
// k_pin_deflate); the pinned origin (colour 7, first vertex) keeps its value
// Element-wise kernels over a blocked field run in storage order, four values of one
// plane per thread (128- and 256-bit accesses); vertices v >= nv are the padding of
// the last block.  One value per thread ran at 2 to 4.7 TB/s.
constexpr int FEB = 256;
__device__ __forceinline__ bool field_quad(long long nv, long long &o, int &q, long long &v) {
    const long long t = blockIdx.x * (long long)FEB + threadIdx.x;  // quad index
    const long long c = t / (FVB / 4);                              // chunk: (vertex block, plane)
    const long long b = c / NF;
    q = (int)(c - b * NF);
    v = b * FVB + (t - c * (FVB / 4)) * 4;
    o = 4 * t;
    return v < nv;
}
static unsigned field_quad_blocks(long long nv) { return (unsigned)((field_floats(nv) / 4 + FEB - 1) / FEB); }

__global__ void __launch_bounds__(FEB) k_update64(long long nv, double *u, const float *__restrict__ e,
                                                 const double *__restrict__ T, long long pin) {
    long long o, v;
    int q;
    if (!field_quad(nv, o, q, v)) return;
    const float4 d = *reinterpret_cast<const float4 *>(e + o);
    double2 *p = reinterpret_cast<double2 *>(u + o);
    double2 a = p[0], b = p[1];
    const double t = T[q];
    if (v != pin) a.x += (double)d.x + t;
    if (v + 1 < nv && v + 1 != pin) a.y += (double)d.y + t;
    if (v + 2 < nv && v + 2 != pin) b.x += (double)d.z + t;
    if (v + 3 < nv && v + 3 != pin) b.y += (double)d.w + t;
    p[0] = a;
    p[1] = b;
}

// ---- rigid-translation deflation of the pinned problem -------------------------
// In the pinned system (rows v != origin, u_origin = 0) the rigid translation t'
// (1 on every vertex but the origin) is the lowest-energy mode: t'^T K t' is only
// the origin's 3x3 self block A_pp.  The FP16 coarse operators misjudge that tiny
// eigenvalue, and once the solution itself is small (near-uniform designs, where
// f nearly cancels) the V-cycle's error in this mode can grow from cycle to cycle.
// After every V-cycle of a solve the translation error is therefore removed
// exactly: s = sum_{v != origin} r_v = F + q with F = sum_{v != origin} f_v and
// q = sum_{d != 0} A_{p,d} u_{p+d} (because the columns of the periodic K sum to
// zero), alpha = A_pp^-1 s per case.  Instead of adding alpha to every vertex the
// shift is kept pending in T and folded into f (f_v += K_{v,p} alpha at the 26
// neighbours of the origin, F -= A_pp alpha), which is the same iteration; T joins
// the solution when it is next folded (k_update64, k_pin_fold).
// state[0..17] = F per (case, component), state[18..35] = T.
// One CTA of PIN_THREADS: thread (n, cr) with n < 26 the neighbour index (d = n,
// or n + 1 past the origin's own d = 13) and cr = 3c + r; the products of each
// neighbour are summed over d in ascending order by one thread per (c, r).
constexpr int PIN_THREADS = 26 * NF;
__device__ __forceinline__ void pin_deflate_block(const FineArgs &a, const KeMat &ke, double *state) {
    __shared__ double qpart[26][NF];
    __shared__ double al[NF];
    __shared__ double Ms[9];
    __shared__ int ok;
    const int tid = threadIdx.x;
    const int n = tid / NF, cr = tid % NF, c = cr / 3, r = cr % 3;
    const int d = n < 13 ? n : n + 1;
    const VertexGeo<7> g(a, 0);
    int Kn;
    bool pinned;
    const unsigned nid = g.nbr(a, d, Kn, pinned);
    float A[9];
    g.block(ke, d, A);
    {
        double t = 0;
        if (!pinned)
            for (int k = 0; k < 3; ++k) t += (double)A[3 * r + k] * (double)a.u[fidx(3 * c + k, nid)];
        qpart[n][cr] = t;
    }
    if (tid == 0) {
        float Af[9];
        g.block(ke, 13, Af);
        for (int k = 0; k < 9; ++k) Ms[k] = (double)Af[k];
    }
    __syncthreads();
    if (tid < NCASE) {
        const int cc = tid;
        const double *M = Ms;
        // inverse of the 3x3 self block by cofactors
        const double c00 = M[4] * M[8] - M[5] * M[7], c01 = M[5] * M[6] - M[3] * M[8], c02 = M[3] * M[7] - M[4] * M[6];
        const double det = M[0] * c00 + M[1] * c01 + M[2] * c02;
        if (cc == 0) ok = det > 0.0;
        if (det > 0.0) {  // otherwise not positive definite: leave the iterate alone
            const double inv[9] = {c00 / det, (M[2] * M[7] - M[1] * M[8]) / det, (M[1] * M[5] - M[2] * M[4]) / det,
                                   c01 / det, (M[0] * M[8] - M[2] * M[6]) / det, (M[2] * M[3] - M[0] * M[5]) / det,
                                   c02 / det, (M[1] * M[6] - M[0] * M[7]) / det, (M[0] * M[4] - M[1] * M[3]) / det};
            double sres[3];
            for (int rr = 0; rr < 3; ++rr) {
                double q = 0;
                for (int m = 0; m < 26; ++m) q += qpart[m][3 * cc + rr];
                sres[rr] = state[3 * cc + rr] + q;
            }
            double a3[3];
            for (int rr = 0; rr < 3; ++rr) a3[rr] = inv[3 * rr] * sres[0] + inv[3 * rr + 1] * sres[1] + inv[3 * rr + 2] * sres[2];
            for (int rr = 0; rr < 3; ++rr) {
                al[3 * cc + rr] = a3[rr];
                state[NF + 3 * cc + rr] += a3[rr];
                state[3 * cc + rr] -= M[3 * rr] * a3[0] + M[3 * rr + 1] * a3[1] + M[3 * rr + 2] * a3[2];
            }
        }
    }
    __syncthreads();
    if (!ok || pinned) return;
    // f at the origin's neighbours: K_{v,p} alpha = A_{p,d}^T alpha
    const double t = (double)A[r] * al[3 * c] + (double)A[3 + r] * al[3 * c + 1] + (double)A[6 + r] * al[3 * c + 2];
    float *fp = const_cast<float *>(a.f) + fidx(3 * c + r, nid);
    *fp = (float)((double)*fp + t);
}

__global__ void __launch_bounds__(PIN_THREADS) k_pin_deflate(FineArgs a, const __grid_constant__ KeMat ke,
                                                              double *state) {
    pin_deflate_block(a, ke, state);
}

// state: F = (plane sums of f) - f at the origin, T = 0
__global__ void k_pin_init(const double *__restrict__ sums, const float *__restrict__ f, long long nv, long long pin,
                           double *state) {
    const int i = threadIdx.x;
    if (i >= NF) return;
    state[i] = sums[i] - (double)f[fidx(i, pin)];
    state[NF + i] = 0.0;
}

// FP32 solutions: u += T on every vertex but the origin
__global__ void __launch_bounds__(FEB) k_pin_fold_u(long long nv, float *u, const double *__restrict__ state,
                                                    long long pin) {
    long long o, v;
    int q;
    if (!field_quad(nv, o, q, v)) return;
    float4 *p = reinterpret_cast<float4 *>(u + o);
    float4 a = *p;
    const double t = state[NF + q];
    if (v != pin) a.x = (float)((double)a.x + t);
    if (v + 1 < nv && v + 1 != pin) a.y = (float)((double)a.y + t);
    if (v + 2 < nv && v + 2 != pin) a.z = (float)((double)a.z + t);
    if (v + 3 < nv && v + 3 != pin) a.w = (float)((double)a.w + t);
    *p = a;
}

// undo the fold of T into f at the origin's neighbours, then T = 0; one thread per
// (neighbour, case, component) as in k_pin_deflate (one thread for all: 130-180 us)
__global__ void __launch_bounds__(PIN_THREADS) k_pin_restore_f(FineArgs a, const __grid_constant__ KeMat ke,
                                                               double *state) {
    __shared__ double T[NF];
    const int tid = threadIdx.x, n = tid / NF, cr = tid % NF, c = cr / 3, r = cr % 3;
    const int d = n < 13 ? n : n + 1;
    if (tid < NF) T[tid] = state[NF + tid];
    const VertexGeo<7> g(a, 0);
    int Kn;
    bool pinned;
    const unsigned nid = g.nbr(a, d, Kn, pinned);
    float A[9];
    g.block(ke, d, A);
    __syncthreads();
    if (tid < NF) state[NF + tid] = 0.0;
    if (pinned) return;
    const double t = (double)A[r] * T[3 * c] + (double)A[3 + r] * T[3 * c + 1] + (double)A[6 + r] * T[3 * c + 2];
    float *fp = const_cast<float *>(a.f) + fidx(3 * c + r, nid);
    *fp = (float)((double)*fp - t);
}

// FP32 field <-> FP64 field (both blocked; the padding holds whatever it held)
__global__ void __launch_bounds__(FEB) k_f32_to_f64(long long nv, const float *__restrict__ s, double *d) {
    long long o, v;
    int q;
    if (!field_quad(nv, o, q, v)) return;
    const float4 a = *reinterpret_cast<const float4 *>(s + o);
    double2 *p = reinterpret_cast<double2 *>(d + o);
    p[0] = make_double2((double)a.x, (double)a.y);
    p[1] = make_double2((double)a.z, (double)a.w);
}

__global__ void __launch_bounds__(FEB) k_f64_to_f32(long long nv, const double *__restrict__ s, float *d) {
    long long o, v;
    int q;
    if (!field_quad(nv, o, q, v)) return;
    const double2 *p = reinterpret_cast<const double2 *>(s + o);
    const double2 a = p[0], b = p[1];
    *reinterpret_cast<float4 *>(d + o) = make_float4((float)a.x, (float)a.y, (float)b.x, (float)b.y);
}

void launch_update64(const Level &L, double *u64, const float *e, const double *T, cudaStream_t s) {
    k_update64<<<field_quad_blocks(L.P.nv), FEB, 0, s>>>(L.P.nv, u64, e, T, L.P.base[7]);
}
void launch_pin_deflate(const Level &L, const float *rho, const KeMat &ke, double *state, cudaStream_t s) {
    k_pin_deflate<<<1, PIN_THREADS, 0, s>>>(make_args(L, rho), ke, state);
}
// level-0 f of a zero FP64 solution: f0 - K 0 = f0 on every vertex but the pinned
// origin, whose residual is 0 (what k_fine_residual64 computes for u64 = 0)
__global__ void __launch_bounds__(FEB) k_rhs_at_zero(long long nv, const float *__restrict__ f0, float *f,
                                                    long long pin) {
    long long o, v;
    int q;
    if (!field_quad(nv, o, q, v)) return;
    float4 a = *reinterpret_cast<const float4 *>(f0 + o);
    if (v == pin) a.x = 0.f;
    else if (v + 1 == pin) a.y = 0.f;
    else if (v + 2 == pin) a.z = 0.f;
    else if (v + 3 == pin) a.w = 0.f;
    *reinterpret_cast<float4 *>(f + o) = a;
}
void launch_rhs_at_zero(const Level &L, const float *f0, float *f, cudaStream_t s) {
    k_rhs_at_zero<<<field_quad_blocks(L.P.nv), FEB, 0, s>>>(L.P.nv, f0, f, L.P.base[7]);
}
void launch_pin_init(const Level &L, const double *sums, double *state, cudaStream_t s) {
    k_pin_init<<<1, 32, 0, s>>>(sums, L.f, L.P.nv, L.P.base[7], state);
}
void launch_pin_fold(const Level &L, const float *rho, const KeMat &ke, double *state, cudaStream_t s) {
    k_pin_fold_u<<<field_quad_blocks(L.P.nv), FEB, 0, s>>>(L.P.nv, L.u, state, L.P.base[7]);
    k_pin_restore_f<<<1, PIN_THREADS, 0, s>>>(make_args(L, rho), ke, state);
}
void launch_convert_field(long long nv, const float *src, double *dst, cudaStream_t s) {
    k_f32_to_f64<<<field_quad_blocks(nv), FEB, 0, s>>>(nv, src, dst);
}
void launch_convert_field(long long nv, const double *src, float *dst, cudaStream_t s) {
    k_f64_to_f32<<<field_quad_blocks(nv), FEB, 0, s>>>(nv, src, dst);
}

// ---- lockstep batches: the level 0 of several designs in one launch per step ----
// Each design owns a slice of the launch's CTAs (BatchSlices) and runs the same
// per-CTA body as its own launch would, with its CTA index inside the slice, so
// every design's fields and norm partials are those of its own launches, to the
// last bit.  A CTA copies its design's arguments to shared memory once; a design
// whose flag in `active` is 0 (converged) returns at once.  All designs of a launch
// share one CTA size, so a design's rows per CTA can differ from its own launch's.
struct FineEnt {
    FineArgs a;
    double *partial;  // the design's norm partials
    double *state;    // its deflation state
    int design;       // its index in the active flags
};
struct FineBatchTab {
    BatchSlices gs;   // CTAs of one sweep launch, three cases per thread
    BatchSlices gs2;  // the same with two cases per thread
    BatchSlices res;  // CTAs of the residual
    FineEnt e[BATCH_MAX];
};

// C cases per thread: launch shape 0 (C = 3, 4 CTAs of 128 threads per SM) or 1 (C = 2, 5)
template <int K0, int C, int TM, int MB>
__global__ void __launch_bounds__(TM, MB) k_fine_gs_batch(const FineBatchTab *__restrict__ t,
                                                        const int *__restrict__ active,
                                                        const __grid_constant__ KeMat ke) {
    __shared__ __align__(16) unsigned buf[(sizeof(FineArgs) + 3) / 4];
    const BatchSlices &sl = C == 3 ? t->gs : t->gs2;
    const int i = batch_slice(sl, blockIdx.x);
    const FineEnt &en = t->e[i];
    if (!__ldg(&active[en.design])) return;
    const FineArgs &a = stage_args(en.a, buf);
    fine_gs_block<K0, C, TM>(a, ke, blockIdx.x - __ldg(&sl.start[i]));
}

template <int TM, int MB>
__global__ void __launch_bounds__(TM, MB) k_fine_residual_batch(const FineBatchTab *__restrict__ t,
                                                              const int *__restrict__ active,
                                                              const __grid_constant__ KeMat ke) {
    __shared__ __align__(16) unsigned buf[(sizeof(FineArgs) + 3) / 4];
    const int i = batch_slice(t->res, blockIdx.x);
    const FineEnt &en = t->e[i];
    if (!__ldg(&active[en.design])) return;
    const FineArgs &a = stage_args(en.a, buf);
    fine_residual_block<CPT, TM>(a, ke, en.partial, blockIdx.x - __ldg(&t->res.start[i]));
}

// one CTA per design
__global__ void __launch_bounds__(PIN_THREADS) k_pin_deflate_batch(const FineBatchTab *__restrict__ t,
                                                                    const int *__restrict__ active,
                                                                    const __grid_constant__ KeMat ke) {
    __shared__ __align__(16) unsigned buf[(sizeof(FineArgs) + 3) / 4];
    const FineEnt &en = t->e[blockIdx.x];
    if (!__ldg(&active[en.design])) return;
    const FineArgs &a = stage_args(en.a, buf);
    pin_deflate_block(a, ke, en.state);
}

int fine_batch_create(const Level *const *lv0, const float *const *rho, double *const *partial,
                      double *const *state, const int *design, int n, bool scratch, BatchTab *out) {
    if (n < 1 || n > BATCH_MAX) return -1;
    FineBatchTab *t = new FineBatchTab();
    t->gs.n = t->gs2.n = t->res.n = n;
    t->gs.start[0] = t->gs2.start[0] = t->res.start[0] = 0;
    int hmax = 0;
    for (int i = 0; i < n; i++) hmax = lv0[i]->P.n[0] / 2 > hmax ? lv0[i]->P.n[0] / 2 : hmax;
    // one CTA size for all: 128 threads, or the longest row's (lockstep rows: h0 < 256)
    const int nt = hmax <= 128 ? 128 : 256;
    for (int i = 0; i < n; i++) {
        t->e[i].a = make_args(*lv0[i], rho[i]);
        t->e[i].a.rows = nt / t->e[i].a.h[0];
        if (scratch) t->e[i].a.u = t->e[i].a.r;
        t->e[i].partial = partial[i];
        t->e[i].state = state[i];
        t->e[i].design = design[i];
        const unsigned rb = pair_blocks(t->e[i].a);
        t->gs.start[i + 1] = t->gs.start[i] + rb * 2;
        t->gs2.start[i + 1] = t->gs2.start[i] + rb * 3;
        t->res.start[i + 1] = t->res.start[i] + rb * (NCASE / CPT) * 4;
    }
    void *d = nullptr;
    int rc = cudaMalloc(&d, sizeof(FineBatchTab)) == cudaSuccess ? 0 : -2;
    if (rc == 0 && cudaMemcpy(d, t, sizeof(FineBatchTab), cudaMemcpyHostToDevice) != cudaSuccess) rc = -2;
    if (rc == 0) {
        out->dev = d;
        out->n = n;
        out->grid[0] = t->gs.start[n];
        out->grid[1] = t->res.start[n];
        out->grid[2] = t->gs2.start[n];
        out->grid[3] = (unsigned)nt;
    } else if (d) {
        cudaFree(d);
    }
    delete t;
    return rc;
}

template <int C, int TM, int MB>
static void fine_sweep_batch(const BatchTab &t, const KeMat &ke, const int *active, bool residual, cudaStream_t s) {
    const FineBatchTab *d = static_cast<const FineBatchTab *>(t.dev);
    const unsigned g = C == 3 ? t.grid[0] : t.grid[2];
    k_fine_gs_batch<0, C, TM, MB><<<g, TM, 0, s>>>(d, active, ke);
    k_fine_gs_batch<2, C, TM, MB><<<g, TM, 0, s>>>(d, active, ke);
    k_fine_gs_batch<4, C, TM, MB><<<g, TM, 0, s>>>(d, active, ke);
    k_fine_gs_batch<6, C, TM, MB><<<g, TM, 0, s>>>(d, active, ke);
    constexpr int MR = TM == 128 ? RES_MINB : RES_MINB / 2;
    if (residual) k_fine_residual_batch<TM, MR><<<t.grid[1], TM, 0, s>>>(d, active, ke);
}

void launch_fine_sweep_batch(const BatchTab &t, const KeMat &ke, const int *active, bool residual, int shape,
                             cudaStream_t s) {
    if (t.grid[3] == 128) {
        if (shape == 1) fine_sweep_batch<2, 128, 5>(t, ke, active, residual, s);
        else fine_sweep_batch<3, 128, 4>(t, ke, active, residual, s);
    } else {
        if (shape == 1) fine_sweep_batch<2, 256, 2>(t, ke, active, residual, s);
        else fine_sweep_batch<3, 256, 2>(t, ke, active, residual, s);
    }
}

void launch_pin_deflate_batch(const BatchTab &t, const KeMat &ke, const int *active, cudaStream_t s) {
    k_pin_deflate_batch<<<t.n, PIN_THREADS, 0, s>>>(static_cast<const FineBatchTab *>(t.dev), active, ke);
}

// mean of each of the 18 planes over unique vertices, removed in place (FP64)
__global__ void __launch_bounds__(256) k_sum18_64(long long nv, const double *__restrict__ v, double *partial) {
    double s[NF];
#pragma unroll
    for (int q = 0; q < NF; ++q) s[q] = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv; i += (long long)gridDim.x * blockDim.x)
#pragma unroll
        for (int q = 0; q < NF; ++q) s[q] += v[fidx(q, i)];
    block_reduce<NF>(s, partial, blockIdx.x);
}

__global__ void __launch_bounds__(256) k_sum18_finish(const double *__restrict__ partial, int nblk, double *out) {
    double s[NF];
#pragma unroll
    for (int c = 0; c < NF; ++c) s[c] = 0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x)
#pragma unroll
        for (int c = 0; c < NF; ++c) s[c] += partial[(long long)b * NF + c];
    block_reduce<NF>(s, out, 0);
}

__global__ void k_sub_mean64(long long nv, double *v, const double *__restrict__ sum18) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const double inv = 1.0 / (double)nv;
#pragma unroll
    for (int q = 0; q < NF; ++q) v[fidx(q, i)] -= sum18[q] * inv;
}

void launch_remove_mean64(const Planes &P, double *v, double *partial, int nblk, cudaStream_t s) {
    double *tot = partial + (long long)nblk * NF;
    k_sum18_64<<<nblk, 256, 0, s>>>(P.nv, v, partial);
    k_sum18_finish<<<1, 256, 0, s>>>(partial, nblk, tot);
    k_sub_mean64<<<(unsigned)((P.nv + 255) / 256), 256, 0, s>>>(P.nv, v, tot);
}

}  // namespace h3d
