// Correlations of forward and backward DFT fields (gradient_F, hess_F) on TMA boxes.
//
// A CTA owns 32 (z) x 8 (x) cells of a plane, two z-adjacent cells a thread, and walks over
// the pairs of field sets (shot and frequency; for the Hessian also receiver). A set is
// six fields, real and imaginary parts of three components; a pair comes in four groups
// of three boxes (F re, B re, F im, B im), each group on its own mbarrier and refilled
// for the next pair as soon as the CTA has taken its derivatives, so the loads of three
// groups run while the fourth is computed.
//
// The kernels this replaces read the 156 neighbours of a cell and pair through L1, one
// cell a thread and eight planes after one another, with the derivatives in shared
// memory: latency-bound at a tenth of the copy bandwidth. Gradient of one 384x256x384
// shot, L = 3, nf = 4: 16.9 -> 6.8 ms; of 16 shots of 64^3, nf = 2: 3.7 -> 0.33 ms.
//
// Expressions and their order are gradient_F's and hess_F's: the same bits.
#pragma once
#include "ifosb_box.cuh"

namespace ifosb {

// planes of a CTA: 1 (85 KB, two CTAs per SM at up to 238 registers) 6.8 ms for 384x256x384, L = 3,
// nf = 4; 2 planes (106 KB, 128 registers with spills) 8.3, one CTA of 2 planes 7.4
constexpr int CYB = 1;
constexpr int CTHR = 16 * 8 * CYB;     // threads: 16 pairs of cells along z
constexpr int CGRP = 3 * StrSm<CYB>::VS;  // floats of a group
constexpr size_t corr_smem() { return 4 * (size_t)4 * CGRP; }

__device__ __forceinline__ float2 two(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 diff2(float b1, float2 p, float2 q, float b2, float2 r, float2 s) {
    return add2(mul2(two(b1), sub2(p, q)), mul2(two(b2), sub2(r, s)));
}
__device__ __forceinline__ float2 diff2z_up(float b1, float b2, const float *p) {
    const float2 c = ld2(p), n = ld2(p + 2);
    const float m = p[-1];
    return add2(mul2(two(b1), make_float2(c.y - c.x, n.x - c.y)), mul2(two(b2), make_float2(n.x - m, n.y - c.x)));
}
__device__ __forceinline__ float2 diff2z_dn(float b1, float b2, const float *p) {
    const float2 c = ld2(p), m = ld2(p - 2);
    const float n = p[2];
    return add2(mul2(two(b1), make_float2(c.x - m.y, c.y - c.x)), mul2(two(b2), make_float2(c.y - m.x, n - m.y)));
}
// a / h with the operator's bits: an exact reciprocal (P2), or div4's division with the
// operator for the operands it sends away
template <bool P2>
__device__ __forceinline__ float2 dvh2(float2 a, float h, float ih) {
    if constexpr (P2) return mul2(two(ih), a);
    const float2 b = two(h), ny = two(-ih), na = mul2(two(-DIV_UP), a), q0 = mul2(na, ny);
    const float2 q1 = fma2(fma2(b, q0, na), ny, q0), q = fma2(fma2(b, q1, na), ny, q1), t = mul2(two(DIV_DOWN), q);
    const float2 off = fma2(t, two(-DIV_UP), q);
    if ((__float_as_uint(off.x) | __float_as_uint(off.y)) == 0u && h >= DIV_B_MIN && h <= DIV_B_MAX) return t;
    return make_float2(__fdiv_rn(a.x, h), __fdiv_rn(a.y, h));
}

struct CorrArgs {
    Geo g;
    int hess;                  // B are receivers' fields, each met by every shot, else the shots' own
    int nshots, nrec, nf;      // nrec: receivers of the Hessian, else 1
    const float *md, *rho;     // model slots pi, u; rho (field layout)
    float fdummy[MAXNF];       // gradient: 1/(4 pi^2 f^2) as gradient_F.c:70-72; Hessian: 1/(2 pi f) as hess_F.c:72-74
    float b1, b2, rdx, rdy, rdz;
    float ihx, ihy, ihz;       // RN(1/DX) etc. (exact for power-of-two spacings)
    float *out;                // gradient or Hessian [3][NY][NX][NZ]
    double *out64;             // the gradient's FP64 sum
    // viscoelastic only: gradients with respect to taup and taus ([2][NY][NX][NZ],
    // FP64), with Phi(omega_l) = sum_m s tau_m / (1 + s tau_m), s = -i omega_l,
    // tau_m = DT / eta_m (the memory-variable relaxation of update_s_ssg.c:108-122)
    double *gradq;
    double rphi[MAXNF], iphi[MAXNF];
    int *tma_err;
};
struct CorrBox {
    CUtensorMap F, B;  // [shot or receiver][6 nf][y][x][z], one field with its halo
    CorrArgs a;
};

// Three components' centres and derivatives (dft_derivs' order) of one group.
struct Set {
    float2 c[3], d[9];
};
template <bool P2, class Args>
__device__ __forceinline__ void take(Set &s, const float *grp, const Args &a, int y, int x, int z) {
    using M = StrSm<CYB>;
    const M m(grp, 0, y, x, z);
    constexpr int I = M::vI(), J = M::vJ();
    const float b1 = a.b1, b2 = a.b2;
    const float *X = m.vx, *Y = m.vy, *Z = m.vz;
    const float2 x0 = ld2(X), y0 = ld2(Y), z0 = ld2(Z);
    s.c[0] = x0; s.c[1] = y0; s.c[2] = z0;
    s.d[0] = dvh2<P2>(diff2(b1, x0, ld2(X - I), b2, ld2(X + I), ld2(X - 2 * I)), a.rdx, a.ihx);
    s.d[1] = dvh2<P2>(diff2(b1, ld2(X + J), x0, b2, ld2(X + 2 * J), ld2(X - J)), a.rdy, a.ihy);
    s.d[2] = dvh2<P2>(diff2z_up(b1, b2, X), a.rdz, a.ihz);
    s.d[3] = dvh2<P2>(diff2(b1, ld2(Y + I), y0, b2, ld2(Y + 2 * I), ld2(Y - I)), a.rdx, a.ihx);
    s.d[4] = dvh2<P2>(diff2(b1, y0, ld2(Y - J), b2, ld2(Y + J), ld2(Y - 2 * J)), a.rdy, a.ihy);
    s.d[5] = dvh2<P2>(diff2z_up(b1, b2, Y), a.rdz, a.ihz);
    s.d[6] = dvh2<P2>(diff2(b1, ld2(Z + I), z0, b2, ld2(Z + 2 * I), ld2(Z - I)), a.rdx, a.ihx);
    s.d[7] = dvh2<P2>(diff2(b1, ld2(Z + J), z0, b2, ld2(Z + 2 * J), ld2(Z - J)), a.rdy, a.ihy);
    s.d[8] = dvh2<P2>(diff2z_dn(b1, b2, Z), a.rdz, a.ihz);
}
__device__ __forceinline__ float at2(const float2 &v, int c) { return c ? v.y : v.x; }

// gradient_F (gradient_F.c:62-139) on one cell: FP32 in the reference's order, the FP64
// sum of the same contributions, and with Q the taup / taus gradient.
template <bool Q>
struct GradCell {
    float r, pp, uu, ur, pr, g1, g2, g3;
    double sqp, squ, h1, h2, h3, qp, qs;
    __device__ void init(const CorrArgs &a, long long c, long long m, long long n) {
        const long long F = a.g.field;
        r = a.rho[c]; pp = a.md[MD_PI * F + c]; uu = a.md[MD_U * F + c];
        ur = uu / r;
        pr = (pp - 2.0f * uu) / r;
        sqp = sqrt((double)(r * pp));
        squ = sqrt((double)(r * uu));
        g1 = a.out[m]; g2 = a.out[n + m]; g3 = a.out[2 * n + m];
        h1 = a.out64[m]; h2 = a.out64[n + m]; h3 = a.out64[2 * n + m];
        qp = qs = 0.0;
        if (Q) { qp = a.gradq[m]; qs = a.gradq[n + m]; }
    }
    __device__ void add(const CorrArgs &a, int l, const Set &F, const Set &B, const Set &G, const Set &C, int z) {
        float fv[9], bv[9], fi[9], bi[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            fv[q] = at2(F.d[q], z); bv[q] = at2(B.d[q], z); fi[q] = at2(G.d[q], z); bi[q] = at2(C.d[q], z);
        }
        const float fdummy = a.fdummy[l];
        float gradlam = (fv[0] + fv[4] + fv[8]) * (bv[0] + bv[4] + bv[8]) + (fi[0] + fi[4] + fi[8]) * (bi[0] + bi[4] + bi[8]);
        gradlam = -gradlam * fdummy;
        float gradmu = 2.0f * fv[0] * bv[0] + 2.0f * fv[4] * bv[4] + 2.0f * fv[8] * bv[8] + 2.0f * fi[0] * bi[0] +
                       2.0f * fi[4] * bi[4] + 2.0f * fi[8] * bi[8] + (fv[1] + fv[3]) * (bv[1] + bv[3]) +
                       (fi[1] + fi[3]) * (bi[1] + bi[3]) + (fv[2] + fv[6]) * (bv[2] + bv[6]) +
                       (fi[2] + fi[6]) * (bi[2] + bi[6]) + (fv[5] + fv[7]) * (bv[5] + bv[7]) +
                       (fi[5] + fi[7]) * (bi[5] + bi[7]);
        gradmu = -gradmu * fdummy;
        const float gradrho = (at2(F.c[0], z) * at2(B.c[0], z) + at2(F.c[1], z) * at2(B.c[1], z) + at2(F.c[2], z) * at2(B.c[2], z)) +
                              (at2(G.c[0], z) * at2(C.c[0], z) + at2(G.c[1], z) * at2(C.c[1], z) + at2(G.c[2], z) * at2(C.c[2], z));
        const double c1 = sqp * 2.0 * (double)gradlam;
        const double c2 = -4.0 * squ * (double)gradlam + 2.0 * squ * (double)gradmu;
        const float c3 = gradrho + ur * gradmu + pr * gradlam;
        g1 = (float)((double)g1 + c1);
        g2 = (float)((double)g2 + c2);
        g3 = g3 + c3;
        h1 += c1;
        h2 += c2;
        h3 += (double)c3;
        if (Q) {
            // complex correlations C = F conj(B) of the lambda and mu terms with
            // gradient_F's factor -fdummy: its gradlam / gradmu are their real
            // parts. A modulus M(1 + tau Phi) perturbed in tau moves the misfit
            // by Re[M Phi C] (lambda part for taup; mu - 2 lambda for taus).
            const double fd = -(double)fdummy;
            const double dfr = (double)fv[0] + fv[4] + fv[8], dfi = (double)fi[0] + fi[4] + fi[8];
            const double dbr = (double)bv[0] + bv[4] + bv[8], dbi = (double)bi[0] + bi[4] + bi[8];
            const double rl = fd * (dfr * dbr + dfi * dbi), il = fd * (dfi * dbr - dfr * dbi);
            double rm = 0.0, im = 0.0;
#pragma unroll
            for (int q = 0; q < 9; q += 4) {  // xx, yy, zz
                rm += 2.0 * ((double)fv[q] * bv[q] + (double)fi[q] * bi[q]);
                im += 2.0 * ((double)fi[q] * bv[q] - (double)fv[q] * bi[q]);
            }
            const int pair[3][2] = {{1, 3}, {2, 6}, {5, 7}};  // xy, xz, yz
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double fr = (double)fv[pair[q][0]] + fv[pair[q][1]], fim = (double)fi[pair[q][0]] + fi[pair[q][1]];
                const double br = (double)bv[pair[q][0]] + bv[pair[q][1]], bim = (double)bi[pair[q][0]] + bi[pair[q][1]];
                rm += fr * br + fim * bim;
                im += fim * br - fr * bim;
            }
            rm *= fd;
            im *= fd;
            const double ph = a.rphi[l], qh = a.iphi[l];
            qp += (double)pp * (ph * rl - qh * il);
            qs += (double)uu * (ph * (rm - 2.0 * rl) - qh * (im - 2.0 * il));
        }
    }
    __device__ void store(const CorrArgs &a, long long m, long long n) const {
        a.out[m] = g1; a.out[n + m] = g2; a.out[2 * n + m] = g3;
        a.out64[m] = h1; a.out64[n + m] = h2; a.out64[2 * n + m] = h3;
        if (Q) {
            a.gradq[m] = qp;
            a.gradq[n + m] = qs;
        }
    }
};

// hess_F (hess_F.c:67-155) on one cell: the diagonal approximate Hessian from the
// forward fields and the receivers' Green's functions, accumulated in FP32 in the
// reference's order: shots, then receivers, then frequencies.
struct HessCell {
    float r, pp, uu, h1, h2, h3;
    __device__ void init(const CorrArgs &a, long long c, long long m, long long n) {
        const long long F = a.g.field;
        r = a.rho[c]; pp = a.md[MD_PI * F + c]; uu = a.md[MD_U * F + c];
        h1 = a.out[m]; h2 = a.out[n + m]; h3 = a.out[2 * n + m];
    }
    __device__ void add(const CorrArgs &a, int l, const Set &F, const Set &B, const Set &G, const Set &C, int z) {
        float fv[9], bv[9], fi[9], bi[9], f[6], b[6];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            fv[q] = at2(F.d[q], z); bv[q] = at2(B.d[q], z); fi[q] = at2(G.d[q], z); bi[q] = at2(C.d[q], z);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            f[q] = at2(F.c[q], z); f[3 + q] = at2(G.c[q], z); b[q] = at2(B.c[q], z); b[3 + q] = at2(C.c[q], z);
        }
        const float fd = a.fdummy[l];
        const float fdiv = fv[0] + fv[4] + fv[8], fidiv = fi[0] + fi[4] + fi[8];
        const float bdiv = bv[0] + bv[4] + bv[8], bidiv = bi[0] + bi[4] + bi[8];
        float relam = fidiv * bdiv + fdiv * bidiv;
        relam = fd * relam;
        float imlam = fidiv * bidiv - fdiv * bdiv;
        imlam = fd * imlam;
        float remu = 2.0f * fi[0] * bv[0] + 2.0f * fi[4] * bv[4] + 2.0f * fi[8] * bv[8] +
                     2.0f * fv[0] * bi[0] + 2.0f * fv[4] * bi[4] + 2.0f * fv[8] * bi[8] +
                     (fi[1] + fi[3]) * (bv[1] + bv[3]) + (fv[1] + fv[3]) * (bi[1] + bi[3]) +
                     (fi[2] + fi[6]) * (bv[2] + bv[6]) + (fv[2] + fv[6]) * (bi[2] + bi[6]) +
                     (fi[5] + fi[7]) * (bv[5] + bv[7]) + (fv[5] + fv[7]) * (bi[5] + bi[7]);
        remu = fd * remu;
        float immu = 2.0f * fi[0] * bi[0] + 2.0f * fi[4] * bi[4] + 2.0f * fi[8] * bi[8] -
                     2.0f * fv[0] * bv[0] - 2.0f * fv[4] * bv[4] - 2.0f * fv[8] * bv[8] +
                     (fi[1] + fi[3]) * (bi[1] + bi[3]) - (fv[1] + fv[3]) * (bv[1] + bv[3]) +
                     (fi[2] + fi[6]) * (bi[2] + bi[6]) - (fv[2] + fv[6]) * (bv[2] + bv[6]) +
                     (fi[5] + fi[7]) * (bi[5] + bi[7]) - (fv[5] + fv[7]) * (bv[5] + bv[7]);
        immu = fd * immu;
        const float rerho = (f[0] * b[0] + f[1] * b[1] + f[2] * b[2]) - (f[3] * b[3] + f[4] * b[4] + f[5] * b[5]);
        const float imrho = (f[0] * b[3] + f[1] * b[4] + f[2] * b[5]) + (f[3] * b[0] + f[4] * b[1] + f[5] * b[2]);
        const float revs = -2.0f * relam + remu;
        const float imvs = -2.0f * imlam + immu;
        const float rerho1 = rerho + relam * (pp - 2.0f * uu) / r + remu * uu / r;
        const float imrho1 = imrho + imlam * (pp - 2.0f * uu) / r + immu * uu / r;
        h1 += (relam * relam + imlam * imlam) * r * pp * 4.0f;
        h2 += (revs * revs + imvs * imvs) * 4.0f * r * uu;
        h3 += rerho1 * rerho1 + imrho1 * imrho1;
    }
    __device__ void store(const CorrArgs &a, long long m, long long n) const {
        a.out[m] = h1; a.out[n + m] = h2; a.out[2 * n + m] = h3;
    }
};

template <class Cell, bool P2>
__global__ void __launch_bounds__(CTHR, 2) k_corr(const __grid_constant__ CorrBox T) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full[4];
    const CorrArgs &a = T.a;
    const Geo &g = a.g;
    float *sm = reinterpret_cast<float *>(smem);
    const int k0 = blockIdx.x * TZ + 1, i0 = blockIdx.y * TX + 1, j0 = blockIdx.z * CYB + 1;
    const int z = (threadIdx.x & 15) * 2, x = (threadIdx.x >> 4) & 7, y = threadIdx.x >> 7;
    const int k = k0 + z, i = i0 + x, j = j0 + y;
    const int nc = i <= g.nx && j <= g.ny ? min(2, g.nz - k + 1) : 0;  // this thread's cells
    const int pairs = a.nshots * a.nrec * a.nf;
    auto issue = [&](int p, int q) {
        const int l = p % a.nf, r = p / a.nf % a.nrec, s = p / a.nf / a.nrec;
        const CUtensorMap *m = q & 1 ? &T.B : &T.F;
        const int e = (q & 1) && a.hess ? r : s, f = 6 * l + 3 * (q >> 1);
        float *d = sm + q * CGRP;
        mbar_expect_tx(&full[q], 4 * 3 * StrSm<CYB>::VN);
        tma_load5(d, m, zc(k0) - HZ, xc(i0) - 2, yc_(j0) - 1, f, e, &full[q]);
        tma_load5(d + StrSm<CYB>::VS, m, zc(k0) - HZ, xc(i0) - 1, yc_(j0) - 2, f + 1, e, &full[q]);
        tma_load5(d + 2 * StrSm<CYB>::VS, m, zc(k0) - HZ, xc(i0) - 1, yc_(j0) - 1, f + 2, e, &full[q]);
    };
    if (threadIdx.x == 0) {
        for (int q = 0; q < 4; ++q) mbar_init(&full[q], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int q = 0; q < 4; ++q) issue(0, q);
    }
    __syncthreads();
    const long long n = (long long)g.nx * g.ny * g.nz, m = ((long long)(j - 1) * g.nx + (i - 1)) * g.nz + (k - 1);
    Cell cell[2];
#pragma unroll
    for (int c = 0; c < 2; ++c)
        if (c < nc) cell[c].init(a, widx(g, j, i, k) + c, m + c, n);
    for (int p = 0; p < pairs; ++p) {
        Set set[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            bool ok = mbar_wait(&full[q], p & 1, WAIT_LIMIT_NS);
            if (!ok) atomicExch(a.tma_err, 1);
            else if (nc > 0) take<P2>(set[q], sm + q * CGRP, a, y, x, z);
            if (!__syncthreads_and(ok)) {  // no copy may still be landing when the CTA ends
                if (threadIdx.x == 0)
                    for (int w = 0; w < 4; ++w) mbar_wait(&full[w], (w < q ? p + (p + 1 < pairs) : p) & 1, WAIT_LIMIT_NS);
                return;
            }
            if (threadIdx.x == 0 && p + 1 < pairs) issue(p + 1, q);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (c < nc) cell[c].add(a, p % a.nf, set[0], set[1], set[2], set[3], c);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
        if (c < nc) cell[c].store(a, m + c, n);
}

// The time-domain kernels' zero-lag correlations of one pair of steps (TdArgs): per shot
// the two sets of running sums come as boxes, the velocities of the cell itself directly.
struct TdBox {
    CUtensorMap F, B;  // forward / adjoint running sums [shot][3][y][x][z], one field with its halo
    TdArgs a;
    int *tma_err;
};
template <bool P2>
__global__ void __launch_bounds__(CTHR, 4) k_td_corr(const __grid_constant__ TdBox T) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full[2];
    const TdArgs &a = T.a;
    const Geo &g = a.g;
    float *sm = reinterpret_cast<float *>(smem);
    const int k0 = blockIdx.x * TZ + 1, i0 = blockIdx.y * TX + 1, j0 = blockIdx.z * CYB + 1;
    const int z = (threadIdx.x & 15) * 2, x = (threadIdx.x >> 4) & 7, y = threadIdx.x >> 7;
    const int k = k0 + z, i = i0 + x, j = j0 + y;
    const int nc = i <= g.nx && j <= g.ny ? min(2, g.nz - k + 1) : 0;  // this thread's cells
    auto issue = [&](int s, int q) {
        const CUtensorMap *m = q ? &T.B : &T.F;
        float *d = sm + q * CGRP;
        mbar_expect_tx(&full[q], 4 * 3 * StrSm<CYB>::VN);
        tma_load5(d, m, zc(k0) - HZ, xc(i0) - 2, yc_(j0) - 1, 0, s, &full[q]);
        tma_load5(d + StrSm<CYB>::VS, m, zc(k0) - HZ, xc(i0) - 1, yc_(j0) - 2, 1, s, &full[q]);
        tma_load5(d + 2 * StrSm<CYB>::VS, m, zc(k0) - HZ, xc(i0) - 1, yc_(j0) - 1, 2, s, &full[q]);
    };
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; ++q) mbar_init(&full[q], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int q = 0; q < 2; ++q) issue(0, q);
    }
    __syncthreads();
    const long long n = (long long)g.nx * g.ny * g.nz, F = g.field, m = ((long long)(j - 1) * g.nx + (i - 1)) * g.nz + (k - 1);
    const long long c = widx(g, j, i, k);
    double kr[2] = {0.0, 0.0}, kl[2] = {0.0, 0.0}, km[2] = {0.0, 0.0}, old[3][2];
#pragma unroll
    for (int w = 0; w < 2; ++w)  // on their way while the boxes land
        if (w < nc) { old[0][w] = a.k[m + w]; old[1][w] = a.k[n + m + w]; old[2][w] = a.k[2 * n + m + w]; }
    for (int s = 0; s < a.nshots; ++s) {
        float2 vf[3], vb[3];
        if (nc > 0) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                vf[q] = ld2(a.seg + (long long)s * a.seg_shot + q * F + c);
                vb[q] = ld2(a.st + (long long)s * a.st_shot + q * F + c);
            }
        }
        Set set[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            bool ok = mbar_wait(&full[q], s & 1, WAIT_LIMIT_NS);
            if (!ok) atomicExch(T.tma_err, 1);
            else if (nc > 0) take<P2>(set[q], sm + q * CGRP, a, y, x, z);
            if (!__syncthreads_and(ok)) {  // no copy may still be landing when the CTA ends
                if (threadIdx.x == 0)
                    for (int w = 0; w < 2; ++w) mbar_wait(&full[w], (w < q ? s + (s + 1 < a.nshots) : s) & 1, WAIT_LIMIT_NS);
                return;
            }
            if (threadIdx.x == 0 && s + 1 < a.nshots) issue(s + 1, q);
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            if (w >= nc) continue;
            float fu[9], bu[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                fu[q] = at2(set[0].d[q], w);
                bu[q] = at2(set[1].d[q], w);
            }
            kr[w] += (double)at2(vf[0], w) * at2(vb[0], w) + (double)at2(vf[1], w) * at2(vb[1], w) +
                     (double)at2(vf[2], w) * at2(vb[2], w);
            kl[w] += ((double)fu[0] + fu[4] + fu[8]) * ((double)bu[0] + bu[4] + bu[8]);
            km[w] += 2.0 * ((double)fu[0] * bu[0] + (double)fu[4] * bu[4] + (double)fu[8] * bu[8]) +
                     ((double)fu[1] + fu[3]) * ((double)bu[1] + bu[3]) + ((double)fu[2] + fu[6]) * ((double)bu[2] + bu[6]) +
                     ((double)fu[5] + fu[7]) * ((double)bu[5] + bu[7]);
        }
    }
#pragma unroll
    for (int w = 0; w < 2; ++w)
        if (w < nc) {
            a.k[m + w] = old[0][w] + kr[w];
            a.k[n + m + w] = old[1][w] + kl[w];
            a.k[2 * n + m + w] = old[2][w] + km[w];
        }
}

}  // namespace ifosb
