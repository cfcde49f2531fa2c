// The time step on quads: the update of the four z-adjacent cells a thread owns, and
// the kernels that read their neighbours straight from global memory. (The box
// kernels, ifosb_box.cuh, stage them in shared memory and share the update.)
//
// Every expression keeps the reference's operand order and promotions.
#pragma once
#include "ifosb_kernels.cuh"
#include "ifosb_quad.cuh"

namespace ifosb {

constexpr int QTHR = 128;      // threads per block, at most
constexpr int QZ = 8, QX = 8;  // quads along z and rows of a block, at most

// This thread's place in its block: quad (cells k..k+3), row i, first plane j.
struct Quad {
    int k, i, j, j1, dj, s, yc;
    int ncell;  // cells of the quad inside the grid (>= 4: all)
    bool active;
};
__device__ __forceinline__ Quad quad_of(const Geo &g, int yb) {
    Quad q;
    const int nq = g.bz / 4, z = threadIdx.x % nq, t = threadIdx.x / nq, x = t % g.by;
    q.k = blockIdx.x * g.bz + 4 * z + 1;
    q.i = blockIdx.y * g.by + x + 1;
    q.yc = blockIdx.z % g.nyc;
    q.s = blockIdx.z / g.nyc;
    q.j = q.yc * g.cy + t / g.by + 1;
    q.j1 = min((q.yc + 1) * g.cy, g.ny);
    q.dj = yb;
    q.ncell = g.nz - q.k + 1;
    q.active = q.ncell > 0 && q.i <= g.nx;
    return q;
}

// One CPML recursion on a quad: psi' = b psi + a d, d' = d / K + psi'.
__device__ __forceinline__ F4 pml4(F4 d, F4 old, float *psi, F4 K, F4 NRK, F4 A, F4 B, bool fast) {
    const F4 v = B * old + A * d;
    st4(psi, v);
    return div4(d, K, NRK, fast) + v;
}
__device__ __forceinline__ F4 pml4(F4 d, F4 old, float *psi, float K, float NRK, float A, float B, bool fast) {
    return pml4(d, old, psi, f4(K), f4(NRK), f4(A), f4(B), fast);
}

// Which of the quad's cells lie in a z face of the CPML frame (bit c: cell k+c).
__device__ __forceinline__ int face_z_mask(const Geo &g, int k) {
    int m = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (k + c <= g.nz && face_z(g, k + c)) m |= 1 << c;
    return m;
}
// the quad's word in a z slab (it never holds cells of both faces: see pzw)
__device__ __forceinline__ long long szq(const Geo &g, int j, int i, int k) {
    return ((long long)(j - 1) * g.nx + (i - 1)) * g.pzw + (k - 1) + (k > g.fw ? g.zfo : 0);
}

// The quad's place in the CPML frame. Its PML memories are asked for before the update
// (prefetch into L1, no registers) and read when their axis is done: held in registers
// from the start, up to nine words a thread, they cost the velocity kernel a fifth of
// its time at 256^3 (128 registers with spills against 115 without).
struct Psi {
    int hx, hy, zm;
    float *px, *py, *pz;
};
__device__ __forceinline__ void prefetch3(const float *p, long long d) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p + d));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 2 * d));
}
__device__ __forceinline__ void psi_find(Psi &q, const Geo &g, const Slabs &sl, float *ps, int j, int i, int k) {
    q.hx = face_x(g, i);
    q.hy = face_y(g, j);
    q.zm = face_z_mask(g, k);
    if (q.hx) {
        q.px = ps + sxi(g, j, q.hx, k);
        prefetch3(q.px, sl.sx);
    }
    if (q.hy) {
        q.py = ps + 3 * sl.sx + syi(g, q.hy, i, k);
        prefetch3(q.py, sl.sy);
    }
    if (q.zm) {
        q.pz = ps + 3 * sl.sx + 3 * sl.sy + szq(g, j, i, k);
        prefetch3(q.pz, sl.sz);
    }
}
// An axis's three memories, read together (a load after a recursion's store waits for it).
struct Psi3 {
    F4 v[3];
    __device__ Psi3(const float *p, long long d) : v{ld4(p), ld4(p + d), ld4(p + 2 * d)} {}
};

// The point forces on a quad's velocities, in list order. pass < 0: the frame's cells
// before their update; pass 0, 1: after it (an interior cell takes one forward pass,
// two adjoint ones; a frame cell one adjoint pass: update_v_ssg_CPML.c:384-393).
template <bool BACK>
__device__ __forceinline__ void quad_points(const VelArgs &a, F4 (&v)[3], int p0, int p1, int j, int i, int k, int nt,
                                            bool row_frame, int zmask, int pass) {
    const long long F = a.g.field;
    for (int q = p0; q < p1; ++q) {
        const Pt pt = a.pts[q];
        const int c = pt.k - k;
        if (pt.j != j || pt.i != i || c < 0 || c > 3) continue;
        const bool frame = row_frame || ((zmask >> c) & 1);
        if (pass < 0 ? !frame : pass >= (frame ? (BACK ? 1 : 0) : (BACK ? 2 : 1))) continue;
        float add[3] = {0.f, 0.f, 0.f};
        double add5[3] = {0.0, 0.0, 0.0};
        int on = 0;  // bit n: component n takes add; 8: all take add5
        if (BACK) {
            const float *s = a.val + (long long)pt.row * a.val_row + (nt - 1);
            add[0] = s[0]; add[1] = s[a.val_comp]; add[2] = s[2 * a.val_comp];
            on = 7;
        } else {
            const float amp = a.val[(long long)pt.row * a.val_row + (nt - 1)];
            const long long m = widx(a.g, j, i, pt.k);
            if (pt.kind == 2) { add[0] = amp * a.md[MD_RIP * F + m]; on = 1; }
            if (pt.kind == 3) { add[2] = amp * a.md[MD_RJP * F + m]; on = 4; }  // rjp for vz as in the reference
            if (pt.kind == 4) { add[1] = amp * a.md[MD_RKP * F + m]; on = 2; }  // rkp for vy as in the reference
            if (pt.kind == 5) {
                add5[0] = a.cf5x * (double)amp; add5[1] = a.cf5y * (double)amp; add5[2] = a.cf5z * (double)amp;
                on = 8;
            }
        }
#pragma unroll
        for (int n = 0; n < 3; ++n)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                if (cc == c) {
                    if (on == 8) set4(v[n], cc, (float)((double)get4(v[n], cc) + add5[n]));
                    else if (on & (1 << n)) set4(v[n], cc, get4(v[n], cc) + add[n]);
                }
    }
}

// Where an update reads its fields: the quad's word of each, and the strides to its x
// and y neighbours. Global memory has one pair of strides; a box has its own per field.
struct VelGlobal {
    const float *xx, *yy, *zz, *xy, *yz, *xz, *rh, *v;
    long long I, J, F;
    __device__ long long xxI() const { return I; }
    __device__ long long xzI() const { return I; }
    __device__ long long xyI() const { return I; }
    __device__ long long xyJ() const { return J; }
    __device__ long long yyJ() const { return J; }
    __device__ long long yzJ() const { return J; }
    __device__ long long rhI() const { return I; }
    __device__ long long rhJ() const { return J; }
    __device__ long long vF() const { return F; }
    static __device__ F4 ld(const float *p) { return ldg4(p); }
};

// Velocity update of one quad: update_v_ssg.c:102-127, update_v_ssg_CPML.c, and the
// point forces of update_v_ssg.c:474-522.
template <bool BACK, class S>
__device__ __forceinline__ void vel_quad(const VelArgs &a, const S &m, Psi &q, int nt, int s, int j, int i, int k, int ncell,
                                         int p0, int p1) {
    const Geo &g = a.g;
    const long long F = g.field;
    const float *cg = a.cpg, *cz = cg + CZ0 + (k - 1);
    const float b1 = a.b1, b2 = a.b2, dx = a.dxr, dy = a.dyr, dz = a.dzr;
    const bool fast = a.fast_div != 0;
    F4 v[3] = {ld4(m.v), ld4(m.v + m.vF()), ld4(m.v + 2 * m.vF())};
    const F4 xy0 = S::ld(m.xy), yz0 = S::ld(m.yz);
    F4 sxx_x = dx * diff4(b1, S::ld(m.xx + m.xxI()), S::ld(m.xx), b2, S::ld(m.xx + 2 * m.xxI()), S::ld(m.xx - m.xxI()));
    F4 sxy_y = dy * diff4(b1, xy0, S::ld(m.xy - m.xyJ()), b2, S::ld(m.xy + m.xyJ()), S::ld(m.xy - 2 * m.xyJ()));
    F4 sxz_z = dz * diffz_dn(b1, b2, m.xz);
    F4 syy_y = dy * diff4(b1, S::ld(m.yy + m.yyJ()), S::ld(m.yy), b2, S::ld(m.yy + 2 * m.yyJ()), S::ld(m.yy - m.yyJ()));
    F4 sxy_x = dx * diff4(b1, xy0, S::ld(m.xy - m.xyI()), b2, S::ld(m.xy + m.xyI()), S::ld(m.xy - 2 * m.xyI()));
    F4 syz_z = dz * diffz_dn(b1, b2, m.yz);
    F4 szz_z = dz * diffz_up(b1, b2, m.zz);
    F4 sxz_x = dx * diff4(b1, S::ld(m.xz), S::ld(m.xz - m.xzI()), b2, S::ld(m.xz + m.xzI()), S::ld(m.xz - 2 * m.xzI()));
    F4 syz_y = dy * diff4(b1, yz0, S::ld(m.yz - m.yzJ()), b2, S::ld(m.yz + m.yzJ()), S::ld(m.yz - 2 * m.yzJ()));
    if (q.hx) {
        const Psi3 o(q.px, a.sl.sx);
        const int h = q.hx;
        const float K = CPG(cg, K_X, h), RK = CPG(cg, RK_X, h), A = CPG(cg, A_X, h), B = CPG(cg, B_X, h);
        sxx_x = pml4(sxx_x, o.v[0], q.px, CPG(cg, KH_X, h), CPG(cg, RKH_X, h), CPG(cg, AH_X, h), CPG(cg, BH_X, h), fast);
        sxy_x = pml4(sxy_x, o.v[1], q.px + a.sl.sx, K, RK, A, B, fast);
        sxz_x = pml4(sxz_x, o.v[2], q.px + 2 * a.sl.sx, K, RK, A, B, fast);
    }
    if (q.hy) {
        const Psi3 o(q.py, a.sl.sy);
        const int h = q.hy;
        const float K = CPG(cg, K_Y, h), RK = CPG(cg, RK_Y, h), A = CPG(cg, A_Y, h), B = CPG(cg, B_Y, h);
        sxy_y = pml4(sxy_y, o.v[0], q.py, K, RK, A, B, fast);
        syy_y = pml4(syy_y, o.v[1], q.py + a.sl.sy, CPG(cg, KH_Y, h), CPG(cg, RKH_Y, h), CPG(cg, AH_Y, h), CPG(cg, BH_Y, h), fast);
        syz_y = pml4(syz_y, o.v[2], q.py + 2 * a.sl.sy, K, RK, A, B, fast);
    }
    if (q.zm) {
        const Psi3 o(q.pz, a.sl.sz);
        const F4 K = ldg4(cz + Z_K * g.pz), RK = ldg4(cz + Z_RK * g.pz), A = ldg4(cz + Z_A * g.pz), B = ldg4(cz + Z_B * g.pz);
        sxz_z = sel4(q.zm, pml4(sxz_z, o.v[0], q.pz, K, RK, A, B, fast), sxz_z);
        syz_z = sel4(q.zm, pml4(syz_z, o.v[1], q.pz + a.sl.sz, K, RK, A, B, fast), syz_z);
        szz_z = sel4(q.zm, pml4(szz_z, o.v[2], q.pz + 2 * a.sl.sz, ldg4(cz + Z_KH * g.pz), ldg4(cz + Z_RKH * g.pz),
                                ldg4(cz + Z_AH * g.pz), ldg4(cz + Z_BH * g.pz), fast), szz_z);
    }
    // av_mat's averaged densities (av_mat.c:63-65) from rho and its +1 neighbours; its
    // double product with 0.5, rounded, is the float product
    const F4 r0 = S::ld(m.rh);
    const F4 rb[3] = {0.5f * (r0 + S::ld(m.rh + m.rhI())), 0.5f * (r0 + S::ld(m.rh + m.rhJ())),
                      0.5f * (r0 + f4(r0.a.y, r0.b.x, r0.b.y, m.rh[4]))};
    const F4 ny[3] = {nrcp4(rb[0]), nrcp4(rb[1]), nrcp4(rb[2])};
    F4 d[3] = {sxx_x + sxy_y + sxz_z, syy_y + sxy_x + syz_z, szz_z + sxz_x + syz_y};
    div4<3>(d, rb, ny, fast);
    // the frame takes its point forces before the update (update_v() runs first)
    const bool rf = q.hx || q.hy;
    if (p1 > p0) quad_points<BACK>(a, v, p0, p1, j, i, k, nt, rf, q.zm, -1);
#pragma unroll
    for (int n = 0; n < 3; ++n) v[n] = v[n] + d[n];
    if (p1 > p0) {
        quad_points<BACK>(a, v, p0, p1, j, i, k, nt, rf, q.zm, 0);
        if (BACK) quad_points<BACK>(a, v, p0, p1, j, i, k, nt, rf, q.zm, 1);
    }
    float *V = a.vout + (long long)s * a.vout_shot + widx(g, j, i, k);
    st4n(V + VX * F, v[0], ncell);
    st4n(V + VY * F, v[1], ncell);
    st4n(V + VZ * F, v[2], ncell);
    if (a.u) {
        // U += v DT beside the update: one pass over U instead of a launch that reads the
        // velocities again and, for a segment, writes what it has just read
        float *U = a.u + (long long)s * 3 * F + widx(g, j, i, k);
        const F4 u[3] = {ld4(U) + a.dt * v[0], ld4(U + F) + a.dt * v[1], ld4(U + 2 * F) + a.dt * v[2]};
        float *G = a.useg ? a.useg + (long long)s * a.useg_shot + widx(g, j, i, k) : nullptr;
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            st4n(U + n * F, u[n], ncell);
            if (G) {
                st4n(G + n * F, v[n], ncell);
                st4n(G + (3 + n) * F, u[n], ncell);
            }
        }
    }
    if (j == a.probe_j && i == a.probe_i && a.probe_k >= k && a.probe_k < k + 4) {
#pragma unroll
        for (int n = 0; n < 4; ++n)
            if (k + n == a.probe_k && isnan(get4(v[1], n))) atomicMin(a.err_step + s, nt);
    }
}

template <bool BACK>
__global__ void __launch_bounds__(QTHR, 4) k_velocity(const __grid_constant__ VelArgs a, int nt, int yb) {
    const Geo &g = a.g;
    const Quad Q = quad_of(g, yb);
    if (!Q.active) return;
    int p0, p1;
    block_points(a.pt_off, g, Q.s, Q.yc, p0, p1);
    const long long F = g.field;
    const float *st = a.st + (long long)Q.s * a.st_shot;
    for (int j = Q.j; j <= Q.j1; j += Q.dj) {
        const long long c = widx(g, j, Q.i, Q.k);
        Psi q;
        psi_find(q, g, a.sl, a.psi + (long long)Q.s * a.psi_shot, j, Q.i, Q.k);
        const float *p = st + c;
        const VelGlobal m{p + SXX * F, p + SYY * F, p + SZZ * F, p + SXY * F, p + SYZ * F, p + SXZ * F, a.rho + c,
                          a.vin + (long long)Q.s * a.vin_shot + c, g.pz, g.plane, F};
        vel_quad<BACK>(a, m, q, nt, Q.s, j, Q.i, Q.k, Q.ncell, p0, p1);
    }
}

// ---------------------------------------------------------------------------
// Stress update and the rest of the time step, in the reference's order:
//   1. update_s_elastic / update_s (L mechanisms) with the CPML psi recursions
//      (update_s_ssg_elastic.c:106-140, update_s_ssg.c:150-230,
//       update_s_ssg_CPML(_elastic).c)
//   2. psource (psource.c:38-52)
//   3. surface_elastic / surface at j=1 (surface_ssg_elastic.c:69-111,
//      surface_ssg.c:117-160), mirror rows j=0,-1 written by the j=1..3 cells
//   4. seismo (seismo_ssg.c:43-50)
// (discfourier, which reads the velocities only, is k_dft.)
template <bool P2>
__device__ __forceinline__ F4 dvs(F4 x, float h, float ih, bool fast) {
    if constexpr (P2) return ih * x;
    else return div4(x, f4(h), f4(-ih), fast);
}
// (float)((double)x * s), the reference's promotion of a modulus times (1.0 + L tau)
__device__ __forceinline__ F4 scale_d(F4 x, double s) {
    return f4((float)((double)x.a.x * s), (float)((double)x.a.y * s), (float)((double)x.b.x * s), (float)((double)x.b.y * s));
}
// the same with a relaxation time per cell
template <int L>
__device__ __forceinline__ F4 scale_t(F4 x, F4 tau) {
    const float Lf = (float)L;
    return f4((float)((double)x.a.x * (1.0 + (double)(Lf * tau.a.x))), (float)((double)x.a.y * (1.0 + (double)(Lf * tau.a.y))),
              (float)((double)x.b.x * (1.0 + (double)(Lf * tau.b.x))), (float)((double)x.b.y * (1.0 + (double)(Lf * tau.b.y))));
}

struct StrGlobal {
    const float *vx, *vy, *vz;  // the quad's velocities
    const float *sg;            // sigma and memory variables from slot SYY, F apart
    const float *md;            // model slots from MD_PI, F apart
    long long I, J, F;
    __device__ long long vI() const { return I; }
    __device__ long long vJ() const { return J; }
    __device__ long long sF() const { return F; }
    __device__ long long mF() const { return F; }
    static __device__ F4 ldv(const float *p) { return ldg4(p); }
};

template <int L, bool P2, class S>
__device__ __forceinline__ void str_quad(const StrArgs &a, const S &m, Psi &pq, int nt, int sample, int s, int j, int i,
                                         int k, int ncell, int p0, int p1) {
    const Geo &g = a.g;
    const long long F = g.field, dJ = g.plane;
    const float *cg = a.cpg, *cz = cg + CZ0 + (k - 1);
    const float b1 = a.b1, b2 = a.b2, DT = a.dt;
    const bool fast = a.fast_div != 0;
    const long long c = widx(g, j, i, k);
    const float *vx = m.vx, *vy = m.vy, *vz = m.vz;
    const auto vI = m.vI(), vJ = m.vJ(), sF = m.sF(), mF = m.mF();
    const F4 vx0 = S::ldv(vx), vy0 = S::ldv(vy), vz0 = S::ldv(vz);
    F4 vxx = dvs<P2>(diff4(b1, vx0, S::ldv(vx - vI), b2, S::ldv(vx + vI), S::ldv(vx - 2 * vI)), a.rdx, a.idx, fast);
    F4 vxy = dvs<P2>(diff4(b1, S::ldv(vx + vJ), vx0, b2, S::ldv(vx + 2 * vJ), S::ldv(vx - vJ)), a.rdy, a.idy, fast);
    F4 vxz = dvs<P2>(diffz_up(b1, b2, vx), a.rdz, a.idz, fast);
    F4 vyx = dvs<P2>(diff4(b1, S::ldv(vy + vI), vy0, b2, S::ldv(vy + 2 * vI), S::ldv(vy - vI)), a.rdx, a.idx, fast);
    F4 vyy = dvs<P2>(diff4(b1, vy0, S::ldv(vy - vJ), b2, S::ldv(vy + vJ), S::ldv(vy - 2 * vJ)), a.rdy, a.idy, fast);
    F4 vyz = dvs<P2>(diffz_up(b1, b2, vy), a.rdz, a.idz, fast);
    F4 vzx = dvs<P2>(diff4(b1, S::ldv(vz + vI), vz0, b2, S::ldv(vz + 2 * vI), S::ldv(vz - vI)), a.rdx, a.idx, fast);
    F4 vzy = dvs<P2>(diff4(b1, S::ldv(vz + vJ), vz0, b2, S::ldv(vz + 2 * vJ), S::ldv(vz - vJ)), a.rdy, a.idy, fast);
    F4 vzz = dvs<P2>(diffz_dn(b1, b2, vz), a.rdz, a.idz, fast);
    const bool surf = g.free_surf && j == 1;
    // the free surface works on the plain derivatives (surface_ssg_elastic.c:91-93)
    F4 hor, svyy;
    if (surf) {
        hor = vxx + vzz;
        svyy = vyy;
    }
    if (pq.hx) {
        const Psi3 o(pq.px, a.sl.sx);
        const int h = pq.hx;
        const float KH = CPG(cg, KH_X, h), RKH = CPG(cg, RKH_X, h), AH = CPG(cg, AH_X, h), BH = CPG(cg, BH_X, h);
        vxx = pml4(vxx, o.v[0], pq.px, CPG(cg, K_X, h), CPG(cg, RK_X, h), CPG(cg, A_X, h), CPG(cg, B_X, h), fast);
        vyx = pml4(vyx, o.v[1], pq.px + a.sl.sx, KH, RKH, AH, BH, fast);
        vzx = pml4(vzx, o.v[2], pq.px + 2 * a.sl.sx, KH, RKH, AH, BH, fast);
    }
    if (pq.hy) {
        const Psi3 o(pq.py, a.sl.sy);
        const int h = pq.hy;
        const float KH = CPG(cg, KH_Y, h), RKH = CPG(cg, RKH_Y, h), AH = CPG(cg, AH_Y, h), BH = CPG(cg, BH_Y, h);
        vxy = pml4(vxy, o.v[0], pq.py, KH, RKH, AH, BH, fast);
        vyy = pml4(vyy, o.v[1], pq.py + a.sl.sy, CPG(cg, K_Y, h), CPG(cg, RK_Y, h), CPG(cg, A_Y, h), CPG(cg, B_Y, h), fast);
        vzy = pml4(vzy, o.v[2], pq.py + 2 * a.sl.sy, KH, RKH, AH, BH, fast);
    }
    if (pq.zm) {
        const Psi3 o(pq.pz, a.sl.sz);
        const F4 KH = ldg4(cz + Z_KHS * g.pz), RKH = ldg4(cz + Z_RKHS * g.pz), AH = ldg4(cz + Z_AH * g.pz), BH = ldg4(cz + Z_BH * g.pz);
        vxz = sel4(pq.zm, pml4(vxz, o.v[0], pq.pz, KH, RKH, AH, BH, fast), vxz);
        vyz = sel4(pq.zm, pml4(vyz, o.v[1], pq.pz + a.sl.sz, KH, RKH, AH, BH, fast), vyz);
        vzz = sel4(pq.zm, pml4(vzz, o.v[2], pq.pz + 2 * a.sl.sz, ldg4(cz + Z_KS * g.pz), ldg4(cz + Z_RKS * g.pz),
                               ldg4(cz + Z_A * g.pz), ldg4(cz + Z_B * g.pz), fast), vzz);
    }
    const F4 vxyyx = vxy + vyx, vyzzy = vyz + vzy, vxzzx = vxz + vzx;
    const F4 vxxyyzz = vxx + vyy + vzz, vyyzz = vyy + vzz, vxxzz = vxx + vzz, vxxyy = vxx + vyy;
    const float *md = m.md, *sg = m.sg;
    const F4 pim = ld4(md + MD_PI * mF), um = ld4(md + MD_U * mF);
    float *S0 = a.st + (long long)s * a.st_shot + c;  // the results' place
    F4 sxx, syy, szz;
    F4 sxy = ld4(sg + (SXY - SYY) * sF), syz = ld4(sg + (SYZ - SYY) * sF), sxz = ld4(sg + (SXZ - SYY) * sF);
    // ---- 1. stress (and memory variables) -----------------------------------
    F4 taus, taup, srx, srz;
    if constexpr (L == 0) {
        const F4 f = 2.f * um, gt = pim * vxxyyzz;
        sxy = sxy + (DT * ld4(md + MD_UIPJP * mF)) * vxyyx;
        syz = syz + (DT * ld4(md + MD_UJPKP * mF)) * vyzzy;
        sxz = sxz + (DT * ld4(md + MD_UIPKP * mF)) * vxzzx;
        sxx = ld4(sg + (SXX - SYY) * sF) + DT * (gt - f * vyyzz);
        syy = ld4(sg) + DT * (gt - f * vxxzz);
        szz = ld4(sg + (SZZ - SYY) * sF) + DT * (gt - f * vxxyy);
    } else {
        const float dth = a.dthalbe;
        const bool ut = a.unif_tau != 0;
        const float *R = sg + 6 * sF;
        float *RO = S0 + NEL * F;
        // shear: one component at a time, its mechanisms' old and new sums
        auto shear = [&](F4 t, F4 e, int slot, int tslot, int q) {
            const F4 mu = ld4(md + slot * mF);
            const F4 tau = ut ? f4(a.uts_avg) : ld4(md + tslot * mF);
            const F4 f = ut ? scale_d(DT * mu, 1.0 + (double)((float)L * a.uts_avg)) : scale_t<L>(DT * mu, tau);
            F4 so, sn;
#pragma unroll
            for (int l = 0; l < L; ++l) {
                const F4 r = ld4(R + (6 * l + q) * sF);
                const F4 n = a.mb[l] * (a.mc[l] * r - (a.eta[l] * mu * tau) * e);
                st4n(RO + (6 * l + q) * F, n, ncell);
                so = l == 0 ? r : so + r;
                sn = l == 0 ? n : sn + n;
            }
            return (t + (f * e + dth * so)) + dth * sn;
        };
        sxy = shear(sxy, vxyyx, MD_UIPJP, MD_TSIPJP, 3);
        syz = shear(syz, vyzzy, MD_UJPKP, MD_TSJPKP, 4);
        sxz = shear(sxz, vxzzx, MD_UIPKP, MD_TSIPKP, 5);
        taus = ut ? f4(a.utaus) : ld4(md + MD_TAUS * mF);
        taup = ut ? f4(a.utaup) : ld4(md + MD_TAUP * mF);
        const F4 gg = ut ? scale_d(pim, 1.0 + (double)((float)L * a.utaup)) : scale_t<L>(pim, taup);
        const F4 f = ut ? scale_d(2.f * um, 1.0 + (double)((float)L * a.utaus)) : scale_t<L>(2.f * um, taus);
        F4 o[3], n[3];
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const F4 e = a.eta[l] * pim * taup, u2 = 2.f * um, et = e * vxxyyzz;
            F4 d;  // ((2.0 um) eta) taus in double, rounded once
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                set4(d, cc, (float)(((double)get4(u2, cc) * (double)a.eta[l]) * (double)get4(taus, cc)));
            const F4 pr[3] = {vyyzz, vxxzz, vxxyy};
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const F4 r = ld4(R + (6 * l + q) * sF);
                const F4 w = a.mb[l] * (a.mc[l] * r - et + d * pr[q]);
                st4n(RO + (6 * l + q) * F, w, ncell);
                o[q] = l == 0 ? r : o[q] + r;
                n[q] = l == 0 ? w : n[q] + w;
            }
        }
        const F4 gt = gg * vxxyyzz;
        sxx = (ld4(sg + (SXX - SYY) * sF) + (DT * (gt - f * vyyzz) + dth * o[0])) + dth * n[0];
        syy = (ld4(sg) + (DT * (gt - f * vxxzz) + dth * o[1])) + dth * n[1];
        szz = (ld4(sg + (SZZ - SYY) * sF) + (DT * (gt - f * vxxyy) + dth * o[2])) + dth * n[2];
        srx = n[0];
        srz = n[2];
    }
    // ---- 2. explosive sources ------------------------------------------------
    for (int q = p0; q < p1; ++q) {
        const Pt pt = a.pts[q];
        if (pt.kind == PT_EXPLOSIVE && pt.j == j && pt.i == i && pt.k >= k && pt.k < k + 4) {
            const float amp = a.amp[(long long)pt.row * a.amp_row + (nt - 1)];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                if (cc == pt.k - k) {
                    set4(sxx, cc, get4(sxx, cc) + amp);
                    set4(syy, cc, get4(syy, cc) + amp);
                    set4(szz, cc, get4(szz, cc) + amp);
                }
        }
    }
    // ---- 3. free surface ---------------------------------------------------
    if (surf) {
        const F4 zero = f4(0.f);
        syy = zero;
        if constexpr (L == 0) {
            F4 spi = pim, su = um;
            if (a.smod) {  // the surface's own moduli (the reference's step-length forwards)
                const float *q = a.smod + (long long)(i - 1) * g.nz + (k - 1);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc)
                    if (cc < ncell) {
                        set4(spi, cc, q[cc]);
                        set4(su, cc, q[(long long)g.nx * g.nz + cc]);
                    }
            }
            const F4 f = 2.f * su, gf = spi - f;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const float gc = get4(gf, cc);
                const float h = -(DT * gc * gc * get4(hor, cc) / get4(spi, cc)) - (DT * gc * get4(svyy, cc));
                set4(sxx, cc, get4(sxx, cc) + h);
                set4(szz, cc, get4(szz, cc) + h);
            }
        } else {
            const float Lf = (float)L, dth = a.dthalbe;
            F4 h, hh, ratio, de;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const float u1 = get4(um, cc), p1_ = get4(pim, cc), ts = get4(taus, cc), tp = get4(taup, cc);
                const float f = (float)(((double)u1 * 2.0) * (1.0 + (double)(Lf * ts)));
                const float gg = (float)((double)p1_ * (1.0 + (double)(Lf * tp)));
                set4(h, cc, -(DT * (gg - f) * (gg - f) * get4(hor, cc) / gg) - (DT * (gg - f) * get4(svyy, cc)));
                set4(ratio, cc, f / gg);
                set4(de, cc, (float)((2.0 * (double)u1) * (double)ts) - p1_ * tp);
            }
            sxx = sxx + (h - dth * srx);
            szz = szz + (h - dth * srz);
            float *R = S0 + NEL * F;
#pragma unroll
            for (int l = 0; l < L; ++l) {
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const double d = (double)get4(de, cc);
                    set4(hh, cc, (float)((double)a.msb[l] * (((d * ((double)get4(ratio, cc) - 1.0)) * (double)get4(hor, cc)) -
                                                            (double)(get4(de, cc) * get4(svyy, cc)))));
                }
                const F4 rx = ld4(R + 6 * l * F) + hh, rz = ld4(R + (6 * l + 2) * F) + hh;
                st4n(R + 6 * l * F, rx, ncell);
                st4n(R + (6 * l + 1) * F, zero, ncell);
                st4n(R + (6 * l + 2) * F, rz, ncell);
                srx = l == 0 ? rx : srx + rx;
                srz = l == 0 ? rz : srz + rz;
            }
            sxx = sxx + dth * srx;
            szz = szz + dth * srz;
        }
    }
    st4n(S0 + SYY * F, syy, ncell); st4n(S0 + SXY * F, sxy, ncell); st4n(S0 + SYZ * F, syz, ncell);
    st4n(S0 + SXX * F, sxx, ncell); st4n(S0 + SZZ * F, szz, ncell); st4n(S0 + SXZ * F, sxz, ncell);
    if (g.free_surf && j <= 3) {
        // image rows above the surface (surface_ssg_elastic.c:80-84)
        const F4 ny = neg4(syy), nxy = neg4(sxy), nyz = neg4(syz);
        if (j == 1) { st4n(S0 + SXY * F - dJ, nxy, ncell); st4n(S0 + SYZ * F - dJ, nyz, ncell); }
        if (j == 2) {
            st4n(S0 + SYY * F - 2 * dJ, ny, ncell);
            st4n(S0 + SXY * F - 3 * dJ, nxy, ncell);
            st4n(S0 + SYZ * F - 3 * dJ, nyz, ncell);
        }
        if (j == 3) st4n(S0 + SYY * F - 4 * dJ, ny, ncell);
    }
    // ---- 4. receivers --------------------------------------------------------
    if (sample >= 0) {
        for (int q = p0; q < p1; ++q) {
            const Pt pt = a.pts[q];
            if (pt.kind != PT_RECEIVER || pt.j != j || pt.i != i || pt.k < k || pt.k > k + 3) continue;
            const int cc = pt.k - k;
            const float *x = vx + cc, *y = vy + cc, *z = vz + cc;
            const long long at = (long long)s * a.sec_shot + (long long)pt.row * a.sec_tr + sample;
            float *o = a.sec + at;
            o[0] = x[0];
            o[a.sec_comp] = y[0];
            o[2 * a.sec_comp] = z[0];
            if (a.seismo >= 2) {
                float pr, dv, cu, s3[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (m == cc) { s3[0] = get4(sxx, m); s3[1] = get4(syy, m); s3[2] = get4(szz, m); }
                seismo_pdc(x[0], x[-vI], x[vJ], x[1], y[0], y[-vJ], y[vI], y[1], z[0], z[-1], z[vI], z[vJ], s3[0], s3[1],
                           s3[2], md[MD_PI * mF + cc], md[MD_U * mF + cc], a.hrx, a.hry, a.hrz, pr, dv, cu);
                float *o2 = a.sec2 + at;
                o2[0] = pr;
                o2[a.sec_comp] = dv;
                o2[2 * a.sec_comp] = cu;
            }
        }
    }
}

template <int L, bool P2>
__global__ void __launch_bounds__(QTHR, 4) k_stress(const __grid_constant__ StrArgs a, int nt, int sample, int yb) {
    const Geo &g = a.g;
    const Quad Q = quad_of(g, yb);
    if (!Q.active) return;
    int p0, p1;
    block_points(a.pt_off, g, Q.s, Q.yc, p0, p1);
    const long long F = g.field;
    for (int j = Q.j; j <= Q.j1; j += Q.dj) {
        const long long c = widx(g, j, Q.i, Q.k);
        Psi q;
        psi_find(q, g, a.sl, a.psi + (long long)Q.s * a.psi_shot + 3 * (a.sl.sx + a.sl.sy + a.sl.sz), j, Q.i, Q.k);
        const float *p = a.st + (long long)Q.s * a.st_shot + c;
        const float *v = a.v + (long long)Q.s * a.v_shot + c;
        const StrGlobal m{v + VX * F, v + VY * F, v + VZ * F, p + SYY * F, a.md + c, g.pz, g.plane, F};
        str_quad<L, P2>(a, m, q, nt, sample, Q.s, j, Q.i, Q.k, Q.ncell, p0, p1);
    }
}

}  // namespace ifosb
