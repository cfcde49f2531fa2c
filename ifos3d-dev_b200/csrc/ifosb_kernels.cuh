// Device kernels of the B200 wavefield engine.
//
// Arithmetic contract: every floating-point expression keeps the operand order
// and the float/double promotions of the reference C code it restates, and the
// library is compiled with --fmad=false (no FMA contraction), IEEE division and
// square root, and denormals preserved. On the same inputs the results are
// therefore bit-identical to the reference built with gcc -O3 on x86-64.
//
// Layout in HBM (per shot, per field): the reference's halo ranges
// j=-2..NY+2, i=-1..NX+2, k=-1..NZ+2, with the z row padded to a pitch that is a
// multiple of 8 floats and k=1 placed at a 32-byte boundary. Fields of a shot are
// contiguous ([shot][field][y][x][z]); the model is one copy shared by all shots.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ifosb_tma.cuh"

namespace ifosb {

constexpr int MAXFW = 64;
constexpr int MAXMECH = 4;
constexpr int MAXNF = 16;
constexpr int BX = 32;  // threads along z (contiguous)

// state field slots of a shot. The stresses with a y derivative in the velocity
// update (syy, sxy, syz) come first, then the in-plane ones (sxx, szz, sxz), then
// the memory variables: the stress kernel takes them all as one TMA box, the velocity
// kernel each stress as a box with the halo its derivatives need.
enum { VX = 0, VY, VZ, SYY, SXY, SYZ, SXX, SZZ, SXZ, NEL };
// memory variables: slot NEL + 6*l + q, q: 0 rxx, 1 ryy, 2 rzz, 3 rxy, 4 ryz, 5 rxz
// model slots (one copy shared by every shot): the stress update's coefficients
// first (5, or 10 with non-uniform relaxation times; one TMA box), then av_mat's
// averaged densities, which the body forces read (the velocity update forms its own
// from rho).
enum { MD_PI = 0, MD_U, MD_UIPJP, MD_UJPKP, MD_UIPKP, MD_TAUS, MD_TAUP, MD_TSIPJP, MD_TSJPKP, MD_TSIPKP, MD_RIP, MD_RJP, MD_RKP, NMODEL };
// CPML coefficient rows
enum { K_X = 0, A_X, B_X, KH_X, AH_X, BH_X, K_Y, A_Y, B_Y, KH_Y, AH_Y, BH_Y, K_Z, A_Z, B_Z, KH_Z, AH_Z, BH_Z,
       RK_X, RKH_X, RK_Y, RKH_Y, NCPG };  // RK: minus the correctly rounded reciprocals of K
// The z faces' coefficients per cell (index k-1; K = 1, a = b = 0 inside), so that a
// thread reads its four cells' as one word. KS, KHS: the stress update's, which takes
// K_y on the front face (update_s_ssg_CPML_elastic.c:104-108).
enum { Z_K = 0, Z_RK, Z_A, Z_B, Z_KH, Z_RKH, Z_AH, Z_BH, Z_KS, Z_RKS, Z_KHS, Z_RKHS, NCZ };
constexpr int CZ0 = NCPG * 2 * MAXFW;  // where they start; row pitch pz

struct Geo {
    int nx, ny, nz, fw, free_surf, nmech;
    int pz;             // z row pitch in floats
    int px;             // rows per plane (NX+4)
    long long plane;    // px*pz
    long long field;    // (NY+5)*plane
    int cy, nyc;        // y planes per block, y chunks
    int ntk, nti;       // blocks along z and x
    int by;             // rows (x) per block: the tile height of the kernels in use
    int pzw, zfo;       // z PML slab: row pitch, and the far face's offset from k-1 (see Slabs)
    int bz;             // cells (z) per block
};

__host__ __device__ __forceinline__ long long widx(const Geo &g, int j, int i, int k) {
    return (long long)(j + 2) * g.plane + (long long)(i + 1) * g.pz + (k + 7);
}

// A source, injection or receiver located in one cell. Lists are grouped per
// (shot, block) and keep the order in which the reference visits them.
struct Pt {
    int j, i, k, kind;  // kind: 1 explosive, 2..5 body force, 6 adjoint injection, 7 receiver
    int row;            // value-table row (forces) or trace number (receivers)
    int pad0, pad1, pad2;
};
enum { PT_EXPLOSIVE = 1, PT_ADJOINT = 6, PT_RECEIVER = 7 };

// z-face slab indices differ between the lanes of a warp; the constant cache would
// serialise them, L1 serves them in one pass
__device__ __forceinline__ float CPG(const float *cpg, int row, int h) { return __ldg(cpg + row * 2 * MAXFW + h - 1); }

// CPML frame membership (CPML_ini_elastic.c:26-71): 1-based slab index or 0.
__device__ __forceinline__ int face_x(const Geo &g, int i) {
    return i <= g.fw ? i : (i > g.nx - g.fw ? i - g.nx + 2 * g.fw : 0);
}
__device__ __forceinline__ int face_y(const Geo &g, int j) {
    return (!g.free_surf && j <= g.fw) ? j : (j > g.ny - g.fw ? j - g.ny + 2 * g.fw : 0);
}
__device__ __forceinline__ int face_z(const Geo &g, int k) {
    return k <= g.fw ? k : (k > g.nz - g.fw ? k - g.nz + 2 * g.fw : 0);
}

// PML memory slabs of a shot: 9 for the stress derivatives (velocity update),
// then 9 for the velocity derivatives (stress update). x: [NY][2FW][z row],
// y: [2FW][NX][z row], z: [NY][NX][2FW], the reference's slabs (ifos3d.c:421-440)
// with rows padded so that the four cells a thread owns (k = 1 mod 4) are one
// 16-byte word: x and y rows are field rows (pitch pz, k = 1 at float 8), a z row
// holds k-1 for the near face and k-1 + zfo for the far one.
struct Slabs {
    long long sx, sy, sz;
};
__device__ __forceinline__ long long sxi(const Geo &g, int j, int h, int k) {
    return ((long long)(j - 1) * 2 * g.fw + (h - 1)) * g.pz + (k + 7);
}
__device__ __forceinline__ long long syi(const Geo &g, int h, int i, int k) {
    return ((long long)(h - 1) * g.nx + (i - 1)) * g.pz + (k + 7);
}
__device__ __forceinline__ long long szi(const Geo &g, int j, int i, int h) {
    return ((long long)(j - 1) * g.nx + (i - 1)) * g.pzw + (h <= g.fw ? h - 1 : h - 1 - 2 * g.fw + g.nz + g.zfo);
}

struct VelArgs {
    Geo g;
    Slabs sl;
    float *st;            // state base (shot 0)
    long long st_shot;    // floats per shot
    const float *vin;     // velocities before the step [shot][3][field], and where the new ones go
    float *vout;          // (a slot of the velocity ring; the same place without one)
    long long vin_shot, vout_shot;
    // time-domain mode: the running sums U += v dt of the new velocities [shot][3][field] (null:
    // none), and where v and U go besides [shot][6][field] (null: nowhere)
    float *u, *useg;
    long long useg_shot;
    float dt;
    const float *md;      // model base
    const float *rho;     // rho in field layout (with matcopy's ghost layers)
    float *psi;           // PML memory base (shot 0)
    long long psi_shot;
    const int *pt_off;    // [nshots][nblocks+1] or null
    const Pt *pts;
    const float *val;     // forces: amp table [row][NT]; adjoint: residual [shot][3][ntr][ns]
    long long val_row, val_comp;
    float dxr, dyr, dzr;  // DT/DX, DT/DY, DT/DZ
    float b1, b2;
    double cf5x, cf5y, cf5z;  // type-5 force direction factors (update_v_ssg.c:498-503)
    const float *cpg;         // global copy of the CPML rows, for lane-divergent (z-face) reads
    int fast_div;         // every density and CPML divisor is in div4's range
    int *err_step;        // [nshots] first step whose probe cell went NaN
    int probe_j, probe_i, probe_k;
};

struct StrArgs {
    Geo g;
    Slabs sl;
    float *st;
    long long st_shot;
    const float *md;
    float *psi;
    long long psi_shot;
    const int *pt_off;
    const Pt *pts;
    const float *amp;     // explosive amplitudes [row][NT]
    long long amp_row;
    float *sec;           // traces [shot][3][ntr][ns]
    long long sec_shot, sec_comp, sec_tr;
    const float *v;       // velocities of this step [shot][3][field]
    long long v_shot;
    float dt, dthalbe, rdx, rdy, rdz;
    float b1, b2;
    float eta[MAXMECH], mb[MAXMECH], mc[MAXMECH], msb[MAXMECH];
    const float *cpg;     // global copy of the CPML rows, for lane-divergent (z-face) reads
    int seismo;           // SEISMO: 1 particle velocities; 2, 3, 4 add p / div, curl (sec2)
    float *sec2;          // [shot][3][ntr][ns]: p, div, curl
    float hrx, hry, hrz;  // 1.0/DX etc. in float (seismo_ssg.c:38-40)
    int fast_div;         // every CPML divisor and spacing is in div4's range
    int unif_tau;         // one relaxation time for all cells (utaus, utaup and the average)
    float utaus, utaup, uts_avg;
    float idx, idy, idz;  // RN(1/DX) etc. (exact for power-of-two spacings)
    const float *smod;    // elastic free surface: pi, u of plane j=1 ([2][NX][NZ]) when they
                          // differ from the propagation model's, else null
};

// seismo (seismo_ssg.c:48-125), SEISMO 2-4: pressure from the cell's new
// stresses; divergence and curl from one-sided velocity differences at the cell.
// The curl's squares are formed in double as the reference's fabs() promotes them.
__device__ __forceinline__ void seismo_pdc(float vx, float vx_im, float vx_jp, float vx_kp, float vy, float vy_jm,
                                           float vy_ip, float vy_kp, float vz, float vz_km, float vz_ip, float vz_jp,
                                           float sxx, float syy, float szz, float pi, float u, float hx, float hy,
                                           float hz, float &p, float &dv, float &cu) {
    p = -sxx - syy - szz;
    const float vxy = (vx_jp - vx) * hy, vxz = (vx_kp - vx) * hz;
    const float vyx = (vy_ip - vy) * hx, vyz = (vy_kp - vy) * hz;
    const float vzx = (vz_ip - vz) * hx, vzy = (vz_jp - vz) * hy;
    const double t1 = (double)(vyz - vzy) * fabs((double)(vyz - vzy));
    const double t2 = (double)(vzx - vxz) * fabs((double)(vzx - vxz));
    const double t3 = (double)(vxy - vyx) * fabs((double)(vxy - vyx));
    const float amp = (float)((double)u * (t1 + t2 + t3));
    cu = (float)((amp < 0.0 ? -1 : 1) * sqrt(fabs((double)amp)));
    const float vxx = (vx - vx_im) * hx, vyy = (vy - vy_jm) * hy, vzz = (vz - vz_km) * hz;
    dv = (float)((double)(vxx + vyy + vzz) * sqrt((double)pi));
}

__device__ __forceinline__ void block_points(const int *pt_off, const Geo &g, int s, int yc, int &p0, int &p1) {
    p0 = p1 = 0;
    if (pt_off) {
        const int nblk = g.ntk * g.nti * g.nyc;
        const int blk = (yc * g.nti + blockIdx.y) * g.ntk + blockIdx.x;
        const int *o = pt_off + (long long)s * (nblk + 1);
        p0 = o[blk];
        p1 = o[blk + 1];
    }
}

// ---------------------------------------------------------------------------
// discfourier (disc_fourier.c:36-57) for P steps at once: every accumulator takes the
// steps' velocities in order, F += v * trig with product and sum in double and a float
// store each time, so the bits are those of one pass per step. A pass reads and writes
// the 6 nf accumulators of a cell (48 nf bytes), which at one pass a step is more than
// a third of an L = 3, nf = 4 step's traffic; over P steps it costs 12 + 48 nf / P
// bytes a step, the 12 being the velocities, kept in a ring for it.
constexpr int MAXRING = 8;
struct DftArgs {
    Geo g;
    const float *v[MAXRING];  // velocities of the steps [shot][3][field]
    long long v_shot[MAXRING];
    const double *trig[MAXRING];  // cos, sin of 2 pi f t, times DT*ntast, [nf][2] of each step
    float *dft;               // [shot][nf][6][field]
    long long dft_shot;
    int nf;
};
// (float)x as a double: x rounded to nearest even at 24 bits, or at 2^-149 below the
// normal floats, by adding and subtracting 1.5 * 2^(e+29) (1.5 * 2^-97 at least), whose
// last place is the float's; a zero keeps x's sign. For |x| < 2^126.
__device__ __forceinline__ double round24(double x) {
    const int hi = __double2hiint(x);
    const double c = __hiloint2double(__viaddmax_s32(hi & 0x7ff00000, 0x01d80000, 0x39e80000), 0);
    const double r = __dadd_rn(__dadd_rn(x, c), -c);
    return __hiloint2double((__double2hiint(r) & 0x7fffffff) | (hi & 0x80000000), __double2loint(r));
}
// One velocity component (blockIdx.y) of two z-adjacent cells a thread: their velocities
// of all P steps stay in registers as doubles, eight blocks share an SM, and the next
// accumulators are on their way while these are updated. The two conversions of every
// (double)(float) bind the pass to the conversion unit when both cells take them, and
// round24's integer work to the issue slots when neither does, so one goes each way.
// 8 steps, nf = 4, 192x160x192: 484 us; 631 (84 % conversion unit) with four
// cells a thread, 15 warps an SM and conversions only, 736 with round24 only.
template <int P>
__global__ void __launch_bounds__(128, 8) k_dft(const __grid_constant__ DftArgs a) {
    __shared__ double trig[P][2 * MAXNF];
    const Geo &g = a.g;
    const int nl = 2 * a.nf;
    pdl_release();
    for (int q = threadIdx.x; q < P * nl; q += 128) trig[q / nl][q % nl] = a.trig[q / nl][q % nl];
    __syncthreads();
    pdl_wait();
    const int nq = (g.nz + 1) / 2, id = blockIdx.x * 128 + threadIdx.x, row = id / nq;
    const int j = row / g.nx + 1, i = row % g.nx + 1, k = 2 * (id % nq) + 1, c = blockIdx.y, s = blockIdx.z;
    if (j > g.ny) return;
    const long long F = g.field, at = (long long)c * F + widx(g, j, i, k);
    double v[P][2];
    float top = 0.f;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const float2 x = __ldg(reinterpret_cast<const float2 *>(a.v[p] + (long long)s * a.v_shot[p] + at));
        v[p][0] = x.x;
        v[p][1] = x.y;
        top = fabsf(x.x) < 0x1p100f && fabsf(x.y) < 0x1p100f ? top : INFINITY;  // (NaN too)
    }
    float *f = a.dft + (long long)s * a.dft_shot + at;
    float2 o = *reinterpret_cast<const float2 *>(f);
    for (int l = 0; l < nl; ++l, f += 3 * F) {  // cos and sin accumulators in turn
        double x0 = o.x, x1 = o.y;
        const bool fine = top == 0.f && fabsf(o.x) < 0x1p100f;  // far from overflow
        if (l + 1 < nl) o = *reinterpret_cast<const float2 *>(f + 3 * F);
        if (fine) {
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const double t = trig[p][l];
                x0 = round24(__dadd_rn(x0, __dmul_rn(v[p][0], t)));
                x1 = (double)(float)__dadd_rn(x1, __dmul_rn(v[p][1], t));
            }
        } else {
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const double t = trig[p][l];
                x0 = (double)(float)__dadd_rn(x0, __dmul_rn(v[p][0], t));
                x1 = (double)(float)__dadd_rn(x1, __dmul_rn(v[p][1], t));
            }
        }
        if (k < g.nz) *reinterpret_cast<float2 *>(f) = make_float2((float)x0, (float)x1);
        else f[0] = (float)x0;
    }
}

// ---------------------------------------------------------------------------
// Time-domain gradient kernels (the optional checkpoint/recompute mode). For a
// forward step n and the adjoint step m = P - n, P = TIME / DT (TIME = (NT-1) DT
// after ifos3d.c:177), the pair whose discfourier phases agree (t_f - t_b =
// n DT - (TIME - m DT) = 0), they add
//   rho: sum_c v_f,c v_b,c                      (gradient_F's gradrho term)
//   lambda: div U_f . div U_b                   (U = running time sum of v times DT)
//   mu: 2 sum_i e_ii,f e_ii,b + sum_i<j (e_ij+e_ji)_f (e_ij+e_ji)_b
// in FP64 over the interior cells, summed over the batch's shots.
struct TdArgs {
    Geo g;
    const float *st;       // adjoint state [shot][slot][field] (v at slots 0..2)
    long long st_shot;
    const float *ub;       // adjoint running sums [shot][3][field]
    const float *seg;      // forward v and running sums of one step [shot][6][field]
    long long seg_shot;
    int nshots;
    float b1, b2, rdx, rdy, rdz;
    float ihx, ihy, ihz;   // 1/DX, 1/DY, 1/DZ (exact for power-of-two spacings)
    double *k;             // [4][NY][NX][NZ]: rho, lambda, mu, dc
};

// The zero-frequency product of the two runs: sum_c U_f,c(NT) U_b,c(NT).
__global__ void k_td_dc(TdArgs a, const float *uf_end) {
    const Geo &g = a.g;
    const long long n = (long long)g.nx * g.ny * g.nz, F = g.field;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(m % g.nz) + 1, i = (int)((m / g.nz) % g.nx) + 1, j = (int)(m / ((long long)g.nz * g.nx)) + 1;
        const long long c = widx(g, j, i, k);
        double d = 0.0;
        for (int s = 0; s < a.nshots; ++s) {
            const float *uf = uf_end + (long long)s * 3 * F, *ub = a.ub + (long long)s * 3 * F;
            d += (double)uf[c] * ub[c] + (double)uf[F + c] * ub[F + c] + (double)uf[2 * F + c] * ub[2 * F + c];
        }
        a.k[3 * n + m] += d;
    }
}

// ---------------------------------------------------------------------------
// av_mat (av_mat.c:45-69) from the ghosted model [NY+2][NX+2][NZ+2] into the
// model slots, plus the per-cell pi, u, taus, taup.
struct AvArgs {
    Geo g;
    const float *rho, *pi, *u, *taus, *taup;  // ghosted
    float *md;
    float *rho_w;                              // rho in field layout (gradient)
};

// rho in field layout over the ghosted box (j, i, k = 0..N+1): the ghost layers
// matcopy left (periodic on one rank) next to the interior, so the velocity
// kernel can form av_mat's averages rip, rjp, rkp from rho and its +1 neighbours.
__global__ void k_rho_field(AvArgs a) {
    const Geo &g = a.g;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    const int j = blockIdx.z;
    if (k > g.nz + 1 || i > g.nx + 1 || j > g.ny + 1) return;
    const long long GX = g.nx + 2, GZ = g.nz + 2;
    a.rho_w[widx(g, j, i, k)] = a.rho[((long long)j * GX + i) * GZ + k];
}

__global__ void k_av_mat(AvArgs a) {
    const Geo &g = a.g;
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int i = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int j = blockIdx.z + 1;
    if (k > g.nz || i > g.nx || j > g.ny) return;
    const long long GX = g.nx + 2, GZ = g.nz + 2;
#define GM(A, jj, ii, kk) ((double)A[((long long)(jj) * GX + (ii)) * GZ + (kk)])
#define GF(A, jj, ii, kk) (A[((long long)(jj) * GX + (ii)) * GZ + (kk)])
    const long long F = g.field, c = widx(g, j, i, k);
    const float *u = a.u, *rho = a.rho;
    a.md[MD_UIPJP * F + c] = (float)(4.0 / ((1.0 / GM(u, j, i, k)) + (1.0 / GM(u, j, i + 1, k)) + (1.0 / GM(u, j + 1, i + 1, k)) +
                                          (1.0 / GM(u, j + 1, i, k))));
    a.md[MD_UJPKP * F + c] = (float)(4.0 / ((1.0 / GM(u, j, i, k)) + (1.0 / GM(u, j, i, k + 1)) + (1.0 / GM(u, j + 1, i, k + 1)) +
                                          (1.0 / GM(u, j + 1, i, k))));
    a.md[MD_UIPKP * F + c] = (float)(4.0 / ((1.0 / GM(u, j, i, k)) + (1.0 / GM(u, j, i, k + 1)) + (1.0 / GM(u, j, i + 1, k + 1)) +
                                          (1.0 / GM(u, j, i + 1, k))));
    if (g.nmech) {
        const float *t = a.taus;
        a.md[MD_TSIPJP * F + c] = (float)(0.25 * (double)(GF(t, j, i, k) + GF(t, j, i + 1, k) + GF(t, j + 1, i + 1, k) + GF(t, j + 1, i, k)));
        a.md[MD_TSJPKP * F + c] = (float)(0.25 * (double)(GF(t, j, i, k) + GF(t, j + 1, i, k) + GF(t, j + 1, i, k + 1) + GF(t, j, i, k + 1)));
        a.md[MD_TSIPKP * F + c] = (float)(0.25 * (double)(GF(t, j, i, k) + GF(t, j, i + 1, k) + GF(t, j, i + 1, k + 1) + GF(t, j, i, k + 1)));
        a.md[MD_TAUS * F + c] = GF(a.taus, j, i, k);
        a.md[MD_TAUP * F + c] = GF(a.taup, j, i, k);
    }
    a.md[MD_RJP * F + c] = (float)(0.5 * (double)(GF(rho, j, i, k) + GF(rho, j + 1, i, k)));
    a.md[MD_RKP * F + c] = (float)(0.5 * (double)(GF(rho, j, i, k) + GF(rho, j, i, k + 1)));
    a.md[MD_RIP * F + c] = (float)(0.5 * (double)(GF(rho, j, i, k) + GF(rho, j, i + 1, k)));
    a.md[MD_PI * F + c] = GF(a.pi, j, i, k);
    a.md[MD_U * F + c] = GF(a.u, j, i, k);
    a.rho_w[c] = GF(rho, j, i, k);
#undef GM
#undef GF
}

// ---------------------------------------------------------------------------
// residual (residual.c:35-60): one thread per (shot, component, trace) runs the
// time-integrated, time-reversed difference; the FP64 sum of squares of each
// trace goes to part[] and is reduced per shot in a fixed order.
__global__ void k_residual(const float *syn, const float *obs, float *diff, double *part, int nshots, int ntr, int ns,
                           float DT) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nshots * 3 * ntr) return;
    const float *sy = syn + (long long)t * ns;
    const float *ob = obs + (long long)t * ns;
    float *o = diff + (long long)t * ns;
    float vdiff = 0.0f;
    double acc = 0.0;
    for (int j = 1; j <= ns; ++j) {
        vdiff += sy[j - 1] - ob[j - 1];
        const float d = DT * vdiff;
        o[ns - j] = d;
        acc += (double)d * (double)d;
    }
    part[t] = acc;
}

// One warp per shot: strided lane sums then a shuffle tree — a fixed order, so
// the FP64 misfit is deterministic.
__global__ void k_misfit(const double *part, double *misfit, int per_shot) {
    const int s = blockIdx.x;
    const double *p = part + (long long)s * per_shot;
    double v = 0.0;
    for (int q = threadIdx.x; q < per_shot; q += 32) v += p[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) misfit[s] = v;
}

// The reference's own float L2 (residual.c:53): a sequential sum per shot.
__global__ void k_l2_ref(const float *diff, float *l2, int nshots, int ntr, int ns) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nshots) return;
    float L2 = 0.0f;
    const float *d = diff + (long long)s * 3 * ntr * ns;
    for (int c = 0; c < 3; ++c)
        for (int t = 0; t < ntr; ++t)
            for (int j = 1; j <= ns; ++j) {
                const float x = d[((long long)c * ntr + t) * ns + (ns - j)];
                L2 = (float)((double)L2 + fabs((double)(x * x)));
            }
    l2[s] = L2;
}

}  // namespace ifosb
