// The time step on TMA boxes (sm_100a).
//
// A CTA updates a box of 32 (z) x 8 (x) x YB (y) cells of one shot, four z-adjacent
// cells a thread. One thread asks the Tensor Memory Accelerator for everything the box
// reads from the wavefield and the model: each field with just the halo its
// derivatives need, every box completing on one mbarrier. The other threads fetch
// their PML memories meanwhile; then the whole update runs out of shared memory and the
// results go straight to HBM as 16-byte words. Nothing waits inside the update, so four
// CTAs per SM keep 100 KB and more of loads in flight, which is what the step needs: it
// moves 2 to 3 bytes per flop.
//
// Why boxes: a version that streamed along y through a six-plane ring (one plane of
// loads in flight behind a producer warp, one cell per thread) spent its time waiting
// for that plane; reading neighbours through L1 instead (ifosb_step.cuh) leaves each
// warp with one or two loads outstanding, since the update needs its registers.
//
// A chunk of more than YB planes per CTA (a launch shape) is done box after box.
// Every mbarrier wait is bounded in time (1 s of %globaltimer): on expiry the thread
// sets the error flag; CTAs that see the flag return without an update.
#pragma once
#include "ifosb_step.cuh"
#include "ifosb_tma.cuh"

namespace ifosb {

constexpr int TZ = 32, TX = 8;               // cells of a box along z and x
constexpr int HZ = 4;                        // z halo (a TMA box starts on 16 bytes)
constexpr int WZ = TZ + 2 * HZ;              // row with both z halos
constexpr int WR = TZ + 4;                   // row with the upper z halo (rho)
constexpr int XH = TX + 3;                   // rows of a fourth-order x difference
__host__ __device__ constexpr int a32(int x) { return (x + 31) & ~31; }  // boxes start on 128 bytes

// Velocity boxes [y][x][z], in floats. Fields without a halo along an axis have none.
template <int YB>
struct VelSm {
    static constexpr int YH = YB + 3;
    static constexpr int XX = 0, ZZ = XX + a32(TZ * XH * YB), XZ = ZZ + a32(WZ * TX * YB), YY = XZ + a32(WZ * XH * YB),
                         XY = YY + a32(TZ * TX * YH), YZ = XY + a32(TZ * XH * YH), V = YZ + a32(WZ * TX * YH),
                         RH = V + 3 * TZ * TX * YB, END = RH + a32(WR * (TX + 1) * (YB + 1));
    static constexpr int BYTES = 4 * (TZ * XH * YB + WZ * TX * YB + WZ * XH * YB + TZ * TX * YH + TZ * XH * YH + WZ * TX * YH +
                                      3 * TZ * TX * YB + WR * (TX + 1) * (YB + 1));
    const float *xx, *yy, *zz, *xy, *yz, *xz, *rh, *v;
    __device__ VelSm(const float *sm, int y, int x, int z)
        : xx(sm + XX + (y * XH + x + 1) * TZ + z), yy(sm + YY + ((y + 1) * TX + x) * TZ + z),
          zz(sm + ZZ + (y * TX + x) * WZ + HZ + z), xy(sm + XY + ((y + 2) * XH + x + 2) * TZ + z),
          yz(sm + YZ + ((y + 2) * TX + x) * WZ + HZ + z), xz(sm + XZ + (y * XH + x + 2) * WZ + HZ + z),
          rh(sm + RH + (y * (TX + 1) + x) * WR + z), v(sm + V + (y * TX + x) * TZ + z) {}
    static __device__ constexpr int xxI() { return TZ; }
    static __device__ constexpr int xzI() { return WZ; }
    static __device__ constexpr int xyI() { return TZ; }
    static __device__ constexpr int xyJ() { return TZ * XH; }
    static __device__ constexpr int yyJ() { return TZ * TX; }
    static __device__ constexpr int yzJ() { return WZ * TX; }
    static __device__ constexpr int rhI() { return WR; }
    static __device__ constexpr int rhJ() { return WR * (TX + 1); }
    static __device__ constexpr int vF() { return TZ * TX * YB; }
    static __device__ F4 ld(const float *p) { return ld4(p); }
};

// Stress boxes: the three velocities with their halo (vx from row i-2, plane j-1; vy
// from i-1, j-2; vz from i-1, j-1), then sigma and the memory variables, then the model.
template <int YB>
struct StrSm {
    static constexpr int VN = WZ * XH * (YB + 3), VS = a32(VN), PT = TZ * TX * YB;
    const float *vx, *vy, *vz, *sg, *md;
    __device__ StrSm(const float *sm, int nsr, int y, int x, int z)
        : vx(sm + ((y + 1) * XH + x + 2) * WZ + HZ + z), vy(sm + VS + ((y + 2) * XH + x + 1) * WZ + HZ + z),
          vz(sm + 2 * VS + ((y + 1) * XH + x + 1) * WZ + HZ + z), sg(sm + 3 * VS + (y * TX + x) * TZ + z),
          md(sg + nsr * PT) {}
    static __device__ constexpr int vI() { return WZ; }
    static __device__ constexpr int vJ() { return WZ * XH; }
    static __device__ constexpr int sF() { return PT; }
    static __device__ constexpr int mF() { return PT; }
    static __device__ F4 ldv(const float *p) { return ld4(p); }
};
template <int YB>
constexpr size_t str_box_bytes(int nsr, int nm) {
    return 4 * ((size_t)3 * StrSm<YB>::VS + (size_t)(nsr + nm) * StrSm<YB>::PT);
}

struct VelBox {
    CUtensorMap xx, zz, xz, yy, xy, yz;  // state, one slot: the boxes of VelSm
    CUtensorMap v;                       // velocities before the step: vx vy vz
    CUtensorMap rho;                     // rho in field layout
    VelArgs a;
    int *tma_err;
    int ahead;
    WaitCtl w;
};
struct StrBox {
    CUtensorMap v;    // velocities of this step, one component with its halo
    CUtensorMap sr;   // state, sigma and memory variables
    CUtensorMap mod;  // model slots
    StrArgs a;
    int nsr, nm;
    int *tma_err;
    int ahead;
    WaitCtl w;
};

// Planes of a box. Four CTAs per SM (16 warps, 8 with mechanisms) that are each at another
// point of their load-update-store sequence beat two larger ones, although the y halo is
// then read from L2 more often: velocity 2 planes (38 KB) 218 us at 256^3, 4 planes 243;
// elastic stress with the DFT at 128^3 2 planes (49 KB) 66.7 us, 4 planes 69.5; L = 3
// stress 1 plane (51 KB) 730 us at 256^3, 2 planes 738.
constexpr int VYB = 2;
__host__ __device__ constexpr int str_yb(int nmech) { return nmech == 0 ? 2 : 1; }

// CTAs resident at once on a B200 at the four per SM of the launch bounds. (A stress box with
// four mechanisms and relaxation times per cell is 62 KB: three fit there, and the limits that
// are counted in waves come a little late.)
constexpr unsigned ONE_WAVE = 4 * 148;

// This thread's cells in a CTA's box, and the chunk's planes.
struct BoxAt {
    int k0, i0, s, yc, j0, j1, zq, x, y, k, i;
    bool inside;
};
__device__ __forceinline__ BoxAt box_at(const Geo &g) {
    BoxAt b;
    b.k0 = blockIdx.x * TZ + 1;
    b.i0 = blockIdx.y * g.by + 1;
    b.yc = blockIdx.z % g.nyc;
    b.s = blockIdx.z / g.nyc;
    b.j0 = b.yc * g.cy + 1;
    b.j1 = min(b.j0 + g.cy - 1, g.ny);
    b.zq = (threadIdx.x & 7) * 4;
    b.x = (threadIdx.x >> 3) & 7;
    b.y = threadIdx.x >> 6;
    b.k = b.k0 + b.zq;
    b.i = b.i0 + b.x;
    b.inside = b.x < g.by && b.i <= g.nx && b.k <= g.nz;
    return b;
}

// The loop over a chunk's boxes. load(j): thread 0 issues the boxes of planes from j;
// fetch(j) (prefetch into L2 alike); before(): a thread's own loads; update(): its cells.
template <int YB, class Load, class Fetch, class Before, class Update>
__device__ __forceinline__ void box_loop(uint64_t *full, int *err, WaitCtl w, int ahead, const BoxAt &b, Load load, Fetch fetch,
                                         Before before, Update update) {
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    const int flag = *(volatile const int *)err;
    const int n = (b.j1 - b.j0 + YB) / YB;
    for (int it = 0; it < n; ++it) {
        const int jb = b.j0 + it * YB, j = jb + b.y;
        const bool issue = w.stop_it < 0 || it < w.stop_it;  // failure-path test: issue nothing more
        if (threadIdx.x == 0) {
            if (issue) load(jb);
            if (ahead > 0 && it + ahead < n) fetch(jb + ahead * YB);
        }
        const bool active = b.inside && j <= b.j1;
        if (active) before(j);
        bool ok = mbar_wait(full, it & 1, w.limit_ns);
        if (!ok) {
            atomicExch(err, 1);
            // no copy may still be landing in shared memory when the CTA ends
            if (threadIdx.x == 0 && issue) mbar_wait(full, it & 1, w.limit_ns);
        }
        ok = ok && flag == 0;
        // the next kernel's CTAs may move in once the boxes of the last wave have landed; a
        // grid of one wave keeps its SMs to itself until it ends
        if (it == 0 && gridDim.x * gridDim.y * gridDim.z > ONE_WAVE) pdl_release();
        if (active && ok) update(j);
        // every thread has read the box before the next one lands in it
        if (it + 1 < n && !__syncthreads_and(ok)) return;
    }
}

template <bool BACK>
__global__ void __launch_bounds__(64 * VYB, 4) k_velocity_box(const __grid_constant__ VelBox T, int nt) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full;
    using M = VelSm<VYB>;
    const VelArgs &a = T.a;
    const Geo &g = a.g;
    const BoxAt b = box_at(g);
    float *sm = reinterpret_cast<float *>(smem);
    int p0, p1;
    block_points(a.pt_off, g, b.s, b.yc, p0, p1);
    float *ps = a.psi + (long long)b.s * a.psi_shot;
    Psi q;
    const int z = zc(b.k0), x = xc(b.i0), s = b.s;
    box_loop<VYB>(
        &full, T.tma_err, T.w, T.ahead, b,
        [&](int j) {
            const int y = yc_(j);
            mbar_expect_tx(&full, M::BYTES);
            tma_load5(sm + M::XX, &T.xx, z, x - 1, y, SXX, s, &full);
            tma_load5(sm + M::ZZ, &T.zz, z - HZ, x, y, SZZ, s, &full);
            tma_load5(sm + M::XZ, &T.xz, z - HZ, x - 2, y, SXZ, s, &full);
            tma_load5(sm + M::YY, &T.yy, z, x, y - 1, SYY, s, &full);
            tma_load5(sm + M::XY, &T.xy, z, x - 2, y - 2, SXY, s, &full);
            tma_load5(sm + M::YZ, &T.yz, z - HZ, x, y - 2, SYZ, s, &full);
            tma_load5(sm + M::V, &T.v, z, x, y, VX, s, &full);
            tma_load3(sm + M::RH, &T.rho, z, x, y, &full);
        },
        [&](int j) {
            const int y = yc_(j);
            tma_prefetch5(&T.xx, z, x - 1, y, SXX, s);
            tma_prefetch5(&T.zz, z - HZ, x, y, SZZ, s);
            tma_prefetch5(&T.xz, z - HZ, x - 2, y, SXZ, s);
            tma_prefetch5(&T.yy, z, x, y - 1, SYY, s);
            tma_prefetch5(&T.xy, z, x - 2, y - 2, SXY, s);
            tma_prefetch5(&T.yz, z - HZ, x, y - 2, SYZ, s);
            tma_prefetch5(&T.v, z, x, y, VX, s);
            tma_prefetch3(&T.rho, z, x, y);
        },
        [&](int j) {
            psi_find(q, g, a.sl, ps, j, b.i, b.k);
            if (a.u) prefetch3(a.u + (long long)s * 3 * g.field + widx(g, j, b.i, b.k), g.field);
        },
        [&](int j) { vel_quad<BACK>(a, M(sm, b.y, b.x, b.zq), q, nt, s, j, b.i, b.k, g.nz - b.k + 1, p0, p1); });
}

template <int L, bool P2>
__global__ void __launch_bounds__(64 * str_yb(L), 4) k_stress_box(const __grid_constant__ StrBox T, int nt, int sample) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full;
    constexpr int YB = str_yb(L);
    using M = StrSm<YB>;
    const StrArgs &a = T.a;
    const Geo &g = a.g;
    const BoxAt b = box_at(g);
    float *sm = reinterpret_cast<float *>(smem);
    int p0, p1;
    block_points(a.pt_off, g, b.s, b.yc, p0, p1);
    float *ps = a.psi + (long long)b.s * a.psi_shot + 3 * (a.sl.sx + a.sl.sy + a.sl.sz);
    Psi q;
    const int z = zc(b.k0), x = xc(b.i0), s = b.s;
    box_loop<YB>(
        &full, T.tma_err, T.w, T.ahead, b,
        [&](int j) {
            const int y = yc_(j);
            mbar_expect_tx(&full, 4 * (3 * M::VN + (T.nsr + T.nm) * M::PT));
            tma_load5(sm, &T.v, z - HZ, x - 2, y - 1, VX, s, &full);
            tma_load5(sm + M::VS, &T.v, z - HZ, x - 1, y - 2, VY, s, &full);
            tma_load5(sm + 2 * M::VS, &T.v, z - HZ, x - 1, y - 1, VZ, s, &full);
            tma_load5(sm + 3 * M::VS, &T.sr, z, x, y, SYY, s, &full);
            tma_load4(sm + 3 * M::VS + T.nsr * M::PT, &T.mod, z, x, y, 0, &full);
        },
        [&](int j) {
            const int y = yc_(j);
            tma_prefetch5(&T.v, z - HZ, x - 2, y - 1, VX, s);
            tma_prefetch5(&T.v, z - HZ, x - 1, y - 2, VY, s);
            tma_prefetch5(&T.v, z - HZ, x - 1, y - 1, VZ, s);
            tma_prefetch5(&T.sr, z, x, y, SYY, s);
            tma_prefetch4(&T.mod, z, x, y, 0);
        },
        [&](int j) { psi_find(q, g, a.sl, ps, j, b.i, b.k); },
        [&](int j) {
            str_quad<L, P2>(a, M(sm, T.nsr, b.y, b.x, b.zq), q, nt, sample, s, j, b.i, b.k, g.nz - b.k + 1, p0, p1);
        });
}

}  // namespace ifosb
