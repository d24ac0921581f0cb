// stencil.cu — tendency, friction, forcing, Adams-Bashforth and pressure
// gradient kernels of the ps3D time step on sm_100a.
//
// K1 (k_step) fuses, per grid point, what the reference does in ~40 full
// passes over memory:
//   buoyancy_advection_2nd            advection.f90:2-48
//   N^2 term                          integrate.f90:21-23
//   momentum_advection_2nd            advection.f90:53-184
//   Coriolis and buoyancy force       integrate.f90:37-54
//   harmonic friction (in place)      mixing.f90:225-274, integrate.f90:59-66
//   set_forcing (wavemaker and
//     background-flow advection)      config.f90:224-237, lee_wave1.f90:232-332
//   Adams-Bashforth 2/3               integrate.f90:87-102
// The block owns a 32 x BY column tile and marches up in z, two neighbouring
// points along x per thread.  Levels k and k+1 of u, v, w, b (and of U_back,
// B_back when present) sit corrected in a four-slot shared-memory ring; level
// k+2 has landed and gets its pending pressure correction while level k is
// stepped, and level k+3 is on its way (16-byte asynchronous copies), so one
// barrier a level is enough and no load is waited for where it is issued.  The
// vertical fluxes and a column's own values pass from level to level in
// registers; only the level's horizontal neighbours are read from the ring.
// Each state word is read once from HBM and each tendency and new value is
// written once.
//
// What bounds it: HBM.  At 256x256x128 it runs 240 us in FP64 (168 B a point,
// 5.9 TB/s) and 210 us in the mixed form (132 B, 5.3 TB/s).  The form it
// replaced (one point a thread, planes loaded through registers behind two
// barriers a level, all fluxes formed from shared memory) took 321 and 292 us:
// it kept the L1/shared data path at 72 % with 257 wavefronts and 632
// instructions per 32 points, against 140 and 365 now.
#include <cstdlib>
#include <type_traits>
#include "engine.h"

namespace ps3d {

constexpr int kTX = 32;

// The ring of state planes, filled by 16-byte asynchronous copies three
// levels ahead of the level that is stepped: levels k and k+1 (corrected,
// read by the stencil), k+2 (landed, being corrected) and k+3 (on its way).
// Tiles start two columns west of the block's first point so that every
// 16-byte pair is aligned (nx is even: a pair never straddles the periodic
// seam); the pressure tile has one row and one pair more, for the
// correction's north and east neighbours.  The level's Adams-Bashforth
// history is copied to a slot of the thread's own.
template <int BY>
struct StepTile {
    static constexpr int NT = kTX / 2 * BY;           // threads: a pair of points along x each
    static constexpr int FP = kTX + 4, FR = BY + 2;   // field tile: columns i0-2 .. i0+33, rows j0-1 .. j0+BY
    static constexpr int PP = kTX + 6, PR = BY + 3;   // pressure tile: columns i0-2 .. i0+35, rows j0-1 .. j0+BY+1
    static constexpr int FCH = FP / 2 * FR, PCH = PP / 2 * PR;   // pairs of a tile
};
template <typename TT> struct pair_t;
template <> struct pair_t<double> { using type = double2; };
template <> struct pair_t<float> { using type = float2; };

template <typename TT, int BY, int NF>
struct __align__(16) StepSmem {
    double pl[4][NF][StepTile<BY>::FP * StepTile<BY>::FR];
    double pp[4][StepTile<BY>::PP * StepTile<BY>::PR];
    double2 hw[2][StepTile<BY>::NT];
    typename pair_t<TT>::type hist[2][3][StepTile<BY>::NT];   // u, v, b
};

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory"); }

// What a thread keeps of its two columns between two levels: its values at
// the level (with u west and v south of them, which the fluxes through the
// level's west and south faces have read one level earlier), the vertical
// fluxes through the level's lower face and w below it.
struct StepCarry {
    double u0[2], v0[2], w0[2], b0[2], uw, vs[2];
    double tb[2], tu[2], tv[2], tw[2];     // lower-face fluxes of b, u, v, w
    double hu[2], hv[2], hw[2], hb[2];     // lower-face harmonic fluxes
    double gu[2], gb[2];                   // lower-face background fluxes of u, b
    double wm[2];
};

// One block's column tile (bx, by) and z chunk / instance bz of the grid
// described by `a`.
template <typename TT, int BY, int HARM, bool WM, bool BG>
__device__ __forceinline__ void step_tile(const StepArgs& a, int kchunk, int bx, int by, int bz) {
    using TW = double;   // stored w tendencies stay FP64 in both paths
    using T2 = typename pair_t<TT>::type;
    using L = StepTile<BY>;
    constexpr int NF = BG ? 6 : 4, NT = L::NT;
    extern __shared__ __align__(16) unsigned char step_smem_raw[];
    StepSmem<TT, BY, NF>& sm = *reinterpret_cast<StepSmem<TT, BY, NF>*>(step_smem_raw);
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int i0 = bx * kTX, j0 = by * BY;
    const int kcnt = a.kcount ? a.kcount : nz;           // levels stepped (a z-slab's interior)
    const int kofs = a.kofs, nzg = a.nzg ? a.nzg : nz;   // global level k + kofs of nzg (rigid-lid masks)
    const int nzc = (kcnt + kchunk - 1) / kchunk;
    const int inst = bz / nzc;
    const int kb = a.kbeg + (bz - inst * nzc) * kchunk;
    const int ke = min(a.kbeg + kcnt, kb + kchunk);
    const long ioff = (long)inst * a.sN;
    const bool active = (i0 + 2 * tx < nx) && (j0 + ty < ny);   // threads past the edge run along, storing nothing
    const unsigned plane = (unsigned)nx * ny;
    const double* src[6] = {a.u + ioff, a.v + ioff, a.w + ioff, a.b + ioff, a.ub, a.bb};
    const double* pc = a.pc ? a.pc + ioff : nullptr;
    const int tid = ty * (kTX / 2) + tx;

    // offset in the plane of the tiles' pair in row r, pair column p (full
    // modulo: tiles may be wider than the grid)
    auto pair_at = [&](int r, int p) -> unsigned {
        const int gi = ((i0 - 2 + 2 * p) % nx + nx) % nx, gj = ((j0 - 1 + r) % ny + ny) % ny;
        return (unsigned)gj * nx + gi;
    };
    // every thread copies (and corrects) its own pair; the halo pairs, the
    // tiles' outer rows and then the outer columns of the rows between, go to
    // the low threads (fields) and to the high ones (pressure)
    constexpr int XF = L::FCH - NT, XP = L::PCH - NT;
    static_assert(XF <= NT && XP <= NT, "two pairs a thread");
    const unsigned gcol = pair_at(ty + 1, tx + 1);
    const int pos = (ty + 1) * L::FP + 2 * tx + 2, posp = (ty + 1) * L::PP + 2 * tx + 2;
    const bool more_f = tid < XF, more_p = pc != nullptr && tid >= NT - XP;
    unsigned gfx, gpx;
    int sfx, spx, cqx;   // cqx: the halo field pair's place in the pressure tile
    {
        constexpr int FC = L::FP / 2, PC = L::PP / 2;
        int r, p, t = more_f ? tid : 0;
        if (t < 2 * FC) { r = t < FC ? 0 : BY + 1; p = t < FC ? t : t - FC; }
        else { t -= 2 * FC; r = 1 + t / 2; p = t % 2 ? FC - 1 : 0; }
        gfx = pair_at(r, p); sfx = r * L::FP + 2 * p; cqx = r * L::PP + 2 * p;
        t = more_p ? tid - (NT - XP) : 0;
        if (t < 3 * PC) { r = t < PC ? 0 : (t < 2 * PC ? BY + 1 : BY + 2); p = t % PC; }
        else { t -= 3 * PC; r = 1 + t / 3; p = t % 3 == 0 ? 0 : PC - 3 + t % 3; }
        gpx = pair_at(r, p); spx = r * L::PP + 2 * p;
    }
    auto copy_fields = [&](int kk) {
        const unsigned o = (unsigned)wrap(kk, nz) * plane;
        double* d = sm.pl[kk & 3][0];
#pragma unroll
        for (int f = 0; f < NF; ++f) cp_async<16>(d + f * (L::FP * L::FR) + pos, src[f] + (o + gcol));
        if (more_f) {
#pragma unroll
            for (int f = 0; f < NF; ++f) cp_async<16>(d + f * (L::FP * L::FR) + sfx, src[f] + (o + gfx));
        }
    };
    auto copy_p = [&](int kk) {
        if (!pc) return;
        const unsigned o = (unsigned)wrap(kk, nz) * plane;
        double* d = sm.pp[kk & 3];
        cp_async<16>(d + posp, pc + (o + gcol));
        if (more_p) cp_async<16>(d + spx, pc + (o + gpx));
    };
    // the previous step's pressure-gradient correction
    // (pressure_solver.f90:98-110) of a landed plane, in place
    auto correct_pair = [&](int kk, int fpos, int ppos, bool lid) {
        const double* q = &sm.pp[kk & 3][ppos];
        const double2 p0 = *reinterpret_cast<const double2*>(q);
        const double pe = q[2];
        const double2 pn = *reinterpret_cast<const double2*>(q + L::PP);
        const double2 pt = *reinterpret_cast<const double2*>(&sm.pp[(kk + 1) & 3][ppos]);
        constexpr int FS = L::FP * L::FR;
        double2* u = reinterpret_cast<double2*>(&sm.pl[kk & 3][0][fpos]);
        double2* v = u + FS / 2;
        double2* w = v + FS / 2;
        double2 x = *u, y = *v, z = *w;
        x.x = x.x - a.dtp * (p0.y - p0.x) * a.rdx;
        x.y = x.y - a.dtp * (pe - p0.y) * a.rdx;
        y.x = y.x - a.dtp * (pn.x - p0.x) * a.rdy;
        y.y = y.y - a.dtp * (pn.y - p0.y) * a.rdy;
        z.x = lid ? 0.0 : z.x - a.dtwp * (pt.x - p0.x) * a.rdz;
        z.y = lid ? 0.0 : z.y - a.dtwp * (pt.y - p0.y) * a.rdz;
        *u = x; *v = y; *w = z;
    };
    auto correct = [&](int kk, bool lid) {
        if (!pc) return;
        correct_pair(kk, pos, posp, lid);
        if (more_f) correct_pair(kk, sfx, cqx, lid);
    };
    auto is_lid = [&](int kk) { return a.rigid && wrap(wrap(kk, nz) + kofs, nzg) == nzg - 1; };
    // field f at the thread's pair (or one point) shifted by (di, dj) in a ring slot
    auto at2 = [&](int s, int f, int dj, double* o) {
        const double2 v = *reinterpret_cast<const double2*>(&sm.pl[s][f][pos + dj * L::FP]);
        o[0] = v.x; o[1] = v.y;
    };
    auto at1 = [&](int s, int f, int di, int dj) -> double { return sm.pl[s][f][pos + dj * L::FP + di]; };

    // the level's Adams-Bashforth history, into the thread's own slot
    const bool h1 = a.do_ab && a.ab1 != 0.0, h2 = a.do_ab && a.ab2 != 0.0;
    auto copy_history = [&](int kk) {
        const long g = (long)(unsigned)((unsigned)kk * plane + gcol) + ioff;
        if (h1) {
            cp_async<sizeof(T2)>(&sm.hist[0][0][tid], (const TT*)a.t1[0] + g);
            cp_async<sizeof(T2)>(&sm.hist[0][1][tid], (const TT*)a.t1[1] + g);
            cp_async<sizeof(T2)>(&sm.hist[0][2][tid], (const TT*)a.t1[3] + g);
            cp_async<16>(&sm.hw[0][tid], (const TW*)a.t1[2] + g);
        }
        if (h2) {
            cp_async<sizeof(T2)>(&sm.hist[1][0][tid], (const TT*)a.t2[0] + g);
            cp_async<sizeof(T2)>(&sm.hist[1][1][tid], (const TT*)a.t2[1] + g);
            cp_async<sizeof(T2)>(&sm.hist[1][2][tid], (const TT*)a.t2[3] + g);
            cp_async<16>(&sm.hw[1][tid], (const TW*)a.t2[2] + g);
        }
    };

    for (int kk = kb - 1; kk <= min(kb + 2, ke); ++kk) copy_fields(kk);
    for (int kk = kb - 1; kk <= min(kb + 2, ke + 1); ++kk) copy_p(kk);
    cp_commit();
    copy_history(kb);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    correct(kb - 1, is_lid(kb - 1));
    __syncthreads();
    if (kb + 2 <= ke) copy_p(kb + 3);   // into level kb-1's place
    cp_commit();
    correct(kb, is_lid(kb));
    correct(kb + 1, is_lid(kb + 1));
    cp_wait<0>();
    __syncthreads();   // three levels corrected; p of level kb+3 has landed
    const double Ro = a.Ro, rdx = a.rdx, rdy = a.rdy, rdz = a.rdz;
    const bool rigid = a.rigid;
    StepCarry c;
    {
        const int s2 = (kb - 1) & 3, s0 = kb & 3;
        const bool bot = rigid && (kb + kofs == 0);   // flux_top(0) = 0
        double um[2], vm[2], bm[2], wn[2], we[2];
        at2(s2, 0, 0, um); at2(s2, 1, 0, vm); at2(s2, 2, 0, c.wm); at2(s2, 3, 0, bm);
        at2(s0, 0, 0, c.u0); at2(s0, 1, 0, c.v0); at2(s0, 2, 0, c.w0); at2(s0, 3, 0, c.b0);
        c.uw = at1(s0, 0, -1, 0);
        at2(s0, 1, -1, c.vs);
        at2(s2, 2, 1, wn);
        we[0] = c.wm[1]; we[1] = at1(s2, 2, 2, 0);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            c.tb[q] = bot ? 0.0 : (bm[q] + c.b0[q]) * c.wm[q];
            c.tu[q] = bot ? 0.0 : (c.u0[q] + um[q]) * (c.wm[q] + we[q]);
            c.tv[q] = bot ? 0.0 : (c.v0[q] + vm[q]) * (c.wm[q] + wn[q]);
            // rigid lid zeroes flux_top(nz-1:nz+2) for w (advection.f90:167-170)
            c.tw[q] = (bot || (rigid && kb + kofs >= nzg - 1)) ? 0.0 : (c.w0[q] + c.wm[q]) * (c.wm[q] + c.w0[q]);
            if constexpr (HARM > 0) {
                c.hu[q] = bot ? 0.0 : a.Av * (c.u0[q] - um[q]) * rdz;
                c.hv[q] = bot ? 0.0 : a.Av * (c.v0[q] - vm[q]) * rdz;
                c.hw[q] = bot ? 0.0 : a.Av * (c.w0[q] - c.wm[q]) * rdz;
            }
            if constexpr (HARM > 1) c.hb[q] = bot ? 0.0 : a.Kv * (c.b0[q] - bm[q]) * rdz;
        }
        if constexpr (BG) {
            double U0[2], Um[2], B0[2], Bm[2];
            at2(s0, 4, 0, U0); at2(s2, 4, 0, Um); at2(s0, 5, 0, B0); at2(s2, 5, 0, Bm);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                c.gu[q] = bot ? 0.0 : 0.25 * (U0[q] + Um[q]) * (c.wm[q] + we[q]);
                c.gb[q] = bot ? 0.0 : 0.5 * (Bm[q] + B0[q]) * c.wm[q];
            }
        }
    }
    __syncthreads();   // level kb-1 is read: its place is filled next
    // one level; LID: the level may touch the rigid lid
    auto level = [&](int k, auto lid_c) {
        constexpr bool LID = decltype(lid_c)::value;
        const int s0 = k & 3, s1 = (k + 1) & 3;
        const long g = (long)(unsigned)((unsigned)k * plane + gcol) + ioff;
        if (k + 3 <= ke) {
            copy_fields(k + 3);
            copy_p(k + 4);
        }
        cp_commit();
        [[maybe_unused]] double2 fr[4], fi[4];   // the wavemaker's fields
        if constexpr (WM) {
            const unsigned gi = (unsigned)k * plane + gcol;   // within the instance
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                fr[f] = a.wr[f] ? __ldg(reinterpret_cast<const double2*>(a.wr[f] + gi)) : make_double2(0.0, 0.0);
                fi[f] = a.wi[f] ? __ldg(reinterpret_cast<const double2*>(a.wi[f] + gi)) : make_double2(0.0, 0.0);
            }
        }
        const int kg = k + kofs;                     // global level
        const bool top = LID && rigid && (kg == nzg - 1);   // flux_top(nz) = 0
        // rows: [0] is the point west of the pair (U, V, W, B and Un, Ut) or the pair's first (others)
        double U[4], V[4], W[4], B[4], Us[2], Un[3], Vs[3], Vn[2], Ws[2], Wn[2], Bs[2], Bn[2];
        double Ut[3], Vt[2], Wt[2], Bt[2], Vst[2];
        U[0] = c.uw; U[1] = c.u0[0]; U[2] = c.u0[1]; U[3] = at1(s0, 0, 2, 0);
        V[0] = at1(s0, 1, -1, 0); V[1] = c.v0[0]; V[2] = c.v0[1]; V[3] = at1(s0, 1, 2, 0);
        W[0] = at1(s0, 2, -1, 0); W[1] = c.w0[0]; W[2] = c.w0[1]; W[3] = at1(s0, 2, 2, 0);
        B[0] = at1(s0, 3, -1, 0); B[1] = c.b0[0]; B[2] = c.b0[1]; B[3] = at1(s0, 3, 2, 0);
        at2(s0, 0, -1, Us); Un[0] = at1(s0, 0, -1, 1); at2(s0, 0, 1, Un + 1);
        Vs[0] = c.vs[0]; Vs[1] = c.vs[1]; Vs[2] = at1(s0, 1, 2, -1); at2(s0, 1, 1, Vn);
        at2(s0, 2, -1, Ws); at2(s0, 2, 1, Wn);
        at2(s0, 3, -1, Bs); at2(s0, 3, 1, Bn);
        Ut[0] = at1(s1, 0, -1, 0); at2(s1, 0, 0, Ut + 1);
        at2(s1, 1, 0, Vt); at2(s1, 1, -1, Vst); at2(s1, 2, 0, Wt); at2(s1, 3, 0, Bt);
        double du[2], dv[2], dw[2], db[2], u1[2], v1[2], w1[2], b1[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double u0 = U[q + 1], v0 = V[q + 1], w0 = W[q + 1], b0 = B[q + 1];
            const double ue = U[q + 2], uw = U[q], ve = V[q + 2], vw = V[q], we = W[q + 2], ww = W[q];
            // ---- buoyancy advection + N^2 (advection.f90:12-47, integrate.f90:21-23)
            // The reference's 0.5 and 0.25 flux factors are powers of two: they
            // are carried in the per-axis factors a.hd* = 0.5/d*, a.qd* = 0.25/d*
            // (and 0.25 f0, 0.5 N0^2, set by the launcher), a multiply saved per
            // flux; scaling by a power of two rounds exactly.  Which of a
            // difference's two fluxes is rounded before the subtraction is
            // written out (a point shares fluxes with its pair and with the
            // level above), so that every form of the kernel gives the same bits.
            if (a.nonlinear) {
                {
                    const double x = __dsub_rn(__dmul_rn(b0 + B[q + 2], u0), __dmul_rn(B[q] + b0, uw));
                    const double y = __fma_rn(-(Bs[q] + b0), Vs[q], __dmul_rn(b0 + Bn[q], v0));
                    const double t = top ? 0.0 : __dmul_rn(b0 + Bt[q], w0);
                    db[q] = -Ro * (x * a.hdx + y * a.hdy + __dsub_rn(t, c.tb[q]) * a.hdz);
                    c.tb[q] = t;
                }
                // ---- zonal momentum (advection.f90:65-100)
                const double uv = __dmul_rn(u0 + Un[q + 1], ve + v0);          // (u_n)(v_e), also v's eastern flux
                const double uw_ = __dmul_rn(Ut[q + 1] + u0, w0 + we);         // (u_t)(w_e), also w's eastern flux
                {
                    const double x = __fma_rn(u0 + ue, ue + u0, -__dmul_rn(uw + u0, u0 + uw));
                    const double y = __fma_rn(-(Us[q] + u0), Vs[q + 1] + Vs[q], uv);
                    const double t = top ? 0.0 : uw_;
                    du[q] = -Ro * (x * a.qdx + y * a.qdy + __dsub_rn(t, c.tu[q]) * a.qdz);
                    c.tu[q] = t;
                }
                // ---- meridional momentum (advection.f90:104-140)
                const double vw_ = __dmul_rn(Vt[q] + v0, w0 + Wn[q]);          // (v_t)(w_n), also w's northern flux
                {
                    const double x = __fma_rn(-(vw + v0), Un[q] + uw, uv);
                    const double y = __fma_rn(v0 + Vn[q], Vn[q] + v0, -__dmul_rn(Vs[q] + v0, v0 + Vs[q]));
                    const double t = top ? 0.0 : vw_;
                    dv[q] = -Ro * (x * a.qdx + y * a.qdy + __dsub_rn(t, c.tv[q]) * a.qdz);
                    c.tv[q] = t;
                }
                // ---- vertical momentum (advection.f90:145-181)
                {
                    const bool wtop = LID && rigid && (kg >= nzg - 2);
                    const double x = __dsub_rn(uw_, __dmul_rn(ww + w0, uw + Ut[q]));
                    const double y = __dsub_rn(vw_, __dmul_rn(Ws[q] + w0, Vs[q] + Vst[q]));
                    const double t = wtop ? 0.0 : __dmul_rn(Wt[q] + w0, w0 + Wt[q]);
                    dw[q] = -a.dsqr * Ro * (x * a.qdx + y * a.qdy + __dsub_rn(t, c.tw[q]) * a.qdz);
                    c.tw[q] = t;
                }
            } else {
                db[q] = du[q] = dv[q] = dw[q] = 0.0;
            }
            db[q] = db[q] - (w0 + c.wm[q]) * a.hN0sq;
            // ---- Coriolis, buoyancy force, rigid-lid mask (integrate.f90:37-54)
            du[q] = du[q] + (v0 + Vs[q] + ve + Vs[q + 1]) * a.qf0;
            dv[q] = dv[q] - (uw + u0 + Un[q] + Un[q + 1]) * a.qf0;
            dw[q] = dw[q] + 0.5 * (b0 + Bt[q]);
            if (top) dw[q] = 0.0;
            // ---- friction, in place before AB (integrate.f90:59-66)
            u1[q] = u0; v1[q] = v0; w1[q] = w0; b1[q] = b0;
            if constexpr (HARM > 0) {
                const double dt = a.dt;
#define HARMONIC(f0, fe, fw, fn, fs, ft, Hm, Vm, low, out)                                     \
    {                                                                                        \
        const double x = __fma_rn(Hm * (fe - f0), rdx, -__dmul_rn(Hm * (f0 - fw), rdx));     \
        const double y = __fma_rn(Hm * (fn - f0), rdy, -__dmul_rn(Hm * (f0 - fs), rdy));     \
        const double t = top ? 0.0 : Vm * (ft - f0) * rdz;                                   \
        out = f0 + dt * (x * rdx + y * rdy + __dsub_rn(t, low) * rdz);                       \
        low = t;                                                                             \
    }
                if (HARM == 1 || a.harm_uvw) {
                    HARMONIC(u0, ue, uw, Un[q + 1], Us[q], Ut[q + 1], a.Ah, a.Av, c.hu[q], u1[q])
                    HARMONIC(v0, ve, vw, Vn[q], Vs[q], Vt[q], a.Ah, a.Av, c.hv[q], v1[q])
                    HARMONIC(w0, we, ww, Wn[q], Ws[q], Wt[q], a.Ah, a.Av, c.hw[q], w1[q])
                    if (top) w1[q] = 0.0;
                }
                if (HARM > 1 && a.harm_b) HARMONIC(b0, B[q + 2], B[q], Bn[q], Bs[q], Bt[q], a.Kh, a.Kv, c.hb[q], b1[q])
#undef HARMONIC
            }
        }
        // ---- set_forcing: background-flow advection (lee_wave1.f90:245-312)
        if constexpr (BG) {
            double P[4], Pn[3], Ps[2], Pt[3], Q[4], Qn[2], Qs[2], Qt[2];   // U_back, B_back
            P[0] = at1(s0, 4, -1, 0); at2(s0, 4, 0, P + 1); P[3] = at1(s0, 4, 2, 0);
            Pn[0] = at1(s0, 4, -1, 1); at2(s0, 4, 1, Pn + 1); at2(s0, 4, -1, Ps);
            Pt[0] = at1(s1, 4, -1, 0); at2(s1, 4, 0, Pt + 1);
            Q[0] = at1(s0, 5, -1, 0); at2(s0, 5, 0, Q + 1); Q[3] = at1(s0, 5, 2, 0);
            at2(s0, 5, 1, Qn); at2(s0, 5, -1, Qs); at2(s1, 5, 0, Qt);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double u0 = U[q + 1], v0 = V[q + 1], w0 = W[q + 1], b0 = B[q + 1];
                {
                    const double x = __fma_rn(-(0.5 * (P[q] + P[q + 1])), u0 + U[q], __dmul_rn(0.5 * (P[q + 1] + P[q + 2]), U[q + 2] + u0));
                    const double y = __fma_rn(0.25 * (P[q + 1] + Pn[q + 1]), V[q + 2] + v0, -__dmul_rn(0.25 * (Ps[q] + P[q + 1]), Vs[q + 1] + Vs[q]));
                    const double t = top ? 0.0 : __dmul_rn(0.25 * (Pt[q + 1] + P[q + 1]), w0 + W[q + 2]);
                    du[q] = du[q] - Ro * (x * rdx + y * rdy + __dsub_rn(t, c.gu[q]) * rdz);
                    c.gu[q] = t;
                }
                {
                    const double x = __fma_rn(0.25 * (v0 + V[q + 2]), Pn[q + 1] + P[q + 1], -__dmul_rn(0.25 * (V[q] + v0), Pn[q] + P[q]));
                    dv[q] = dv[q] - Ro * x * rdx;
                }
                {
                    const double x = __fma_rn(0.25 * (w0 + W[q + 2]), P[q + 1] + Pt[q + 1], -__dmul_rn(0.25 * (W[q] + w0), P[q] + Pt[q]));
                    dw[q] = dw[q] - a.dsqr * Ro * x * rdx;
                }
                {
                    const double e = __fma_rn(0.5 * (b0 + B[q + 2]), P[q + 1], __dmul_rn(0.5 * (Q[q + 1] + Q[q + 2]), u0));
                    const double em = __fma_rn(0.5 * (B[q] + b0), P[q], __dmul_rn(0.5 * (Q[q] + Q[q + 1]), U[q]));
                    const double y = __dsub_rn(__dmul_rn(0.5 * (Q[q + 1] + Qn[q]), v0), __dmul_rn(0.5 * (Qs[q] + Q[q + 1]), Vs[q]));
                    const double t = top ? 0.0 : __dmul_rn(0.5 * (Q[q + 1] + Qt[q]), w0);
                    db[q] = db[q] - Ro * (__dsub_rn(e, em) * rdx + y * rdy + __dsub_rn(t, c.gb[q]) * rdz);
                    c.gb[q] = t;
                }
            }
        }
        // ---- set_forcing: wavemaker (config.f90:224-237)
        if constexpr (WM) {
            const double dt = a.dt, cw = a.wm_c, sw = a.wm_s;
            double* o[4] = {u1, v1, w1, b1};
#pragma unroll
            for (int f = 0; f < 4; ++f)
                if (a.wr[f] || a.wi[f]) {
                    o[f][0] = o[f][0] + dt * (cw * fr[f].x + sw * fi[f].x);
                    o[f][1] = o[f][1] + dt * (cw * fr[f].y + sw * fi[f].y);
                }
        }
        // ---- store tendency of time level tau
        if (active) {
            T2 t;
            t.x = (TT)du[0]; t.y = (TT)du[1]; *reinterpret_cast<T2*>((TT*)a.t0[0] + g) = t;
            t.x = (TT)dv[0]; t.y = (TT)dv[1]; *reinterpret_cast<T2*>((TT*)a.t0[1] + g) = t;
            *reinterpret_cast<double2*>((TW*)a.t0[2] + g) = make_double2(dw[0], dw[1]);
            t.x = (TT)db[0]; t.y = (TT)db[1]; *reinterpret_cast<T2*>((TT*)a.t0[3] + g) = t;
        }
        // ---- Adams-Bashforth (integrate.f90:87-102)
        if (a.do_ab) {
            const double dt = a.dt, dtw = a.dtw;
            const double c0 = a.ab0, c1 = a.ab1, c2 = a.ab2;
            // the current tendency enters at full precision; only the
            // stored history (FP32 in the mixed path) is rounded
            double tu[2], tv[2], tw[2], tb[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) { tu[q] = c0 * du[q]; tv[q] = c0 * dv[q]; tw[q] = c0 * dw[q]; tb[q] = c0 * db[q]; }
            cp_wait<1>();   // this level's history has landed (the thread's own copies)
            auto add = [&](double cc, int l) {
                const T2 hu = sm.hist[l][0][tid], hv = sm.hist[l][1][tid], hb = sm.hist[l][2][tid];
                const double2 hw = sm.hw[l][tid];
                tu[0] = tu[0] + cc * (double)hu.x; tu[1] = tu[1] + cc * (double)hu.y;
                tv[0] = tv[0] + cc * (double)hv.x; tv[1] = tv[1] + cc * (double)hv.y;
                tw[0] = tw[0] + cc * hw.x; tw[1] = tw[1] + cc * hw.y;
                tb[0] = tb[0] + cc * (double)hb.x; tb[1] = tb[1] + cc * (double)hb.y;
            };
            if (h1) add(c1, 0);
            if (h2) add(c2, 1);
            if (k + 1 < ke) copy_history(k + 1);
            cp_commit();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                u1[q] = u1[q] + dt * tu[q]; v1[q] = v1[q] + dt * tv[q];
                w1[q] = w1[q] + dtw * tw[q]; b1[q] = b1[q] + dt * tb[q];
            }
        }
        if (active) {
            *reinterpret_cast<double2*>(a.uo + g) = make_double2(u1[0], u1[1]);
            *reinterpret_cast<double2*>(a.vo + g) = make_double2(v1[0], v1[1]);
            *reinterpret_cast<double2*>(a.wo + g) = make_double2(w1[0], w1[1]);
            *reinterpret_cast<double2*>(a.bo + g) = make_double2(b1[0], b1[1]);
        }
        c.uw = Ut[0];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            c.wm[q] = W[q + 1];
            c.u0[q] = Ut[q + 1]; c.v0[q] = Vt[q]; c.w0[q] = Wt[q]; c.b0[q] = Bt[q]; c.vs[q] = Vst[q];
        }
        if (k + 2 <= ke) correct(k + 2, LID && is_lid(k + 2));
        if (a.do_ab) cp_wait<1>();   // the planes; the next level's history may be on its way
        else cp_wait<0>();
        __syncthreads();
    };
    // levels whose planes stay below the lid go in pairs (the carried values
    // change registers by name instead of by moves), the others one by one
    const int km = rigid ? min(ke, nzg - 3 - kofs) : ke;
    int k = kb;
#pragma unroll 1
    for (; k + 1 < km; k += 2) {
        level(k, std::false_type());
        level(k + 1, std::false_type());
    }
#pragma unroll 1
    for (; k < ke; ++k) level(k, std::true_type());
}

// Blocks an SM the step kernels are built for: the plain and the u, v, w
// friction forms fit 168 registers without a spill and run three (held to two
// they took 9 % longer in FP64 and 11 % mixed at 256x256x128), the others would
// spill and run two.
constexpr int step_blocks(int harm, bool wm, bool bg) { return harm > 1 || wm || bg ? 2 : 3; }

template <typename TT, int BY, int HARM, bool WM, bool BG>
__global__ void __launch_bounds__(kTX / 2 * BY, step_blocks(HARM, WM, BG)) k_step(const StepArgs a, int kchunk) {
    pdl_trigger();
    pdl_wait();   // the state, p and history were written by the preceding kernels
    step_tile<TT, BY, HARM, WM, BG>(a, kchunk, blockIdx.x, blockIdx.y, blockIdx.z);
}

// One launch over the grids of several groups (an ensemble's members of
// uneven sizes): block b belongs to the group g with blk0[g] <= b <
// blk0[g+1] and runs that group's tile as k_step would.  The table rides in
// the kernel's parameter space (captured by value into a CUDA graph).
template <typename TT, int BY, int HARM, bool WM, bool BG>
__global__ void __launch_bounds__(kTX / 2 * BY, step_blocks(HARM, WM, BG)) k_step_groups(const __grid_constant__ StepGroups m) {
    pdl_trigger();
    pdl_wait();
    int g = 0;
    while (g + 1 < m.n && (int)blockIdx.x >= m.blk0[g + 1]) ++g;
    const int l = blockIdx.x - m.blk0[g];
    const int gx = m.gx[g], gy = m.gy[g];
    step_tile<TT, BY, HARM, WM, BG>(m.a[g], m.a[g].kchunk, l % gx, (l / gx) % gy, l / (gx * gy));
}

// ---------------------------------------------------------------------------
// Generic friction stages with the reference's stale-halo semantics: the
// biharmonic operators of mixing.f90:96-217 run after harmonic() without a
// halo exchange, so any neighbour outside the interior still holds the
// start-of-step value.  `cur` is the field after the previous stage, `old`
// the start-of-step field; out = cur + dt*op(.).
// ---------------------------------------------------------------------------
__global__ void k_biharmonic_h(const double* __restrict__ cur, const double* __restrict__ old,
                               double* __restrict__ out, int nx, int ny, int nz,
                               double Hmix, double rdx, double rdy, double dt) {
    const long N = (long)nx * ny * nz;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < N; g += (long)gridDim.x * blockDim.x) {
        const int i = (int)(g % nx), j = (int)((g / nx) % ny), k = (int)(g / ((long)nx * ny));
        const long pk = (long)k * nx * ny;
        auto P = [&](int di, int dj) -> double {
            const int ii = i + di, jj = j + dj;
            const bool in = ii >= 0 && ii < nx && jj >= 0 && jj < ny;
            const long gg = pk + (long)wrap(jj, ny) * nx + wrap(ii, nx);
            return in ? cur[gg] : old[gg];
        };
        auto del2 = [&](int di, int dj) -> double {
            const double fe = -Hmix * (P(di + 1, dj) - P(di, dj)) * rdx;
            const double fem = -Hmix * (P(di, dj) - P(di - 1, dj)) * rdx;
            const double fn = -Hmix * (P(di, dj + 1) - P(di, dj)) * rdy;
            const double fnm = -Hmix * (P(di, dj) - P(di, dj - 1)) * rdy;
            return (fe - fem) * rdx + (fn - fnm) * rdy;
        };
        const double d0 = del2(0, 0);
        const double fe = (del2(1, 0) - d0) * rdx, fem = (d0 - del2(-1, 0)) * rdx;
        const double fn = (del2(0, 1) - d0) * rdy, fnm = (d0 - del2(0, -1)) * rdy;
        out[g] = cur[g] + dt * ((fe - fem) * rdx + (fn - fnm) * rdy);
    }
}

__global__ void k_biharmonic_v(const double* __restrict__ cur, const double* __restrict__ old,
                               double* __restrict__ out, int nx, int ny, int nz, int rigid,
                               double Vmix, double rdz, double dt) {
    const long N = (long)nx * ny * nz;
    const long plane = (long)nx * ny;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < N; g += (long)gridDim.x * blockDim.x) {
        const int k = (int)(g / plane);
        const long col = g - (long)k * plane;
        // 1-based level kr = k+1; flux_top(kr) lives between levels kr and kr+1
        auto P = [&](int kk) -> double {   // kk: 0-based level, may be outside
            const bool in = kk >= 0 && kk < nz;
            const long gg = (long)wrap(kk, nz) * plane + col;
            return in ? cur[gg] : old[gg];
        };
        auto ft1 = [&](int kr) -> double {  // first-stage flux at 1-based level kr
            if (rigid && (kr <= 0 || kr >= nz)) return 0.0;
            return -Vmix * (P(kr) - P(kr - 1)) * rdz;
        };
        auto del2 = [&](int kr) -> double { return (ft1(kr) - ft1(kr - 1)) * rdz; };
        auto ft2 = [&](int kr) -> double {
            if (rigid && (kr <= 0 || kr >= nz)) return 0.0;
            return (del2(kr + 1) - del2(kr)) * rdz;
        };
        const int kr = k + 1;
        out[g] = cur[g] + dt * ((ft2(kr) - ft2(kr - 1)) * rdz);
    }
}

// ---------------------------------------------------------------------------
// Biharmonic friction of all four fields, wavemaker and Adams-Bashforth in one
// pass over the step kernel's output (mixing.f90:96-217, config.f90:224-237,
// integrate.f90:68-102), where the stages above are a pass over memory each.
// A block marches up in z with the planes of the harmonic-updated fields in a
// three-slot ring (16-byte asynchronous copies, two points of halo); a thread
// applies the horizontal operator to its pair of points as a plane arrives
// and keeps the five levels that the vertical operator needs in registers.
// A neighbour outside the interior is read from the start-of-step field, as
// the reference's unexchanged halos hold it.
// 160 B a point (fields and three tendency levels read, fields written);
// 128x128x64 takes 47 us (3.6 TB/s; two blocks of 240 registers an SM wait on
// their FP64 chains), where eight friction passes, the wavemaker and
// Adams-Bashforth pass and the correction pass took 243 us.
// ---------------------------------------------------------------------------
template <int BY>
struct FrictionTile {
    static constexpr int NT = kTX / 2 * BY;
    static constexpr int FP = kTX + 4, FR = BY + 4, FS = FP * FR;   // columns i0-2 .. i0+33, rows j0-2 .. j0+BY+1
    static constexpr int XF = FP / 2 * FR - NT;                     // halo pairs
};

template <int BY>
__global__ void __launch_bounds__(kTX / 2 * BY, 2) k_friction_ab(const FrictionArgs a) {
    using L = FrictionTile<BY>;
    constexpr int NT = L::NT;
    static_assert(L::XF <= NT, "one halo pair a thread");
    pdl_trigger();
    pdl_wait();   // inputs written by the preceding kernels
    __shared__ __align__(16) double ring[3][4][L::FS];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * (kTX / 2) + tx;
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int i0 = blockIdx.x * kTX, j0 = blockIdx.y * BY;
    const int kb = blockIdx.z * a.kchunk, ke = min(nz, kb + a.kchunk);
    const bool active = (i0 + 2 * tx < nx) && (j0 + ty < ny);   // threads past the edge run along, storing nothing
    const unsigned plane = (unsigned)nx * ny;
    auto pair_at = [&](int r, int p, bool& in) -> unsigned {
        const int x = i0 - 2 + 2 * p, y = j0 - 2 + r;
        in = x >= 0 && x < nx && y >= 0 && y < ny;
        return (unsigned)((y % ny + ny) % ny) * nx + (x % nx + nx) % nx;
    };
    bool in0, inx;
    const unsigned gcol = pair_at(ty + 2, tx + 1, in0);
    const int pos = (ty + 2) * L::FP + 2 * tx + 2;
    const bool more = tid < L::XF;
    unsigned gx;
    int sx;
    {
        constexpr int FC = L::FP / 2;
        int r, p, t = more ? tid : 0;
        if (t < 4 * FC) { r = t / FC; p = t - r * FC; r = r < 2 ? r : BY + r; }
        else { t -= 4 * FC; r = 2 + t / 2; p = t % 2 ? FC - 1 : 0; }
        gx = pair_at(r, p, inx);
        sx = r * L::FP + 2 * p;
    }
    auto copy_plane = [&](int m) {
        const bool lin = m >= 0 && m < nz;
        const unsigned o = (unsigned)wrap(m, nz) * plane;
        double* d = ring[(m + 3) % 3][0];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            cp_async<16>(d + f * L::FS + pos, (lin && in0 ? a.h[f] : a.old[f]) + (o + gcol));
            if (more) cp_async<16>(d + f * L::FS + sx, (lin && inx ? a.h[f] : a.old[f]) + (o + gx));
        }
    };
    const double rdx2 = a.rdx * a.rdx, rdy2 = a.rdy * a.rdy, rdz = a.rdz, dt = a.dt;
    // the pair of field f at a landed level after the horizontal operator
    auto horizontal = [&](const double* t, double H, double* g) {
        const double2 c = *reinterpret_cast<const double2*>(t);
        g[0] = c.x; g[1] = c.y;
        if (H > 0.) {
            // rows j-2 .. j+2 of the pair and its neighbours: [2], [3] are the pair
            double r0[6], rn[4], rs[4];
            {
                const double2 w = *reinterpret_cast<const double2*>(t - 2), e = *reinterpret_cast<const double2*>(t + 2);
                r0[0] = w.x; r0[1] = w.y; r0[2] = c.x; r0[3] = c.y; r0[4] = e.x; r0[5] = e.y;
                const double2 n = *reinterpret_cast<const double2*>(t + L::FP), q = *reinterpret_cast<const double2*>(t - L::FP);
                rn[0] = t[L::FP - 1]; rn[1] = n.x; rn[2] = n.y; rn[3] = t[L::FP + 2];
                rs[0] = t[-L::FP - 1]; rs[1] = q.x; rs[2] = q.y; rs[3] = t[-L::FP + 2];
            }
            const double2 nn = *reinterpret_cast<const double2*>(t + 2 * L::FP);
            const double2 ss = *reinterpret_cast<const double2*>(t - 2 * L::FP);
            const double cx = -H * rdx2, cy = -H * rdy2;
            auto lap = [&](double w, double m, double e, double lo, double hi) {
                return ((e - m) - (m - w)) * cx + ((hi - m) - (m - lo)) * cy;
            };
            double d[4];   // first Laplacian at the pair and the points west and east of it
#pragma unroll
            for (int q = 0; q < 4; ++q) d[q] = lap(r0[q], r0[q + 1], r0[q + 2], rs[q], rn[q]);
            const double dn[2] = {lap(rn[0], rn[1], rn[2], c.x, nn.x), lap(rn[1], rn[2], rn[3], c.y, nn.y)};
            const double ds[2] = {lap(rs[0], rs[1], rs[2], ss.x, c.x), lap(rs[1], rs[2], rs[3], ss.y, c.y)};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double m = d[q + 1];
                g[q] = g[q] + dt * (((d[q + 2] - m) - (m - d[q])) * rdx2 + ((dn[q] - m) - (m - ds[q])) * rdy2);
            }
        }
    };
    double w[4][5][2];   // levels k-2 .. k+2 of the pair
    copy_plane(kb - 2);
    cp_commit();
    copy_plane(kb - 1);
    cp_commit();
    for (int m = kb - 2; m <= ke + 1; ++m) {
        cp_wait<1>();
        __syncthreads();   // plane m has landed; plane m-1 is read
        if (m + 2 <= ke + 1) copy_plane(m + 2);
        cp_commit();
        const int k = m - 2;
        const unsigned g = (unsigned)max(k, 0) * plane + gcol;
        double2 t0[4], t1[4], t2[4];
        const bool h1 = a.ab1 != 0.0, h2 = a.ab2 != 0.0;
        if (k >= kb) {
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                t0[f] = __ldg(reinterpret_cast<const double2*>(a.t0[f] + g));
                t1[f] = h1 ? __ldg(reinterpret_cast<const double2*>(a.t1[f] + g)) : make_double2(0.0, 0.0);
                t2[f] = h2 ? __ldg(reinterpret_cast<const double2*>(a.t2[f] + g)) : make_double2(0.0, 0.0);
            }
        }
        const double* pl = ring[(m + 3) % 3][0] + pos;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
#pragma unroll
            for (int q = 0; q < 4; ++q) { w[f][q][0] = w[f][q + 1][0]; w[f][q][1] = w[f][q + 1][1]; }
            // a level outside the interior holds the start-of-step value
            horizontal(pl + f * L::FS, m >= 0 && m < nz ? a.hmix[f] : 0.0, w[f][4]);
        }
        if (k < kb) continue;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            double o[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                double x = w[f][2][q];
                const double V = a.vmix[f];
                if (V > 0.) {
                    // fluxes between the window's levels; none through a rigid lid or bottom
                    double f1[4], d2[3];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        f1[j] = a.rigid && (k - 1 + j <= 0 || k - 1 + j >= nz) ? 0.0 : -V * (w[f][j + 1][q] - w[f][j][q]) * rdz;
#pragma unroll
                    for (int j = 0; j < 3; ++j) d2[j] = (f1[j + 1] - f1[j]) * rdz;
                    const double lo = a.rigid && k <= 0 ? 0.0 : (d2[1] - d2[0]) * rdz;
                    const double hi = a.rigid && k + 1 >= nz ? 0.0 : (d2[2] - d2[1]) * rdz;
                    x = x + dt * ((hi - lo) * rdz);
                    if (f == 2 && a.rigid && k == nz - 1) x = 0.0;   // w(:,:,nz:nz+2) = 0 after biharmonic_v(w)
                }
                o[q] = x;
            }
            if (a.wm_on && (a.wr[f] || a.wi[f])) {
                const double2 r = a.wr[f] ? __ldg(reinterpret_cast<const double2*>(a.wr[f] + g)) : make_double2(0.0, 0.0);
                const double2 i = a.wi[f] ? __ldg(reinterpret_cast<const double2*>(a.wi[f] + g)) : make_double2(0.0, 0.0);
                o[0] = o[0] + dt * (a.wm_c * r.x + a.wm_s * i.x);
                o[1] = o[1] + dt * (a.wm_c * r.y + a.wm_s * i.y);
            }
            const double h = f == 2 ? a.dtw : dt;
            double tx_ = a.ab0 * t0[f].x, ty_ = a.ab0 * t0[f].y;
            if (h1) { tx_ = tx_ + a.ab1 * t1[f].x; ty_ = ty_ + a.ab1 * t1[f].y; }
            if (h2) { tx_ = tx_ + a.ab2 * t2[f].x; ty_ = ty_ + a.ab2 * t2[f].y; }
            if (active) *reinterpret_cast<double2*>(a.out[f] + g) = make_double2(o[0] + h * tx_, o[1] + h * ty_);
        }
    }
}

// background-flow forcing on the friction-updated state (generic path).
// set_forcing runs after the in-place friction with no halo exchange, so a
// neighbour outside the interior still holds its start-of-step value: those
// reads go to the old fields (a.uo..bo hold the start-of-step state here,
// a.u..b the friction-updated one).
__global__ void k_forcing_background(StepArgs a) {
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const long N = (long)nx * ny * nz, plane = (long)nx * ny;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < N; g += (long)gridDim.x * blockDim.x) {
        const int i = (int)(g % nx), j = (int)((g / nx) % ny), k = (int)(g / plane);
        auto at = [&](const double* f, int di, int dj, int dk) -> double {
            return f[(long)wrap(k + dk, nz) * plane + (long)wrap(j + dj, ny) * nx + wrap(i + di, nx)];
        };
        auto st = [&](int fld, int di, int dj, int dk) -> double {
            const bool in = i + di >= 0 && i + di < nx && j + dj >= 0 && j + dj < ny && k + dk >= 0 && k + dk < nz;
            const double* cur = fld == 0 ? a.u : fld == 1 ? a.v : fld == 2 ? a.w : a.b;
            const double* old = fld == 0 ? a.uo : fld == 1 ? a.vo : fld == 2 ? a.wo : a.bo;
            return at(in ? cur : old, di, dj, dk);
        };
        const double *ub = a.ub, *bb = a.bb;
        const bool top = a.rigid && k == nz - 1, bot = a.rigid && k == 0;
        const double Ro = a.Ro, rdx = a.rdx, rdy = a.rdy, rdz = a.rdz;
        double* const* T0 = (double* const*)a.t0;
        double du_ = T0[0][g], dv_ = T0[1][g], dw_ = T0[2][g], db_ = T0[3][g];
        {
            const double e = 2 * 0.25 * (at(ub, 0, 0, 0) + at(ub, 1, 0, 0)) * (st(0, 1, 0, 0) + st(0, 0, 0, 0));
            const double em = 2 * 0.25 * (at(ub, -1, 0, 0) + at(ub, 0, 0, 0)) * (st(0, 0, 0, 0) + st(0, -1, 0, 0));
            const double n = 0.25 * (at(ub, 0, 0, 0) + at(ub, 0, 1, 0)) * (st(1, 1, 0, 0) + st(1, 0, 0, 0));
            const double nm = 0.25 * (at(ub, 0, -1, 0) + at(ub, 0, 0, 0)) * (st(1, 1, -1, 0) + st(1, 0, -1, 0));
            const double t = top ? 0.0 : 0.25 * (at(ub, 0, 0, 1) + at(ub, 0, 0, 0)) * (st(2, 0, 0, 0) + st(2, 1, 0, 0));
            const double tm = bot ? 0.0 : 0.25 * (at(ub, 0, 0, 0) + at(ub, 0, 0, -1)) * (st(2, 0, 0, -1) + st(2, 1, 0, -1));
            du_ = du_ - Ro * ((e - em) * rdx + (n - nm) * rdy + (t - tm) * rdz);
        }
        {
            const double e = 0.25 * (st(1, 0, 0, 0) + st(1, 1, 0, 0)) * (at(ub, 0, 1, 0) + at(ub, 0, 0, 0));
            const double em = 0.25 * (st(1, -1, 0, 0) + st(1, 0, 0, 0)) * (at(ub, -1, 1, 0) + at(ub, -1, 0, 0));
            dv_ = dv_ - Ro * (e - em) * rdx;
        }
        {
            const double e = 0.25 * (st(2, 0, 0, 0) + st(2, 1, 0, 0)) * (at(ub, 0, 0, 0) + at(ub, 0, 0, 1));
            const double em = 0.25 * (st(2, -1, 0, 0) + st(2, 0, 0, 0)) * (at(ub, -1, 0, 0) + at(ub, -1, 0, 1));
            dw_ = dw_ - a.dsqr * Ro * (e - em) * rdx;
        }
        {
            const double e = 0.5 * (st(3, 0, 0, 0) + st(3, 1, 0, 0)) * at(ub, 0, 0, 0) + 0.5 * (at(bb, 0, 0, 0) + at(bb, 1, 0, 0)) * st(0, 0, 0, 0);
            const double em = 0.5 * (st(3, -1, 0, 0) + st(3, 0, 0, 0)) * at(ub, -1, 0, 0) + 0.5 * (at(bb, -1, 0, 0) + at(bb, 0, 0, 0)) * st(0, -1, 0, 0);
            const double n = 0.5 * (at(bb, 0, 0, 0) + at(bb, 0, 1, 0)) * st(1, 0, 0, 0);
            const double nm = 0.5 * (at(bb, 0, -1, 0) + at(bb, 0, 0, 0)) * st(1, 0, -1, 0);
            const double t = top ? 0.0 : 0.5 * (at(bb, 0, 0, 0) + at(bb, 0, 0, 1)) * st(2, 0, 0, 0);
            const double tm = bot ? 0.0 : 0.5 * (at(bb, 0, 0, -1) + at(bb, 0, 0, 0)) * st(2, 0, 0, -1);
            db_ = db_ - Ro * ((e - em) * rdx + (n - nm) * rdy + (t - tm) * rdz);
        }
        T0[0][g] = du_; T0[1][g] = dv_; T0[2][g] = dw_; T0[3][g] = db_;
    }
}

// wavemaker + Adams-Bashforth, pointwise, in place on the state (generic path)
__global__ void k_wavemaker_ab(StepArgs a, int do_wm) {
    const long N = (long)a.nx * a.ny * a.nz;
    double* fld[4] = {a.uo, a.vo, a.wo, a.bo};
    const double* const* t0 = (const double* const*)a.t0;
    const double* const* t1 = (const double* const*)a.t1;
    const double* const* t2 = (const double* const*)a.t2;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < N; g += (long)gridDim.x * blockDim.x) {
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            double x = fld[f][g];
            if (do_wm && (a.wr[f] || a.wi[f]))
                x = x + a.dt * (a.wm_c * (a.wr[f] ? a.wr[f][g] : 0.0) + a.wm_s * (a.wi[f] ? a.wi[f][g] : 0.0));
            double t = a.ab0 * t0[f][g];
            if (a.ab1 != 0.0) t = t + a.ab1 * t1[f][g];
            if (a.ab2 != 0.0) t = t + a.ab2 * t2[f][g];
            fld[f][g] = x + (f == 2 ? a.dtw : a.dt) * t;
        }
    }
}

// ---------------------------------------------------------------------------
// pressure gradient correction, pressure_solver.f90:98-110 (and the rigid-lid
// ghost levels :82-93, which make the w correction vanish at level nz)
// ---------------------------------------------------------------------------
// levels kbeg .. kbeg+kcnt-1 of each instance; the rigid lid is global level
// nzg-1 with global level k + kofs
__global__ void k_correct(double* __restrict__ u, double* __restrict__ v, double* __restrict__ w,
                          const double* __restrict__ p, int nx, int ny, int nz, int rigid,
                          double dt, double dtw, double rdx, double rdy, double rdz, int batch,
                          int kbeg, int kcnt, int kofs, int nzg) {
    const long plane = (long)nx * ny, N = plane * nz, NW = plane * kcnt, NB = NW * batch;
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < NB; q += (long)gridDim.x * blockDim.x) {
        const long inst = q / NW, r = q - inst * NW;
        const long g = inst * N + (long)kbeg * plane + r;
        const int i = (int)(r % nx), j = (int)((r / nx) % ny), k = kbeg + (int)(r / plane);
        const double p0 = p[g];
        const double pe = p[g - i + wrap(i + 1, nx)];
        const double pn = p[g + (long)(wrap(j + 1, ny) - j) * nx];
        u[g] = u[g] - dt * (pe - p0) * rdx;
        v[g] = v[g] - dt * (pn - p0) * rdy;
        if (rigid && wrap(k + kofs, nzg) == nzg - 1) {
            w[g] = 0.0;
        } else {
            const double pt = p[g + (long)(wrap(k + 1, nz) - k) * plane];
            w[g] = w[g] - dtw * (pt - p0) * rdz;
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// the launcher-derived fields of a step and its grid of blocks
static dim3 prep_step(StepArgs& a, int by) {
    a.hdx = 0.5 * a.rdx; a.hdy = 0.5 * a.rdy; a.hdz = 0.5 * a.rdz;
    a.qdx = 0.25 * a.rdx; a.qdy = 0.25 * a.rdy; a.qdz = 0.25 * a.rdz;
    a.qf0 = 0.25 * a.f0; a.hN0sq = 0.5 * a.N0sq;
    const int kcnt = a.kcount ? a.kcount : a.nz;
    a.kchunk = a.kchunk > 0 ? std::min(a.kchunk, kcnt) : (kcnt <= 16 ? kcnt : 8);
    while ((long)((kcnt + a.kchunk - 1) / a.kchunk) * std::max(1, a.batch) > 65535 && a.kchunk < kcnt) ++a.kchunk;   // the grid's z limit
    return dim3((a.nx + kTX - 1) / kTX, (a.ny + by - 1) / by, ((kcnt + a.kchunk - 1) / a.kchunk) * std::max(1, a.batch));
}

template <typename TT, int BY, int HARM, bool WM, bool BG>
static cudaError_t launch_step_t(const StepArgs& a0, cudaStream_t s) {
    StepArgs a = a0;
    const dim3 grid = prep_step(a, BY);
    return launch_pdl(k_step<TT, BY, HARM, WM, BG>, grid, dim3(kTX / 2, BY), sizeof(StepSmem<TT, BY, BG ? 6 : 4>), s, a,
                      a.kchunk);
}

template <typename TT, int BY, int HARM, bool WM, bool BG>
static cudaError_t launch_step_groups_t(const StepArgs* in, int n, cudaStream_t s) {
    static_assert(sizeof(StepGroups) <= 32000, "grouped step table exceeds the kernel parameter space");
    StepGroups m{};
    m.n = n;
    long blocks = 0;
    for (int g = 0; g < n; ++g) {
        m.a[g] = in[g];
        const dim3 gr = prep_step(m.a[g], BY);
        m.gx[g] = (int)gr.x; m.gy[g] = (int)gr.y;
        m.blk0[g] = (int)blocks;
        blocks += (long)gr.x * gr.y * gr.z;
    }
    if (blocks > 0x7fffffffL) return cudaErrorInvalidValue;
    m.blk0[n] = (int)blocks;
    return launch_pdl(k_step_groups<TT, BY, HARM, WM, BG>, dim3((unsigned)blocks), dim3(kTX / 2, BY),
                      sizeof(StepSmem<TT, BY, BG ? 6 : 4>), s, m);
}

// friction of u, v, w alone (1) or of b as well (2), wavemaker, background flow
int step_flavour(const StepArgs& a) {
    return (a.harm_b ? 2 : (a.harm_uvw ? 1 : 0)) | (a.wm_on ? 4 : 0) | (a.ub ? 8 : 0);
}
// F(harm, wm, bg) for the instantiation that a flavour runs
#define PS3D_STEP_DISPATCH(flavour, F)                                                            \
    switch (flavour) {                                                                           \
        case 0: F(0, false, false); break;                                                       \
        case 1: F(1, false, false); break;                                                       \
        case 2: F(2, false, false); break;                                                       \
        case 4: F(0, true, false); break;                                                        \
        case 5: F(1, true, false); break;                                                        \
        case 6: F(2, true, false); break;                                                        \
        case 8: F(0, false, true); break;                                                        \
        case 9: F(1, false, true); break;                                                        \
        case 10: F(2, false, true); break;                                                       \
        case 12: F(0, true, true); break;                                                        \
        case 13: F(1, true, true); break;                                                        \
        default: F(2, true, true); break;                                                        \
    }

template <typename TT>
static cudaError_t launch_step_groups_tt(const StepArgs* a, int n, cudaStream_t s) {
    if (n < 1 || n > kMaxStepGroups) return cudaErrorInvalidValue;
    const int fl = step_flavour(a[0]);
    for (int g = 1; g < n; ++g)
        if (step_flavour(a[g]) != fl) return cudaErrorInvalidValue;
#define L(H, W, G) return launch_step_groups_t<TT, 8, H, W, G>(a, n, s)
    PS3D_STEP_DISPATCH(fl, L)
#undef L
    return cudaErrorInvalidValue;
}

cudaError_t launch_step_groups(const StepArgs* a, int n, bool fp32_tendencies, cudaStream_t s) {
    return fp32_tendencies ? launch_step_groups_tt<float>(a, n, s) : launch_step_groups_tt<double>(a, n, s);
}

template <typename TT>
static cudaError_t launch_step_tt(const StepArgs& a, cudaStream_t s) {
#define L(H, W, G) return launch_step_t<TT, 8, H, W, G>(a, s)
    PS3D_STEP_DISPATCH(step_flavour(a), L)
#undef L
    return cudaErrorInvalidValue;
}

template <typename TT>
static cudaError_t step_setup_tt() {
    cudaError_t e;
    // PS3D_STEP_CARVEOUT=<percent>: the shared-memory share of the unified
    // L1/shared storage the step kernels ask for (a hint to the driver)
    const char* cv = std::getenv("PS3D_STEP_CARVEOUT");
    const int carve = cv ? std::atoi(cv) : -1;
#define S(H, W, G)                                                                                        \
    if ((e = cudaFuncSetAttribute(k_step<TT, 8, H, W, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                                  (int)sizeof(StepSmem<TT, 8, G ? 6 : 4>))))                              \
        return e;                                                                                         \
    if ((e = cudaFuncSetAttribute(k_step_groups<TT, 8, H, W, G>,                                       \
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,                            \
                                  (int)sizeof(StepSmem<TT, 8, G ? 6 : 4>))))                              \
        return e;                                                                                         \
    if (carve >= 0 &&                                                                                     \
        (e = cudaFuncSetAttribute(k_step<TT, 8, H, W, G>, cudaFuncAttributePreferredSharedMemoryCarveout,  \
                                  carve)))                                                                \
        return e;
    for (int fl = 0; fl < 15; ++fl) {
        if (fl % 4 == 3) continue;
        PS3D_STEP_DISPATCH(fl, S)
    }
#undef S
    return cudaSuccess;
}
// opts the step kernels in to their dynamic shared memory (above 48 KB with
// the background fields)
cudaError_t step_setup() {
    cudaError_t e = step_setup_tt<double>();
    return e != cudaSuccess ? e : step_setup_tt<float>();
}

// resident blocks per SM of the fused step kernel that launch_step(a) runs
template <typename TT>
static int step_resident_tt(const StepArgs& a) {
    int n = 0;
    cudaError_t e = cudaSuccess;
#define R(H, W, G)                                                                                            \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_step<TT, 8, H, W, G>, kTX / 2 * 8,                   \
                                                      sizeof(StepSmem<TT, 8, G ? 6 : 4>));
    PS3D_STEP_DISPATCH(step_flavour(a), R)
#undef R
    if (e != cudaSuccess) { cudaGetLastError(); return 1; }
    return n > 0 ? n : 1;
}
int step_resident(const StepArgs& a, bool fp32_tendencies) {
    return fp32_tendencies ? step_resident_tt<float>(a) : step_resident_tt<double>(a);
}

cudaError_t launch_step(const StepArgs& a, bool fp32_tendencies, cudaStream_t s) {
    return fp32_tendencies ? launch_step_tt<float>(a, s) : launch_step_tt<double>(a, s);
}

static inline int grid_for(long n, int threads) {
    long b = (n + threads - 1) / threads;
    return (int)std::min<long>(b, 148L * 16);
}

// The z chunk minimises waves x (levels + 6): the march loads four planes more
// than it writes, and starting costs about two.
cudaError_t launch_friction(const FrictionArgs& a0, cudaStream_t s) {
    FrictionArgs a = a0;
    static const int per_sm = [] {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_friction_ab<8>, kTX / 2 * 8, 0) != cudaSuccess) cudaGetLastError();
        return n > 0 ? n : 1;
    }();
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long slots = (long)sms * per_sm, tiles = (long)((a.nx + kTX - 1) / kTX) * ((a.ny + 7) / 8);
    double best = 1e300;
    for (int kc = (a.nz + 65534) / 65535; kc <= std::min(a.nz, 64); ++kc) {
        const double c = (double)((tiles * ((a.nz + kc - 1) / kc) + slots - 1) / slots) * (kc + 6);
        if (c < best) { best = c; a.kchunk = kc; }
    }
    return launch_pdl(k_friction_ab<8>, dim3((a.nx + kTX - 1) / kTX, (a.ny + 7) / 8, (a.nz + a.kchunk - 1) / a.kchunk),
                      dim3(kTX / 2, 8), 0, s, a);
}

cudaError_t launch_biharmonic_h(const double* cur, const double* old, double* out, int nx, int ny, int nz,
                                double Hmix, double rdx, double rdy, double dt, cudaStream_t s) {
    const long N = (long)nx * ny * nz;
    k_biharmonic_h<<<grid_for(N, 256), 256, 0, s>>>(cur, old, out, nx, ny, nz, Hmix, rdx, rdy, dt);
    return cudaGetLastError();
}
cudaError_t launch_biharmonic_v(const double* cur, const double* old, double* out, int nx, int ny, int nz,
                                int rigid, double Vmix, double rdz, double dt, cudaStream_t s) {
    const long N = (long)nx * ny * nz;
    k_biharmonic_v<<<grid_for(N, 256), 256, 0, s>>>(cur, old, out, nx, ny, nz, rigid, Vmix, rdz, dt);
    return cudaGetLastError();
}
cudaError_t launch_forcing_background(const StepArgs& a, cudaStream_t s) {
    const long N = (long)a.nx * a.ny * a.nz;
    k_forcing_background<<<grid_for(N, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}
cudaError_t launch_wavemaker_ab(const StepArgs& a, int do_wm, cudaStream_t s) {
    const long N = (long)a.nx * a.ny * a.nz;
    k_wavemaker_ab<<<grid_for(N, 256), 256, 0, s>>>(a, do_wm);
    return cudaGetLastError();
}
cudaError_t launch_correct(double* u, double* v, double* w, const double* p, int nx, int ny, int nz, int rigid,
                           double dt, double dtw, double rdx, double rdy, double rdz, cudaStream_t s, int batch,
                           int kbeg, int kcount, int kofs, int nzg) {
    const int kcnt = kcount ? kcount : nz;
    const long N = (long)nx * ny * kcnt * batch;
    k_correct<<<grid_for(N, 256), 256, 0, s>>>(u, v, w, p, nx, ny, nz, rigid, dt, dtw, rdx, rdy, rdz, batch, kbeg, kcnt,
                                              kofs, nzg ? nzg : nz);
    return cudaGetLastError();
}

}  // namespace ps3d
