// swe_step.cu -- fused FP32 step of the DiffSWE2d finite-volume solver on
// sm_100a, and its C ABI (include/swe_b200.h).
//
// One SWE2D.step (src/solver.py:572-663) is two kernel launches:
//   stage 1: tendency k1 of the state U (spatial_operator, solver.py:448-531)
//            and the global maxima of the x/y face wave speeds (solver.py:
//            527-530), reduced in-kernel with warp max + one atomicMax per
//            warp into the step's reduction words;
//   stage 2: every block derives dt from those maxima (solver.py:620-626),
//            forms the predictor clean(U, U + dt/2 k1) on its tile plus a
//            two-cell halo, the tendency k2 of the predictor on its tile,
//            the corrector clean(U, U + dt k2) and the friction update
//            (solver.py:639-661), and writes U_out.
// The global reduction between the two stages is why the step is two
// launches: dt depends on every face of the grid.
//
// Two forms of the IEEE stages give the same bits.  In the tile form
// (stage_kernel, small and medium grids) each block owns a TX x TY tile: it
// stages the tile and a two-cell halo (ghost cells of add_ghost_cells,
// src/boundary.py:150-413, evaluated on the fly at the domain edge) in
// shared memory as per-cell primitives, then computes per-cell face-side
// values in both directions, then the HLL face fluxes, then each cell's
// tendency.  In the sweep form (sweep_kernel, large grids and ensembles)
// each warp walks down a strip of columns.  All arithmetic is FP32 on the CUDA
// cores (swe_math.cuh) in the reference's operation order.
#include <cuda_runtime.h>

#include <mutex>
#include <stdlib.h>
#include <string.h>

#include "swe_common.cuh"
#include "swe_sweep.cuh"
#include "swe_ensemble.cuh"

namespace swe {
namespace {

constexpr int TX = 32, TY = 8, NT = TX * TY;
constexpr int RX = TX + 4, RY = TY + 4;
constexpr int NXS = TY * (TX + 2);  // x-direction side cells per tile
constexpr int NYS = (TY + 2) * TX;  // y-direction side cells per tile
constexpr int NXF = TY * (TX + 1);  // x faces per tile
constexpr int NYF = (TY + 1) * TX;  // y faces per tile


// State of interior cell (j, i) as the stage sees it: U for stage 1, the
// predictor clean(U, U + hdt*k1) (solver.py:639) for stage 2.
template <int STAGE>
__device__ __forceinline__ State interior_state(const StepArgs& a, int b, int j, int i, float hdt) {
    const size_t plane = (size_t)a.ny * a.nx;
    const size_t o = at3(b, 0, j, i, a.ny, a.nx);
    State u{a.U[o], a.U[o + plane], a.U[o + 2 * plane]};
    if (STAGE == 1) return u;
    State c{u.h + hdt * a.tend[o], u.hu + hdt * a.tend[o + plane], u.hv + hdt * a.tend[o + 2 * plane]};
    return clean_and_limit(u, c, a.kc, a.positivity != 0);
}


// Padded cell (j, i) (interior coordinates, -2 <= j < ny+2) with the ghost
// rules of add_ghost_cells.  Only the four "arms" of the padding are ever
// used by the stencil (corner ghosts feed no face of an interior row or
// column), so a cell outside the interior in both directions, or beyond the
// two-cell padding, gets its clamped neighbour's value and is never read.
template <int STAGE>
__device__ __forceinline__ void region_cell(const StepArgs& a, int b, int j, int i, float hdt,
                                            State& s, float& z) {
    const int ny = a.ny, nx = a.nx;
    const bool jin = (unsigned)j < (unsigned)ny, iin = (unsigned)i < (unsigned)nx;
    const int jc = min(max(j, 0), ny - 1), ic = min(max(i, 0), nx - 1);
    if (jin && iin) {
        s = interior_state<STAGE>(a, b, j, i, hdt);
        z = bed_at(a, b, j, i);
        return;
    }
    const bool xarm = jin && i >= -2 && i < nx + 2;
    const bool yarm = iin && j >= -2 && j < ny + 2;
    if (!xarm && !yarm) {
        s = interior_state<STAGE>(a, b, jc, ic, hdt);
        z = bed_at(a, b, jc, ic);
        return;
    }
    int side, jm, im, jp, ip;
    if (xarm) {
        side = i < 0 ? 0 : 1;
        jm = j;
        im = i < 0 ? -1 - i : 2 * nx - 1 - i;  // flip of the first/last two columns
        jp = j;
        ip = i < 0 ? nx + i : i - nx;
    } else {
        side = j < 0 ? 2 : 3;
        im = i;
        jm = j < 0 ? -1 - j : 2 * ny - 1 - j;
        ip = i;
        jp = j < 0 ? ny + j : j - ny;
    }
    const int code = a.bc[side];
    if (code == SWE_BC_PERIODIC) {  // boundary.py:247-257, :301-302
        s = interior_state<STAGE>(a, b, jp, ip, hdt);
        z = bed_at(a, b, jp, ip);
        return;
    }
    z = bed_at(a, b, jc, ic);  // replicate padding of the bed, boundary.py:234-238
    if (code == SWE_BC_CONSTANT) {  // boundary.py:304-305
        s = State{a.cval, a.cval, a.cval};
        return;
    }
    s = interior_state<STAGE>(a, b, jc, ic, hdt);  // replicate padding, boundary.py:228-232
    const float lev = a.level[a.levelB == 1 ? 0 : b];
    if (code == SWE_BC_WATER_LEVEL) {  // boundary.py:279-282, :307-310
        s.h = fmaxf(lev - z, 0.0f);
    } else if (code == SWE_BC_WALL) {  // boundary.py:312-316
        State m = (jm == jc && im == ic) ? s : interior_state<STAGE>(a, b, jm, im, hdt);
        if (xarm) s.hu = -m.hu;
        else s.hv = -m.hv;
    } else if (code == SWE_BC_ABSORBING) {  // boundary.py:318-328
        const float hr = fmaxf(lev - z, 0.0f);
        const float hg = s.h;
        const float hc = hr > a.kc.absorb_lim ? hr : hg;
        const float c = sqrtf(a.kc.g981 * fmaxf(hc, a.kc.absorb_min));
        const float cc = (side == 0 || side == 2) ? -c : c;
        const float val = cc * (hg - hr);
        if (xarm) s.hu = val;
        else s.hv = val;
    }
}

template <int STAGE>
__global__ void __launch_bounds__(NT) stage_kernel(const StepArgs a) {
    __shared__ float s_h[RY][RX], s_u[RY][RX], s_v[RY][RX], s_eta[RY][RX], s_z[RY][RX];
    __shared__ Side s_xp[TY][TX + 2], s_xm[TY][TX + 2];
    __shared__ Side s_yp[TY + 2][TX], s_ym[TY + 2][TX];
    __shared__ FaceFlux s_fx[TY][TX + 1], s_fy[TY + 1][TX];

    chain_start();
    if (clock_row<STAGE>(a)) return;
    const SweConsts& kc = a.kc;
    const int tid = threadIdx.x;
    const int b = blockIdx.z;
    const int i0 = blockIdx.x * TX, j0 = tile_row<STAGE>(a) * TY;

    if (a.clk != nullptr && !a.clk->active) {
        // A step after the end of the call: the state is carried over unchanged.
        if (STAGE == 2) {
            const int j = j0 + tid / TX, i = i0 + tid % TX;
            if (j < a.ny && i < a.nx) {
                const size_t plane = (size_t)a.ny * a.nx;
                const size_t o = at3(b, 0, j, i, a.ny, a.nx);
                a.U_out[o] = a.U[o];
                a.U_out[o + plane] = a.U[o + plane];
                a.U_out[o + 2 * plane] = a.U[o + 2 * plane];
            }
        }
        return;
    }

    float dt = 0.0f, hdt = 0.0f;
    if (STAGE == 2) {
        // solver.py:620-626; torch.minimum propagates a NaN stable dt.
        const float st = stable_dt(u2f(a.red[0]), u2f(a.red[1]), kc);
        const float max_dt = a.clk != nullptr ? a.clk->max_dt : a.max_dt;
        dt = st != st ? st : fminf(st, max_dt);
        hdt = 0.5f * dt;
        if (tid == 0 && i0 == 0 && j0 == 0 && b == 0) {
            const uint32_t st_bits = dt_status(dt);
            if (st_bits) atomicOr(&a.red[2], st_bits);
            a.red[3] = f2u(dt);
        }
    }

    // Phase 0: primitives of the tile and its two-cell halo.
    bool bad = false;
    for (int r = tid; r < RY * RX; r += NT) {
        const int ry = r / RX, rx = r - ry * RX;
        const int j = j0 + ry - 2, i = i0 + rx - 2;
        State s;
        float z;
        region_cell<STAGE>(a, b, j, i, hdt, s, z);
        if (STAGE == 1 && (unsigned)j < (unsigned)a.ny && (unsigned)i < (unsigned)a.nx)
            bad |= !(isfinite(s.h) && isfinite(s.hu) && isfinite(s.hv));
        const Prim p = make_prim(s.h, s.hu, s.hv, z, kc);
        s_h[ry][rx] = p.h;
        s_u[ry][rx] = p.u;
        s_v[ry][rx] = p.v;
        s_eta[ry][rx] = p.eta;
        s_z[ry][rx] = p.z;
    }
    if (STAGE == 1 && __any_sync(0xffffffffu, bad) && (tid & 31) == 0) atomicOr(&a.red[2], SWE_S_NONFINITE_STATE);
    __syncthreads();

    // Phase 1: face-side values (reconstruction.py:26-96) in x and y.
    const bool wsr = a.wsr != 0;
    // (where a cell and both neighbours hold no water its sides feed no face)
    for (int w = tid; w < NXS + NYS; w += NT) {
        if (w < NXS) {
            const int ty = w / (TX + 2), sx = w - ty * (TX + 2);
            const int ry = ty + 2, cx = sx + 1;
            if (no_water(s_h[ry][cx - 1], s_eta[ry][cx - 1]) && no_water(s_h[ry][cx], s_eta[ry][cx]) &&
                no_water(s_h[ry][cx + 1], s_eta[ry][cx + 1]))
                continue;
            const Prim pa{s_h[ry][cx - 1], s_u[ry][cx - 1], s_v[ry][cx - 1], s_eta[ry][cx - 1], s_z[ry][cx - 1]};
            const Prim pc{s_h[ry][cx], s_u[ry][cx], s_v[ry][cx], s_eta[ry][cx], s_z[ry][cx]};
            const Prim pb{s_h[ry][cx + 1], s_u[ry][cx + 1], s_v[ry][cx + 1], s_eta[ry][cx + 1], s_z[ry][cx + 1]};
            const Sides sd = make_sides(pa, pc, pb, kc, wsr);
            s_xp[ty][sx] = sd.p;
            s_xm[ty][sx] = sd.m;
        } else {
            const int w2 = w - NXS;
            const int sy = w2 / TX, tx = w2 - sy * TX;
            const int cy = sy + 1, rx = tx + 2;
            if (no_water(s_h[cy - 1][rx], s_eta[cy - 1][rx]) && no_water(s_h[cy][rx], s_eta[cy][rx]) &&
                no_water(s_h[cy + 1][rx], s_eta[cy + 1][rx]))
                continue;
            const Prim pa{s_h[cy - 1][rx], s_u[cy - 1][rx], s_v[cy - 1][rx], s_eta[cy - 1][rx], s_z[cy - 1][rx]};
            const Prim pc{s_h[cy][rx], s_u[cy][rx], s_v[cy][rx], s_eta[cy][rx], s_z[cy][rx]};
            const Prim pb{s_h[cy + 1][rx], s_u[cy + 1][rx], s_v[cy + 1][rx], s_eta[cy + 1][rx], s_z[cy + 1][rx]};
            const Sides sd = make_sides(pa, pc, pb, kc, wsr);
            s_yp[sy][tx] = sd.p;
            s_ym[sy][tx] = sd.m;
        }
    }
    __syncthreads();

    // Phase 2: HLL fluxes of the faces of the tile (riemann.py:41-105).
    uint32_t axb = 0u, ayb = 0u;
    for (int w = tid; w < NXF + NYF; w += NT) {
        if (w < NXF) {
            const int ty = w / (TX + 1), fx = w - ty * (TX + 1);
            const int ry = ty + 2;
            FaceFlux F{};
            if (!(no_water(s_h[ry][fx + 1], s_eta[ry][fx + 1]) && no_water(s_h[ry][fx + 2], s_eta[ry][fx + 2])))
                F = face_flux(s_xp[ty][fx], s_h[ry][fx + 1], s_z[ry][fx + 1], s_xm[ty][fx + 1],
                                         s_h[ry][fx + 2], s_z[ry][fx + 2], false, kc);
            s_fx[ty][fx] = F;
            if (STAGE == 1 && j0 + ty < a.ny && i0 + fx <= a.nx) axb = max(axb, F.speed_bits);
        } else {
            const int w2 = w - NXF;
            const int fy = w2 / TX, tx = w2 - fy * TX;
            const int rx = tx + 2;
            FaceFlux F{};
            if (!(no_water(s_h[fy + 1][rx], s_eta[fy + 1][rx]) && no_water(s_h[fy + 2][rx], s_eta[fy + 2][rx])))
                F = face_flux(s_yp[fy][tx], s_h[fy + 1][rx], s_z[fy + 1][rx], s_ym[fy + 1][tx],
                                         s_h[fy + 2][rx], s_z[fy + 2][rx], true, kc);
            s_fy[fy][tx] = F;
            if (STAGE == 1 && j0 + fy <= a.ny && i0 + tx < a.nx) ayb = max(ayb, F.speed_bits);
        }
    }
    if (STAGE == 1) {
        axb = warp_max_u32(axb);
        ayb = warp_max_u32(ayb);
        if ((tid & 31) == 0) {
            if (axb) atomicMax(&a.red[0], axb);
            if (ayb) atomicMax(&a.red[1], ayb);
        }
    }
    __syncthreads();

    // Phase 3: tendency of each tile cell (solver.py:511-525), then for stage 2
    // the corrector, clean-up and friction (solver.py:646-661).
    const int ty = tid / TX, tx = tid - (tid / TX) * TX;
    const int j = j0 + ty, i = i0 + tx;
    if (j >= a.ny || i >= a.nx) return;
    const float rain = forcing(a.rain, a.rain_mode, a.rain_batch, b, j, i, a.ny, a.nx);
    const float loss = fmaxf(forcing(a.infil, a.infil_mode, a.infil_batch, b, j, i, a.ny, a.nx), 0.0f);
    const Rhs r = cell_rhs(s_fx[ty][tx], s_fx[ty][tx + 1], s_fy[ty][tx], s_fy[ty + 1][tx], kc, rain, loss);
    const size_t plane = (size_t)a.ny * a.nx;
    const size_t o = at3(b, 0, j, i, a.ny, a.nx);
    if (STAGE == 1) {
        a.tend[o] = r.r0;
        a.tend[o + plane] = r.r1;
        a.tend[o + 2 * plane] = r.r2;
    } else {
        if (a.k2_out != nullptr) {
            a.k2_out[o] = r.r0;
            a.k2_out[o + plane] = r.r1;
            a.k2_out[o + 2 * plane] = r.r2;
        }
        const State u{a.U[o], a.U[o + plane], a.U[o + 2 * plane]};
        const State c{u.h + dt * r.r0, u.hu + dt * r.r1, u.hv + dt * r.r2};
        State upd = clean_and_limit(u, c, kc, a.positivity != 0);
        if (a.friction && upd.h > kc.dry) {  // dry cells have no momentum left
            const float nv = a.n[at1(a.nB == 1 ? 0 : b, j, i, a.ny, a.nx)];
            upd = a.friction_model == 0 ? manning(upd, nv, dt, kc) : roughness_friction(upd, nv, dt, kc);
        }
        a.U_out[o] = upd.h;
        a.U_out[o + plane] = upd.hu;
        a.U_out[o + 2 * plane] = upd.hv;
        if (a.hmax != nullptr) {  // torch.maximum(hmax, U[:, 0]), NaN-propagating
            float& m = a.hmax[at1(b, j, i, a.ny, a.nx)];
            m = (upd.h > m || upd.h != upd.h) ? upd.h : m;
        }
    }
}

// Stage-2 predictor of the IEEE kernels: clean(U, U + hdt*k1) in the
// reference's operation order (solver.py:639).
struct ExactPredict {
    static __device__ __forceinline__ State predict(const State& u, float k0, float k1, float k2,
                                                    float hdt, const SweConsts& k, int positivity) {
        const State c{u.h + hdt * k0, u.hu + hdt * k1, u.hv + hdt * k2};
        return clean_and_limit(u, c, k, positivity != 0);
    }
};

// ---------------------------------------------------------------------------
// Row-sweep form of the two stages.
//
// Each warp owns a strip of 32 columns -- 28 output columns plus the 2-cell
// halo either side -- and SW_ROWS output rows, and sweeps down the strip one
// row at a time.  The y-direction stencil lives in a rolling window of
// registers (primitives of three rows, the previous y-face side and flux);
// x-direction neighbours are exchanged with warp shuffles.  Per output cell
// the warp computes one primitive, one x-side, one y-side, one x-face and
// one y-face (plus 4/28 of a column and 4/SW_ROWS of a row of halo), with no
// shared memory and no block barrier.

// FRIC: 0 no friction, 1 Manning, 2 roughness length (stage 2 only).
// One tile of the sweep: SW_WARPS strips side by side (tile column bx) times
// `rows` output rows (tile row by) of batch member b.  The whole block calls
// it; warps whose strip lies beyond the grid return at once.
// CG is the persistent ensemble kernel: state written by other blocks is read
// through L2, and dry rows are not skipped there: its blocks wait for their
// slowest warp, whose chain the branch lengthens (64 members of 122 x 196:
// 8.4 ms a run, 9.2 with the skip; a 4096 x 4096 step alone 1,968 -> 1,839
// us with it).
template <int STAGE, int FRIC, bool CG>
__device__ __forceinline__ void sweep_tile(const StepArgs& a, int bx, int by, int b, int rows) {
    const SweConsts& kc = a.kc;
    const int lane = threadIdx.x & 31;
    const int strip = bx * SW_WARPS + (threadIdx.x >> 5);
    const int i0 = strip * SW_OUT;
    const int j0 = by * rows;
    if (i0 >= a.nx) return;  // whole warp
    const int c = i0 - 2 + lane;  // this lane's column
    const bool out_lane = lane >= 2 && lane < 2 + SW_OUT && c < a.nx;
    const int jend = min(j0 + rows, a.ny);  // one past the last output row
    const size_t plane = (size_t)a.ny * a.nx;

    if (a.clk != nullptr && !a.clk->active) {
        if (STAGE == 2 && out_lane)
            for (int j = j0; j < jend; ++j) {
                const size_t o = at3(b, 0, j, c, a.ny, a.nx);
                a.U_out[o] = a.U[o];
                a.U_out[o + plane] = a.U[o + plane];
                a.U_out[o + 2 * plane] = a.U[o + 2 * plane];
            }
        return;
    }

    float dt = 0.0f, hdt = 0.0f;
    if (STAGE == 2) {
        dt = stage2_dt<CG>(a, threadIdx.x == 0 && bx == 0 && by == 0 && b == 0);
        hdt = 0.5f * dt;
    }

    const bool wsr = a.wsr != 0;
    Prim pm2{}, pm1{}, p0{};      // primitives of rows k-2, k-1, k
    State um2{}, um1{}, u0{};     // raw U of those rows (stage 2)
    Side sy_prev_p{};              // "p" side of row k-2 in y
    float fy_m = 0.0f, fy_nR = 0.0f, fy_t = 0.0f;  // face above row k-2
    uint32_t axb = 0u, ayb = 0u;
    bool bad = false;
    bool dry2 = false, dry1 = false, dry0 = false;  // rows k-2, k-1, k: no water on any lane
    for (int k = j0 - 2, it = 0; k < jend + 2; ++k, ++it) {
        State s, ur;
        float z;
        sweep_cell<STAGE, CG, ExactPredict>(a, b, k, c, hdt, s, z, ur);
        if (STAGE == 1 && (unsigned)k < (unsigned)a.ny && (unsigned)c < (unsigned)a.nx)
            bad |= !(isfinite(s.h) && isfinite(s.hu) && isfinite(s.hv));
        pm2 = pm1;
        pm1 = p0;
        p0 = make_prim(s.h, s.hu, s.hv, z, kc);
        dry2 = dry1;
        dry1 = dry0;
        dry0 = !CG && warp_no_water(p0.h, p0.eta);
        if (STAGE == 2) {
            um2 = um1;
            um1 = u0;
            u0 = ur;
        }
        if (it < 2) continue;
        // y-sides of row k-1, y-face between rows k-2 and k-1, x-sides and faces
        // of row k-2: nothing where the three rows are dry.  One branch for
        // all, so that the two directions' chains overlap where there is water.
        Sides sy{};
        FaceFlux fy{}, fx{}, fxl{};
        if (!(dry2 && dry1 && dry0)) {
            sy = make_sides(pm2, pm1, p0, kc, wsr);  // reconstruction.py:26-96 along y
            if (it >= 3) fy = face_flux(sy_prev_p, pm2.h, pm2.z, sy.m, pm1.h, pm1.z, true, kc);
            if (it >= 4) {
                // x-sides need the neighbours' primitives, x-faces the right
                // neighbour's side
                const Prim xl{shfl_up1(pm2.h), shfl_up1(pm2.u), shfl_up1(pm2.v), shfl_up1(pm2.eta),
                              shfl_up1(pm2.z)};
                const Prim xr{shfl_dn1(pm2.h), shfl_dn1(pm2.u), shfl_dn1(pm2.v), shfl_dn1(pm2.eta),
                              shfl_dn1(pm2.z)};
                const Sides sx = make_sides(xl, pm2, xr, kc, wsr);
                const Side rm{shfl_dn1(sx.m.hlin), shfl_dn1(sx.m.eta), shfl_dn1(sx.m.bed),
                              shfl_dn1(sx.m.u), shfl_dn1(sx.m.v)};
                fx = face_flux(sx.p, pm2.h, pm2.z, rm, xr.h, xr.z, false, kc);
                if (STAGE == 1 && lane >= 1 && lane < 2 + SW_OUT && c >= -1 && c < a.nx)
                    axb = max(axb, fx.speed_bits);
                fxl = FaceFlux{shfl_up1(fx.fmass), 0.0f, shfl_up1(fx.fnorm_R), shfl_up1(fx.ftan), 0u};
            }
        }
        if (it >= 3) {
            if (STAGE == 1 && out_lane && k - 1 >= 0 && k - 1 <= a.ny) ayb = max(ayb, fy.speed_bits);
            if (it >= 4) {
                const int o = k - 2;  // the output row, complete
                const FaceFlux fyt{fy_m, 0.0f, fy_nR, fy_t, 0u};
                if (out_lane) {
                    const float rain = forcing(a.rain, a.rain_mode, a.rain_batch, b, o, c, a.ny, a.nx);
                    const float loss =
                        fmaxf(forcing(a.infil, a.infil_mode, a.infil_batch, b, o, c, a.ny, a.nx), 0.0f);
                    const Rhs r = cell_rhs(fxl, fx, fyt, fy, kc, rain, loss);
                    const size_t oo = at3(b, 0, o, c, a.ny, a.nx);
                    if (STAGE == 1) {
                        a.tend[oo] = r.r0;
                        a.tend[oo + plane] = r.r1;
                        a.tend[oo + 2 * plane] = r.r2;
                    } else {
                        if (a.k2_out != nullptr) {
                            a.k2_out[oo] = r.r0;
                            a.k2_out[oo + plane] = r.r1;
                            a.k2_out[oo + 2 * plane] = r.r2;
                        }
                        const float nv = FRIC != 0 ? a.n[at1(a.nB == 1 ? 0 : b, o, c, a.ny, a.nx)] : 0.0f;
                        const State u = um2;
                        const State cand{u.h + dt * r.r0, u.hu + dt * r.r1, u.hv + dt * r.r2};
                        State upd = clean_and_limit(u, cand, kc, a.positivity != 0);
                        if (FRIC != 0 && (CG || upd.h > kc.dry))  // dry cells have no momentum left
                            upd = FRIC == 1 ? manning(upd, nv, dt, kc) : roughness_friction(upd, nv, dt, kc);
                        a.U_out[oo] = upd.h;
                        a.U_out[oo + plane] = upd.hu;
                        a.U_out[oo + 2 * plane] = upd.hv;
                        if (a.hmax != nullptr) {
                            float* mp = a.hmax + at1(b, o, c, a.ny, a.nx);
                            const float m = ld_state<CG>(mp);
                            *mp = (upd.h > m || upd.h != upd.h) ? upd.h : m;
                        }
                    }
                }
            }
            fy_m = fy.fmass;
            fy_nR = fy.fnorm_R;
            fy_t = fy.ftan;
        }
        sy_prev_p = sy.p;
    }
    if (STAGE == 1) {
        axb = warp_max_u32(axb);
        ayb = warp_max_u32(ayb);
        if (lane == 0) {
            if (axb) atomicMax(&a.red[0], axb);
            if (ayb) atomicMax(&a.red[1], ayb);
        }
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&a.red[2], SWE_S_NONFINITE_STATE);
    }
}

// Eight 128-thread blocks per SM for both stages: stage 2 then fits in 64
// registers with a few dozen bytes of spills and measured 5 % faster than at
// six blocks (80 registers); ten blocks spill too much.
template <int STAGE, int FRIC>
__global__ void __launch_bounds__(SW_WARPS * 32, 8) sweep_kernel(const StepArgs a) {
    chain_start();
    if (clock_row<STAGE>(a)) return;
    sweep_tile<STAGE, FRIC, false>(a, blockIdx.x, tile_row<STAGE>(a), blockIdx.z, a.rows);
}


// Persistent ensemble kernel (scheduler in swe_ensemble.cuh) over the IEEE
// sweep tiles.
struct ExactTile {
    template <int STAGE, int FRIC>
    static __device__ __forceinline__ void run(const StepArgs& a, int bx, int by, int rows) {
        sweep_tile<STAGE, FRIC, true>(a, bx, by, 0, rows);
    }
};

template <int FRIC>
__global__ void __launch_bounds__(SW_WARPS * 32, 6)
ensemble_kernel(const StepArgs* __restrict__ args, EnsCtl* ctl, int count, EnsGlobal* g,
                unsigned long long stall_ns) {
    ensemble_body<FRIC, ExactTile>(args, ctl, count, g, stall_ns);
}

// One block of >= count threads (count <= 1024).
__global__ void ensemble_init_kernel(EnsCtl* ctl, int count, EnsGlobal* g) {
    const int t = threadIdx.x;
    if (t == 0) {
        g->finished = 0u;
        g->error = 0u;
        g->progress = 0u;
    }
    __syncthreads();
    if (t < count) {
        EnsCtl* c = ctl + t;
        c->claim = 0ull;
        c->done = 0u;
        for (int w = 0; w < SWE_RED_WORDS; ++w) c->red[w] = 0u;
        c->step = 0;
        c->finished = c->steps > 0 ? 0 : 1;
        c->status = 0u;
        c->time = 0.0;
        c->dt_last = 0.0f;
        if (c->n_out > 0) {
            c->chunk = 0;
            c->elapsed = 0.0;
            c->max_dt_cur = (float)((c->cap > 0.0 && c->cap < c->out_dt) ? c->cap : c->out_dt);
            c->level = c->out_levels[0];
        } else {
            c->level = ens_level(*c);
        }
        if (c->finished) atomicAdd(&g->finished, 1u);
    }
}

// Output rows per sweep tile for the single-grid kernels (tuning knob set by
// swe_tune_sweep_rows, 0: sweep_rows_for's choice; the ensemble carries one
// value per scenario).
int g_sweep_rows = 0;

// Tile height of a launch while the knob is 0.  A warp walks
// r + 4 rows one after another, so a stage takes about
// (r + 4) (1 + W(r) / 2500) row times, W(r) the launch's warps: the first
// term is one warp's chain (a small grid: short tiles), the second the
// chip's rate once warps queue (a large grid: the 4 halo rows want tall
// tiles).  Against the best of twelve heights, measured from 40 x 40 to
// 4096 x 4096 in both arithmetics, the height this picks is within 6 %; 64
// rows everywhere took 171 us a step at 64 x 96 in the tolerance mode (15 us at
// one row), 172 at 244 x 393 (21 at two) and 789 at 4096^2 (754 at 32).
int sweep_rows_for(int B, int ny, int nx) {
    if (g_sweep_rows != 0) return g_sweep_rows;
    const double strips = (double)((nx + SW_OUT - 1) / SW_OUT) * B;
    int best = SW_ROWS;
    double best_cost = INFINITY;
    for (int r : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, SW_ROWS}) {
        const int tiles = (ny + r - 1) / r;
        if (tiles > 65535) continue;  // grid.y
        const double cost = (r + 4) * (1.0 + strips * tiles / 2500.0);
        if (cost < best_cost) {
            best_cost = cost;
            best = r;
        }
    }
    return best;
}

bool fill_common(StepArgs& a, const float* U, const float* bed, int B, int bedB, int ny, int nx,
                 const swe_params* p, const float* level, int levelB) {
    if (!U || !bed || !level || !valid_params(p)) return false;
    if (B < 1 || ny < 2 || nx < 2) return false;  // boundary.py:98-102 (ng = 2)
    if (bedB != 1 && bedB != B) return false;
    if (levelB != 1 && levelB != B) return false;
    if ((long long)ny * nx * 3 * B >= (1ll << 40)) return false;
    if ((ny + TY - 1) / TY > 65535 || B > 65535) return false;
    if ((long long)((nx + SW_OUT - 1) / SW_OUT + SW_WARPS - 1) / SW_WARPS > 2147483647LL) return false;
    a.U = U;
    a.bed = bed;
    a.level = level;
    a.B = B;
    a.bedB = bedB;
    a.levelB = levelB;
    a.ny = ny;
    a.nx = nx;
    a.bc[0] = p->bc_left;
    a.bc[1] = p->bc_right;
    a.bc[2] = p->bc_top;
    a.bc[3] = p->bc_bottom;
    a.cval = (float)p->constant_value;
    a.wsr = p->water_slope_reset;
    a.positivity = p->positivity_limiter;
    a.friction = p->apply_friction;
    a.friction_model = p->friction_model;
    a.kc = make_consts(*p);
    a.rows = sweep_rows_for(B, ny, nx);
    return true;
}

bool valid_forcing(const float* f, int mode, int fb, int B) {
    if (mode == SWE_FORCING_NONE) return true;
    if (!f) return false;
    if (mode == SWE_FORCING_SCALAR) return true;
    if (mode == SWE_FORCING_FIELD) return fb == 1 || fb == B;
    return false;
}

dim3 grid_of(const StepArgs& a) { return dim3((a.nx + TX - 1) / TX, (a.ny + TY - 1) / TY, a.B); }

dim3 sweep_grid_of(const StepArgs& a) {
    const int strips = (a.nx + SW_OUT - 1) / SW_OUT;
    return dim3((strips + SW_WARPS - 1) / SW_WARPS, (a.ny + a.rows - 1) / a.rows, a.B);
}

// Kernel form of the IEEE stages.  The shared-memory tile evaluates a cell
// per thread (no serial chain, fewer halo cells than short sweep tiles) and
// is the faster form up to about 1.5 million cells; above that the row sweep
// with tall tiles is (a step of an all-wet state, tile / best sweep: 244 x 393
// 36 / 45 us, 4 x 244 x 393 78 / 97, 1021 x 1019 168 / 189, 1200^2 221 / 235,
// 2048^2 605 / 570, 4096^2 2341 / 1968; both gain alike from dry land).  SWE_STEP_KERNEL=tiled or =sweep fixes the
// form, read once per process.  Both give the same bits.
constexpr long long kTiledMaxCells = 3ll << 19;

bool use_tiled_kernels(const StepArgs& a) {
    static const int form = [] {
        const char* v = getenv("SWE_STEP_KERNEL");
        return v == nullptr ? 0 : strcmp(v, "tiled") == 0 ? 1 : strcmp(v, "sweep") == 0 ? 2 : 0;
    }();
    if (form != 0) return form == 1;
    return (long long)a.B * a.ny * a.nx <= kTiledMaxCells;
}

}  // namespace
}  // namespace swe

using namespace swe;

extern "C" int swe_spatial_operator_f32(const float* U, const float* bed, int B, int bedB, int ny,
                                        int nx, const swe_params* p, const float* level, int levelB,
                                        const float* rain, int rain_mode, int rain_batch,
                                        const float* infil, int infil_mode, int infil_batch,
                                        float* rhs, uint32_t* red, void* stream) {
    StepArgs a{};
    if (!fill_common(a, U, bed, B, bedB, ny, nx, p, level, levelB) || !rhs || !red) return SWE_EARG;
    if (!valid_forcing(rain, rain_mode, rain_batch, B) || !valid_forcing(infil, infil_mode, infil_batch, B))
        return SWE_EARG;
    a.rain = rain;
    a.rain_mode = rain_mode;
    a.rain_batch = rain_batch;
    a.infil = infil;
    a.infil_mode = infil_mode;
    a.infil_batch = infil_batch;
    a.tend = rhs;
    a.red = red;
    cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemsetAsync(red, 0, SWE_RED_WORDS * sizeof(uint32_t), s) != cudaSuccess) return SWE_ECUDA;
    // the stage-1 kernel of the step computes exactly this (tendency + maxima)
    if (p->arithmetic == SWE_ARITH_FAST) return fast_launch_stages(1, a, sweep_grid_of(a), s);
    const cudaError_t e =
        use_tiled_kernels(a) ? launch_chained(stage_kernel<1>, grid_of(a), dim3(NT), s, a)
                             : launch_chained(sweep_kernel<1, 0>, sweep_grid_of(a), dim3(SW_WARPS * 32), s, a);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

namespace swe {
namespace {

// Where stage 2 leaves the clock of the following step.
struct NextClock {
    swe_clock* clock;
    uint32_t* red;
    float* level;
    const float* series_t;
    const float* series_w;
    int nseries;
};

int launch_step(int stage, const float* U, const float* bed, int bedB, const float* n, int nB, int B,
                int ny, int nx, const swe_params* p, const float* level, int levelB, float max_dt,
                const swe_clock* clk, const float* rain, int rain_mode, int rain_batch,
                const float* infil, int infil_mode, int infil_batch, float* scratch_k, uint32_t* red,
                float* U_out, float* hmax, void* stream, float* k2_out = nullptr,
                const NextClock* next = nullptr) {
    StepArgs a{};
    if (stage != 1 && stage != 2 && stage != 3) return SWE_EARG;
    if (!fill_common(a, U, bed, B, bedB, ny, nx, p, level, levelB)) return SWE_EARG;
    if (!scratch_k || !red || !U_out || (p->apply_friction && !n)) return SWE_EARG;
    if (p->apply_friction && nB != 1 && nB != B) return SWE_EARG;
    if (!valid_forcing(infil, infil_mode, infil_batch, B)) return SWE_EARG;
    if (!valid_forcing(rain, rain_mode, rain_batch, B)) return SWE_EARG;
    a.n = n;
    a.nB = nB;
    a.infil = infil;
    a.infil_mode = infil_mode;
    a.infil_batch = infil_batch;
    a.rain = rain;
    a.rain_mode = rain_mode;
    a.rain_batch = rain_batch;
    a.tend = scratch_k;
    a.U_out = U_out;
    a.red = red;
    a.max_dt = max_dt;
    a.clk = clk;
    a.hmax = hmax;
    a.k2_out = k2_out;
    if (next != nullptr) {
        a.next_clk = next->clock;
        a.next_red = next->red;
        a.next_level = next->level;
        a.series_t = next->series_t;
        a.series_w = next->series_w;
        a.nseries = next->nseries;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const bool fast = p->arithmetic == SWE_ARITH_FAST;
    const bool tiled = !fast && use_tiled_kernels(a);
    dim3 g = tiled ? grid_of(a) : sweep_grid_of(a);
    if (next != nullptr && g.y >= 65535u) return SWE_EARG;  // no room for the clock's row
    // A clocked step's reduction words are cleared when the clock is advanced.
    if ((stage & 1) && !clk && cudaMemsetAsync(red, 0, SWE_RED_WORDS * sizeof(uint32_t), s) != cudaSuccess)
        return SWE_ECUDA;
    if (fast) return fast_launch_stages(stage, a, g, s);
    const dim3 th(SW_WARPS * 32);
    cudaError_t e = cudaSuccess;
    if (stage & 1) {
        if (tiled) e = launch_chained(stage_kernel<1>, g, dim3(NT), s, a);
        else e = launch_chained(sweep_kernel<1, 0>, g, th, s, a);
    }
    if ((stage & 2) && e == cudaSuccess) {
        if (next != nullptr) g.y += 1;
        if (tiled) {
            e = launch_chained(stage_kernel<2>, g, dim3(NT), s, a);
        } else if (!a.friction) {
            e = launch_chained(sweep_kernel<2, 0>, g, th, s, a);
        } else if (a.friction_model == 0) {
            e = launch_chained(sweep_kernel<2, 1>, g, th, s, a);
        } else {
            e = launch_chained(sweep_kernel<2, 2>, g, th, s, a);
        }
    }
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

}  // namespace
}  // namespace swe

extern "C" int swe_step_stage_f32(int stage, const float* U, const float* bed, int bedB,
                                  const float* n, int nB, int B, int ny, int nx,
                                  const swe_params* p, const float* level, int levelB,
                                  float max_dt, const float* infil, int infil_mode,
                                  int infil_batch, float* scratch_k, uint32_t* red, float* U_out,
                                  void* stream) {
    return launch_step(stage, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, max_dt, nullptr,
                       nullptr, SWE_FORCING_NONE, 1, infil, infil_mode, infil_batch, scratch_k, red,
                       U_out, nullptr, stream);
}

extern "C" int swe_step_stage_forced_f32(int stage, const float* U, const float* bed, int bedB,
                                         const float* n, int nB, int B, int ny, int nx,
                                         const swe_params* p, const float* level, int levelB,
                                         float max_dt, const float* rain, int rain_mode,
                                         int rain_batch, const float* infil, int infil_mode,
                                         int infil_batch, float* scratch_k, uint32_t* red,
                                         float* U_out, void* stream) {
    return launch_step(stage, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, max_dt, nullptr,
                       rain, rain_mode, rain_batch, infil, infil_mode, infil_batch, scratch_k, red,
                       U_out, nullptr, stream);
}

extern "C" int swe_step_clocked_f32(int stage, const float* U, const float* bed, int bedB,
                                    const float* n, int nB, int B, int ny, int nx,
                                    const swe_params* p, const float* level, int levelB,
                                    const swe_clock* clock, const float* infil, int infil_mode,
                                    int infil_batch, float* scratch_k, uint32_t* red, float* U_out,
                                    float* hmax, void* stream) {
    if (!clock) return SWE_EARG;
    return launch_step(stage, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, 0.0f, clock, nullptr,
                       SWE_FORCING_NONE, 1, infil, infil_mode, infil_batch, scratch_k, red, U_out, hmax,
                       stream);
}

extern "C" int swe_step_clocked_next_f32(const float* U, const float* bed, int bedB, const float* n, int nB, int B,
                                         int ny, int nx, const swe_params* p, const float* level, int levelB,
                                         const swe_clock* clock, const float* infil, int infil_mode,
                                         int infil_batch, float* scratch_k, uint32_t* red, float* U_out,
                                         float* hmax, swe_clock* next_clock, uint32_t* next_red,
                                         const float* series_t, const float* series_w, int nseries,
                                         float* next_level, void* stream) {
    if (!clock || !next_clock || next_clock == clock || !next_red || next_red == red || nseries < 0) return SWE_EARG;
    if (nseries > 0 && (!series_t || !series_w || !next_level || next_level == level)) return SWE_EARG;
    const NextClock next{next_clock, next_red, next_level, series_t, series_w, nseries};
    return launch_step(3, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, 0.0f, clock, nullptr,
                       SWE_FORCING_NONE, 1, infil, infil_mode, infil_batch, scratch_k, red, U_out, hmax,
                       stream, nullptr, &next);
}

extern "C" int swe_step_clocked_k2_f32(int stage, const float* U, const float* bed, int bedB,
                                       const float* n, int nB, int B, int ny, int nx,
                                       const swe_params* p, const float* level, int levelB,
                                       const swe_clock* clock, const float* infil, int infil_mode,
                                       int infil_batch, float* scratch_k, uint32_t* red,
                                       float* U_out, float* hmax, float* k2_out, void* stream) {
    if (!clock || !k2_out || !(stage & 2)) return SWE_EARG;
    return launch_step(stage, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, 0.0f, clock, nullptr,
                       SWE_FORCING_NONE, 1, infil, infil_mode, infil_batch, scratch_k, red, U_out, hmax,
                       stream, k2_out);
}

extern "C" int swe_step_f32(const float* U, const float* bed, int bedB, const float* n, int nB,
                            int B, int ny, int nx, const swe_params* p, const float* level,
                            int levelB, float max_dt, const float* infil, int infil_mode,
                            int infil_batch, float* scratch_k, uint32_t* red, float* U_out,
                            void* stream) {
    return swe_step_stage_f32(3, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, max_dt, infil,
                              infil_mode, infil_batch, scratch_k, red, U_out, stream);
}

// ---------------------------------------------------------------------------
// Step without allocation: scratch in a static device array.
//
// For callers that cannot allocate device memory (their device memory is
// owned by another allocator, or they may not allocate after start-up), the
// stage-1 tendency and the reduction words live in this array instead of
// caller buffers.  Layout: words [0, 64) reduction/status (SWE_RED_WORDS
// used, the rest keeps the tendency 256-byte aligned), then 3 planes of
// SWE_NOALLOC_MAX_CELLS floats for the tendency.  In host code the name
// g_noalloc_scratch is only a host-side stand-in; the device address is
// looked up once per device with cudaGetSymbolAddress.
namespace {

constexpr size_t kNoallocRedWords = 64;
constexpr size_t kNoallocWords = kNoallocRedWords + 3 * (size_t)SWE_NOALLOC_MAX_CELLS;

static __device__ __align__(256) float g_noalloc_scratch[kNoallocWords];

constexpr int kMaxDevices = 128;
std::mutex g_noalloc_mutex;
float* g_noalloc_base[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device (looked up on
// the first call per device, then cached).
int noalloc_scratch(float** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SWE_ECUDA;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_base[dev]) {
        void* addr = nullptr;
        if (cudaGetSymbolAddress(&addr, g_noalloc_scratch) != cudaSuccess || !addr) return SWE_ECUDA;
        g_noalloc_base[dev] = static_cast<float*>(addr);
    }
    *out = g_noalloc_base[dev];
    return SWE_OK;
}

}  // namespace

extern "C" int swe_step_noalloc_f32(const float* U, const float* bed, int bedB, const float* n,
                                    int nB, int B, int ny, int nx, const swe_params* p,
                                    const float* level, int levelB, float max_dt,
                                    const float* infil, int infil_mode, int infil_batch,
                                    float* U_out, uint32_t* status_dt, void* stream) {
    if (!status_dt || B < 1 || ny < 1 || nx < 1) return SWE_EARG;
    if ((long long)B * ny * nx > (long long)SWE_NOALLOC_MAX_CELLS) return SWE_ETOOLARGE;
    float* base = nullptr;
    const int rc0 = noalloc_scratch(&base);
    if (rc0 != SWE_OK) return rc0;
    uint32_t* red = reinterpret_cast<uint32_t*>(base);
    float* scratch_k = base + kNoallocRedWords;
    const int rc = swe_step_stage_f32(3, U, bed, bedB, n, nB, B, ny, nx, p, level, levelB, max_dt,
                                      infil, infil_mode, infil_batch, scratch_k, red, U_out, stream);
    if (rc != SWE_OK) return rc;
    if (cudaMemcpyAsync(status_dt, red + 2, 2 * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                        (cudaStream_t)stream) != cudaSuccess)
        return SWE_ECUDA;
    return SWE_OK;
}

// ---------------------------------------------------------------------------
// Ensemble entry points.
namespace swe {
namespace {

size_t ens_offset_ctl(int count) { return ((size_t)count * sizeof(StepArgs) + 255) / 256 * 256; }
size_t ens_offset_global(int count) {
    return ens_offset_ctl(count) + ((size_t)count * sizeof(EnsCtl) + 255) / 256 * 256;
}

}  // namespace
}  // namespace swe

extern "C" long long swe_ensemble_workspace_bytes(int count) {
    if (count < 1 || count > 1024) return -1;
    return (long long)(ens_offset_global(count) + sizeof(EnsGlobal));
}

extern "C" int swe_ensemble_prepare_f32(const swe_ensemble_member* members, int count,
                                        void* workspace, void* stream) {
    if (!members || !workspace || count < 1 || count > 1024) return SWE_EARG;
    StepArgs* args = (StepArgs*)malloc(sizeof(StepArgs) * count);
    EnsCtl* ctl = (EnsCtl*)malloc(sizeof(EnsCtl) * count);
    if (!args || !ctl) {
        free(args);
        free(ctl);
        return SWE_EARG;
    }
    char* ws = (char*)workspace;
    EnsCtl* ctl_dev = (EnsCtl*)(ws + ens_offset_ctl(count));
    int rc = SWE_OK;
    const int fric0 = members[0].params.apply_friction ? 1 + members[0].params.friction_model : 0;
    const int arith0 = members[0].params.arithmetic;
    for (int m = 0; m < count && rc == SWE_OK; ++m) {
        const swe_ensemble_member& e = members[m];
        StepArgs a{};
        const int fric = e.params.apply_friction ? 1 + e.params.friction_model : 0;
        const bool interval = e.n_out > 0;
        if (fric != fric0 || e.params.arithmetic != arith0 || !e.U_a || !e.U_b || !e.k1 || e.steps < 0 || e.rows < 1 ||
            (!interval && e.nseries > 0 && (!e.series_t || !e.series_w)) || e.n_out < 0 ||
            (interval && (!(e.out_dt > 0.0) || !e.out_levels || e.ngauge < 0 ||
                          (e.ngauge > 0 && (!e.gauge_cells || !e.gauge_out)))) ||
            !fill_common(a, e.U_a, e.bed, 1, 1, e.ny, e.nx, &e.params, e.U_a, 1) ||
            (e.params.apply_friction && !e.n)) {
            rc = SWE_EARG;
            break;
        }
        a.n = e.n;
        a.nB = 1;
        a.rain_mode = SWE_FORCING_NONE;
        a.infil_mode = SWE_FORCING_NONE;
        a.tend = e.k1;
        a.U_out = e.U_b;
        a.hmax = e.hmax;
        a.max_dt = (float)e.max_dt;
        a.rows = e.rows;
        a.level = &ctl_dev[m].level;  // the ensemble's current level of this member
        a.red = ctl_dev[m].red;
        args[m] = a;
        EnsCtl c{};
        const int strips = (e.nx + SW_OUT - 1) / SW_OUT;
        c.nbx = (strips + SW_WARPS - 1) / SW_WARPS;
        c.rows = e.rows;
        c.tiles = c.nbx * ((e.ny + e.rows - 1) / e.rows);
        c.steps = e.steps;
        c.nseries = e.nseries;
        c.series_t = e.series_t;
        c.series_w = e.series_w;
        c.level = e.level;
        c.start = e.start_time;
        c.Ua = e.U_a;
        c.Ub = e.U_b;
        c.max_dt_cur = (float)e.max_dt;
        if (interval) {
            // gauge cells must lie in the grid (read back once per member)
            int32_t cells[2 * SWE_ENSEMBLE_MAX_GAUGES];
            if (e.ngauge > SWE_ENSEMBLE_MAX_GAUGES) {
                rc = SWE_EARG;
            } else if (e.ngauge > 0) {
                if (cudaMemcpy(cells, e.gauge_cells, sizeof(int32_t) * 2 * e.ngauge,
                               cudaMemcpyDeviceToHost) != cudaSuccess)
                    rc = SWE_ECUDA;
                for (int q = 0; q < e.ngauge && rc == SWE_OK; ++q)
                    if (cells[2 * q] < 0 || cells[2 * q] >= e.ny || cells[2 * q + 1] < 0 ||
                        cells[2 * q + 1] >= e.nx)
                        rc = SWE_EARG;
            }
            c.n_out = e.n_out;
            c.out_dt = e.out_dt;
            c.tol = e.out_dt * 1e-12 > 1e-12 ? e.out_dt * 1e-12 : 1e-12;
            c.cap = e.max_dt;
            c.ngauge = e.ngauge;
            c.nx = e.nx;
            c.out_levels = e.out_levels;
            c.gauge_cells = e.gauge_cells;
            c.gauge_out = e.gauge_out;
            c.bed = e.bed;
        }
        ctl[m] = c;
    }
    if (rc == SWE_OK) {
        if (cudaMemcpy(ws, args, sizeof(StepArgs) * count, cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(ctl_dev, ctl, sizeof(EnsCtl) * count, cudaMemcpyHostToDevice) != cudaSuccess)
            rc = SWE_ECUDA;
    }
    free(args);
    free(ctl);
    if (rc != SWE_OK) return rc;
    return swe_ensemble_reset_f32(workspace, count, stream);
}

extern "C" int swe_ensemble_reset_f32(void* workspace, int count, void* stream) {
    if (!workspace || count < 1 || count > 1024) return SWE_EARG;
    char* ws = (char*)workspace;
    ensemble_init_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(
        (EnsCtl*)(ws + ens_offset_ctl(count)), count, (EnsGlobal*)(ws + ens_offset_global(count)));
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int swe_ensemble_run_f32(void* workspace, int count, int friction, int arithmetic,
                                    int blocks, long long stall_ns, void* stream) {
    if (!workspace || count < 1 || count > 1024 || blocks < 1 || friction < 0 || friction > 2 ||
        (arithmetic != SWE_ARITH_EXACT && arithmetic != SWE_ARITH_FAST) || stall_ns < 0)
        return SWE_EARG;
    char* ws = (char*)workspace;
    const StepArgs* args = (const StepArgs*)ws;
    EnsCtl* ctl = (EnsCtl*)(ws + ens_offset_ctl(count));
    EnsGlobal* g = (EnsGlobal*)(ws + ens_offset_global(count));
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned long long limit = stall_ns > 0 ? (unsigned long long)stall_ns : EnsStallNsDefault;
    if (arithmetic == SWE_ARITH_FAST)
        return fast_launch_ensemble(friction, blocks, args, ctl, count, g, limit, s);
    if (friction == 0) ensemble_kernel<0><<<blocks, SW_WARPS * 32, 0, s>>>(args, ctl, count, g, limit);
    else if (friction == 1) ensemble_kernel<1><<<blocks, SW_WARPS * 32, 0, s>>>(args, ctl, count, g, limit);
    else ensemble_kernel<2><<<blocks, SW_WARPS * 32, 0, s>>>(args, ctl, count, g, limit);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

namespace swe {
namespace {
__global__ void ensemble_results_kernel(const EnsCtl* ctl, int count, const EnsGlobal* g,
                                        swe_ensemble_result* out, uint32_t* error) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < count) {
        out[t].steps = ctl[t].step;
        out[t].finished = ctl[t].finished;
        out[t].status = ctl[t].status;
        out[t].dt_last = ctl[t].dt_last;
        out[t].time = ctl[t].time;
    }
    if (t == 0) *error = g->error;
}
}  // namespace
}  // namespace swe

extern "C" int swe_ensemble_results_f32(const void* workspace, int count, swe_ensemble_result* out,
                                        uint32_t* error, void* stream) {
    if (!workspace || !out || !error || count < 1 || count > 1024) return SWE_EARG;
    const char* ws = (const char*)workspace;
    ensemble_results_kernel<<<(count + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        (const EnsCtl*)(ws + ens_offset_ctl(count)), count,
        (const EnsGlobal*)(ws + ens_offset_global(count)), out, error);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int swe_tune_sweep_rows(int rows) {
    if (rows < 0 || rows > 4096) return SWE_EARG;
    g_sweep_rows = rows;
    return SWE_OK;
}

extern "C" int swe_sweep_rows(void) { return g_sweep_rows; }

extern "C" int swe_launch_rows(int B, int ny, int nx, int arithmetic) {
    if (B < 1 || ny < 2 || nx < 2) return -1;
    StepArgs a{};
    a.B = B;
    a.ny = ny;
    a.nx = nx;
    return arithmetic != SWE_ARITH_FAST && use_tiled_kernels(a) ? 0 : sweep_rows_for(B, ny, nx);
}

extern "C" int swe_load_kernels(void) {
    // Touching each kernel loads its module now (CUDA lazy loading), so that
    // no first load happens inside a stream capture.
    cudaFuncAttributes at;
    const void* fns[] = {
        (const void*)stage_kernel<1>,        (const void*)stage_kernel<2>,
        (const void*)sweep_kernel<1, 0>,     (const void*)sweep_kernel<2, 0>,
        (const void*)sweep_kernel<2, 1>,     (const void*)sweep_kernel<2, 2>,
        (const void*)ensemble_kernel<0>,     (const void*)ensemble_kernel<1>,
        (const void*)ensemble_kernel<2>,     (const void*)ensemble_init_kernel,
        (const void*)ensemble_results_kernel,
    };
    for (const void* f : fns)
        if (cudaFuncGetAttributes(&at, f) != cudaSuccess) return SWE_ECUDA;
    return fast_load_kernels();
}
