// swe_adjoint_kernels.cuh -- kernels of the step adjoint, templated on the
// arithmetic policy M of swe_adjoint.cuh and instantiated twice: with
// ExactMath in swe_adjoint.cu (IEEE flags) and with FastMath in
// swe_adjoint_fast.cu (compiled like the tolerance-mode step).
//
// The spatial-operator adjoint is two launches.  adj_tile_kernel owns a tile
// of cells per block and keeps everything between the state and its adjoint
// in shared memory: primitives of the tile and a three-cell halo, the face
// sides of its cells in both directions, the reverse mode of each face
// (swe_adjoint.cuh) written over the sides it read, each cell's reverse mode
// of its two sides written over those, and their sums.  The adjoints of
// ghost cells go to a small buffer; adj_edge_kernel folds them back into the
// cells and boundary level they were made from (the adjoint of
// add_ghost_cells, src/boundary.py:150-413) and finishes the two-cell frame
// along the sides; adj_level_kernel sums the level's adjoint.  Stage 2 goes on through the predictor's adjoint in both.
// No float atomics: results are deterministic.  On request the ghosts that
// depend on the level and the cells next to them are done face by face
// instead (level bands, below), in two more launches.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "swe_adjoint.cuh"
#include "swe_common.cuh"

namespace swe {

constexpr int ADJ_THREADS = 256;
constexpr int ADJ_TX = 32;  // tile columns
// Blocks per SM the tile kernel is compiled for (80 registers, no spills).
// Measured with 16-row tiles at 4 x 244 x 393, stage 2 / stage 1: three
// 58.5 / 52.0 us, two 69 / 60; with 8-row tiles (37 KB instead of 65) at
// three, four and five blocks 67 / 59, 64 / 57 and 66 / 59, all with every
// cell evaluated; where zero cotangents are skipped 8 rows and four blocks
// come out level (44 / 39 against 45 / 39).
#ifndef SWE_ADJ_TILE_MINB
#define SWE_ADJ_TILE_MINB 3
#endif

struct AdjArgs {
    const float* S;      // state whose tendency is differentiated, [B,3,ny,nx]; with the
                         // predictor fused in: P, or null to form it from U and k1
    const float* bed;    // [bedB,1,ny,nx]
    const float* level;  // [levelB]
    const float* lrhs;   // adjoint of the tendency, [B,3,ny,nx]
    float* gx;           // adjoints of the x ghosts [B][left, right][1st, 2nd][ny][4]
    float* gy;           // adjoints of the y ghosts [B][top, bottom][1st, 2nd][nx][4]
    float* frame;        // adjoints of the frame's cells before the folds [B][4][ny][nx] (the
                         // fourth plane: the bed's, then the cell's share of the level's)
    int bands;           // along level sides, sums face by face (level bands, below)
    float* bandx;        // face records along the level's x sides, or null: no records
    float* bandy;        // the same along its y sides
    float* lS;           // adjoint of S, accumulated (+=)
    float* llevel_part;  // partial level adjoints [B][level_blocks]
    int level_blocks, direct_level;  // the latter: written by adj_edge_kernel's own blocks
    float* lbed;         // adjoint of the bed [B,ny,nx], accumulated (+=); BEDG only
    int B, bedB, levelB, ny, nx;
    int bc[4];
    float cval;
    int wsr;
    SweConsts kc;
    // Predictor adjoint fused in (PRED; S is then the predictor
    // P = clean(U, U + dt/2 k1)): the cell's adjoint of P is not stored but
    // taken through the clean-up's adjoint at once.
    const float* U;       // step input [B,3,ny,nx]
    const float* k1;      // stage-1 tendency [B,3,ny,nx]
    const float* dt_dev;  // the step's dt in device memory, or null: dt
    float dt;
    float* lU;            // adjoint of U, accumulated (+=)
    float* lk1;           // adjoint of k1 (written)
    int positivity;
};

struct PwArgs {
    const float* U;     // step input
    const float* k;     // tendency (k2 for modes 0 and 3, k1 for modes 1 and 2)
    const float* n;     // roughness (modes 0, 3)
    const float* lout;  // adjoint of the step output (modes 0, 3) or of P (mode 1)
    float* lU;          // adjoint of U, accumulated (+=; written in mode 3)
    float* lk;          // adjoint of the tendency (written)
    float* ln;          // adjoint of the roughness field, accumulated (+=) [nB,ny,nx]
    float* P;           // mode 2: predictor output
    float scale;        // dt (modes 0, 3) or dt/2 (modes 1, 2)
    float dt;
    const float* dt_dev;  // if set: dt read from device memory (scale derived here)
    int B, nB, ny, nx, mode, positivity, friction, friction_model;
    SweConsts kc;
};

namespace {

__device__ __forceinline__ size_t a3(int b, int c, int j, int i, int ny, int nx) {
    return (((size_t)b * 3 + c) * ny + j) * nx + i;
}

__device__ __forceinline__ float bed_of(const AdjArgs& a, int b, int j, int i) {
    return a.bed[((size_t)(a.bedB == 1 ? 0 : b) * a.ny + j) * a.nx + i];
}

// _clean_and_limit (solver.py:547-570) in the arithmetic M.
template <class M>
__device__ __forceinline__ State clean_fwd(const State& o, State c, const SweConsts& k, bool positivity) {
    if (positivity) {
        const float d0 = c.h - o.h, d1 = c.hu - o.hu, d2 = c.hv - o.hv;
        const float safe = fmaxf(-d0, k.eps);
        const float th = d0 < 0.0f ? fminf(M::div(o.h, safe, M::rcp(safe)), 1.0f) : 1.0f;
        c.h = o.h + th * d0;
        c.hu = o.hu + th * d1;
        c.hv = o.hv + th * d2;
    }
    State r;
    r.h = fmaxf(c.h, 0.0f);
    const bool wet = r.h > k.dry;
    r.hu = wet ? c.hu : 0.0f;
    r.hv = wet ? c.hv : 0.0f;
    return r;
}

// Adjoint of _clean_and_limit (solver.py:547-570): returns lam_old, lam_cand.
template <class M>
__device__ void clean_bwd(const State& o, const State& c, const State& lout, const SweConsts& k,
                          bool positivity, State& lold, State& lcand) {
    State cp = c;
    float d0 = 0.0f, d1 = 0.0f, d2 = 0.0f, th = 1.0f, ratio = 0.0f, safe = 0.0f, ysafe = 0.0f;
    bool theta_branch = false;
    if (positivity) {
        d0 = c.h - o.h;
        d1 = c.hu - o.hu;
        d2 = c.hv - o.hv;
        safe = fmaxf(-d0, k.eps);
        ysafe = M::rcp(safe);
        ratio = M::div(o.h, safe, ysafe);
        theta_branch = d0 < 0.0f;
        th = theta_branch ? fminf(ratio, 1.0f) : 1.0f;
        cp.h = o.h + th * d0;
        cp.hu = o.hu + th * d1;
        cp.hv = o.hv + th * d2;
    }
    const float h = fmaxf(cp.h, 0.0f);
    const bool wet = h > k.dry;
    State lcp;
    lcp.h = cp.h >= 0.0f ? lout.h : 0.0f;
    lcp.hu = wet ? lout.hu : 0.0f;
    lcp.hv = wet ? lout.hv : 0.0f;
    if (!positivity) {
        lold = State{0.0f, 0.0f, 0.0f};
        lcand = lcp;
        return;
    }
    // cand' = old + th * delta
    const float l_th = lcp.h * d0 + lcp.hu * d1 + lcp.hv * d2;
    float ld0 = lcp.h * th, ld1 = lcp.hu * th, ld2 = lcp.hv * th;
    lold = lcp;
    if (theta_branch && ratio <= 1.0f) {  // th = clamp(old_h / safe, max=1)
        lold.h += M::div(l_th, safe, ysafe);
        const float l_safe = -l_th * M::div(ratio, safe, ysafe);
        if (-d0 >= k.eps) ld0 -= l_safe;  // safe = clamp(-dh, min=eps)
    }
    lcand = State{ld0, ld1, ld2};
    lold.h -= ld0;
    lold.hu -= ld1;
    lold.hv -= ld2;
}

// State of interior cell (j, i): S, or the predictor formed from U and k1.
template <bool PRED, class M>
__device__ __forceinline__ State cell_state(const AdjArgs& a, int b, int j, int i, float scale) {
    const size_t plane = (size_t)a.ny * a.nx;
    const size_t o = a3(b, 0, j, i, a.ny, a.nx);
    if (!PRED || a.S != nullptr) return State{a.S[o], a.S[o + plane], a.S[o + 2 * plane]};
    const State u{a.U[o], a.U[o + plane], a.U[o + 2 * plane]};
    const State cand{u.h + scale * a.k1[o], u.hu + scale * a.k1[o + plane], u.hv + scale * a.k1[o + 2 * plane]};
    return clean_fwd<M>(u, cand, a.kc, a.positivity != 0);
}

// Padded cell (j, i) with the ghost rules (arm cells only: in the interior
// along one direction, at most two cells outside along the other).
template <bool PRED, class M>
__device__ State padded_state(const AdjArgs& a, int b, int j, int i, float scale, float& z) {
    const int ny = a.ny, nx = a.nx;
    const bool jin = (unsigned)j < (unsigned)ny, iin = (unsigned)i < (unsigned)nx;
    int js = min(max(j, 0), ny - 1), is = min(max(i, 0), nx - 1);
    const bool xarm = jin && !iin, yarm = iin && !jin;
    int code = -1, side = 0;
    if (xarm || yarm) {
        side = xarm ? (i < 0 ? 0 : 1) : (j < 0 ? 2 : 3);
        code = a.bc[side];
        if (code == SWE_BC_PERIODIC) {
            if (xarm) is = i < 0 ? nx + i : i - nx;
            else js = j < 0 ? ny + j : j - ny;
        }
    }
    State s = cell_state<PRED, M>(a, b, js, is, scale);
    z = bed_of(a, b, js, is);
    if (code < 0) return s;
    const float lev = a.level[a.levelB == 1 ? 0 : b];
    if (code == SWE_BC_CONSTANT) {
        s = State{a.cval, a.cval, a.cval};
    } else if (code == SWE_BC_WATER_LEVEL) {
        s.h = fmaxf(lev - z, 0.0f);
    } else if (code == SWE_BC_WALL) {
        const int jm = xarm ? j : (j < 0 ? -1 - j : 2 * ny - 1 - j);
        const int im = xarm ? (i < 0 ? -1 - i : 2 * nx - 1 - i) : i;
        const State m = cell_state<PRED, M>(a, b, jm, im, scale);
        if (xarm) s.hu = -m.hu;
        else s.hv = -m.hv;
    } else if (code == SWE_BC_ABSORBING) {
        const float hr = fmaxf(lev - z, 0.0f);
        const float hg = s.h;
        const float hc = hr > a.kc.absorb_lim ? hr : hg;
        const float c = M::sqrt(a.kc.g981 * fmaxf(hc, a.kc.absorb_min));
        const float val = ((side == 0 || side == 2) ? -c : c) * (hg - hr);
        if (xarm) s.hu = val;
        else s.hv = val;
    }
    return s;
}

// ------------------------------------------------------------ level bands
// Along a side whose ghosts depend on the level, the adjoints of its ghosts
// and of the two lines of cells next to it are summed from face records
// (swe_adjoint.cuh, namespace line): of the faces normal to the side, d = 0
// to 3 lines away from it, and of the faces along each line of cells, e = 0,
// 1.  (The cells because a second call's ghosts take their cotangents from
// what this one makes of them.)  A record holds the face's contributions to its
// four cells, 4 x (U0, U1, U2, Z).  Grids too small for the scratch buffers
// (either side below BAND_MIN cells) keep none: there every face is evaluated
// where it is summed (FLY below), the same values in the same order.
constexpr int BAND_MIN = 32;
constexpr int BAND_REC = 16;

__host__ __device__ inline long long band_faces(int n) { return 4LL * n + 2LL * (n + 1); }
__host__ __device__ inline long long band_floats(int B, int n) { return 2LL * B * band_faces(n) * BAND_REC; }
__host__ __device__ inline bool level_side(const AdjArgs& a, int side) {
    return a.bands && (a.bc[side] == SWE_BC_WATER_LEVEL || a.bc[side] == SWE_BC_ABSORBING);
}

struct LevelBand {
    float* base;  // this side's records of batch member b
    int n;        // cells along the side
    __device__ LevelBand(const AdjArgs& a, int b, int side) {
        n = side < 2 ? a.ny : a.nx;
        base = (side < 2 ? a.bandx : a.bandy) + ((long long)b * 2 + (side & 1)) * band_faces(n) * BAND_REC;
    }
    __device__ float* normal(int d, int pos) const { return base + ((long long)d * n + pos) * BAND_REC; }
    __device__ float* along(int e, int face) const {
        return base + (4LL * n + (long long)e * (n + 1) + face) * BAND_REC;
    }
};

// One face of a band: the x face f of row `row`, or the y face f of column `row`.
template <bool BEDG, bool PRED, class M>
__device__ void band_face(const AdjArgs& a, int b, bool diry, int f, int row, float scale, float* rec) {
    const int ny = a.ny, nx = a.nx;
    const size_t plane = (size_t)ny * nx;
    line::PrimRec P[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        float z;
        const State q = diry ? padded_state<PRED, M>(a, b, f - 2 + s, row, scale, z)
                             : padded_state<PRED, M>(a, b, row, f - 2 + s, scale, z);
        P[s] = line::prim_rec<M>(q.h, q.hu, q.hv, z, a.kc);
    }
    const float d = diry ? a.kc.dy : a.kc.dx, rd = diry ? a.kc.rdy : a.kc.rdx;
    const int n = diry ? ny : nx;
    float rp[3] = {0.0f, 0.0f, 0.0f}, rm[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (f < n) rp[c] = M::div(a.lrhs[(diry ? a3(b, 0, f, row, ny, nx) : a3(b, 0, row, f, ny, nx)) + c * plane], d, rd);
        if (f >= 1)
            rm[c] = M::div(a.lrhs[(diry ? a3(b, 0, f - 1, row, ny, nx) : a3(b, 0, row, f - 1, ny, nx)) + c * plane], d, rd);
    }
    line::CellAdj out[4];
    line::face_vjp<BEDG, M>(P, rp[0] - rm[0], diry ? -rm[2] : -rm[1], diry ? rp[2] : rp[1],
                            diry ? rp[1] - rm[1] : rp[2] - rm[2], diry, a.kc, a.wsr != 0, out);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        rec[4 * s] = out[s].U0;
        rec[4 * s + 1] = out[s].U1;
        rec[4 * s + 2] = out[s].U2;
        rec[4 * s + 3] = BEDG ? out[s].Z : 0.0f;
    }
}

// Faces of all bands of a batch member.
__host__ __device__ inline long long side_items(const AdjArgs& a, int side) {
    return a.bandx != nullptr && level_side(a, side) ? band_faces(side < 2 ? a.ny : a.nx) : 0;
}
__host__ __device__ inline long long band_items(const AdjArgs& a) {
    return side_items(a, 0) + side_items(a, 1) + side_items(a, 2) + side_items(a, 3);
}

// The bands' faces, one per thread.  (In the tile kernel's grid their code
// cost every tile 8 to 25 %; here 10.6 and 8.7 us at 2 x 244 x 393.)
template <bool BEDG, bool PRED, class M>
__global__ void __launch_bounds__(64) adj_band_kernel(const AdjArgs a) {
    chain_start();
    const int b = blockIdx.y;
    float scale = 0.0f;
    if (PRED) scale = 0.5f * (a.dt_dev != nullptr ? *a.dt_dev : a.dt);
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int side = 0;
    while (side < 4 && t >= side_items(a, side)) t -= side_items(a, side++);
    if (side == 4) return;
    const int n = side < 2 ? a.ny : a.nx, m = side < 2 ? a.nx : a.ny;  // along, across
    const LevelBand band(a, b, side);
    const bool far = (side & 1) != 0, normal = t < 4LL * n;
    if (!normal) t -= 4LL * n;
    const int len = normal ? n : n + 1;
    const int d = (int)(t / len), pos = (int)(t - (long long)d * len);  // d: or the line of cells
    const int across = far ? (normal ? m - d : m - 1 - d) : d;
    band_face<BEDG, PRED, M>(a, b, normal == (side >= 2), normal ? across : pos, normal ? pos : across, scale,
                             normal ? band.normal(d, pos) : band.along(d, pos));
}

// Sum over the band's faces along one axis of what they contribute to padded
// cell `pos` (its index along that axis, n interior cells; `line` its index
// along the other), in the faces' order.  normal: the axis is the side's
// normal; e: the band's line of cells.
__device__ __noinline__ void band_sum(const LevelBand& band, bool normal, bool far, int e, int line, int pos,
                                      int n, float l[4]) {
    float v[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // all loads first: a face that is not there adds zero
        int f = pos - 1 + q;
        const bool ok = f >= 0 && f <= n;
        f = min(max(f, max(pos - 1, 0)), min(pos + 2, n));
        const float* r = (normal ? band.normal(far ? n - f : f, line) : band.along(e, f)) + 4 * (3 - q);
#pragma unroll
        for (int c = 0; c < 4; ++c) v[q][c] = ok ? r[c] : 0.0f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) l[c] = (((0.0f + v[0][c]) + v[1][c]) + v[2][c]) + v[3][c];
}

// The same sum with the faces evaluated here, one by each of four lanes that
// share a cell (q: this lane's): along x of row `line`, or along y of column
// `line`.  (A cell's lane evaluating all four takes the edge kernel 74 and 81
// us in the two stages at 2 x 24 x 30, four lanes 38 and 43; tile sums 6.)
template <bool BEDG, bool PRED, class M>
__device__ __noinline__ void face_sum(const AdjArgs& a, int b, bool diry, int line, int pos, int n, float scale,
                                      int q, float l[4]) {
    const int f = pos - 1 + q, lane = threadIdx.x & 31;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (f >= 0 && f <= n) {
        float r[BAND_REC];
        band_face<BEDG, PRED, M>(a, b, diry, f, line, scale, r);
#pragma unroll
        for (int s = 0; s < 4; ++s)  // (a constant index keeps the record in registers)
            if (s == 3 - q)
                for (int c = 0; c < 4; ++c) v[c] = r[4 * s + c];
    }
    const unsigned group = 0xfu << (lane & 28);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        l[c] = 0.0f;
        for (int k = 0; k < 4; ++k) l[c] += __shfl_sync(group, v[c], (lane & 28) + k);
    }
}

// Floats per cell of the sides' and adjoints' slots (see adj_tile_kernel).
template <bool BEDG>
__host__ __device__ constexpr int adj_slots() { return BEDG ? 14 : 10; }

template <bool BEDG, int TY>
__host__ __device__ constexpr int adj_tile_smem() {
    return (int)sizeof(float) * (5 * (TY + 6) * (ADJ_TX + 6) + adj_slots<BEDG>() * TY * (ADJ_TX + 4) +
                                 adj_slots<BEDG>() * (TY + 4) * ADJ_TX);
}

// A line of cells through the tile in one direction: the primitives and the
// slots of its cells, `ps` and `ss` floats apart from one cell to the next,
// `pf` and `sf` from one field or slot to the next.
//
// Slots of a cell: the sides p (0-4: hlin, eta, bed, u, v) and m (5-9), over
// which each face writes its adjoints of the sides it read (p: 0 hlin, 1 eta,
// 2 the cell's h, 3 u, 4 v, BEDG: 10 bed, 11 the cell's z; m: 5-9, 12, 13),
// over which each cell writes what its sides contribute to its left
// neighbour (0 h, 1 u, 2 v, BEDG 10 z), itself (3 h, 4 safe, 5 u, 6 v, 11 z)
// and its right neighbour (7 h, 8 u, 9 v, 12 z).
struct Line {
    const float* prim;
    float* slot;
    int pf, sf;
};

__device__ __forceinline__ CellPrim prim_at(const Line& l, int off) {
    const float* p = l.prim + off;
    return CellPrim{p[0], p[l.pf], p[2 * l.pf], p[3 * l.pf], p[4 * l.pf]};
}

template <class M>
__device__ __forceinline__ void line_sides(const Line& l, int ps, const SweConsts& k, bool wsr) {
    const SidePair s = side_pair<M>(prim_at(l, -ps), prim_at(l, 0), prim_at(l, ps), k, wsr);
    float* q = l.slot;
    const int f = l.sf;
    q[0] = s.p.hlin;
    q[f] = s.p.eta;
    q[2 * f] = s.p.bed;
    q[3 * f] = s.p.u;
    q[4 * f] = s.p.v;
    q[5 * f] = s.m.hlin;
    q[6 * f] = s.m.eta;
    q[7 * f] = s.m.bed;
    q[8 * f] = s.m.u;
    q[9 * f] = s.m.v;
}

// The face between the line's cell and the next one.  lo / hi: the
// tendency's cotangents (mass, normal, tangential, already over d) of the
// two cells (zero outside the grid).  tame: see kTame.
template <bool BEDG, class M>
__device__ __forceinline__ void line_face(const Line& l, int ps, int ss, bool exists, const float lo[3],
                                          const float hi[3], bool normal_y, bool tame, const SweConsts& k) {
    float* qp = l.slot;
    float* qm = l.slot + ss;
    const int f = l.sf;
    SideAdj lL{}, lR{};
    if (exists) {
        const Side L{qp[0], qp[f], qp[2 * f], qp[3 * f], qp[4 * f]};
        const Side R{qm[5 * f], qm[6 * f], qm[7 * f], qm[8 * f], qm[9 * f]};
        const float* p = l.prim;
        // (F_right(f) - F_left(f + 1)) / d
        const float l_mass = hi[0] - lo[0], l_tan = hi[2] - lo[2];
        // a face without water on either side carries no flux, whatever the
        // cotangents of its mass and tangential momentum
        const bool idle = lo[1] == 0.0f && hi[1] == 0.0f &&
                          ((l_mass == 0.0f && l_tan == 0.0f) || (L.hlin <= 0.0f && R.hlin <= 0.0f));
        if (!(tame && idle))
            face_adj<BEDG, M>(L, p[0], p[4 * l.pf], R, p[ps], p[4 * l.pf + ps], l_mass, -lo[1], hi[1], l_tan,
                              normal_y, k, lL, lR);
    }
    qp[0] = lL.hlin;
    qp[f] = lL.eta;
    qp[2 * f] = lL.dh;
    qp[3 * f] = lL.u;
    qp[4 * f] = lL.v;
    qm[5 * f] = lR.hlin;
    qm[6 * f] = lR.eta;
    qm[7 * f] = lR.dh;
    qm[8 * f] = lR.u;
    qm[9 * f] = lR.v;
    if (BEDG) {
        qp[10 * f] = lL.bed;
        qp[11 * f] = lL.dz;
        qm[12 * f] = lR.bed;
        qm[13 * f] = lR.dz;
    }
}

template <bool BEDG, class M>
__device__ __forceinline__ void line_cell(const Line& l, int ps, bool exists, bool tame, const SweConsts& k,
                                          bool wsr) {
    float* q = l.slot;
    const int f = l.sf;
    LineAdj left{}, right{};
    PrimAdj own{};
    if (exists) {
        SideAdj lp{q[0], q[f], q[3 * f], q[4 * f], q[2 * f], 0.0f, 0.0f};
        SideAdj lm{q[5 * f], q[6 * f], q[8 * f], q[9 * f], q[7 * f], 0.0f, 0.0f};
        if (BEDG) {
            lp.bed = q[10 * f];
            lp.dz = q[11 * f];
            lm.bed = q[12 * f];
            lm.dz = q[13 * f];
        }
        const bool idle = lp.hlin == 0.0f && lp.eta == 0.0f && lp.u == 0.0f && lp.v == 0.0f && lp.dh == 0.0f &&
                          lm.hlin == 0.0f && lm.eta == 0.0f && lm.u == 0.0f && lm.v == 0.0f && lm.dh == 0.0f &&
                          (!BEDG || (lp.bed == 0.0f && lp.dz == 0.0f && lm.bed == 0.0f && lm.dz == 0.0f));
        if (tame && idle) return;  // its slots hold the zeros already
        side_pair_bwd<BEDG, M>(prim_at(l, -ps), prim_at(l, 0), prim_at(l, ps), lp, lm, k, wsr, left, own, right);
    }
    q[0] = left.h;
    q[f] = left.u;
    q[2 * f] = left.v;
    q[3 * f] = own.h;
    q[4 * f] = own.safe;
    q[5 * f] = own.u;
    q[6 * f] = own.v;
    q[7 * f] = right.h;
    q[8 * f] = right.u;
    q[9 * f] = right.v;
    if (BEDG) {
        q[10 * f] = left.z;
        q[11 * f] = own.z;
        q[12 * f] = right.z;
    }
}

// Adds what reaches a cell's primitives along a line: its own slots and, if
// they are there, its neighbours'.
template <bool BEDG>
__device__ __forceinline__ void line_sum(const Line& l, int ss, bool self, bool lower, bool upper, PrimAdj& t) {
    const float* q = l.slot;
    const int f = l.sf;
    if (self) {
        t.h += q[3 * f];
        t.safe += q[4 * f];
        t.u += q[5 * f];
        t.v += q[6 * f];
        if (BEDG) t.z += q[11 * f];
    }
    if (lower) {
        const float* r = q - ss;
        t.h += r[7 * f];
        t.u += r[8 * f];
        t.v += r[9 * f];
        if (BEDG) t.z += r[12 * f];
    }
    if (upper) {
        const float* r = q + ss;
        t.h += r[0];
        t.u += r[f];
        t.v += r[2 * f];
        if (BEDG) t.z += r[10 * f];
    }
}

__device__ __forceinline__ bool in_frame(const AdjArgs& a, int j, int i) {
    return i < 2 || i >= a.nx - 2 || j < 2 || j >= a.ny - 2;
}

// The reverse mode is linear in the cotangents, so where they are exactly
// zero its results are too, as long as no factor is infinite or NaN: values
// up to kTame in magnitude leave the factors (products of at most four of
// them, quotients by clamped depths) far inside the range of a float.  A
// gauge misfit's gradient is zero ahead of the front that has left the
// gauges, four cells a step, and on dry land (the clean-up passes no
// momentum cotangent of a dry cell).  Over a run of 112 steps at 4 x 244 x
// 393 the tile kernels took 45 + 39 us a step with the zeros skipped and 58 +
// 52 without; where nothing is zero the test costs them 5 %.
constexpr float kTame = 1e8f;
__device__ __forceinline__ bool tame3(float x, float y, float z) {
    return fabsf(x) <= kTame && fabsf(y) <= kTame && fabsf(z) <= kTame;
}

// What becomes of a cell's adjoint lam of S (or of P).
template <bool PRED, class M>
__device__ __forceinline__ void finish_cell(const AdjArgs& a, size_t o, size_t plane, const float lam[3],
                                            float scale) {
    if (PRED) {  // predictor P = clean(U, U + dt/2 k1), solver.py:639
        const State u{a.U[o], a.U[o + plane], a.U[o + 2 * plane]};
        const State cand{u.h + scale * a.k1[o], u.hu + scale * a.k1[o + plane], u.hv + scale * a.k1[o + 2 * plane]};
        State lold, lcand;
        clean_bwd<M>(u, cand, State{lam[0], lam[1], lam[2]}, a.kc, a.positivity != 0, lold, lcand);
        a.lU[o] += lold.h + lcand.h;
        a.lU[o + plane] += lold.hu + lcand.hu;
        a.lU[o + 2 * plane] += lold.hv + lcand.hv;
        a.lk1[o] = lcand.h * scale;
        a.lk1[o + plane] = lcand.hu * scale;
        a.lk1[o + 2 * plane] = lcand.hv * scale;
    } else {
        a.lS[o] += lam[0];
        a.lS[o + plane] += lam[1];
        a.lS[o + 2 * plane] += lam[2];
    }
}

// A tile whose cotangents are all zero: adds nothing, and writes the zeros
// that the edges or the next kernel read.
template <bool PRED>
__device__ __forceinline__ void zero_tile(const AdjArgs& a, int b, int j0, int i0, int rows) {
    const int ny = a.ny, nx = a.nx;
    const size_t plane = (size_t)ny * nx;
    for (int w = threadIdx.x; w < rows * ADJ_TX; w += ADJ_THREADS) {
        const int j = j0 + w / ADJ_TX, i = i0 + w % ADJ_TX;
        if (j >= ny || i >= nx) continue;
        if (in_frame(a, j, i)) {
            float* fr = a.frame + (size_t)b * 4 * plane + (size_t)j * nx + i;
            fr[0] = fr[plane] = fr[2 * plane] = fr[3 * plane] = 0.0f;
        } else if (PRED) {
            float* q = a.lk1 + a3(b, 0, j, i, ny, nx);
            q[0] = q[plane] = q[2 * plane] = 0.0f;
        }
    }
    for (int w = threadIdx.x; w < 4 * rows; w += ADJ_THREADS) {  // [left, right][1st, 2nd][row]
        const int q = w / rows, j = j0 + w % rows;
        if ((q < 2 ? i0 == 0 : nx - i0 <= ADJ_TX) && j < ny)
            for (int c = 0; c < 4; ++c) a.gx[4 * (((size_t)b * 4 + q) * ny + j) + c] = 0.0f;
    }
    for (int w = threadIdx.x; w < 4 * ADJ_TX; w += ADJ_THREADS) {  // [top, bottom][1st, 2nd][column]
        const int q = w / ADJ_TX, i = i0 + w % ADJ_TX;
        if ((q < 2 ? j0 == 0 : ny - j0 <= rows) && i < nx)
            for (int c = 0; c < 4; ++c) a.gy[4 * (((size_t)b * 4 + q) * nx + i) + c] = 0.0f;
    }
}

// Instruction and latency bound (its operands fit in L2 at the grids it runs
// on).  Each cell's limiters and each face's reverse mode are evaluated once
// per direction and a cell's primitives once per pass; 16 rows keep the halo
// work at 1.1 (x) to 1.2 (y) times the tile's.  The form it replaces ran a
// thread per face (both cells' sides and four cells' primitives again for
// each) and moved 24 floats per cell through memory to a gather kernel: 114
// us for the faces and 18 to 21 for the gather of one launch pair at 4 x 244
// x 393 in the IEEE arithmetic, against 58.5 (stage 2) and 52 (stage 1) here
// plus 8 for the edges.
template <bool BEDG, bool PRED, class M, int TY>
__global__ void __launch_bounds__(ADJ_THREADS, SWE_ADJ_TILE_MINB) adj_tile_kernel(const AdjArgs a) {
    constexpr int TX = ADJ_TX, RX = TX + 6, RY = TY + 6, SX = TX + 4, SY = TY + 4, NS = adj_slots<BEDG>();
    extern __shared__ float s_mem[];
    float* const s_p = s_mem;                    // primitives [5][RY][RX], cell (ry, rx) = (j0 - 3 + ry, i0 - 3 + rx)
    float* const s_x = s_p + 5 * RY * RX;        // x slots [NS][TY][SX], columns from i0 - 2
    float* const s_y = s_x + NS * TY * SX;       // y slots [NS][SY][TX], rows from j0 - 2
    chain_start();
    const int ny = a.ny, nx = a.nx, tid = threadIdx.x, b = blockIdx.y;
    float scale = 0.0f;
    if (PRED) scale = 0.5f * (a.dt_dev != nullptr ? *a.dt_dev : a.dt);
    const int ntx = (nx + TX - 1) / TX;
    const int i0 = (int)(blockIdx.x % (unsigned)ntx) * TX, j0 = (int)(blockIdx.x / (unsigned)ntx) * TY;
    const size_t plane = (size_t)ny * nx;
    const SweConsts& kc = a.kc;
    const bool wsr = a.wsr != 0;

    // primitives of the tile's cross: rows of the tile with three columns
    // either side, columns of the tile with three rows either side
    bool wild = false, idle = true;
    for (int w = tid; w < RY * RX; w += ADJ_THREADS) {
        const int ry = w / RX, rx = w - ry * RX;
        const int j = j0 + ry - 3, i = i0 + rx - 3;
        const bool xin = ry >= 3 && ry < TY + 3 && j < ny && i >= -2 && i <= nx + 1;
        const bool yin = rx >= 3 && rx < TX + 3 && i < nx && j >= -2 && j <= ny + 1;
        CellPrim p{};
        if (xin || yin) {
            float z;
            const State s = padded_state<PRED, M>(a, b, j, i, scale, z);
            p = cell_prim<M>(s.h, s.hu, s.hv, z, kc);
            wild |= !(tame3(p.h, p.u, p.v) && fabsf(p.eta) <= kTame);
            if ((unsigned)j < (unsigned)ny && (unsigned)i < (unsigned)nx) {
                const float* q = a.lrhs + (size_t)b * 3 * plane + (size_t)j * nx + i;
                idle &= q[0] == 0.0f && q[plane] == 0.0f && q[2 * plane] == 0.0f;
            }
        }
        s_p[w] = p.h;
        s_p[RY * RX + w] = p.u;
        s_p[2 * RY * RX + w] = p.v;
        s_p[3 * RY * RX + w] = p.eta;
        s_p[4 * RY * RX + w] = p.z;
    }
    const bool tame = !__syncthreads_or(wild);
    bool quiet = !__syncthreads_or(!idle) && tame;
    if (PRED && quiet) {  // the predictor's adjoint takes U and U + dt/2 k1, of which dry cells show nothing
        bool odd = false;
        for (int w = tid; w < TY * TX; w += ADJ_THREADS) {
            const int ty = w / TX, tx = w % TX, j = j0 + ty, i = i0 + tx;
            if (j >= ny || i >= nx || s_p[(ty + 3) * RX + tx + 3] > kc.dry) continue;
            const size_t o = a3(b, 0, j, i, ny, nx);
            for (int c = 0; c < 3; ++c) {
                const float u = a.U[o + c * plane];
                odd |= !(fabsf(u) <= kTame && fabsf(u + scale * a.k1[o + c * plane]) <= kTame);
            }
        }
        quiet = !__syncthreads_or(odd);
    }
    if (quiet) {
        zero_tile<PRED>(a, b, j0, i0, TY);
        return;
    }

    // x line of row ty, slot column sx; y line of column tx, slot row sy
    auto xline = [&](int ty, int sx) {
        return Line{s_p + (ty + 3) * RX + sx + 1, s_x + ty * SX + sx, RY * RX, TY * SX};
    };
    auto yline = [&](int sy, int tx) {
        return Line{s_p + (sy + 1) * RX + tx + 3, s_y + sy * TX + tx, RY * RX, SY * TX};
    };

    for (int w = tid; w < TY * SX + SY * TX; w += ADJ_THREADS) {
        if (w < TY * SX) line_sides<M>(xline(w / SX, w % SX), 1, kc, wsr);
        else line_sides<M>(yline((w - TY * SX) / TX, (w - TY * SX) % TX), RX, kc, wsr);
    }
    __syncthreads();

    // x faces between slot columns fx and fx + 1, y faces between slot rows
    constexpr int NFX = TY * (SX - 1), NFY = (SY - 1) * TX;
    for (int w = tid; w < NFX + NFY; w += ADJ_THREADS) {
        const bool isx = w < NFX;
        const int v = isx ? w : w - NFX;
        const int line = isx ? v / (SX - 1) : v / TX, pos = isx ? v - line * (SX - 1) : v - line * TX;
        // first of the face's two cells
        const int j = isx ? j0 + line : j0 - 2 + line, i = isx ? i0 - 2 + pos : i0 + pos;
        const bool exists = isx ? j < ny && i >= -1 && i < nx : i < nx && j >= -1 && j < ny;
        float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
        const float rd = isx ? kc.rdx : kc.rdy;
        const size_t cn = isx ? plane : 2 * plane, ct = isx ? 2 * plane : plane;  // normal, tangential channels
        const float* q = a.lrhs + (size_t)b * 3 * plane + (ptrdiff_t)j * nx + i;
        if (exists && (isx ? i : j) >= 0) {
            lo[0] = q[0] * rd;
            lo[1] = q[cn] * rd;
            lo[2] = q[ct] * rd;
        }
        if (exists && (isx ? i + 1 < nx : j + 1 < ny)) {
            q += isx ? 1 : nx;
            hi[0] = q[0] * rd;
            hi[1] = q[cn] * rd;
            hi[2] = q[ct] * rd;
        }
        if (isx) line_face<BEDG, M>(xline(line, pos), 1, 1, exists, lo, hi, false, tame, kc);
        else line_face<BEDG, M>(yline(line, pos), RX, TX, exists, lo, hi, true, tame, kc);
    }
    __syncthreads();

    // cells whose sides have adjoints: the tile's and one more either side
    constexpr int NCX = TY * (TX + 2), NCY = (TY + 2) * TX;
    for (int w = tid; w < NCX + NCY; w += ADJ_THREADS) {
        if (w < NCX) {
            const int ty = w / (TX + 2), sx = 1 + w - ty * (TX + 2), i = i0 - 2 + sx;
            line_cell<BEDG, M>(xline(ty, sx), 1, j0 + ty < ny && i <= nx, tame, kc, wsr);
        } else {
            const int v = w - NCX, sy = 1 + v / TX, tx = v % TX, j = j0 - 2 + sy;
            line_cell<BEDG, M>(yline(sy, tx), RX, i0 + tx < nx && j <= ny, tame, kc, wsr);
        }
    }
    __syncthreads();

    for (int w = tid; w < TY * TX; w += ADJ_THREADS) {
        const int ty = w / TX, tx = w - ty * TX, j = j0 + ty, i = i0 + tx;
        if (j >= ny || i >= nx) continue;
        PrimAdj t{};
        line_sum<BEDG>(xline(ty, tx + 2), 1, true, true, true, t);
        line_sum<BEDG>(yline(ty + 2, tx), TX, true, true, true, t);
        const size_t o = a3(b, 0, j, i, ny, nx);
        const bool pass = PRED || a.S[o] >= 0.0f;  // a cleaned depth is never negative
        float lam[3];
        prim_bwd<M>(prim_at(xline(ty, tx + 2), 0), pass, t, kc, lam[0], lam[1], lam[2]);
        if (in_frame(a, j, i)) {
            const size_t c = (size_t)j * nx + i;
            float* fr = a.frame + (size_t)b * 4 * plane + c;
            fr[0] = lam[0];
            fr[plane] = lam[1];
            fr[2 * plane] = lam[2];
            if (BEDG) fr[3 * plane] = t.z;
            continue;
        }
        finish_cell<PRED, M>(a, o, plane, lam, scale);
        if (BEDG) a.lbed[(size_t)b * plane + (size_t)j * nx + i] += t.z;
    }

    // the ghosts along the sides that this tile touches: the first one has
    // slots of its own, the second only what the first's increments give it
    auto ghost = [&](const Line& l, int ss, int dir, bool second, int j, int i, float* out) {
        PrimAdj t{};
        // dir: -1 below / left of the grid, +1 above / right of it
        if (!second) line_sum<BEDG>(l, ss, true, dir > 0, dir < 0, t);
        else line_sum<BEDG>(l, ss, false, dir > 0, dir < 0, t);
        float z, l0, l1, l2;
        const State s = padded_state<PRED, M>(a, b, j, i, scale, z);
        prim_bwd<M>(cell_prim<M>(s.h, s.hu, s.hv, z, kc), s.h >= 0.0f, t, kc, l0, l1, l2);
        out[0] = l0;
        out[1] = l1;
        out[2] = l2;
        out[3] = t.z;
    };
    const bool sides[4] = {i0 == 0, nx - i0 <= TX, j0 == 0, ny - j0 <= TY};
    for (int w = tid; w < 4 * TY; w += ADJ_THREADS) {
        const int side = w / (2 * TY), second = (w / TY) & 1, ty = w % TY, j = j0 + ty;
        if (!sides[side] || j >= ny) continue;
        const int i = side == 0 ? -1 - second : nx + second;
        ghost(xline(ty, i - i0 + 2), 1, side == 0 ? -1 : 1, second != 0, j, i,
              a.gx + 4 * ((((size_t)b * 2 + side) * 2 + second) * ny + j));
    }
    for (int w = tid; w < 4 * TX; w += ADJ_THREADS) {
        const int side = w / (2 * TX), second = (w / TX) & 1, tx = w % TX, i = i0 + tx;
        if (!sides[2 + side] || i >= nx) continue;
        const int j = side == 0 ? -1 - second : ny + second;
        ghost(yline(j - j0 + 2, tx), TX, side == 0 ? -1 : 1, second != 0, j, i,
              a.gy + 4 * ((((size_t)b * 2 + side) * 2 + second) * nx + i));
    }
}

// Folds the adjoint lg of ghost g (side `side`; g its column for left/right,
// row for top/bottom) into cell (j, i) if the ghost was made from it, and
// adds the level adjoint once per ghost (in the thread of the ghost's
// clamped source cell).  BEDG: lg[3] is the ghost's bed adjoint, folded into
// the cell its bed was copied from (replicate, or periodic), plus the bed
// terms of the forced ghost depth max(level - z, 0) -> lzc.
template <bool BEDG, bool PRED, class M>
__device__ void fold_ghost(const AdjArgs& a, int b, int side, int g, const float* lg, int j, int i,
                           float scale, float lam[3], float& llev, float& lzc) {
    const int ny = a.ny, nx = a.nx;
    const bool xs = side < 2;
    const int n = xs ? nx : ny;
    const int pos = xs ? i : j;  // this cell's index along the side's direction
    const int clamp_src = g < 0 ? 0 : n - 1;
    const int mirror = g < 0 ? -1 - g : 2 * n - 1 - g;
    const int periodic = g < 0 ? n + g : g - n;
    const int normal = xs ? 1 : 2;  // momentum channel reflected by a wall
    const int code = a.bc[side];
    if (BEDG && pos == (code == SWE_BC_PERIODIC ? periodic : clamp_src)) lzc += lg[3];
    switch (code) {
    case SWE_BC_TRANSMISSIVE:
        if (pos == clamp_src) {
            lam[0] += lg[0];
            lam[1] += lg[1];
            lam[2] += lg[2];
        }
        break;
    case SWE_BC_PERIODIC:
        if (pos == periodic) {
            lam[0] += lg[0];
            lam[1] += lg[1];
            lam[2] += lg[2];
        }
        break;
    case SWE_BC_CONSTANT:
        break;
    case SWE_BC_WATER_LEVEL:
        if (pos == clamp_src) {
            lam[1] += lg[1];
            lam[2] += lg[2];
            const float z = bed_of(a, b, xs ? j : clamp_src, xs ? clamp_src : i);
            const float lev = a.level[a.levelB == 1 ? 0 : b];
            if (lev - z >= 0.0f) {  // clamp(level - z, min=0)
                llev += lg[0];
                if (BEDG) lzc -= lg[0];
            }
        }
        break;
    case SWE_BC_WALL:
        if (pos == clamp_src) {
            lam[0] += lg[0];
            lam[3 - normal] += lg[3 - normal];
        }
        if (pos == mirror) lam[normal] -= lg[normal];
        break;
    case SWE_BC_ABSORBING:
        if (pos == clamp_src) {
            lam[3 - normal] += lg[3 - normal];
            lam[0] += lg[0];
            // value = s c (hg - hr), hr = max(level - z, 0),
            // c = sqrt(9.81 max(where(hr > 1e-4, hr, hg), 1e-6))
            const int jj = xs ? j : clamp_src, ii = xs ? clamp_src : i;
            const float hg = cell_state<PRED, M>(a, b, jj, ii, scale).h;
            const float z = bed_of(a, b, jj, ii);
            const float lev = a.level[a.levelB == 1 ? 0 : b];
            const float hr = fmaxf(lev - z, 0.0f);
            const bool use_hr = hr > a.kc.absorb_lim;
            const float hc = use_hr ? hr : hg;
            const float cm = fmaxf(hc, a.kc.absorb_min);
            const float c = M::sqrt(a.kc.g981 * cm);
            const float s = (side == 0 || side == 2) ? -1.0f : 1.0f;
            const float lv = lg[normal];
            const float l_c = lv * (s * (hg - hr));
            const float l_diff = lv * (s * c);
            float l_hc = 0.0f;
            if (hc >= a.kc.absorb_min) {
                const float c2 = 2.0f * c;
                l_hc = a.kc.g981 * M::div(l_c, c2, M::rcp(c2));
            }
            float l_hg = l_diff + (use_hr ? 0.0f : l_hc);
            float l_hr = -l_diff + (use_hr ? l_hc : 0.0f);
            lam[0] += l_hg;
            if (lev - z >= 0.0f) {
                llev += l_hr;
                if (BEDG) lzc -= l_hr;
            }
        }
        break;
    default:
        break;
    }
}

// Sum over a block in a fixed order (valid in thread 0).
__device__ __forceinline__ float block_sum(float v) {
    __shared__ float s_part[ADJ_THREADS / 32];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
    __syncthreads();
    float sum = 0.0f;
    if (threadIdx.x == 0)
        for (int w = 0; w < ADJ_THREADS / 32; ++w) sum += s_part[w];
    return sum;
}

// The frame: cells within two of a side, numbered along the top and bottom
// pairs of rows, then down the left and right pairs of columns.
__host__ __device__ __forceinline__ long long frame_cells(int ny, int nx) {
    return (ny <= 4 || nx <= 4) ? (long long)ny * nx : 4LL * nx + 4LL * (ny - 4);
}
__device__ __forceinline__ void frame_cell(int ny, int nx, long long t, int& j, int& i) {
    if (ny <= 4 || nx <= 4) {
        j = (int)(t / nx);
        i = (int)(t - (long long)j * nx);
    } else if (t < 4LL * nx) {
        const int r = (int)(t / nx);
        j = r < 2 ? r : ny - 4 + r;
        i = (int)(t - (long long)r * nx);
    } else {
        t -= 4LL * nx;
        const int c = (int)(t & 3);
        j = 2 + (int)(t >> 2);
        i = c < 2 ? c : nx - 4 + c;
    }
}

// Finishes the frame, a cell per thread.  A few warps run through it once,
// so its time is that of its instruction fetches and load chains: one copy
// of each part, no ghost read in vain.  FLY: level bands without records,
// four lanes per cell.
template <bool BEDG, bool PRED, bool FLY, class M>
__global__ void __launch_bounds__(ADJ_THREADS) adj_edge_kernel(const AdjArgs a) {
    chain_start();
    const int ny = a.ny, nx = a.nx, b = blockIdx.y;
    const size_t plane = (size_t)ny * nx;
    float scale = 0.0f;
    if (PRED) scale = 0.5f * (a.dt_dev != nullptr ? *a.dt_dev : a.dt);
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int face = FLY ? (int)(t & 3) : 0;
    if (FLY) t >>= 2;
    float level = 0.0f;
    if (t < frame_cells(ny, nx)) {
        int j, i;
        frame_cell(ny, nx, t, j, i);
        float llev = 0.0f;
        // the band this cell lies in, if any
        int bs = -1;
        for (int side = 3; side >= 0; --side) {
            const int dist = side == 0 ? i : side == 1 ? nx - 1 - i : side == 2 ? j : ny - 1 - j;
            if (dist < 2 && level_side(a, side)) bs = side;
        }
        const LevelBand band(a, b, bs < 0 ? 0 : bs);
        const bool far = (bs & 1) != 0;
        const int e = bs < 2 ? (far ? nx - 1 - i : i) : (far ? ny - 1 - j : j);
        float lam[4], lz = 0.0f, l[4];
        float* fr = a.frame + (size_t)b * 4 * plane + (size_t)j * nx + i;
        if (bs < 0) {
            lam[0] = fr[0];
            lam[1] = fr[plane];
            lam[2] = fr[2 * plane];
            if (BEDG) lz = fr[3 * plane];
        } else {
            if (FLY) {
                face_sum<BEDG, PRED, M>(a, b, false, j, i, nx, scale, face, lam);
                face_sum<BEDG, PRED, M>(a, b, true, i, j, ny, scale, face, l);
            } else {
                band_sum(band, bs < 2, far, e, j, i, nx, lam);
                band_sum(band, bs >= 2, far, e, i, j, ny, l);
            }
            lam[0] += l[0];
            lam[1] += l[1];
            lam[2] += l[2];
            if (BEDG) lz = lam[3] + l[3];
        }
#pragma unroll 1
        for (int q = 0; q < 8; ++q) {  // ghosts -1, -2, nx, nx + 1, then the rows'
            const int side = q >> 1, second = q & 1;
            const bool yax = side >= 2;
            const int n = yax ? ny : nx, pos = yax ? j : i;
            const int g = (side & 1) ? n + second : -1 - second;
            const int code = a.bc[side], edge = (side & 1) ? n - 1 : 0;
            const int mirror = g < 0 ? -1 - g : 2 * n - 1 - g, periodic = g < 0 ? n + g : g - n;
            const bool touches = code == SWE_BC_PERIODIC ? pos == periodic
                                                         : pos == edge || (code == SWE_BC_WALL && pos == mirror);
            if (!touches || (code == SWE_BC_CONSTANT && !BEDG)) continue;
            // a band holds the records of its own side's ghosts and of those
            // at the ends of its two lines
            if (FLY && (level_side(a, side) || (bs >= 0 && (bs < 2) == yax))) {
                face_sum<BEDG, PRED, M>(a, b, yax, yax ? i : j, g, n, scale, face, l);
            } else if (level_side(a, side)) {
                band_sum(LevelBand(a, b, side), true, (side & 1) != 0, 0, yax ? i : j, g, n, l);
            } else if (bs >= 0 && (bs < 2) == yax) {
                band_sum(band, false, far, e, yax ? i : j, g, n, l);
            } else {
                const float* gl = yax ? a.gy + 4 * (((size_t)b * 4 + (q - 4)) * nx + i)
                                      : a.gx + 4 * (((size_t)b * 4 + q) * ny + j);
                for (int c = 0; c < 4; ++c) l[c] = gl[c];
            }
            fold_ghost<BEDG, PRED, M>(a, b, side, g, l, j, i, scale, lam, llev, lz);
        }
        if (face == 0) {
            finish_cell<PRED, M>(a, a3(b, 0, j, i, ny, nx), plane, lam, scale);
            if (BEDG) a.lbed[(size_t)b * plane + (size_t)j * nx + i] += lz;
            fr[3 * plane] = level = llev;
        }
    }
    if (a.direct_level) {
        const float sum = block_sum(level);
        if (threadIdx.x == 0) {
            float* part = a.llevel_part + (size_t)b * a.level_blocks;
            part[blockIdx.x] = sum;
            for (int k = blockIdx.x + gridDim.x; k < a.level_blocks; k += gridDim.x) part[k] = 0.0f;
        }
    }
}

// Partial sums of the level's adjoint with bands: one cell of the grid per
// thread, so that their order does not depend on how the frame is dealt out.
static __global__ void __launch_bounds__(ADJ_THREADS, 8) adj_level_kernel(const float* frame, float* part, int ny,
                                                                         int nx) {
    chain_start();
    const int b = blockIdx.y;
    const size_t plane = (size_t)ny * nx;
    float llev = 0.0f;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)plane;
         t += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(t / nx), i = (int)(t - (long long)j * nx);
        if (i < 2 || i >= nx - 2 || j < 2 || j >= ny - 2) llev += frame[((size_t)b * 4 + 3) * plane + t];
    }
    const float sum = block_sum(llev);
    if (threadIdx.x == 0) part[(size_t)b * gridDim.x + blockIdx.x] = sum;
}

// Adjoint of the friction update (friction.py:12-131) w.r.t. its input state
// and the roughness field.
template <class M>
__device__ void friction_bwd(const State& s0, float n, float dt, int model, const SweConsts& k,
                             const State& lout, State& ls, float& ln) {
    const float h = fmaxf(s0.h, 0.0f);
    const bool wet = h > k.dry;
    if (!wet && fabsf(n) <= kTame && fabsf(dt) <= kTame) {  // no speed, so no friction
        ls = State{lout.h, 0.0f, 0.0f};
        ln = 0.0f;
        return;
    }
    const float safe = fmaxf(h, k.fr_vs);
    const float ys = M::rcp(safe);
    const float u = M::div(wet ? s0.hu : 0.0f, safe, ys), v = M::div(wet ? s0.hv : 0.0f, safe, ys);
    const float sp2 = u * u + v * v;
    const bool moving = wet && sp2 > 0.0f;
    const float S = fmaxf(sp2, k.fr_e2);
    const float speed = moving ? M::sqrt(S) : 0.0f;
    float cf;
    // cf and d cf / d h, d cf / d n (as autograd evaluates them)
    float dcf_dpre = 0.0f, dcf_dn = 0.0f, hpre = 0.0f;
    bool h_pass = false, n_pass = false;
    if (model == 0) {
        const float nn = fmaxf(n, 0.0f);
        hpre = fmaxf(h, k.fr_e);
        float pw, pwd;
        M::pow2(hpre, k.third, k.third - 1.0f, pw, pwd);
        const float num = k.g981 * (nn * nn);
        const float ypw = M::rcp(pw);
        cf = M::div(num, pw, ypw);
        // d/d pw: -cf / pw ; d pw / d hpre = third * hpre^(third - 1)
        const float dpw = k.third * pwd;
        dcf_dpre = -M::div(cf, pw, ypw) * dpw;
        dcf_dn = M::div(k.g981 * (2.0f * nn), pw, ypw);
        h_pass = h >= k.fr_e;
        n_pass = n >= 0.0f;
    } else {
        const float zz = fmaxf(n, k.fr_e);
        hpre = fmaxf(h, k.fr_e);
        const float yzz = M::rcp(zz);
        const float ratio = M::div(hpre, zz, yzz);
        const float shallow_den = fmaxf(0.46f * ratio, k.fr_e);
        const float rc = fmaxf(ratio, k.fr_e);
        const float lg = M::ln(rc);
        const float inv_rc = M::inv(rc);
        const float lt = 2.5f * ((lg - 1.0f) + inv_rc * 1.359f);
        const float deep_den = fmaxf(lt * lt, k.fr_e);
        const bool shallow_b = ratio < 2.71828182845904523536f;
        cf = shallow_b ? M::inv(shallow_den) : M::inv(deep_den);
        float dcf_dratio;
        if (shallow_b) {
            dcf_dratio = (0.46f * ratio >= k.fr_e) ? -(cf * cf) * 0.46f : 0.0f;
        } else {
            float dlt = 0.0f;
            if (ratio >= k.fr_e) dlt = 2.5f * (inv_rc - 1.359f * inv_rc * inv_rc);
            dcf_dratio = (lt * lt >= k.fr_e) ? -(cf * cf) * (2.0f * lt) * dlt : 0.0f;
        }
        dcf_dpre = M::div(dcf_dratio, zz, yzz);
        dcf_dn = -dcf_dratio * M::div(ratio, zz, yzz);
        h_pass = h >= k.fr_e;
        n_pass = n >= k.fr_e;
    }
    const float X = M::div((cf * speed) * dt, safe, ys);
    const float fac = M::inv(1.0f + X);
    ls.h = lout.h;
    ls.hu = wet ? lout.hu * fac : 0.0f;
    ls.hv = wet ? lout.hv * fac : 0.0f;
    float l_fac = wet ? lout.hu * s0.hu + lout.hv * s0.hv : 0.0f;
    const float l_D = -l_fac * (fac * fac);
    const float l_num = M::div(l_D, safe, ys);  // d/d((cf speed) dt)
    float l_safe = -l_D * M::div(X, safe, ys);
    const float l_cs = l_num * dt;
    const float l_cf = l_cs * speed;
    const float l_speed = l_cs * cf;
    float l_u = 0.0f, l_v = 0.0f;
    if (moving) {
        const float s2 = 2.0f * speed;
        const float l_S = M::div(l_speed, s2, M::rcp(s2));
        if (sp2 >= k.fr_e2) {
            l_u = l_S * (2.0f * u);
            l_v = l_S * (2.0f * v);
        }
    }
    if (wet) {
        ls.hu += M::div(l_u, safe, ys);
        ls.hv += M::div(l_v, safe, ys);
    }
    l_safe -= l_u * M::div(u, safe, ys) + l_v * M::div(v, safe, ys);
    float l_h = 0.0f;
    if (h >= k.fr_vs) l_h += l_safe;
    if (h_pass) l_h += l_cf * dcf_dpre;
    ln = n_pass ? l_cf * dcf_dn : 0.0f;
    if (s0.h >= 0.0f) ls.h += l_h;
}

// ------------------------------------------------------- pointwise adjoints

// Instruction bound (some 900 instructions a cell with friction, 60 % of the
// issue slots): 17.5 us a step at 4 x 244 x 393 with one logarithm for both
// powers and the skips of cells without a cotangent or without speed, 19.7
// without these.
template <class M>
__global__ void __launch_bounds__(ADJ_THREADS) adj_pointwise_kernel(const PwArgs a) {
    chain_start();
    const long long plane = (long long)a.ny * a.nx;
    const long long total = plane * a.B;
    float dt = a.dt, scale = a.scale;
    if (a.dt_dev != nullptr) {
        dt = *a.dt_dev;
        scale = (a.mode == 0 || a.mode == 3) ? dt : 0.5f * dt;
    }
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        // (a 64-bit quotient is some eighty instructions)
        const int b = total <= 0xffffffffll ? (int)((unsigned)t / (unsigned)plane) : (int)(t / plane);
        const long long i = t - (long long)b * plane;
        const size_t o = (size_t)b * 3 * plane + i;
        const State u{a.U[o], a.U[o + plane], a.U[o + 2 * plane]};
        const State cand{u.h + scale * a.k[o], u.hu + scale * a.k[o + plane],
                         u.hv + scale * a.k[o + 2 * plane]};
        if (a.mode == 2) {  // predictor forward, solver.py:639
            const State p = clean_fwd<M>(u, cand, a.kc, a.positivity != 0);
            a.P[o] = p.h;
            a.P[o + plane] = p.hu;
            a.P[o + 2 * plane] = p.hv;
            continue;
        }
        State lq{a.lout[o], a.lout[o + plane], a.lout[o + 2 * plane]};
        if (lq.h == 0.0f && lq.hu == 0.0f && lq.hv == 0.0f && tame3(u.h, u.hu, u.hv) &&
            tame3(cand.h, cand.hu, cand.hv) &&
            ((a.mode != 0 && a.mode != 3) || !a.friction ||
             (fabsf(dt) <= kTame && fabsf(a.n[(size_t)(a.nB == 1 ? 0 : b) * plane + i]) <= kTame))) {
            if (a.mode == 3) a.lU[o] = a.lU[o + plane] = a.lU[o + 2 * plane] = 0.0f;
            a.lk[o] = a.lk[o + plane] = a.lk[o + 2 * plane] = 0.0f;
            continue;
        }
        if ((a.mode == 0 || a.mode == 3) && a.friction) {
            const State q = clean_fwd<M>(u, cand, a.kc, a.positivity != 0);
            const size_t on = (size_t)(a.nB == 1 ? 0 : b) * plane + i;
            State lqi;
            float ln = 0.0f;
            friction_bwd<M>(q, a.n[on], dt, a.friction_model, a.kc, lq, lqi, ln);
            lq = lqi;
            if (a.nB == 1 && a.B > 1) atomicAdd(&a.ln[on], ln);
            else a.ln[on] += ln;
        }
        State lold, lcand;
        clean_bwd<M>(u, cand, lq, a.kc, a.positivity != 0, lold, lcand);
        // cand = U + scale * k; mode 3 writes the adjoint of U instead of adding to it
        if (a.mode == 3) {
            a.lU[o] = lold.h + lcand.h;
            a.lU[o + plane] = lold.hu + lcand.hu;
            a.lU[o + 2 * plane] = lold.hv + lcand.hv;
        } else {
            a.lU[o] += lold.h + lcand.h;
            a.lU[o + plane] += lold.hu + lcand.hu;
            a.lU[o + 2 * plane] += lold.hv + lcand.hv;
        }
        a.lk[o] = lcand.h * scale;
        a.lk[o + plane] = lcand.hu * scale;
        a.lk[o + 2 * plane] = lcand.hv * scale;
    }
}

inline int blocks_for(long long n) {
    long long b = (n + ADJ_THREADS - 1) / ADJ_THREADS;
    if (b < 1) b = 1;
    return (int)(b > 148LL * 32 ? 148LL * 32 : b);
}

// Tile kernel of height TY, its shared-memory limit raised once per device.
template <bool BEDG, bool PRED, class M, int TY>
cudaError_t launch_tiles(const AdjArgs& a, cudaStream_t s) {
    static std::atomic<uint64_t> set{0};
    constexpr int smem = adj_tile_smem<BEDG, TY>();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(set.load(std::memory_order_acquire) >> dev & 1)) {
        e = cudaFuncSetAttribute(adj_tile_kernel<BEDG, PRED, M, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev < 64) set.fetch_or(1ull << dev, std::memory_order_release);
    }
    const dim3 g((unsigned)((a.nx + ADJ_TX - 1) / ADJ_TX) * (unsigned)((a.ny + TY - 1) / TY), a.B);
    return launch_chained_smem(adj_tile_kernel<BEDG, PRED, M, TY>, g, dim3(ADJ_THREADS), smem, s, a);
}

// Enqueue the spatial adjoint of a (a.lbed set: with the bed's adjoint;
// pred: the stage-2 form, the predictor adjoint fused in).
template <bool BEDG, bool PRED, class M>
cudaError_t launch_adj_forms(AdjArgs a, cudaStream_t s) {
    const dim3 th(ADJ_THREADS);
    const dim3 ge((unsigned)((frame_cells(a.ny, a.nx) + ADJ_THREADS - 1) / ADJ_THREADS), a.B);
    const dim3 gf((unsigned)((4 * frame_cells(a.ny, a.nx) + ADJ_THREADS - 1) / ADJ_THREADS), a.B);
    const long long items = band_items(a);
    const bool level = level_side(a, 0) || level_side(a, 1) || level_side(a, 2) || level_side(a, 3);
    cudaError_t e = cudaSuccess;
    if (items > 0)
        e = launch_chained(adj_band_kernel<BEDG, PRED, M>, dim3((unsigned)((items + 63) / 64), a.B), dim3(64), s, a);
    a.direct_level = !level && a.level_blocks >= (int)ge.x;
    if (e == cudaSuccess) e = launch_tiles<BEDG, PRED, M, 16>(a, s);
    if (e == cudaSuccess)
        e = level && items == 0 ? launch_chained(adj_edge_kernel<BEDG, PRED, true, M>, gf, th, s, a)
                                : launch_chained(adj_edge_kernel<BEDG, PRED, false, M>, ge, th, s, a);
    if (e == cudaSuccess && !a.direct_level)
        e = launch_chained(adj_level_kernel, dim3(a.level_blocks, a.B), th, s, a.frame, a.llevel_part, a.ny, a.nx);
    return e;
}

// Enqueue the spatial adjoint of a (a.lbed set: with the bed's adjoint;
// pred: the stage-2 form, the predictor adjoint fused in).
template <class M>
int launch_adj_spatial(const AdjArgs& a, bool pred, cudaStream_t s) {
    const cudaError_t e =
        a.lbed ? (pred ? launch_adj_forms<true, true, M>(a, s) : launch_adj_forms<true, false, M>(a, s))
               : (pred ? launch_adj_forms<false, true, M>(a, s) : launch_adj_forms<false, false, M>(a, s));
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

template <class M>
int launch_adj_pointwise(const PwArgs& a, cudaStream_t s) {
    const cudaError_t e = launch_chained(adj_pointwise_kernel<M>, dim3(blocks_for((long long)a.B * a.ny * a.nx)),
                                         dim3(ADJ_THREADS), s, a);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

}  // namespace

// The FastMath instantiations (swe_adjoint_fast.cu).
int fast_launch_adj_spatial(const AdjArgs& a, bool pred, cudaStream_t s);
int fast_launch_adj_pointwise(const PwArgs& a, cudaStream_t s);

}  // namespace swe
