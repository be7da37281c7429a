// vh_step.cu -- the kernels of one hydro timestep (Hydro::performStep,
// src/hdo.cpp:1016-1134) on a structure-of-arrays FP64 grid.
//
// Data-parallel restructuring of the reference's sequential loops:
//  * face kernels compute each HLLE face flux once (two con2prims per face)
//    into a per-direction face array; a cell kernel then gathers the six
//    faces in the reference's accumulation order (x-, x+, y-, y+, z-, z+,
//    source), which keeps every cell's FP64 sum identical to the reference;
//  * the viscous part stores the two cell-centred con2prims that every
//    viscous stage re-derives (Qh at tau_n + dt/2 and Qh at tau_{n+1}) once
//    per cell and reuses them, which is exact because the reference
//    recomputes them from identical inputs;
//  * ghost cells are a gather from a per-dimension source map simulated on
//    the host from the reference's copy sequence (z, then y, then x).
#include <cuda_runtime.h>

#include <algorithm>

#include "vh_physics.cuh"
#include "vh_step.cuh"

namespace vh {

// resident blocks of 128 threads per SM, from sweeps (us per step at the
// stated counts): the face kernel 5 / 6 / 7 / 8 blocks 151 / 149 / 146 / 143 on
// the 101x101x51 event; the update on a list 6 / 8 / 10 / 12: 79 / 64 / 75 / 83
// there (two passes, 30 steps in), 49 / 51 / 60 / 66 early in it, 170 / 156 /
// 198 / 204 on 201x201x101, 155 / 139 / 150 / 181 on 101x101x51 cells full of
// matter; on every cell of the 2+1D grid of 101x101 4 / 5 / 6: 36 / 37 / 40;
// the viscous primitives 6 / 7 / 8: 30.8 / 31.5 / 33.1
constexpr int kFaceMinBlocks = 8, kUpdateMinBlocks = 8, kUpdateFewMinBlocks = 4, kPrimsMinBlocks = 6;

// -------------------------------------------------------------- updateM
// Fluid::updateM, src/fld.cpp:384-423 (both passes; out of place).
__device__ __forceinline__ void d_update_m(const Geo& g, const double* __restrict__ m,
                                           double* __restrict__ mo, const double* __restrict__ clk,
                                           int* __restrict__ fcount, int* __restrict__ nactive,
                                           long long blk) {
  const double tau = clk[0], dt = clk[1];  // the step's clock (device)
  const long long i = blk * blockDim.x + threadIdx.x;
  // the step's list counters, filled by later kernels
  if (i < 9) fcount[i] = 0;
  if (i == 0 && nactive) *nactive = 0;
  if (i >= g.N) return;
  int ix, iy, iz;
  coords(g, i, ix, iy, iz);
  const long long N = g.N;
  double d0 = 0., d1 = 0., d2 = 0.;
  if (maxM(m, N, i) < 1.) {
    // the loads of a stage together: as short-circuits they were a chain (us
    // per step, 101x101x51 18.4 and 15.8, 201x201x101 91.8 and 66.2)
    auto full = [&](int dx, int dy, int dz, int k) {
      return m[k * N + cidx(g, ix + dx, iy + dy, iz + dz)] >= 1.;
    };
    const bool fx = full(1, 0, 0, 0) | full(-1, 0, 0, 0);
    const bool fy = full(0, 1, 0, 1) | full(0, -1, 0, 1);
    const bool fz = full(0, 0, 1, 2) | full(0, 0, -1, 2);
    if (fx) d0 = dt / g.dx;
    if (fy) d1 = dt / g.dy;
    if (fz) d2 = dt / g.dz / tau;
    if (d0 == 0. && d1 == 0.) {
      auto most = [&](int dx, int dy) {
        return maxM(m, N, cidx(g, ix + dx, iy + dy, iz)) >= 1.;
      };
      if (most(1, 1) | most(1, -1) | most(-1, 1) | most(-1, -1)) {
        d0 = 0.707 * dt / g.dx;
        d1 = 0.707 * dt / g.dy;
      }
    }
  }
  // Cell::addM, src/cll.h:147-151, for X, Y, Z in turn
  double a0 = m[i], a1 = m[N + i], a2 = m[2 * N + i];
  a0 += d0;
  if (a0 > 0.9) a0 = a1 = a2 = 1.;
  a1 += d1;
  if (a1 > 0.9) a0 = a1 = a2 = 1.;
  a2 += d2;
  if (a2 > 0.9) a0 = a1 = a2 = 1.;
  mo[i] = a0;
  mo[N + i] = a1;
  mo[2 * N + i] = a2;
}
__global__ void k_update_m(Geo g, const double* __restrict__ m, double* __restrict__ mo,
                           const double* __restrict__ clk, int* __restrict__ fcount,
                           int* __restrict__ nactive) {
  d_update_m(g, m, mo, clk, fcount, nactive, blockIdx.x);
}


// ------------------------------------------------------- cells with matter
// i joins the list: one atomic for the lanes that arrive together
__device__ __forceinline__ void append(int* __restrict__ list, int* __restrict__ n, int i) {
  const unsigned with = __activemask();
  const int lane = threadIdx.x & 31, first = __ffs((int)with) - 1;
  int base = 0;
  if (lane == first) base = atomicAdd(n, __popc(with));
  base = __shfl_sync(with, base, first);
  list[base + __popc(with & ((1u << lane) - 1u))] = i;
}
// The same for the whole block (every thread calls it): one atomic, and the
// block's entries in thread order, so that a list keeps the grid's runs (with
// one atomic per warp the relaxation over the list took 112 instead of 101 us
// at 101x101x51).
__device__ __forceinline__ void append_block(int* __restrict__ list, int* __restrict__ n, int i,
                                             bool with) {
  __shared__ int cnt[4], first;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const unsigned bal = __ballot_sync(0xffffffffu, with);
  __syncthreads();  // an earlier call's reads
  if (lane == 0) cnt[warp] = __popc(bal);
  __syncthreads();
  if (threadIdx.x == 0) {
    int c = 0;
    for (int w = 0; w < nw; w++) c += cnt[w];
    first = c ? atomicAdd(n, c) : 0;
  }
  __syncthreads();
  if (!with) return;
  int at = first + __popc(bal & ((1u << lane) - 1u));
  for (int w = 0; w < warp; w++) at += cnt[w];
  list[at] = i;
}
// the cells the ghost copy writes (Fluid::correctImagCells: the two outermost
// of every side)
__device__ __forceinline__ bool is_ghost(const Geo& g, int ix, int iy, int iz) {
  return ix < 2 || ix >= g.nx - 2 || iy < 2 || iy >= g.ny - 2 || iz < 2 || iz >= g.nz - 2;
}
// what the viscous stages read of an empty cell: e and v at the half step, e
// at the full one
__device__ __forceinline__ void empty_prims(double* __restrict__ pA, double* __restrict__ pD,
                                            long long N, long long i) {
  pA[i] = 0.;
#pragma unroll
  for (int k = 5; k < 8; k++) pA[k * N + i] = 0.;
  pD[i] = 0.;
}

// ------------------------------------------------------------ face lists
// The faces that can carry a flux, one list per direction (cell i for its
// face on the + side).  Most of a grid is vacuum (80 to 92 % of the cells of
// the 3D events in their first steps, 30 % late), and a face between two
// empty edges, or between two cells that are not filled yet, adds nothing
// (src/hdo.cpp:118-144): with the faces taken in grid order the root finds
// ran on 39 to 51 % of their warps' lanes, on packed lists on 87 %.  A face
// off the list has no flux in memory either (fact), so its 56 bytes are
// neither written nor read.
//
// Exact: an edge with Q_t <= 0 is vacuum to transform_pv; hlle_flux returns
// for two vacuum edges, and for two unfilled cells unless it stops the run
// for e > 1e10, which e <= Q_t / tau rules out.  Lists are in block order,
// which varies; no face's flux depends on it.
//
// With `rows` the same kernel settles the cells whose own Q_t and six
// neighbours' are 0: nothing flows into them and they have no source, so their
// update is a copy of the row (predictor) or nothing (corrector).  The others
// are listed for the update, which so runs on full warps, and without the
// vacuum's memory traffic at its low occupancy: lists, faces and update took
// 247 us per step on the 101x101x51 event and take 226 (the update 95 and 54),
// 891 and 804 on 201x201x101.  One cell per thread: with two or four (an
// atomic per 256 or 512 cells) 2 to 15 % slower.
__device__ __forceinline__ void d_face_list(const Geo& g, const Fields& f, bool predict,
                                            bool rows, bool viscous, double* __restrict__ nbB,
                                            const double* __restrict__ clk, long long blk) {
  __shared__ int wcnt[4][4], base[4];
  const double* __restrict__ QT = predict ? f.Q : f.Qh;
  const double* __restrict__ m = f.m2;
  int* fcount = f.fcount + (predict ? 0 : 3);
  int* ucount = f.fcount + (predict ? 7 : 8);
  const long long i = blk * blockDim.x + threadIdx.x;
  const long long N = g.N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  unsigned act = 0;  // bit 3: the update list
  if (i < N) {
    int ix, iy, iz;
    coords(g, i, ix, iy, iz);
    const int cc[3] = {ix, iy, iz}, nn[3] = {g.nx, g.ny, g.nz};
    const long long ss[3] = {1, g.nx, (long long)g.nx * g.ny};
    const double x1 = QT[i], huge = 0.9e10 * clk[0];
    double up[3], dn[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      up[d] = cc[d] < nn[d] - 1 ? QT[i + ss[d]] : 0.;
      dn[d] = cc[d] > 0 ? QT[i - ss[d]] : 0.;
    }
    const bool far = rows && x1 == 0. && up[0] == 0. && up[1] == 0. && up[2] == 0. && dn[0] == 0. &&
                     dn[1] == 0. && dn[2] == 0. && QT[3 * N + i] == 0.;
    if (far) {
      const bool ghost = is_ghost(g, ix, iy, iz);
      if (predict) {
#pragma unroll
        for (int k = 0; k < 7; k++) {
          const double q = QT[k * N + i];
          f.Qprev[k * N + i] = q;
          f.Qh[k * N + i] = q;
        }
        // pB (the predictor's state at rest) is read of cells with matter at
        // the half step: not of this one, unless the ghost copy puts it there
        if (viscous && ghost) {
          f.pBC[i] = 1.;
#pragma unroll
          for (int k = 1; k < 5; k++) f.pBC[k * N + i] = 0.;
          if (nbB) nbB[i] = 0.;
        }
      } else if (viscous && !ghost) {
        empty_prims(f.pA, f.pD, N, i);
      }
    } else {
      act = rows ? 8u : 0u;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const double x2 = up[d];
        // two empty cells have two empty edges (a slope takes the smaller side)
        if (cc[d] >= nn[d] - 1 || (x1 == 0. && x2 == 0.)) continue;
        const long long st = ss[d];
        const bool dry = m[d * N + i] < 1. && m[d * N + i + st] < 1.;
        if (x1 > 0. && x2 > 0. && !dry) {  // matter on both sides: edges > 0
          act |= 1u << d;
          continue;
        }
        const double x0 = cc[d] > 0 ? dn[d] : x1, x3 = cc[d] < nn[d] - 2 ? QT[i + 2 * st] : x2;
        const double el = x1 + minmod((x2 - x1) / 2., (x1 - x0) / 2.);
        const double er = x2 - minmod((x3 - x2) / 2., (x2 - x1) / 2.);
        if (el <= 0. && er <= 0.) continue;
        if (dry && el <= huge) continue;
        act |= 1u << d;
      }
    }
    f.fact[i] = (unsigned char)(act & 7u);
  }
  unsigned bal[4];
#pragma unroll
  for (int d = 0; d < 4; d++) {
    bal[d] = __ballot_sync(0xffffffffu, (act >> d) & 1u);
    if (lane == 0) wcnt[d][warp] = __popc(bal[d]);
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    int n = 0;
    for (int w = 0; w < nw; w++) n += wcnt[threadIdx.x][w];
    base[threadIdx.x] = n ? atomicAdd(threadIdx.x < 3 ? fcount + threadIdx.x : ucount, n) : 0;
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 4; d++) {
    if (!((act >> d) & 1u)) continue;
    int at = base[d] + __popc(bal[d] & ((1u << lane) - 1u));
    for (int w = 0; w < warp; w++) at += wcnt[d][w];
    if (d < 3)
      f.flist[d * N + at] = (int)i;
    else
      f.ulist[at] = (int)i;
  }
}
__global__ void __launch_bounds__(128) k_face_list(Geo g, Fields f, bool predict, bool rows,
                                                   bool viscous, double* nbB,
                                                   const double* __restrict__ clk) {
  d_face_list(g, f, predict, rows, viscous, nbB, clk, blockIdx.x);
}

// ------------------------------------------------------------ face flux
// One HLLE face between cell i and its neighbour on the + side along a
// direction (Hydro::hlle_flux with Cell::getPrimVarRight / getPrimVarLeft or
// their H variants, src/cll.cpp:106-204), for the listed faces.  F[c*N + i]
// holds the flux of the face on the + side of cell i (0 where the reference
// adds nothing).
//
// A block of B threads takes B / 2 faces of one direction: thread t < B/2
// reconstructs and solves the left state of face t, thread t + B/2 its right
// state, the primitives meet in shared memory, and the first half of the
// block forms the fluxes.  One launch holds the faces of every direction
// (the direction of a block a run-time number), so the directions share one
// instruction stream, and there is one ragged end per pass instead of three.
// A thread that solved both states of a face (three kernels of 16 thousand
// warps) spent 5.6 of 14 cycles per issue waiting for instructions; in this
// form it is 0.5 of 9.  101x101x51, two passes, 20 % of the cells with
// matter: 492 us a step in that form, 280 in this one over the whole grid,
// 144 over the lists (with the list kernels).
//
// A state's 21 loads go out together, also for vacuum edges (with Q_t first
// and the rest behind its test 147 us), and what the root find does not need
// waits in shared memory (640 / 896 bytes of spills without, 532 / 792 so).
// A grid without any empty cell gains least from this form: lists, faces and
// hlle_flux of 101x101x51 cells 570 us a step in the three kernels, 553 here,
// but with charge 590 and 640, and 3950 and 4240, 4190 and 4900 of 201x201x101.
// Tried for those: both states of a face by one thread in turn (no barrier)
// even without charge, 4 % slower with; the flux one component at a time (324
// / 304 bytes of spills) 4 % slower; 5, 6 and 7 blocks per SM 3 to 8 % slower.
struct FaceBatch {
  int cnt[3], blocks[3];  // listed faces, and blocks of B / 2 of them, per direction
};
// without lists every cell stands for its faces
__device__ __forceinline__ FaceBatch face_batch(const Geo& g, const int* __restrict__ fcount) {
  FaceBatch b;
  const int half = blockDim.x >> 1;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    b.cnt[d] = fcount ? fcount[d] : (d < 2 || g.nz > 1 ? (int)g.N : 0);
    b.blocks[d] = (b.cnt[d] + half - 1) / half;
  }
  return b;
}
template <int EK>
__device__ __forceinline__ void d_face(const Geo& g, const EosDev& E, bool predict,
                                       const FaceBatch& fb, const double* __restrict__ QQ,
                                       const double* __restrict__ m, double* __restrict__ Fx,
                                       double* __restrict__ Fy, double* __restrict__ Fz,
                                       const int* __restrict__ flist,
                                       const double* __restrict__ clk, unsigned* err, int b) {
  __shared__ double sp[8][128];
  const int half = blockDim.x >> 1, t = threadIdx.x;
  const bool right = t >= half;
  const int dir = b < fb.blocks[0] ? X_ : (b < fb.blocks[0] + fb.blocks[1] ? Y_ : Z_);
  const int first = dir == X_ ? 0 : (dir == Y_ ? fb.blocks[0] : fb.blocks[0] + fb.blocks[1]);
  const int at = (b - first) * half + (right ? t - half : t);
  const int cnt = dir == X_ ? fb.cnt[0] : (dir == Y_ ? fb.cnt[1] : fb.cnt[2]);
  const double tau = clk[0], dt = clk[1];  // the step's clock (device)
  const long long N = g.N;
  const long long st = dir == X_ ? 1 : (dir == Y_ ? g.nx : (long long)g.nx * g.ny);
  bool face = at < cnt;
  const long long i = !face ? 0 : (flist ? flist[(dir - 1) * N + at] : at);
  int c = 0, n = 0;
  if (face) {
    int ix, iy, iz;
    coords(g, i, ix, iy, iz);
    c = dir == X_ ? ix : (dir == Y_ ? iy : iz);
    n = dir == X_ ? g.nx : (dir == Y_ ? g.ny : g.nz);
    face = c < n - 1;
  }
  if (face) {
    // the cell whose edge this is, and its neighbours (clamped as getCell)
    if (right) c++;
    const long long cell = i + (right ? st : 0);
    const long long lo = cell - (c > 0 ? st : 0), hi = cell + (c < n - 1 ? st : 0);
    // the reconstructed state, then divided by tau as one batch
    double q[7], M;
#pragma unroll
    for (int k = 0; k < 7; k++) {
      const double x0 = QQ[k * N + lo], x1 = QQ[k * N + cell], x2 = QQ[k * N + hi];
      const double dQ = minmod((x2 - x1) / 2., (x1 - x0) / 2.);
      q[k] = x1 + (right ? -dQ : dQ);
    }
    Prim p{0., 0., 0., 0., 0., 0., 0., 0.};
    if (!(q[T_] <= 0.)) {
      div_batch<7>(q, tau, 1.0 / tau, crm::mk_den_ok(tau));
      if (c2p_start(q, M)) {
        // what the root find does not need waits in the thread's own slots of sp
        volatile double* park = &sp[0][t];
        const int keep[5] = {X_, Y_, Z_, NQ_, NS_};
#pragma unroll
        for (int k = 0; k < 5; k++) park[128 * k] = q[keep[k]];
        double v, e, pr;
        c2p_root<EK>(E, q[T_], q[NB_], M, c2p_guess(E, cell), v, e, pr);
#pragma unroll
        for (int k = 0; k < 5; k++) q[keep[k]] = park[128 * k];
        c2p_state(q, M, v, e, pr, p);
      }
    }
    sp[0][t] = p.e;
    sp[1][t] = p.p;
    sp[2][t] = p.nb;
    sp[3][t] = p.nq;
    sp[4][t] = p.ns;
    sp[5][t] = p.vx;
    sp[6][t] = p.vy;
    sp[7][t] = p.vz;
  }
  double mL = 0., mR = 0.;  // before the barrier, whose wait covers the loads
  if (face && !right) {
    mL = m[(dir - 1) * N + i];
    mR = m[(dir - 1) * N + i + st];
  }
  __syncthreads();
  if (right || !face) return;
  auto prim = [&](int s) {
    return Prim{sp[0][s], sp[1][s], sp[2][s], sp[3][s], sp[4][s], sp[5][s], sp[6][s], sp[7][s]};
  };
  const double dxdir = dir == X_ ? g.dx : (dir == Y_ ? g.dy : g.dz);
  double* F = dir == X_ ? Fx : (dir == Y_ ? Fy : Fz);
  double fl[7];
  unsigned e = 0;
  const bool ok = hlle_face(dir, predict, tau, dt, dxdir, prim(t), prim(t + half),
                            mL, mR, fl, e);
  if (e) atomicOr(err, e);
#pragma unroll
  for (int k = 0; k < 7; k++) F[k * N + i] = ok ? fl[k] : 0.;
}
// resident blocks that walk the listed faces (their number is known on the
// device only); flist and fcount null: every face
template <int EK>
__global__ void __launch_bounds__(128, kFaceMinBlocks) k_face(
    Geo g, EosDev E, bool predict, const double* __restrict__ QQ, const double* __restrict__ m,
    double* __restrict__ Fx, double* __restrict__ Fy, double* __restrict__ Fz,
    const int* __restrict__ flist, const int* __restrict__ fcount, const double* __restrict__ clk,
    unsigned* err) {
  const FaceBatch fb = face_batch(g, fcount);
  const int nb = fb.blocks[0] + fb.blocks[1] + fb.blocks[2];
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    d_face<EK>(g, E, predict, fb, QQ, m, Fx, Fy, Fz, flist, clk, err, b);
    __syncthreads();  // the shared primitives are read
  }
}


// --------------------------------------------------- ideal cell update
// Gathers the six face fluxes and the Milne source (Hydro::source_step,
// src/hdo.cpp:307-353), then Cell::updateQtoQhByFlux (predictor) or
// Cell::updateByFlux (corrector), src/cll.cpp:70-88.
template <bool PRED, int EK>
__device__ __forceinline__ void d_update(const Geo& g, const EosDev& E, double* __restrict__ Q,
                                         double* __restrict__ Qh, double* __restrict__ Qprev,
                                         const double* __restrict__ Fx,
                                         const double* __restrict__ Fy,
                                         const double* __restrict__ Fz,
                                         const unsigned char* __restrict__ fact,
                                         const double* __restrict__ clk, unsigned* err,
                                         double* __restrict__ pB, double* __restrict__ pA,
                                         double* __restrict__ nbB, double* __restrict__ pD,
                                         int* __restrict__ wet, int* __restrict__ nwet,
                                         long long i) {
  const double tau = clk[0], dt = clk[1];  // the step's clock (device)
  const long long N = g.N;
  const bool in = i < N;  // (the whole block calls)
  int ix = 0, iy = 0, iz = 0;
  if (in) coords(g, i, ix, iy, iz);
  const bool ghost = is_ghost(g, ix, iy, iz);
  // the viscous stages' cells; the ghost copy settles its own
  const bool prims = !PRED && pA && in && !ghost;
  if (!PRED && pA) append_block(wet, nwet, (int)i, prims && !(Qh[i] <= 0.));
  if (!in) return;
  const long long sy = g.nx, sz = (long long)g.nx * g.ny;
  const double* field = PRED ? Q : Qh;
  const double tau1 = PRED ? tau : tau + 0.5 * dt;
  const double _dt = PRED ? dt / 2. : dt;
  // which of the six faces carry a flux (d_face_list; without lists all)
  bool xm = ix > 0, ym = iy > 0, zm = iz > 0;
  bool xp = ix < g.nx - 1, yp = iy < g.ny - 1, zp = iz < g.nz - 1;
  if (fact) {
    const unsigned fi = fact[i];
    xp = fi & 1u;
    yp = fi & 2u;
    zp = fi & 4u;
    if (xm) xm = fact[i - 1] & 1u;
    if (ym) ym = fact[i - sy] & 2u;
    if (zm) zm = fact[i - sz] & 4u;
  }
  const bool faces = xm | xp | ym | yp | zm | zp;
  double q[7], qin[7];
  qin[T_] = field[i];
  qin[Z_] = field[3 * N + i];
  // vacuum that nothing flows into: no flux, no source, the row stays
  const bool still = !faces && qin[T_] <= 0. && qin[Z_] == 0.;
  if (!PRED && still) {
    if (prims) empty_prims(pA, pD, N, i);
    return;
  }
#pragma unroll
  for (int k = 1; k < 7; k++)
    if (k != Z_) qin[k] = field[k * N + i];
  if (PRED && still) {
#pragma unroll
    for (int k = 0; k < 7; k++) {
      Qprev[k * N + i] = qin[k];
      Qh[k * N + i] = qin[k];
    }
    // pB is read of cells with matter at the half step: not of this one,
    // unless the ghost copy puts matter there
    if (pB && ghost) {
      pB[i] = 1.;
#pragma unroll
      for (int k = 1; k < 5; k++) pB[k * N + i] = 0.;
      if (nbB) nbB[i] = 0.;
    }
    return;
  }
  double fl[7];
#pragma unroll
  for (int k = 0; k < 7; k++) {
    double a = 0.;
    if (xm) a += Fx[k * N + i - 1];
    if (xp) a += -Fx[k * N + i];
    if (ym) a += Fy[k * N + i - sy];
    if (yp) a += -Fy[k * N + i];
    if (zm) a += Fz[k * N + i - sz];
    if (zp) a += -Fz[k * N + i];
    fl[k] = a;
  }
  q_over(qin, tau1, q);
  Prim pp;
  transform_pv<EK>(E, q, pp, c2p_guess(E, i));
  if (prims && qin[T_] <= 0.) empty_prims(pA, pD, N, i);
  if (prims && !(qin[T_] <= 0.)) {
    // con2prim(Qh / (tau_n + dt/2)) is the viscous stage's A =
    // con2prim(Qh / (tau_{n+1} - dt/2)) for every cell that the ghost copy
    // does not overwrite, whenever the divisors agree bit for bit
    pA[0 * N + i] = pp.e;
    pA[1 * N + i] = pp.p;
    pA[2 * N + i] = pp.nb;
    pA[3 * N + i] = pp.nq;
    pA[4 * N + i] = pp.ns;
    pA[5 * N + i] = pp.vx;
    pA[6 * N + i] = pp.vy;
    pA[7 * N + i] = pp.vz;
  }
  if (PRED && pB) {
    // con2prim(Q_n / tau_n) is the viscous stage's B = con2prim(Qprev /
    // (tau_{n+1} - dt)) whenever (tau_n + dt) - dt == tau_n: kept for it
    // as its four-velocity and e (the same arithmetic as k_visc_prims)
    const double ut = 1.0 / sqrt(1.0 - pp.vx * pp.vx - pp.vy * pp.vy - pp.vz * pp.vz);
    pB[0 * N + i] = ut;
    pB[1 * N + i] = ut * pp.vx;
    pB[2 * N + i] = ut * pp.vy;
    pB[3 * N + i] = ut * pp.vz;
    pB[4 * N + i] = pp.e;
    if (nbB) nbB[i] = pp.nb;  // with the vorticity on: B's T needs it
  }
  double kk[7];
  kk[T_] = -q[T_] * pp.vz * pp.vz - pp.p * (1. + pp.vz * pp.vz);
  kk[X_] = 0.;
  kk[Y_] = 0.;
  kk[Z_] = -q[Z_];
  kk[NB_] = 0.;
  kk[NQ_] = 0.;
  kk[NS_] = 0.;
#pragma unroll
  for (int k = 0; k < 7; k++) kk[k] *= _dt;
  if (kk[NB_] != kk[NB_]) {
    atomicOr(err, (unsigned)ERR_SOURCE_NAN);
  } else {
#pragma unroll
    for (int k = 0; k < 7; k++) fl[k] += kk[k];
  }
  if (PRED) {
#pragma unroll
    for (int k = 0; k < 7; k++) {
      Qprev[k * N + i] = qin[k];
      Qh[k * N + i] = qin[k] + fl[k];
    }
  } else {
    if (!(Q[i] + fl[0] < 0.)) {
#pragma unroll
      for (int k = 0; k < 7; k++) Q[k * N + i] += fl[k];
    }
  }
}
// LIST: the cells d_face_list listed; else every cell
template <bool PRED, int EK, bool LIST>
__global__ void __launch_bounds__(128, LIST ? kUpdateMinBlocks : kUpdateFewMinBlocks)
k_update(Geo g, EosDev E, double* __restrict__ Q, double* __restrict__ Qh,
         double* __restrict__ Qprev, const double* __restrict__ Fx, const double* __restrict__ Fy,
         const double* __restrict__ Fz, const unsigned char* __restrict__ fact,
         const double* __restrict__ clk, unsigned* err, double* __restrict__ pB,
         double* __restrict__ pA, double* __restrict__ nbB, double* __restrict__ pD,
         int* __restrict__ wet, int* __restrict__ nwet, const int* __restrict__ ulist,
         const int* __restrict__ ucount) {
  if (!LIST) {
    d_update<PRED, EK>(g, E, Q, Qh, Qprev, Fx, Fy, Fz, fact, clk, err, pB, pA, nbB, pD, wet, nwet,
                       (long long)blockIdx.x * blockDim.x + threadIdx.x);
    return;
  }
  const int n = *ucount;
  for (int b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
    const int idx = b + threadIdx.x;
    d_update<PRED, EK>(g, E, Q, Qh, Qprev, Fx, Fy, Fz, fact, clk, err, pB, pA, nbB, pD, wet, nwet,
                       idx < n ? ulist[idx] : g.N);
  }
}

// ------------------------------------------------------------- ghosts
// Fluid::correctImagCells (HALF: Q and Qh) and correctImagCellsFull (FULL:
// Q, pi, Pi), src/fld.cpp:211-382, as a gather from the per-dimension source
// maps, over the cells that are copied into only (78 of 520 thousand at
// 101x101x51); copies into a ghost zero the row when Q_t < 0 (Cell::setQ /
// setQh).  An ideal step, where nothing lies between the two, does both at
// once.  HALF in a viscous step (wet not null) also settles the copied
// cells for the viscous stages; FULL, the step's last kernel, advances the
// clock (which it does not read).
struct Shell {  // the copied-into cells: the z planes, then rows, then ends
  int gx, gy, gz, iy, iz;
  long long a, b, n;
};
__host__ __device__ inline Shell ghost_shell(const Geo& g) {
  Shell s;
  s.gx = g.nx < 4 ? g.nx : 4;
  s.gy = g.ny < 4 ? g.ny : 4;
  s.gz = g.nz < 4 ? g.nz : 4;
  s.iy = g.ny - s.gy;
  s.iz = g.nz - s.gz;
  s.a = (long long)s.gz * g.nx * g.ny;
  s.b = s.a + (long long)s.iz * s.gy * g.nx;
  s.n = s.b + (long long)s.iz * s.iy * s.gx;
  return s;
}
// Row i becomes row s (read before), or zeros where its Q_t is negative.  A
// cell that is its own source keeps its row, and may be read by other threads
// meanwhile (sides of 4 or fewer, where the sources are copied into too):
// zeroed, it stores Q_t last.  So a reader that finds a negative Q_t stores
// zeros whatever else it found, one that finds another Q_t but 0 has a row
// that nobody writes, and one that finds 0 beside anything but zeros reads
// again, behind a fence, what was stored before that 0.
__device__ __forceinline__ void ghost_read(const double* F, long long N, long long s, double q[7]) {
  q[0] = *(const volatile double*)(F + s);
#pragma unroll
  for (int k = 1; k < 7; k++) q[k] = F[k * N + s];
}
__device__ __forceinline__ void ghost_store(double* F, long long N, long long i, long long s,
                                            double q[7]) {
  const bool neg = q[0] < 0.;
  if (s == i) {
    if (!neg) return;
#pragma unroll
    for (int k = 1; k < 7; k++) F[k * N + i] = 0.;
    __threadfence();
    *(volatile double*)(F + i) = 0.;
    return;
  }
  bool rest = false;
#pragma unroll
  for (int k = 1; k < 7; k++) rest |= q[k] != 0.;
  if (q[0] == 0. && rest) {
    __threadfence();
#pragma unroll
    for (int k = 1; k < 7; k++) q[k] = *(const volatile double*)(F + k * N + s);
  }
#pragma unroll
  for (int k = 0; k < 7; k++) F[k * N + i] = neg ? 0. : q[k];
}
__device__ __forceinline__ int ghost_index(int k, int n) { return k < 2 || n <= 4 ? k : n - 4 + k; }

template <bool HALF, bool FULL>
__device__ __forceinline__ void d_ghost(const Geo& g, const int* __restrict__ src,
                                        const Fields& f, int* wet, double* tick, long long blk) {
  const long long t = blk * blockDim.x + threadIdx.x;
  if (FULL && tick && t == 0) tick[0] += tick[1];  // tau += dt (src/hdo.cpp:1095)
  const Shell sh = ghost_shell(g);
  if (t >= sh.n) return;
  int ix, iy, iz;
  if (t < sh.a) {
    const unsigned r = (unsigned)t, p = (unsigned)(g.nx * g.ny), k = r / p, q = r - k * p;
    iy = (int)(q / (unsigned)g.nx);
    ix = (int)(q - iy * (unsigned)g.nx);
    iz = ghost_index((int)k, g.nz);
  } else if (t < sh.b) {
    const unsigned r = (unsigned)(t - sh.a), p = (unsigned)(sh.gy * g.nx), k = r / p, q = r - k * p;
    const unsigned w = q / (unsigned)g.nx;
    ix = (int)(q - w * (unsigned)g.nx);
    iy = ghost_index((int)w, g.ny);
    iz = 2 + (int)k;
  } else {
    const unsigned r = (unsigned)(t - sh.b), p = (unsigned)(sh.iy * sh.gx), k = r / p, q = r - k * p;
    const unsigned w = q / (unsigned)sh.gx;
    ix = ghost_index((int)(q - w * (unsigned)sh.gx), g.nx);
    iy = 2 + (int)w;
    iz = 2 + (int)k;
  }
  const int* sx = src;
  const int* sy = src + g.nx;
  const int* sz = src + g.nx + g.ny;
  const long long N = g.N;
  const long long i = (long long)ix + (long long)g.nx * (iy + (long long)g.ny * iz);
  const long long s = (long long)sx[ix] + (long long)g.nx * (sy[iy] + (long long)g.ny * sz[iz]);
  double q[7], h[7], p[11];  // the loads of all rows together
  ghost_read(f.Q, N, s, q);
  if (HALF) ghost_read(f.Qh, N, s, h);
  if (FULL) {
#pragma unroll
    for (int k = 0; k < 10; k++) p[k] = f.pi[k * N + s];
    p[10] = f.Pi[s];
  }
  ghost_store(f.Q, N, i, s, q);
  if (HALF) {
    ghost_store(f.Qh, N, i, s, h);
    if (wet) {
      if (!(h[0] <= 0.))
        append(wet, f.fcount + 6, (int)i);
      else
        empty_prims(f.pA, f.pD, N, i);
    }
  }
  if (FULL && s != i) {
#pragma unroll
    for (int k = 0; k < 10; k++) f.pi[k * N + i] = p[k];
    f.Pi[i] = p[10];
  }
}
template <bool HALF, bool FULL>
__global__ void k_ghost(Geo g, Fields f, int* wet, double* tick) {
  d_ghost<HALF, FULL>(g, f.gsrc, f, wet, tick, blockIdx.x);
}


// ------------------------------------------------ viscous cell prims
// Per-cell inputs of the viscous stages over the list that the corrector and
// the ghost copy made of the cells with Qh_t > 0 (in grid order the root finds
// ran on 17 of a warp's 32 lanes at 101x101x51 with 80 % vacuum).  Two threads
// per cell, in the two halves of a block: the first takes A, D and the
// thermodynamics, the second B and C.  A cell is a chain of root finds, which
// the few cells of a coarse grid do not hide (us per step with one thread and
// with two: 47x61x23 24.9 and 20.0, 101x101x51 32.6 and 33.5, 201x201x101 90.7
// and 90.6; 101x101x51 with charge 35.4 and 37.8):
//  A  = con2prim(Qh / (tau - dt/2))  (getPrimVarHCenter in ISformal, NSquant,
//                                     visc_flux, visc_source_step),
//  D  = con2prim(Qh / tau), e and u  (the six NSquant neighbour velocities),
//  thermodynamics at A: T, muB, p, s, eta/s, zeta/s, tau_pi, tau_Pi, 9/70/p
//                                    (src/hdo.cpp:427-432, 727-749),
//  B  = con2prim(Qprev / (tau - dt)), C = con2prim(Q / tau) as four-velocities
//                                    (NSquant's time derivative,
//                                     src/hdo.cpp:419-446), only where
//                                     NSquant reaches them (matter, no vacuum
//                                     neighbour).
__device__ __forceinline__ double maxM_at(const Geo& g, const double* __restrict__ m, int ix,
                                          int iy, int iz);

__device__ __forceinline__ Prim loadA(const double* __restrict__ pA, long long N, long long i) {
  Prim a;
  a.e = pA[i];
  a.p = pA[N + i];
  a.nb = pA[2 * N + i];
  a.nq = pA[3 * N + i];
  a.ns = pA[4 * N + i];
  a.vx = pA[5 * N + i];
  a.vy = pA[6 * N + i];
  a.vz = pA[7 * N + i];
  return a;
}

// VORT: also T of the states that the vorticity's rows divide by (TD at D,
// TB at B, TC at C), so that it solves nothing again.
template <int EK, bool VORT>
__device__ __forceinline__ void d_visc_prims(const Geo& g, const EosDev& E, const TrDev& tr,
                                             const double* __restrict__ Q,
                                             const double* __restrict__ Qprev,
                                             const double* __restrict__ Qh,
                                             const double* __restrict__ m, double* __restrict__ pA,
                                             double* __restrict__ pD, double* __restrict__ pTh,
                                             double* __restrict__ pBC,
                                             const double* __restrict__ clk,
                                             int* __restrict__ active,
                                             int* __restrict__ nactive, double* __restrict__ TD,
                                             double* __restrict__ TB, double* __restrict__ TC,
                                             long long i, bool in, bool second) {
  const double dt = clk[1], tau = clk[0] + dt;  // tau_{n+1} (src/hdo.cpp:1095)
  const long long N = g.N;
  double q[7], qh[7];
  const double tA = tau - dt / 2.;
  Prim a{0., 0., 0., 0., 0., 0., 0., 0.};
  // the first half solves A, the second looks for vacuum beside the cell
  __shared__ double ea[64];
  __shared__ bool beside[64];
  const int half = blockDim.x >> 1, slot = second ? threadIdx.x - half : threadIdx.x;
  bool vac = false;
  if (in) {
    int gx, gy, gz;
    coords(g, i, gx, gy, gz);
    if (second) {
      vac = maxM_at(g, m, gx + 1, gy, gz) <= 0.9 || maxM_at(g, m, gx, gy + 1, gz) <= 0.9 ||
            maxM_at(g, m, gx - 1, gy, gz) <= 0.9 || maxM_at(g, m, gx, gy - 1, gz) <= 0.9 ||
            maxM_at(g, m, gx + 1, gy + 1, gz) <= 0.9 ||
            maxM_at(g, m, gx + 1, gy - 1, gz) <= 0.9 ||
            maxM_at(g, m, gx - 1, gy + 1, gz) <= 0.9 || maxM_at(g, m, gx - 1, gy - 1, gz) <= 0.9;
      beside[slot] = vac;
    } else {
      // A is the corrector's con2prim (k_update<false> stored it in pA) when
      // its divisor tau_n + dt/2 equals tA bit for bit and the ghost copy has
      // not changed this cell's Qh since
      if (tA == clk[0] + 0.5 * dt && !is_ghost(g, gx, gy, gz)) {
        a = loadA(pA, N, i);
      } else {
#pragma unroll
        for (int k = 0; k < 7; k++) qh[k] = Qh[k * N + i];
        q_over(qh, tA, q);
        transform_pv<EK>(E, q, a, c2p_guess(E, i));
        pA[0 * N + i] = a.e;
        pA[1 * N + i] = a.p;
        pA[2 * N + i] = a.nb;
        pA[3 * N + i] = a.nq;
        pA[4 * N + i] = a.ns;
        pA[5 * N + i] = a.vx;
        pA[6 * N + i] = a.vy;
        pA[7 * N + i] = a.vz;
      }
      ea[slot] = a.e;
    }
  }
  __syncthreads();
  if (in && second) a.e = ea[slot];
  if (in && !second) vac = beside[slot];
  {
    // the list of cells with matter, for the relaxation and the advection
    // (the complement of a cell next to vacuum, which NSquant leaves alone);
    // every cell's result depends on that cell alone, not on the order
    append_block(active, nactive, vac ? ~(int)i : (int)i, in && !second && !(a.e <= 0.));
  }
  if (!in || (second && (a.e <= 0. || vac))) return;
  // D from Qh, or C from Q (only where NSquant reaches it), both at tau
  {
    const double* src = second ? Q : Qh;
    double qs[7];
#pragma unroll
    for (int k = 0; k < 7; k++) qs[k] = src[k * N + i];
    q_over(qs, tau, q);
    Prim P;
    transform_pv<EK>(E, q, P, c2p_guess(E, i));
    const double ut = 1.0 / sqrt(1.0 - P.vx * P.vx - P.vy * P.vy - P.vz * P.vz);
    double* o = second ? pBC + 5 * N + i : pD + N + i;
    o[0] = ut;
    o[N] = ut * P.vx;
    o[2 * N] = ut * P.vy;
    o[3 * N] = ut * P.vz;
    if (!second) pD[i] = P.e;
    if (VORT) {
      double T, mub, p;
      eos_eval<EK>(E, P.e, P.nb, T, mub, p);
      (second ? TC : TD)[i] = T;
    }
  }
  if (!second) {
    if (a.e <= 0.) return;
    double T, mub, mus, p;
    eos_eval<EK>(E, a.e, a.nb, T, mub, mus, p);
    // EoS::s at the same point (eos_s, muq = 0) from this lookup
    const double s = T > 0.0 ? ddivp(a.e + p - mub * a.nb - 0. * a.nq - mus * a.ns, T) : 0.;
    const double etaS = tr_etaS(tr, a.e, a.nb, T, mub, s, p);
    const double zetaS = tr_zetaS(tr, a.e, T, s, p);
    double taupi, tauPi;
    tr_getTau_from(a.e, T, s, p, etaS, zetaS, taupi, tauPi);
    pTh[0 * N + i] = T;
    pTh[1 * N + i] = mub;
    pTh[2 * N + i] = p;
    pTh[3 * N + i] = s;
    pTh[4 * N + i] = etaS;
    pTh[5 * N + i] = zetaS;
    pTh[6 * N + i] = taupi;
    pTh[7 * N + i] = tauPi;
    pTh[8 * N + i] = 9. / 70. / p;  // eos_p at the same point is this p
    return;
  }
  // B is the predictor's con2prim when the divisors agree bit for bit
  // (k_update<true> stored it in pBC); otherwise computed here
  double eB, nbB;
  if ((clk[0] + dt) - dt == clk[0]) {
    if (!VORT) return;
    eB = pBC[4 * N + i];
    nbB = TB[i];  // held until here for this
  } else {
    double qs[7];
#pragma unroll
    for (int k = 0; k < 7; k++) qs[k] = Qprev[k * N + i];
    q_over(qs, tau - dt, q);
    Prim P;
    transform_pv<EK>(E, q, P, c2p_guess(E, i));
    const double ut = 1.0 / sqrt(1.0 - P.vx * P.vx - P.vy * P.vy - P.vz * P.vz);
    pBC[0 * N + i] = ut;
    pBC[1 * N + i] = ut * P.vx;
    pBC[2 * N + i] = ut * P.vy;
    pBC[3 * N + i] = ut * P.vz;
    pBC[4 * N + i] = P.e;
    eB = P.e;
    nbB = P.nb;
  }
  if (VORT) {
    double T, mub, p;
    eos_eval<EK>(E, eB, nbB, T, mub, p);
    TB[i] = T;
  }
}
template <int EK, bool VORT>
__global__ void __launch_bounds__(128, kPrimsMinBlocks) k_visc_prims(Geo g, EosDev E, TrDev tr,
                                                    const double* __restrict__ Q,
                                                    const double* __restrict__ Qprev,
                                                    const double* __restrict__ Qh,
                                                    const double* __restrict__ m,
                                                    double* __restrict__ pA,
                                                    double* __restrict__ pD,
                                                    double* __restrict__ pTh,
                                                    double* __restrict__ pBC, const double* __restrict__ clk,
                                                    const int* __restrict__ wet,
                                                    const int* __restrict__ nwet,
                                                    int* __restrict__ active,
                                                    int* __restrict__ nactive,
                                                    double* __restrict__ TD,
                                                    double* __restrict__ TB,
                                                    double* __restrict__ TC) {
  const int n = *nwet, half = blockDim.x >> 1;
  const bool second = (int)threadIdx.x >= half;
  for (int b = blockIdx.x * half; b < n; b += gridDim.x * half) {
    const int idx = b + (second ? threadIdx.x - half : threadIdx.x);
    d_visc_prims<EK, VORT>(g, E, tr, Q, Qprev, Qh, m, pA, pD, pTh, pBC, clk, active, nactive, TD, TB,
                           TC, idx < n ? wet[idx] : 0, idx < n, second);
  }
}


__device__ __forceinline__ double maxM_at(const Geo& g, const double* __restrict__ m, int ix,
                                          int iy, int iz) {
  return maxM(m, g.N, cidx(g, ix, iy, iz));
}

// ------------------------------------------------ ISformal, loop #1
// Hydro::ISformal loop 1 with Hydro::NSquant (src/hdo.cpp:381-652,
// 690-864): Navier-Stokes shear/bulk from the velocity gradients, then the
// two-stage Israel-Stewart relaxation with Christoffel and cross terms.
// Writes pi0/piH0/Pi0/PiH0 and the first flux contribution
// (+(tau-dt) * delta Q_n) of the cells with matter; the zeros of the empty
// ones (src/hdo.cpp:697-708) are left to their readers, which see e <= 0
// (writing them, 208 bytes a cell, took 25 us of a 988 us step at 101x101x51
// with 80 % vacuum).  One thread per cell, every index a compile-time
// constant; the con2prims and the thermodynamics come precomputed from
// k_visc_prims.  Three 128-thread blocks per SM (168
// registers): with four (128 registers, 450 bytes of spills) 112 instead of
// 89 us a step at 101x101x51 and 298 instead of 259 at 201x201x101, with two
// (no spills) 97 and 301.
constexpr int kRelaxMinBlocks = 3;

constexpr int kRelaxBlock = 128;
// shared-memory rows of k_is_relax's relaxation loops: pi, sigma, u, h0, f0,
// and phi7 h0^{kl} - tau_pipi sigma^{kl} of the second loop (dynamic shared
// memory: 55 KB per block)
constexpr int kSmPI = 0, kSmSIG = 10, kSmU = 20, kSmH = 24, kSmF = 34, kSmY = 44, kSmRows = 54;
constexpr size_t kRelaxSmem = sizeof(double) * kSmRows * kRelaxBlock;

// The relaxation of one cell with every division checked for its range
// (div_batch, ddiv): the form for cells that relax_fast gives back.
__device__ __noinline__ void relax_general(
    const Geo& g, const double* __restrict__ pA, const double* __restrict__ pD,
    const double* __restrict__ pTh, const double* __restrict__ pBC, const double* __restrict__ pi,
    const double* __restrict__ Pi, double* __restrict__ pi0, double* __restrict__ piH0,
    double* __restrict__ Pi0, double* __restrict__ PiH0, double* __restrict__ flux,
    const double* __restrict__ clk, unsigned* err, long long i, bool vac) {
  const double dt = clk[1], tau = clk[0] + dt;  // tau_{n+1} (src/hdo.cpp:1095)
  const long long N = g.N;
  const double e = pA[i];
  int ix, iy, iz;
  coords(g, i, ix, iy, iz);
  const double gmumu[4] = {1., -1., -1., -1.};
  double cpi[10];
#pragma unroll
  for (int k = 0; k < 10; k++) cpi[k] = pi[k * N + i];
  const double cPi = Pi[i];
#define PI(a, b) cpi[index44(a, b)]
  const double vx = pA[5 * N + i], vy = pA[6 * N + i], vz = pA[7 * N + i];
  const double gamma = 1.0 / sqrt(1.0 - vx * vx - vy * vy - vz * vz);
  // the ~600 divisions by gamma go through crm::mk_div (bit-identical to
  // the divide) in batches whose numerators are all in its range
  const double rg = 1.0 / gamma;
  const bool gfast = crm::mk_den_ok(gamma);
  double u[4];
  u[0] = gamma;
  u[1] = u[0] * vx;
  u[2] = u[0] * vy;
  u[3] = u[0] * vz;
  {
    double f[4];
#pragma unroll
    for (int k = 0; k < 4; k++) f[k] = (tau - dt) * (PI(0, k) + cPi * u[0] * u[k]);
    f[0] += -(tau - dt) * cPi;
#pragma unroll
    for (int k = 0; k < 4; k++) flux[k * N + i] = 0. + f[k];
  }
  const double s = pTh[3 * N + i];
  const double etaS = pTh[4 * N + i];
  const double zetaS = pTh[5 * N + i];

  // ------------------------------------------------------ NSquant
  double piNS[10], PiNS, du;
  double dmu[4][4];
  if (vac) {
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) dmu[a][b] = 0.;
#pragma unroll
    for (int k = 0; k < 10; k++) piNS[k] = 0.;
    PiNS = du = 0.;
  } else {
    const double VMIN = 1e-2;
    const double UDIFF = 3.0;
    const double e0 = pBC[4 * N + i], e1 = e;
    double ut0 = pBC[0 * N + i], ux0 = pBC[1 * N + i], uy0 = pBC[2 * N + i], uz0 = pBC[3 * N + i];
    double ut1 = pBC[5 * N + i], ux1 = pBC[6 * N + i], uy1 = pBC[7 * N + i], uz1 = pBC[8 * N + i];
    const double* uuu = u;
    dmu[0][0] = ddivp(ddivp((ut1 * ut1 - ut0 * ut0) / 2., uuu[0]), dt);
    dmu[0][1] = ddivp(ddiv((ux1 * ux1 - ux0 * ux0) / 2., uuu[1]), dt);
    dmu[0][2] = ddivp(ddiv((uy1 * uy1 - uy0 * uy0) / 2., uuu[2]), dt);
    dmu[0][3] = ddivp(ddiv((uz1 * uz1 - uz0 * uz0) / 2., uuu[3]), dt);
    if (fabs(ddivp(0.5 * (ut1 + ut0), ut1)) > UDIFF) dmu[0][0] = ddivp(ut1 - ut0, dt);
    if (fabs(uuu[1]) < VMIN || fabs(ddiv(0.5 * (ux1 + ux0), ux1)) > UDIFF)
      dmu[0][1] = ddivp(ux1 - ux0, dt);
    if (fabs(uuu[2]) < VMIN || fabs(ddiv(0.5 * (uy1 + uy0), uy1)) > UDIFF)
      dmu[0][2] = ddivp(uy1 - uy0, dt);
    if (fabs(uuu[3]) < VMIN || fabs(ddiv(0.5 * (uz1 + uz0), uz1)) > UDIFF)
      dmu[0][3] = ddivp(uz1 - uz0, dt);
    if (e1 <= 0. || e0 <= 0.) dmu[0][0] = dmu[0][1] = dmu[0][2] = dmu[0][3] = 0.;
#pragma unroll
    for (int d = 1; d <= 3; d++) {
      long long ip, im;
      if (d == 1) {
        ip = cidx(g, ix + 1, iy, iz);
        im = cidx(g, ix - 1, iy, iz);
      } else if (d == 2) {
        ip = cidx(g, ix, iy + 1, iz);
        im = cidx(g, ix, iy - 1, iz);
      } else {
        ip = cidx(g, ix, iy, iz + 1);
        im = cidx(g, ix, iy, iz - 1);
      }
      const double ep = pD[ip], em = pD[im];
      if (ep > 0. && em > 0.) {
        ut0 = pD[N + im], ux0 = pD[2 * N + im], uy0 = pD[3 * N + im], uz0 = pD[4 * N + im];
        ut1 = pD[N + ip], ux1 = pD[2 * N + ip], uy1 = pD[3 * N + ip], uz1 = pD[4 * N + ip];
        if (d < 3) {
          const double h = d == 1 ? g.dx : g.dy;
          dmu[d][0] = ddivp(ddivp(0.25 * (ut1 * ut1 - ut0 * ut0), uuu[0]), h);
          dmu[d][1] = ddivp(ddiv(0.25 * (ux1 * ux1 - ux0 * ux0), uuu[1]), h);
          dmu[d][2] = ddivp(ddiv(0.25 * (uy1 * uy1 - uy0 * uy0), uuu[2]), h);
          dmu[d][3] = ddivp(ddiv(0.25 * (uz1 * uz1 - uz0 * uz0), uuu[3]), h);
          if (fabs(ddivp(0.5 * (ut1 + ut0), uuu[0])) > UDIFF) dmu[d][0] = ddivp(0.5 * (ut1 - ut0), h);
          if (fabs(uuu[1]) < VMIN || fabs(ddiv(0.5 * (ux1 + ux0), uuu[1])) > UDIFF)
            dmu[d][1] = ddivp(0.5 * (ux1 - ux0), h);
          if (fabs(uuu[2]) < VMIN || fabs(ddiv(0.5 * (uy1 + uy0), uuu[2])) > UDIFF)
            dmu[d][2] = ddivp(0.5 * (uy1 - uy0), h);
          if (fabs(uuu[3]) < VMIN || fabs(ddiv(0.5 * (uz1 + uz0), uuu[3])) > UDIFF)
            dmu[d][3] = ddivp(0.5 * (uz1 - uz0), h);
        } else {
          const double dz = g.dz, th = tau + 0.5 * dt;
          dmu[3][0] = ddivp(ddivp(ddivp(0.25 * (ut1 * ut1 - ut0 * ut0), uuu[0]), dz), th);
          dmu[3][1] = ddivp(ddivp(ddiv(0.25 * (ux1 * ux1 - ux0 * ux0), uuu[1]), dz), th);
          dmu[3][2] = ddivp(ddivp(ddiv(0.25 * (uy1 * uy1 - uy0 * uy0), uuu[2]), dz), th);
          dmu[3][3] = ddivp(ddivp(ddiv(0.25 * (uz1 * uz1 - uz0 * uz0), uuu[3]), dz), th);
          if (fabs(ddivp(0.5 * (ut1 + ut0), uuu[0])) > UDIFF)
            dmu[3][0] = ddivp(ddivp(0.5 * (ut1 - ut0), dz), th);
          if (fabs(uuu[1]) < VMIN || fabs(ddiv(0.5 * (ux1 + ux0), uuu[1])) > UDIFF)
            dmu[3][1] = ddivp(ddivp(0.5 * (ux1 - ux0), dz), th);
          if (fabs(uuu[2]) < VMIN || fabs(ddiv(0.5 * (uy1 + uy0), uuu[2])) > UDIFF)
            dmu[3][2] = ddivp(ddivp(0.5 * (uy1 - uy0), dz), th);
          if (fabs(uuu[3]) < VMIN || fabs(ddiv(0.5 * (uz1 + uz0), uuu[3])) > UDIFF)
            dmu[3][3] = ddivp(ddivp(0.5 * (uz1 - uz0), dz), th);
        }
      } else {
        dmu[d][0] = dmu[d][1] = dmu[d][2] = dmu[d][3] = 0.;
      }
    }
    dmu[3][0] += ddivp(uuu[3], tau - 0.5 * dt);
    dmu[3][3] += ddivp(uuu[0], tau - 0.5 * dt);
    const double gdiag[4] = {1., -1., -1., -1.};
    const double r5068 = 1.0 / 5.068;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b <= a; b++) {
        double n[16];  // the (k, l) terms, divided by 5.068 as a batch
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int l = 0; l < 4; l++) {
            double Z = 0.0;
            const double gak = (a == k) ? gdiag[a] : 0.;
            const double gbk = (b == k) ? gdiag[b] : 0.;
            const double gab = (a == b) ? gdiag[a] : 0.;
            if (b == l) Z += 0.5 * (gak - uuu[a] * uuu[k]);
            if (a == l) Z += 0.5 * (gbk - uuu[b] * uuu[k]);
            if (k == l) Z -= ddivp(gab - uuu[a] * uuu[b], 3.0);
            n[4 * k + l] = Z * dmu[k][l] * 2.0 * etaS * s;
          }
        div_batch<16>(n, 5.068, r5068, true);
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 16; j++) acc += n[j];
        piNS[index44(a, b)] = acc;
      }
    PiNS = ddivp(-zetaS * s * (dmu[0][0] + dmu[1][1] + dmu[2][2] + dmu[3][3]), 5.068);
    du = dmu[0][0] + dmu[1][1] + dmu[2][2] + dmu[3][3];
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 10; k++) bad |= isinf(piNS[k]) || isnan(piNS[k]);
    if (bad) atomicOr(err, (unsigned)ERR_NSQUANT_NAN);
  }
#define PINS(a, b) piNS[index44(a, b)]

  // ------------------------------------------------ ISformal loop 1 body
  const double eta = etaS * s;
  double sig[10];
#pragma unroll
  for (int k = 0; k < 10; k++) sig[k] = 0.5 * piNS[k];
  div_batch<10, true>(sig, eta, 1.0 / eta, crm::mk_den_ok(eta));  // ddiv's quotients
#pragma unroll
  for (int k = 0; k < 10; k++) {
    sig[k] = sig[k] * 5.068;
    if (eta <= 0.0) sig[k] = 0.0;
  }
#define SIG(a, b) sig[index44(a, b)]
  const double taupi = pTh[6 * N + i], tauPi = pTh[7 * N + i];
  double deltapipi = 4. / 3., taupipi = 10. / 7., lambdapiPi = 6. / 5.;
  double phi7 = pTh[8 * N + i];
  if (isinf(phi7)) phi7 = 0.0;
  phi7 = ddiv(phi7, taupi);
  if (taupi < 0.5 * dt) deltapipi = taupipi = lambdapiPi = phi7 = 0.0;
  double delPiPi = 2. / 3.;
  double lamPipi = 8. / 5. * (1. / 3. - 1. / 3.);
  if (tauPi < 0.5 * dt) delPiPi = lamPipi = 0.0;
  double Delta[10];
  double h0[10];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b <= a; b++) {
      const int k = index44(a, b);
      Delta[k] = -u[a] * u[b];
      if (a == b) Delta[k] += gmumu[a];
    }
  if (taupi > 0.5 * dt) {
    double n[10];
#pragma unroll
    for (int k = 0; k < 10; k++) n[k] = (cpi[k] - piNS[k]) * dt / 2.0;
    div_batch<10>(n, gamma, rg, gfast);
    div_batch<10>(n, taupi, 1.0 / taupi, crm::mk_den_ok(taupi));
#pragma unroll
    for (int k = 0; k < 10; k++) h0[k] = cpi[k] - n[k];
  } else {
#pragma unroll
    for (int k = 0; k < 10; k++) h0[k] = piNS[k];
  }
  double H0;
  if (tauPi > 0.5 * dt)
    H0 = cPi - ddivp(ddivp((cPi - PiNS) * dt / 2.0, gamma), tauPi);
  else
    H0 = PiNS;
  double tau1 = tau - dt * 0.75;
  h0[index44(0, 0)] += ddivp(-2. * vz * PI(0, 3), tau1) * dt / 2.;
  h0[index44(3, 3)] += -(ddivp(2. * vz, tau1) * PI(0, 3)) * dt / 2.;
  h0[index44(3, 0)] += -(ddivp(vz, tau1) * PI(0, 0) + ddivp(vz, tau1) * PI(3, 3)) * dt / 2.;
  h0[index44(1, 0)] += ddivp(-vz, tau1) * PI(1, 3) * dt / 2.;
  h0[index44(2, 0)] += ddivp(-vz, tau1) * PI(2, 3) * dt / 2.;
  h0[index44(3, 1)] += -(ddivp(vz, tau1) * PI(0, 1)) * dt / 2.;
  h0[index44(3, 2)] += -(ddivp(vz, tau1) * PI(0, 2)) * dt / 2.;
  // The relaxation sums over (a, b) run as a loop with (a, b) known only at
  // run time, so that its body (36 divisions by gamma) is fetched once per
  // warp instead of ten times unrolled: the unrolled kernel's instruction
  // stream outgrew the instruction caches.  Operands indexed by a or b come
  // from shared memory ([component][thread]); the arithmetic of every term
  // is the reference's, in its order.
  extern __shared__ double relax_smem[];
  double(*sm)[kRelaxBlock] = reinterpret_cast<double(*)[kRelaxBlock]>(relax_smem);
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    sm[kSmPI + k][t] = cpi[k];
    sm[kSmSIG + k][t] = sig[k];
    sm[kSmH + k][t] = h0[k];
  }
#pragma unroll
  for (int k = 0; k < 4; k++) sm[kSmU + k][t] = u[k];
  // phi7 pi^{kl} - tau_pipi sigma^{kl}, the same for every (a, b): in the
  // rows loop 2 uses for f0 later
#pragma unroll
  for (int k = 0; k < 10; k++) sm[kSmF + k][t] = phi7 * cpi[k] - taupipi * sig[k];
#pragma unroll 1
  for (int ab = 0; ab < 10; ab++) {
    const int a = ab >= 6 ? 3 : ab >= 3 ? 2 : ab >= 1 ? 1 : 0;
    const int b = ab - a * (a + 1) / 2;
    const double ua = sm[kSmU + a][t], ub = sm[kSmU + b][t];
    double dab = -ua * ub;  // Delta[index44(a, b)]
    if (a == b) dab += a == 0 ? 1. : -1.;
    double acc = sm[kSmH + ab][t];
    acc += ddivp(-deltapipi * sm[kSmPI + ab][t] * du + lambdapiPi * cPi * sm[kSmSIG + ab][t],
                 gamma) *
           0.5 * dt;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double gk = gmumu[k];
      const double pak = sm[kSmPI + index44(a, k)][t], pbk = sm[kSmPI + index44(b, k)][t];
      const double sak = sm[kSmSIG + index44(a, k)][t], sbk = sm[kSmSIG + index44(b, k)][t];
      double n[9];  // numerators of the k term and of its four (x, y) l terms
      n[0] = phi7 * pak * pbk * gk - taupipi * 0.5 * (pak * sbk * gk + pbk * sak * gk);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        n[1 + 2 * l] = (-pak * ub - pbk * ua) * u[l] * dmu[l][k] * gk;
        n[2 + 2 * l] = 1. / 3. * dab * PI(k, l) * sm[kSmF + index44(k, l)][t] * gk * gmumu[l];
      }
      div_batch<9>(n, gamma, rg, gfast);
      acc += n[0] * 0.5 * dt;
#pragma unroll
      for (int l = 0; l < 4; l++) acc += n[1 + 2 * l] * 0.5 * dt - n[2 + 2 * l] * 0.5 * dt;
    }
    sm[kSmH + ab][t] = acc;
  }
#pragma unroll
  for (int k = 0; k < 10; k++) h0[k] = sm[kSmH + k][t];
  {
    double n[16];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int l = 0; l < 4; l++) n[4 * k + l] = lamPipi * PI(k, l) * SIG(k, l) * gmumu[k] * gmumu[l];
    div_batch<16>(n, gamma, rg, gfast);
#pragma unroll
    for (int j = 0; j < 16; j++) H0 += n[j] * 0.5 * dt;
  }
  H0 += ddivp(-delPiPi * cPi * du, gamma) * 0.5 * dt;
#define H(a, b) h0[index44(a, b)]
  double f0[10];
  if (taupi > 0.5 * dt) {
    double n[10];
#pragma unroll
    for (int k = 0; k < 10; k++) n[k] = (h0[k] - piNS[k]) * dt;
    div_batch<10>(n, gamma, rg, gfast);
    div_batch<10>(n, taupi, 1.0 / taupi, crm::mk_den_ok(taupi));
#pragma unroll
    for (int k = 0; k < 10; k++) f0[k] = cpi[k] - n[k];
  } else {
#pragma unroll
    for (int k = 0; k < 10; k++) f0[k] = piNS[k];
  }
  double F0;
  if (tauPi > 0.5 * dt)
    F0 = cPi - ddivp(ddivp((H0 - PiNS) * dt, gamma), tauPi);
  else
    F0 = PiNS;
  tau1 = tau - dt * 0.5;
  f0[index44(0, 0)] += ddivp(-2. * vz, tau1) * H(0, 3) * dt;
  f0[index44(3, 3)] += -(ddivp(2. * vz, tau1) * H(0, 3)) * dt;
  f0[index44(3, 0)] += -(ddivp(vz, tau1) * H(0, 0) + ddivp(vz, tau1) * H(3, 3)) * dt;
  f0[index44(1, 0)] += ddivp(-vz, tau1) * H(1, 3) * dt;
  f0[index44(2, 0)] += ddivp(-vz, tau1) * H(2, 3) * dt;
  f0[index44(3, 1)] += -(ddivp(vz, tau1) * H(0, 1)) * dt;
  f0[index44(3, 2)] += -(ddivp(vz, tau1) * H(0, 2)) * dt;
#pragma unroll
  for (int k = 0; k < 10; k++) sm[kSmF + k][t] = f0[k];
#pragma unroll
  for (int k = 0; k < 10; k++) sm[kSmY + k][t] = phi7 * h0[k] - taupipi * sig[k];
#pragma unroll 1
  for (int ab = 0; ab < 10; ab++) {
    const int a = ab >= 6 ? 3 : ab >= 3 ? 2 : ab >= 1 ? 1 : 0;
    const int b = ab - a * (a + 1) / 2;
    const double ua = sm[kSmU + a][t], ub = sm[kSmU + b][t];
    double dab = -ua * ub;  // Delta[index44(a, b)]
    if (a == b) dab += a == 0 ? 1. : -1.;
    double acc = sm[kSmF + ab][t];
    acc += ddivp(-deltapipi * sm[kSmH + ab][t] * du + lambdapiPi * H0 * sm[kSmSIG + ab][t],
                 gamma) *
           dt;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double gk = gmumu[k];
      const double pak = sm[kSmPI + index44(a, k)][t];
      const double hak = sm[kSmH + index44(a, k)][t], hbk = sm[kSmH + index44(b, k)][t];
      const double sak = sm[kSmSIG + index44(a, k)][t], sbk = sm[kSmSIG + index44(b, k)][t];
      double n[5];  // numerators of the k term and of its four l terms
      n[0] = phi7 * pak * hbk * gk - taupipi * 0.5 * (hak * sbk * gk + hbk * sak * gk);
#pragma unroll
      for (int l = 0; l < 4; l++)
        n[1 + l] = (-hak * ub - hbk * ua) * u[l] * dmu[l][k] * gk -
                   1. / 3. * dab * H(k, l) * sm[kSmY + index44(k, l)][t] * gk * gmumu[l];
      div_batch<5>(n, gamma, rg, gfast);
      acc += n[0] * dt;
#pragma unroll
      for (int l = 0; l < 4; l++) acc += n[1 + l] * dt;
    }
    sm[kSmF + ab][t] = acc;
  }
#pragma unroll
  for (int k = 0; k < 10; k++) f0[k] = sm[kSmF + k][t];
  {
    double n[16];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int l = 0; l < 4; l++) n[4 * k + l] = lamPipi * H(k, l) * SIG(k, l) * gmumu[k] * gmumu[l];
    div_batch<16>(n, gamma, rg, gfast);
#pragma unroll
    for (int j = 0; j < 16; j++) F0 += n[j] * dt;
  }
  F0 += ddivp(-delPiPi * H0 * du, gamma) * dt;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    piH0[k * N + i] = h0[k];
    pi0[k * N + i] = f0[k];
  }
  PiH0[i] = H0;
  Pi0[i] = F0;
#undef PI
#undef PINS
#undef SIG
#undef H
}

// y / b by crm::mk_div's three operations for operands known to be in its
// range (a zero y may lose its sign)
__device__ __forceinline__ double mk_raw(double y, double b, double r) {
  const double q0 = y * r;
  return fma(fma(-q0, b, y), r, q0);
}
// x = +-0 or 2^-B <= |x| < 2^(B+1): integer operations on the exponent
template <int B>
__device__ __forceinline__ bool exp_ok(double x) {
  const unsigned h = crm::mk_hi(x) & 0x7fffffffu;
  return h - ((1023u - B) << 20) < ((2u * B + 1u) << 20) || (h | crm::mk_lo(x)) == 0u;
}

// The relaxation of one cell, or false (with nothing but flux written) for a
// cell that has a nonzero quantity outside the ranges below, which
// relax_general then takes.
//
// The relaxation is bound by the number of instructions it issues (57 % of
// them were not FP64: range tests of the ~600 quotients, sign fixes,
// shared-memory reads), so the ranges are tested once, on the quantities the
// quotients are made of.  With pi, u, dmu, phi7, piNS, sigma and h0 zero or
// in 2^+-140 (pi and h0 in 2^+-300 where the second-order terms are off,
// as in the dilute cells at the edge), and eta zero or in 2^+-100, every
// numerator below is zero or in [2^-860, 2^710]: a product of n such factors
// is above 2^-140n, a difference of two of them is zero or a multiple of the
// smaller one's last bit, and no numerator has more than five factors and two
// differences.  Every quotient is then Markstein's without a test.  The same
// ranges make these rewritings exact, value for value:
//   x * 0.5 * dt = x * (0.5 dt), and Z * dmu * 2 = (2 Z) * dmu;
//   NSquant's terms with Z = 0, and those of lamPipi = 8/5 (1/3 - 1/3) = 0,
//   are +-0 and left out;
//   the terms pi^{kl} Y^{kl} of (k, l) and (l, k) are one value, +- the sign
//   of g_kk g_ll, divided once;
//   |a / b| > 3 as |a| - 3 |b| > 2^-52 |b| (the difference is exact near 3).
__device__ __forceinline__ bool relax_fast(
    const Geo& g, const double* __restrict__ pA, const double* __restrict__ pD,
    const double* __restrict__ pTh, const double* __restrict__ pBC, const double* __restrict__ pi,
    const double* __restrict__ Pi, double* __restrict__ pi0, double* __restrict__ piH0,
    double* __restrict__ Pi0, double* __restrict__ PiH0, double* __restrict__ flux,
    const double* __restrict__ clk, long long i, bool vac) {
  const double dt = clk[1], tau = clk[0] + dt;  // tau_{n+1} (src/hdo.cpp:1095)
  const long long N = g.N;
  const double e = pA[i];
  double cpi[10];
#pragma unroll
  for (int k = 0; k < 10; k++) cpi[k] = pi[k * N + i];
  const double cPi = Pi[i];
#define PI(a, b) cpi[index44(a, b)]
  const double vx = pA[5 * N + i], vy = pA[6 * N + i], vz = pA[7 * N + i];
  const double gamma = 1.0 / sqrt(1.0 - vx * vx - vy * vy - vz * vz);
  const double rg = 1.0 / gamma;
  double u[4];
  u[0] = gamma;
  u[1] = u[0] * vx;
  u[2] = u[0] * vy;
  u[3] = u[0] * vz;
  {
    double f[4];
#pragma unroll
    for (int k = 0; k < 4; k++) f[k] = (tau - dt) * (PI(0, k) + cPi * u[0] * u[k]);
    f[0] += -(tau - dt) * cPi;
#pragma unroll
    for (int k = 0; k < 4; k++) flux[k * N + i] = 0. + f[k];
  }
  const double s = pTh[3 * N + i];
  const double etaS = pTh[4 * N + i];
  const double zetaS = pTh[5 * N + i];
  const double taupi = pTh[6 * N + i], tauPi = pTh[7 * N + i];
  const double eta = etaS * s;
  // (the clock and the cell sizes are the grid's: uniform)
  bool ok = gamma <= 0x1p100 && dt >= 0x1p-60 && tau - dt >= 0x1p-60 && tau <= 0x1p60 &&
            crm::mk_den_ok(g.dx) && crm::mk_den_ok(g.dy) && taupi >= 0. && taupi <= 0x1p60 &&
            (eta == 0. || crm::mk_den_ok(eta)) && exp_ok<140>(etaS) &&
            exp_ok<140>(s) && exp_ok<140>(u[1]) && exp_ok<140>(u[2]) && exp_ok<140>(u[3]) &&
            exp_ok<140>(vz);
  // no relaxation time (below 1 GeV/fm^3 or 100 MeV, most cells): the
  // second-order terms are +-0, and a warp of such cells leaves them out
  const bool still = taupi < 0.5 * dt;
#pragma unroll
  for (int k = 0; k < 10; k++) ok = ok && (still ? exp_ok<300>(cpi[k]) : exp_ok<140>(cpi[k]));

  // ------------------------------------------------------ NSquant
  double piNS[10], PiNS, du;
  double dmu[4][4];
  if (vac) {
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) dmu[a][b] = 0.;
#pragma unroll
    for (int k = 0; k < 10; k++) piNS[k] = 0.;
    PiNS = du = 0.;
  } else {
    const double VMIN = 1e-2;
    // quotients by u^k are used where |u^k| >= VMIN only
    double ud[4], ru[4];
    bool slowu[4];
    ud[0] = gamma;
    ru[0] = rg;
    slowu[0] = false;
#pragma unroll
    for (int k = 1; k < 4; k++) {
      slowu[k] = fabs(u[k]) < VMIN;
      ud[k] = slowu[k] ? 1.0 : u[k];
      ru[k] = 1.0 / ud[k];
    }
    auto over3 = [](double a, double b) {  // |a / b| > UDIFF = 3
      return fma(-3., fabs(b), fabs(a)) > 0x1p-52 * fabs(b);
    };
    {  // the time row: u at tau - dt (B) and at tau (C)
      const double e0 = pBC[4 * N + i];
      const double rdt = 1.0 / dt;
      const bool zero = e <= 0. || e0 <= 0.;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const double u0 = pBC[k * N + i], u1 = pBC[(5 + k) * N + i];
        const bool diff = slowu[k] || over3(0.5 * (u1 + u0), u1);
        const double z = diff ? u1 - u0 : (u1 * u1 - u0 * u0) / 2.;
        ok = ok && exp_ok<500>(z);
        const double x = mk_raw(diff ? z : mk_raw(z, ud[k], ru[k]), dt, rdt);
        dmu[0][k] = zero ? 0. : x;
      }
    }
    int ix, iy, iz;
    coords(g, i, ix, iy, iz);
#pragma unroll
    for (int d = 1; d <= 3; d++) {
      long long ip, im;
      double h;
      if (d == 1) {
        ip = cidx(g, ix + 1, iy, iz);
        im = cidx(g, ix - 1, iy, iz);
        h = g.dx;
      } else if (d == 2) {
        ip = cidx(g, ix, iy + 1, iz);
        im = cidx(g, ix, iy - 1, iz);
        h = g.dy;
      } else {
        ip = cidx(g, ix, iy, iz + 1);
        im = cidx(g, ix, iy, iz - 1);
        h = g.dz;
      }
      const double ep = pD[ip], em = pD[im];
      if (ep > 0. && em > 0.) {
        const double rh = 1.0 / h;
        const double th = tau + 0.5 * dt, rth = d == 3 ? 1.0 / th : 0.;
        // (an infinite dz, one cell in eta, divides the ordinary way)
        const bool fin = d < 3 || crm::mk_den_ok(h);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const double u0 = pD[(1 + k) * N + im], u1 = pD[(1 + k) * N + ip];
          const bool diff = slowu[k] || over3(0.5 * (u1 + u0), u[k]);
          const double z = diff ? 0.5 * (u1 - u0) : 0.25 * (u1 * u1 - u0 * u0);
          ok = ok && exp_ok<500>(z);
          const double y = diff ? z : mk_raw(z, ud[k], ru[k]);
          double x = fin ? mk_raw(y, h, rh) : y / h;
          if (d == 3) x = mk_raw(x, th, rth);
          dmu[d][k] = x;
        }
      } else {
        dmu[d][0] = dmu[d][1] = dmu[d][2] = dmu[d][3] = 0.;
      }
    }
    dmu[3][0] += ddivp(u[3], tau - 0.5 * dt);
    dmu[3][3] += ddivp(u[0], tau - 0.5 * dt);
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) ok = ok && exp_ok<140>(dmu[a][b]);
    const double gdiag[4] = {1., -1., -1., -1.};
    const double r5068 = 1.0 / 5.068, r3 = 1.0 / 3.0;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b <= a; b++) {
        const double gab = (a == b) ? gdiag[a] : 0.;
        const double trace = 2.0 * mk_raw(gab - u[a] * u[b], 3.0, r3);
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int l = 0; l < 4; l++) {
            if (b != l && a != l && k != l) continue;  // Z = 0
            double Z = 0.0;  // 2 Z
            const double gak = (a == k) ? gdiag[a] : 0.;
            const double gbk = (b == k) ? gdiag[b] : 0.;
            if (b == l) Z += gak - u[a] * u[k];
            if (a == l) Z += gbk - u[b] * u[k];
            if (k == l) Z -= trace;
            acc += mk_raw(Z * dmu[k][l] * etaS * s, 5.068, r5068);
          }
        piNS[index44(a, b)] = acc;
      }
    PiNS = ddivp(-zetaS * s * (dmu[0][0] + dmu[1][1] + dmu[2][2] + dmu[3][3]), 5.068);
    du = dmu[0][0] + dmu[1][1] + dmu[2][2] + dmu[3][3];
#pragma unroll
    for (int k = 0; k < 10; k++) ok = ok && exp_ok<140>(piNS[k]);
    ok = ok && exp_ok<140>(du);
  }
  double phi7 = pTh[8 * N + i];
  if (isinf(phi7)) phi7 = 0.0;
  phi7 = ddiv(phi7, taupi);
  if (taupi < 0.5 * dt) phi7 = 0.0;

  // ------------------------------------------------ ISformal loop 1 body
  double sig[10];
  const double reta = 1.0 / (eta == 0. ? 1.0 : eta);
#pragma unroll
  for (int k = 0; k < 10; k++) {
    sig[k] = eta == 0. ? 0. : mk_raw(0.5 * piNS[k], eta, reta) * 5.068;
    ok = ok && exp_ok<140>(sig[k]);
  }
  if (!ok || !exp_ok<140>(phi7)) return false;
  const double deltapipi = still ? 0. : 4. / 3., taupipi = still ? 0. : 10. / 7.;
  const double lambdapiPi = still ? 0. : 6. / 5.;
  const double delPiPi = tauPi < 0.5 * dt ? 0. : 2. / 3.;
  const double hdt = 0.5 * dt;
  const double rtaupi = taupi > 0.5 * dt ? 1.0 / taupi : 0.;
  double h0[10];
#pragma unroll
  for (int k = 0; k < 10; k++)
    h0[k] = taupi > 0.5 * dt
                ? cpi[k] - mk_raw(mk_raw((cpi[k] - piNS[k]) * dt / 2.0, gamma, rg), taupi, rtaupi)
                : piNS[k];
  double H0;
  if (tauPi > 0.5 * dt)
    H0 = cPi - ddivp(ddivp((cPi - PiNS) * dt / 2.0, gamma), tauPi);
  else
    H0 = PiNS;
  double tau1 = tau - dt * 0.75;
  double vt = ddivp(vz, tau1);
  h0[index44(0, 0)] += ddivp(-2. * vz * PI(0, 3), tau1) * dt / 2.;
  h0[index44(3, 3)] += -(2. * vt * PI(0, 3)) * dt / 2.;
  h0[index44(3, 0)] += -(vt * PI(0, 0) + vt * PI(3, 3)) * dt / 2.;
  h0[index44(1, 0)] += -vt * PI(1, 3) * dt / 2.;
  h0[index44(2, 0)] += -vt * PI(2, 3) * dt / 2.;
  h0[index44(3, 1)] += -(vt * PI(0, 1)) * dt / 2.;
  h0[index44(3, 2)] += -(vt * PI(0, 2)) * dt / 2.;
  // The relaxation sums over (a, b) run as a loop with (a, b) known only at
  // run time, so that its body is fetched once per warp instead of ten times
  // unrolled: the unrolled kernel's instruction stream outgrew the
  // instruction caches.  Operands indexed by a or b come from shared memory
  // ([component][thread]); the arithmetic of every term is the reference's,
  // in its order.
  extern __shared__ double relax_smem[];
  double(*sm)[kRelaxBlock] = reinterpret_cast<double(*)[kRelaxBlock]>(relax_smem);
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    sm[kSmPI + k][t] = cpi[k];
    sm[kSmSIG + k][t] = sig[k];
    sm[kSmH + k][t] = h0[k];
    sm[kSmY + k][t] = phi7 * cpi[k] - taupipi * sig[k];
  }
#pragma unroll
  for (int k = 0; k < 4; k++) sm[kSmU + k][t] = u[k];
  const double htp = taupipi * 0.5;
#pragma unroll 1
  for (int ab = 0; ab < 10; ab++) {
    const int a = ab >= 6 ? 3 : ab >= 3 ? 2 : ab >= 1 ? 1 : 0;
    const int b = ab - a * (a + 1) / 2;
    const double ua = sm[kSmU + a][t], ub = sm[kSmU + b][t];
    double dab = -ua * ub;  // Delta[index44(a, b)]
    if (a == b) dab += a == 0 ? 1. : -1.;
    const double d3 = 1. / 3. * dab;
    double w[10];  // the pi^{kl} Y^{kl} terms
#pragma unroll
    for (int k = 0; k < 10; k++) w[k] = 0.;
    double acc = sm[kSmH + ab][t];
    if (!still) {
#pragma unroll
      for (int k = 0; k < 10; k++)
        w[k] = mk_raw(d3 * sm[kSmPI + k][t] * sm[kSmY + k][t], gamma, rg) * hdt;
      acc += ddivp(-deltapipi * sm[kSmPI + ab][t] * du + lambdapiPi * cPi * sm[kSmSIG + ab][t],
                   gamma) *
             0.5 * dt;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double gk = k == 0 ? 1. : -1.;
      const double pak = sm[kSmPI + index44(a, k)][t], pbk = sm[kSmPI + index44(b, k)][t];
      if (!still) {
        const double sak = sm[kSmSIG + index44(a, k)][t], sbk = sm[kSmSIG + index44(b, k)][t];
        const double n0 = phi7 * pak * pbk * gk - htp * (pak * sbk * gk + pbk * sak * gk);
        acc += mk_raw(n0, gamma, rg) * hdt;
      }
      const double c = -pak * ub - pbk * ua;
#pragma unroll
      for (int l = 0; l < 4; l++) {
        const double n1 = c * u[l] * dmu[l][k] * gk;
        const double gl = l == 0 ? 1. : -1.;
        acc += mk_raw(n1, gamma, rg) * hdt - w[index44(k, l)] * (gk * gl);
      }
    }
    sm[kSmH + ab][t] = acc;
  }
#pragma unroll
  for (int k = 0; k < 10; k++) {
    h0[k] = sm[kSmH + k][t];
    ok = ok && (still ? exp_ok<300>(h0[k]) : exp_ok<140>(h0[k]));
  }
  H0 += 0.;  // lamPipi = 0
  H0 += ddivp(-delPiPi * cPi * du, gamma) * 0.5 * dt;
  if (!ok || isinf(H0) || isnan(H0)) return false;
#define H(a, b) h0[index44(a, b)]
  double f0[10];
#pragma unroll
  for (int k = 0; k < 10; k++)
    f0[k] = taupi > 0.5 * dt
                ? sm[kSmPI + k][t] - mk_raw(mk_raw((h0[k] - piNS[k]) * dt, gamma, rg), taupi, rtaupi)
                : piNS[k];
  double F0;
  if (tauPi > 0.5 * dt)
    F0 = cPi - ddivp(ddivp((H0 - PiNS) * dt, gamma), tauPi);
  else
    F0 = PiNS;
  tau1 = tau - dt * 0.5;
  vt = ddivp(vz, tau1);
  f0[index44(0, 0)] += -2. * vt * H(0, 3) * dt;
  f0[index44(3, 3)] += -(2. * vt * H(0, 3)) * dt;
  f0[index44(3, 0)] += -(vt * H(0, 0) + vt * H(3, 3)) * dt;
  f0[index44(1, 0)] += -vt * H(1, 3) * dt;
  f0[index44(2, 0)] += -vt * H(2, 3) * dt;
  f0[index44(3, 1)] += -(vt * H(0, 1)) * dt;
  f0[index44(3, 2)] += -(vt * H(0, 2)) * dt;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    sm[kSmF + k][t] = f0[k];
    sm[kSmY + k][t] = phi7 * h0[k] - taupipi * sm[kSmSIG + k][t];
  }
#pragma unroll 1
  for (int ab = 0; ab < 10; ab++) {
    const int a = ab >= 6 ? 3 : ab >= 3 ? 2 : ab >= 1 ? 1 : 0;
    const int b = ab - a * (a + 1) / 2;
    const double ua = sm[kSmU + a][t], ub = sm[kSmU + b][t];
    double dab = -ua * ub;  // Delta[index44(a, b)]
    if (a == b) dab += a == 0 ? 1. : -1.;
    const double d3 = 1. / 3. * dab;
    double w[10];
#pragma unroll
    for (int k = 0; k < 10; k++) w[k] = 0.;
    double acc = sm[kSmF + ab][t];
    if (!still) {
#pragma unroll
      for (int k = 0; k < 10; k++) w[k] = d3 * sm[kSmH + k][t] * sm[kSmY + k][t];
      acc += ddivp(-deltapipi * sm[kSmH + ab][t] * du + lambdapiPi * H0 * sm[kSmSIG + ab][t],
                   gamma) *
             dt;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double gk = k == 0 ? 1. : -1.;
      const double hak = sm[kSmH + index44(a, k)][t], hbk = sm[kSmH + index44(b, k)][t];
      if (!still) {
        const double pak = sm[kSmPI + index44(a, k)][t];
        const double sak = sm[kSmSIG + index44(a, k)][t], sbk = sm[kSmSIG + index44(b, k)][t];
        const double n0 = phi7 * pak * hbk * gk - htp * (hak * sbk * gk + hbk * sak * gk);
        acc += mk_raw(n0, gamma, rg) * dt;
      }
      const double c = -hak * ub - hbk * ua;
#pragma unroll
      for (int l = 0; l < 4; l++) {
        const double gl = l == 0 ? 1. : -1.;
        const double n = c * u[l] * dmu[l][k] * gk - w[index44(k, l)] * (gk * gl);
        acc += mk_raw(n, gamma, rg) * dt;
      }
    }
    sm[kSmF + ab][t] = acc;
  }
  F0 += 0.;  // lamPipi = 0
  F0 += ddivp(-delPiPi * H0 * du, gamma) * dt;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    piH0[k * N + i] = sm[kSmH + k][t];
    pi0[k * N + i] = sm[kSmF + k][t];
  }
  PiH0[i] = H0;
  Pi0[i] = F0;
#undef PI
#undef H
  return true;
}


__device__ __forceinline__ void d_is_relax(
    const Geo& g, const double* __restrict__ pA, const double* __restrict__ pD,
    const double* __restrict__ pTh, const double* __restrict__ pBC, const double* __restrict__ pi,
    const double* __restrict__ Pi, double* __restrict__ pi0, double* __restrict__ piH0,
    double* __restrict__ Pi0, double* __restrict__ PiH0, double* __restrict__ flux,
    const double* __restrict__ clk, unsigned* err, const int* __restrict__ active,
    const int* __restrict__ nactive, long long blk) {
  const long long idx = blk * blockDim.x + threadIdx.x;
  if (idx >= *nactive) return;
  const int entry = active[idx];  // a cell with matter (k_visc_prims)
  const bool vac = entry < 0;     // next to vacuum
  const long long i = vac ? ~entry : entry;
  if (!relax_fast(g, pA, pD, pTh, pBC, pi, Pi, pi0, piH0, Pi0, PiH0, flux, clk, i, vac))
    relax_general(g, pA, pD, pTh, pBC, pi, Pi, pi0, piH0, Pi0, PiH0, flux, clk, err, i, vac);
}
__global__ void __launch_bounds__(kRelaxBlock, kRelaxMinBlocks) k_is_relax(
    Geo g, const double* __restrict__ pA, const double* __restrict__ pD,
    const double* __restrict__ pTh, const double* __restrict__ pBC, const double* __restrict__ pi,
    const double* __restrict__ Pi, double* __restrict__ pi0, double* __restrict__ piH0,
    double* __restrict__ Pi0, double* __restrict__ PiH0, double* __restrict__ flux,
    const double* __restrict__ clk, unsigned* err, const int* __restrict__ active,
    const int* __restrict__ nactive) {
  d_is_relax(g, pA, pD, pTh, pBC, pi, Pi, pi0, piH0, Pi0, PiH0, flux, clk, err, active, nactive,
             blockIdx.x);
}


// ------------------------------------------------ ISformal, loop #2
// Semi-Lagrangian advection of pi0/piH0 from the 2x2x2 upwind cells, the
// viscous-correction limiter and the -(tau) * delta Q_{n+1} flux
// (src/hdo.cpp:866-962).  Bound by the latency of its 176 scattered loads a
// cell.  Two threads per cell (pi and piH apart, 64 registers, 8 blocks per
// SM) were slower: 49 against 42 us at 101x101x51, 206 against 118 at
// 201x201x101.
__device__ __forceinline__ double sgn(double x) {
  if (x > 0) return 1.;
  if (x < 0.) return -1.;
  return 0.;
}

__device__ __forceinline__ void d_is_advect(const Geo& g, const double* __restrict__ pA,
                                            const double* __restrict__ pi0,
                                            const double* __restrict__ piH0,
                                            const double* __restrict__ Pi0,
                                            const double* __restrict__ PiH0,
                                            double* __restrict__ pi, double* __restrict__ piH,
                                            double* __restrict__ Pi, double* __restrict__ PiH,
                                            double* __restrict__ vcc, double* __restrict__ flux,
                                            const double* __restrict__ clk,
                                            const int* __restrict__ active,
                                            const int* __restrict__ nactive, long long blk) {
  const double dt = clk[1], tau = clk[0] + dt;  // tau_{n+1} (src/hdo.cpp:1095)
  // the cells with matter only (k_visc_prims); the empty ones are left as
  // they are, as the reference's loop 2 leaves them (e <= 0)
  const int idx = (int)(blk * blockDim.x + threadIdx.x);
  if (idx >= *nactive) return;
  const int entry = active[idx];
  const long long i = entry < 0 ? ~entry : entry;
  int ix, iy, iz;
  coords(g, i, ix, iy, iz);
  const long long N = g.N;
  const Prim A = loadA(pA, N, i);
  const double e = A.e, p = A.p, vx = A.vx, vy = A.vy, vz = A.vz;
  const double xm = ddivp(-vx * dt, g.dx);
  const double ym = ddivp(-vy * dt, g.dy);
  const double zm = ddivp(ddivp(-vz * dt, g.dz), tau - 0.5 * dt);
  const double xmH = ddivp(-vx * dt, g.dx) / 2.0;
  const double ymH = ddivp(-vy * dt, g.dy) / 2.0;
  const double zmH = ddivp(ddivp(-vz * dt, g.dz), tau - 0.5 * dt) / 2.0;
  const double wx[2] = {(1. - fabs(xm)), fabs(xm)};
  const double wy[2] = {(1. - fabs(ym)), fabs(ym)};
  const double wz[2] = {(1. - fabs(zm)), fabs(zm)};
  const double wxH[2] = {(1. - fabs(xmH)), fabs(xmH)};
  const double wyH[2] = {(1. - fabs(ymH)), fabs(ymH)};
  const double wzH[2] = {(1. - fabs(zmH)), fabs(zmH)};
  const int sx = (int)sgn(xm), sy = (int)sgn(ym), sz = (int)sgn(zm);
  double a[10], aH[10], P = 0.0, PH = 0.0;
#pragma unroll
  for (int k = 0; k < 10; k++) a[k] = aH[k] = 0.0;
#pragma unroll
  for (int jx = 0; jx < 2; jx++)
#pragma unroll
    for (int jy = 0; jy < 2; jy++)
#pragma unroll
      for (int jz = 0; jz < 2; jz++) {
        const long long c1 = cidx(g, ix + jx * sx, iy + jy * sy, iz + jz * sz);
        if (jx + jy + jz > 0 && pA[c1] <= 0.) continue;  // an empty cell: zeros
        const double w = wx[jx] * wy[jy] * wz[jz];
        const double wH = wxH[jx] * wyH[jy] * wzH[jz];
#pragma unroll
        for (int k = 0; k < 10; k++) {
          a[k] += w * pi0[k * N + c1];
          aH[k] += wH * piH0[k * N + c1];
        }
        P += w * Pi0[c1];
        PH += wH * PiH0[c1];
      }
  const double maxT0 = smax(ddivp(e + p, 1. - vx * vx - vy * vy - vz * vz) - p,
                            ddivp((e + p) * (vx * vx + vy * vy + vz * vz), 1. - vx * vx - vy * vy - vz * vz) + p);
  double maxpi = 0.;
#pragma unroll
  for (int k = 0; k < 10; k++)
    if (fabs(a[k]) > maxpi) maxpi = fabs(a[k]);
  bool rescaled = false;
  if (ddiv(maxT0, maxpi) < 1.0) {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      a[k] = ddiv(0.1 * a[k] * maxT0, maxpi);
      aH[k] = ddiv(0.1 * aH[k] * maxT0, maxpi);
    }
    rescaled = true;
  }
  if (fabs(P) > p) {
    if (P != 0.) P = 1 * P / fabs(P) * p;
    if (PH != 0.) PH = 1 * PH / fabs(PH) * p;
    rescaled = true;
  }
  vcc[i] = rescaled ? ddiv(maxT0, maxpi) : 1.;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    pi[k * N + i] = a[k];
    piH[k * N + i] = aH[k];
  }
  Pi[i] = P;
  PiH[i] = PH;
  const double gamma = 1.0 / sqrt(1.0 - vx * vx - vy * vy - vz * vz);
  double u[4];
  u[0] = gamma;
  u[1] = u[0] * vx;
  u[2] = u[0] * vy;
  u[3] = u[0] * vz;
  double f[4];
#pragma unroll
  for (int k = 0; k < 4; k++) f[k] = -tau * (a[index44(0, k)] + P * u[0] * u[k]);
  f[0] += tau * P;
#pragma unroll
  for (int k = 0; k < 4; k++) flux[k * N + i] += f[k];
}
__global__ void __launch_bounds__(128) k_is_advect(Geo g, const double* __restrict__ pA,
                                                   const double* __restrict__ pi0,
                                                   const double* __restrict__ piH0,
                                                   const double* __restrict__ Pi0,
                                                   const double* __restrict__ PiH0,
                                                   double* __restrict__ pi, double* __restrict__ piH,
                                                   double* __restrict__ Pi, double* __restrict__ PiH,
                                                   double* __restrict__ vcc,
                                                   double* __restrict__ flux, const double* __restrict__ clk,
                                                   const int* __restrict__ active,
                                                   const int* __restrict__ nactive) {
  d_is_advect(g, pA, pi0, piH0, Pi0, PiH0, pi, piH, Pi, PiH, vcc, flux, clk, active, nactive,
              blockIdx.x);
}


// --------------------------------------------- viscous flux + update
// Hydro::visc_flux (src/hdo.cpp:966-1014) for the six faces of the cell,
// visc_source_step (src/hdo.cpp:355-375) and Cell::updateByViscFlux
// (src/cll.cpp:76-84).
// the face's cell size along dir (eta: dz (tau + dt/2), src/hdo.cpp:971-976)
__device__ __forceinline__ double visc_dxa(int dir, double tau, double dt, const Geo& g) {
  if (dir == X_) return g.dx;
  if (dir == Y_) return g.dy;
  return g.dz * (tau + 0.5 * dt);
}

// rdxa = RN(1 / dxa): the four quotients by dxa go through div_batch
__device__ __forceinline__ bool visc_face(int dir, double tau, double dt, const Geo& g,
                                          const double* __restrict__ pA,
                                          const double* __restrict__ piH,
                                          const double* __restrict__ PiH,
                                          const double* __restrict__ m, long long L, long long R,
                                          double dxa, double rdxa, double f[4]) {
  const long long N = g.N;
  if (m[(dir - 1) * N + L] < 1. && m[(dir - 1) * N + R] < 1.) return false;
  double vxl = pA[5 * N + L], vyl = pA[6 * N + L], vzl = pA[7 * N + L];
  const double vxr = pA[5 * N + R], vyr = pA[6 * N + R], vzr = pA[7 * N + R];
  vxl = 0.5 * (vxl + vxr);
  vyl = 0.5 * (vyl + vyr);
  vzl = 0.5 * (vzl + vzr);
  const double v = sqrt(vxl * vxl + vyl * vyl + vzl * vzl);
  if (v > 1.) {
    vxl = ddivp(0.99 * vxl, v);
    vyl = ddivp(0.99 * vyl, v);
    vzl = ddivp(0.99 * vzl, v);
  }
  const double gamma = 1. / sqrt(1. - v * v);
  const double uuu[4] = {gamma, gamma * vxl, gamma * vyl, gamma * vzl};
  const double gmumu[4] = {1., -1., -1., -1.};
  const double PL = PiH[L], PR = PiH[R];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const int k = index44(a, dir);
    double x = 0.5 * (piH[k * N + L] + piH[k * N + R]);
    if (a == dir) x += -0.5 * (PL + PR) * gmumu[a];
    x += 0.5 * (PL + PR) * uuu[a] * uuu[dir];
    f[a] = x * (tau - 0.5 * dt) * dt;
  }
  div_batch<4>(f, dxa, rdxa, crm::mk_den_ok(dxa));
  return true;
}

__device__ __forceinline__ void d_visc_update(const Geo& g, const double* __restrict__ pA,
                                              const double* __restrict__ piH,
                                              const double* __restrict__ PiH,
                                              const double* __restrict__ m,
                                              const double* __restrict__ flux,
                                              double* __restrict__ Q,
                                              const double* __restrict__ clk, long long blk) {
  const double dt = clk[1], tau = clk[0] + dt;  // tau_{n+1} (src/hdo.cpp:1095)
  const long long i = blk * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  int ix, iy, iz;
  coords(g, i, ix, iy, iz);
  const long long N = g.N;
  // an empty cell has no flux so far, and between unfilled cells none comes
  const double e = pA[i];
  const bool empty = e <= 0.;
  double f[4];
  const long long st[3] = {1, g.nx, (long long)g.nx * g.ny};
  const int cc[3] = {ix, iy, iz};
  const int nn[3] = {g.nx, g.ny, g.nz};
  if (empty) {
    // (the nine loads together, as in d_update_m: 201x201x101 133 -> 123 us)
    bool any = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double* md = m + d * N;
      const bool in0 = cc[d] > 0, in1 = cc[d] < nn[d] - 1;
      const double m0 = md[in0 ? i - st[d] : i], m1 = md[in1 ? i + st[d] : i];
      const bool own = !(md[i] < 1.);
      any |= (in0 & (own | !(m0 < 1.))) | (in1 & (own | !(m1 < 1.)));
    }
    if (!any) return;
  }
  double fl[4];
#pragma unroll
  for (int k = 0; k < 4; k++) fl[k] = empty ? 0. : flux[k * N + i];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double dxa = visc_dxa(d + 1, tau, dt, g), rdxa = 1.0 / dxa;
    if (cc[d] > 0 && visc_face(d + 1, tau, dt, g, pA, piH, PiH, m, i - st[d], i, dxa, rdxa, f)) {
#pragma unroll
      for (int k = 0; k < 4; k++) fl[k] += f[k];
    }
    if (cc[d] < nn[d] - 1 &&
        visc_face(d + 1, tau, dt, g, pA, piH, PiH, m, i, i + st[d], dxa, rdxa, f)) {
#pragma unroll
      for (int k = 0; k < 4; k++) fl[k] += -f[k];
    }
  }
  if (!empty) {
    const double vx = pA[5 * N + i], vy = pA[6 * N + i], vz = pA[7 * N + i];
    double uuu[4];
    uuu[0] = 1. / sqrt(1. - vx * vx - vy * vy - vz * vz);
    uuu[1] = uuu[0] * vx;
    uuu[2] = uuu[0] * vy;
    uuu[3] = uuu[0] * vz;
    const double PH = PiH[i];
    double k0 = -piH[index44(3, 3) * N + i] + PH * (-1.0 - uuu[3] * uuu[3]);
    double k3 = -(piH[index44(0, 3) * N + i] + PH * uuu[0] * uuu[3]);
    k0 *= dt;
    k3 *= dt;
    fl[0] += k0;
    fl[1] += 0. * dt;
    fl[2] += 0. * dt;
    fl[3] += k3;
  }
  const double q0 = Q[i];
  if (fabs(fl[0]) <= 0.5 * q0) {
#pragma unroll
    for (int k = 0; k < 4; k++) Q[k * N + i] += fl[k];
#pragma unroll
    for (int k = 4; k < 7; k++) Q[k * N + i] += 0.;
  } else if (fl[0] != 0.) {
    const double fac = fabs(ddiv(0.5 * q0, fl[0]));
#pragma unroll
    for (int k = 0; k < 4; k++) Q[k * N + i] += fac * fl[k];
#pragma unroll
    for (int k = 4; k < 7; k++) Q[k * N + i] += fac * 0.;
  }
}
__global__ void __launch_bounds__(128, 8) k_visc_update(Geo g, const double* __restrict__ pA,
                                                     const double* __restrict__ piH,
                                                     const double* __restrict__ PiH,
                                                     const double* __restrict__ m,
                                                     const double* __restrict__ flux,
                                                     double* __restrict__ Q, const double* __restrict__ clk) {
  d_visc_update(g, pA, piH, PiH, m, flux, Q, clk, blockIdx.x);
}


// --------------------------------------------------- batched transformPV
__global__ void k_transform_pv(EosDev E, const double* __restrict__ Q, long long n,
                               double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double q[7];
#pragma unroll
  for (int k = 0; k < 7; k++) q[k] = Q[k * n + i];
  Prim o;
  transform_pv(E, q, o);
  out[0 * n + i] = o.e;
  out[1 * n + i] = o.p;
  out[2 * n + i] = o.nb;
  out[3 * n + i] = o.nq;
  out[4 * n + i] = o.ns;
  out[5 * n + i] = o.vx;
  out[6 * n + i] = o.vy;
  out[7 * n + i] = o.vz;
}

// ------------------------------------------------------------ launcher
static inline unsigned nblk(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

static long long face_blocks(const Geo& g, int bs) {
  return (g.nz > 1 ? 3LL : 2LL) * nblk(g.N, bs / 2);
}
static long long face_resident(int bs) { return 148LL * kFaceMinBlocks * (128 / bs); }
// Where the faces do not fill one resident set of blocks the step is a chain
// of latencies, and the lists (a kernel more in it, and the emptiest warps
// of a grid that leaves the chip idle anyway) do not pay: 101x101x1, 320
// blocks of 1184, 48 us a step with lists and 39 without; 47x61x23, 3093
// blocks, 192 with and 223 without.  Two directions in place of three gain
// less for the same two list kernels: on 201x201x1, 1264 blocks, an event takes
// 120 us viscous and 50.5 ideal with lists, 119 and 47.8 without, on 251x251x1,
// 1970 blocks, 129 and 54, 141 and 63.
// A grid without empty cells is slower with lists in every case, and the host
// cannot tell.  The conformal EoS in 2+1D, whose root finds are the cheapest,
// is used for such flow (Gubser's): without lists full grids of 251x251 and
// 401x401 take 63 and 134 us and not 71 and 154 (70 and 137 in the form before
// the lists), events, mostly vacuum, 56 and 101 and not 48 and 75 (69 and 106).
bool face_lists(const Geo& g, int bs, int eos_kind) {
  if (g.nz == 1)
    return eos_kind != 0 && face_blocks(g, bs) > face_resident(bs) * 3 / 2;
  return face_blocks(g, bs) > face_resident(bs);
}
// The stage-batched form makes lists for every event but those of the conformal
// EoS in 2+1D (64 Gubser events of 101x101: 643 us a step with lists, 604
// without).
Fields batch_fields(const Fields& f, const Geo& g, int eos_kind) {
  Fields b = f;
  if (g.nz == 1 && eos_kind == 0) {
    b.flist = b.ulist = nullptr;
    b.fact = nullptr;
  }
  return b;
}


const char* const kKernelNames[KK_COUNT] = {
    "k_update_m", "k_face", "k_update", "k_ghost",
    "k_visc_prims", "k_is_relax", "k_is_advect", "k_visc_update",
    "vorticity (k_vort_*, 5 kernels)"};


template <int EK>
static int launch_step_ek(const StepArgs& a, cudaStream_t s, LaunchMarker* mk) {
  const Geo& g = a.g;
  const int bs = a.block == 64 ? 64 : 128;
  const unsigned nb = nblk(g.N, bs);
  const unsigned nb128 = nblk(g.N, 128);
  // one resident set of blocks for the faces
  const long long fblocks = face_blocks(g, bs), resident = face_resident(bs);
  const bool lists = face_lists(g, bs, a.eos.kind);
  const unsigned nface = (unsigned)std::min(fblocks, resident);
  const unsigned rset = 148 * kUpdateMinBlocks * (128u / bs);
  // the update runs on a list where its blocks do not fit one resident set
  // (1184): 101x101x51, 4065 blocks, 446 us a step with the list and 463
  // without; 47x61x23, 516 blocks, 169 with and 161 without; 61x61x31, 902
  // blocks, 80 to 100 % matter, 152 and 173 with, 148 and 156 without
  const bool rows = lists && nb > rset;
  const unsigned nupd = rows ? rset : nb;
  const bool vort = a.vort && a.viscous;
  const unsigned wide = 128 / bs;
  const unsigned nprims = std::min(2 * nb, 148 * kPrimsMinBlocks * wide);
  const unsigned ngh = nblk(ghost_shell(g).n, bs);
  int launches = 0;
  const Fields& F = a.f;
  auto done = [&](int kind) {
    launches++;
    if (mk) mk->after(kind);
  };
  k_update_m<<<nb, bs, 0, s>>>(g, F.m, F.m2, a.clk, F.fcount, a.viscous ? F.nactive : nullptr);
  done(KK_UPDATE_M);
  const double* m = F.m2;  // the updated fill fractions
  // predictor (src/hdo.cpp:1023-1060) and corrector (src/hdo.cpp:1062-1094)
  for (int pass = 0; pass < 2; pass++) {
    const bool pred = pass == 0;
    const double* QQ = pred ? F.Q : F.Qh;
    int* fcount = lists ? F.fcount + 3 * pass : nullptr;
    if (lists) {
      k_face_list<<<nb, bs, 0, s>>>(g, F, pred, rows, a.viscous, vort ? a.vort->TB : nullptr, a.clk);
      launches++;
    }
    k_face<EK><<<nface, bs, 0, s>>>(g, a.eos, pred, QQ, m, F.Fx, F.Fy, F.Fz,
                                    lists ? F.flist : nullptr, fcount, a.clk, F.err);
    done(KK_FACE);
    auto update = pred ? (rows ? k_update<true, EK, true> : k_update<true, EK, false>)
                       : (rows ? k_update<false, EK, true> : k_update<false, EK, false>);
    update<<<nupd, bs, 0, s>>>(g, a.eos, F.Q, F.Qh, F.Qprev, F.Fx, F.Fy, F.Fz, lists ? F.fact : nullptr,
                               a.clk, F.err, pred && a.viscous ? F.pBC : nullptr,
                               !pred && a.viscous ? F.pA : nullptr,
                               pred && vort ? a.vort->TB : nullptr, F.pD, F.wet, F.fcount + 6,
                               F.ulist, F.fcount + 7 + pass);
    done(KK_UPDATE);
  }
  if (!a.viscous) {
    k_ghost<true, true><<<ngh, bs, 0, s>>>(g, F, nullptr, a.tick);
    done(KK_GHOST);
  } else {
    k_ghost<true, false><<<ngh, bs, 0, s>>>(g, F, F.wet, nullptr);
    done(KK_GHOST);
    if (vort)
      k_visc_prims<EK, true><<<nprims, bs, 0, s>>>(g, a.eos, a.tr, F.Q, F.Qprev, F.Qh, m, F.pA, F.pD,
                                               F.pTh, F.pBC, a.clk, F.wet, F.fcount + 6, F.active, F.nactive,
                                               a.vort->TD, a.vort->TB, a.vort->TC);
    else
      k_visc_prims<EK, false><<<nprims, bs, 0, s>>>(g, a.eos, a.tr, F.Q, F.Qprev, F.Qh, m, F.pA, F.pD,
                                                F.pTh, F.pBC, a.clk, F.wet, F.fcount + 6, F.active, F.nactive,
                                                nullptr, nullptr, nullptr);
    done(KK_VISC_PRIMS);
    if (vort) {
      launches += launch_vorticity(a, s) - 1;
      done(KK_VORT);
    }
    // the relaxation on full warps of cells with matter
    k_is_relax<<<nb128, kRelaxBlock, kRelaxSmem, s>>>(g, F.pA, F.pD, F.pTh, F.pBC, F.pi, F.Pi,
                                                      F.pi0, F.piH0, F.Pi0, F.PiH0, F.flux, a.clk,
                                                      F.err, F.active, F.nactive);
    done(KK_IS_RELAX);
    k_is_advect<<<nb, bs, 0, s>>>(g, F.pA, F.pi0, F.piH0, F.Pi0, F.PiH0, F.pi, F.piH, F.Pi, F.PiH,
                                  F.vcc, F.flux, a.clk, F.active, F.nactive);
    done(KK_IS_ADVECT);
    k_visc_update<<<nb, bs, 0, s>>>(g, F.pA, F.piH, F.PiH, m, F.flux, F.Q, a.clk);
    done(KK_VISC_UPDATE);
    k_ghost<false, true><<<ngh, bs, 0, s>>>(g, F, nullptr, a.tick);
    done(KK_GHOST);
  }
  return launches;
}

int launch_step(const StepArgs& a, cudaStream_t s, LaunchMarker* mk) {
  const bool chiral = a.eos.kind == 2;
  if (a.eos.kind == 3) return launch_step_ek<EK_TABLE3>(a, s, mk);  // EoS3f (no slope method)
  if (a.eos.kind == 6) return launch_step_ek<EK_AZH>(a, s, mk);     // EoSAZH (no slope method)
  if (a.eos.kind == 7) return launch_step_ek<EK_CMFE>(a, s, mk);    // EoSCMFe (no slope method)
  if (a.eos.slope)
    return chiral ? launch_step_ek<EK_CHIRAL_SL>(a, s, mk) : launch_step_ek<EK_TABLE_SL>(a, s, mk);
  return chiral ? launch_step_ek<EK_CHIRAL>(a, s, mk) : launch_step_ek<EK_TABLE>(a, s, mk);
}

void launch_transform_pv(const EosDev& E, const double* Q, long long n, double* out,
                         cudaStream_t s) {
  k_transform_pv<<<nblk(n, 128), 128, 0, s>>>(E, Q, n, out);
}

// TransportCoeff::getEta + getTau (src/trancoeff.cpp:68-100) on arrays:
// in[6][n] = e, nb, T, muB, s, p -> out[4][n] = eta/s, zeta/s, tau_pi, tau_Pi
__global__ void k_transport(TrDev tr, const double* __restrict__ in, long long n,
                            double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double e = in[i], nb = in[n + i], T = in[2 * n + i], mub = in[3 * n + i],
               s = in[4 * n + i], p = in[5 * n + i];
  double taupi, tauPi;
  tr_getTau(tr, e, nb, T, mub, s, p, taupi, tauPi);
  out[i] = tr_etaS(tr, e, nb, T, mub, s, p);
  out[n + i] = tr_zetaS(tr, e, T, s, p);
  out[2 * n + i] = taupi;
  out[3 * n + i] = tauPi;
}

void launch_transport(const TrDev& tr, const double* in, long long n, double* out,
                      cudaStream_t s) {
  k_transport<<<nblk(n, 128), 128, 0, s>>>(tr, in, n, out);
}

// EoS::eos with muS, EoS::p and EoS::s (nq = ns = 0) on arrays:
// e[n], nb[n] -> out[6][n] = p, T, muB, muS, p(), s
__global__ void k_eos_eval(EosDev E, const double* __restrict__ e, const double* __restrict__ nb,
                           long long n, double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double T, mub, mus, p;
  eos_eval(E, e[i], nb[i], T, mub, mus, p);
  out[i] = p;
  out[n + i] = T;
  out[2 * n + i] = mub;
  out[3 * n + i] = mus;
  out[4 * n + i] = eos_p(E, e[i], nb[i]);
  out[5 * n + i] = eos_s(E, e[i], nb[i], 0., 0.);
}

void launch_eos_eval(const EosDev& E, const double* e, const double* nb, long long n, double* out,
                     cudaStream_t s) {
  k_eos_eval<<<nblk(n, 128), 128, 0, s>>>(E, e, nb, n, out);
}

// ------------------------------------------------------------ clock
// The step kernels read (tau, dt) from a two-double device clock, so that a
// captured step stays valid from one step to the next.
__global__ void k_clock_set(double* clk, double tau, double dt) {
  clk[0] = tau;
  clk[1] = dt;
}
// the substep divide (dt / n) and restore (dt * n) of the driver loop
// (src/main.cpp:411,415), in the host's order
__global__ void k_clock_op(double* clk, int op, int n) {
  if (op == 1)
    clk[1] = clk[1] / n;
  else
    clk[1] = clk[1] * n;
}

// ------------------------------------------------- stage-batched step
// The step kernels' bodies over a work table: block b of the launch is
// block items[b].blk of event items[b].ev, whose arguments come from
// evs[items[b].ev] (the small structures copied into registers, the
// field pointers loaded once).  Each event's cells see exactly the
// operations of its own launch_step; events are independent, so the order
// of blocks across events does not matter.
#define VH_ITEM                              \
  const BItem it = items[blockIdx.x];        \
  const StepDev& A = evs[it.ev];             \
  const Geo g = A.g;                         \
  const long long blk = it.blk;

__global__ void kb_update_m(const StepDev* __restrict__ evs, const BItem* __restrict__ items) {
  VH_ITEM
  d_update_m(g, A.f.m, A.f.m2, A.clk, A.f.fcount, A.f.nactive, blk);
}

__global__ void __launch_bounds__(128) kb_face_list(const StepDev* __restrict__ evs,
                                                    const BItem* __restrict__ items,
                                                    bool predict) {
  VH_ITEM
  if (!A.f.flist) return;  // (batch_fields)
  d_face_list(g, A.f, predict, true, A.viscous, nullptr, A.clk, blk);
}

// a work item of kBatchBlock cells stands for six blocks (grid.y) of its
// event's faces: all there can be
template <int EK>
__global__ void __launch_bounds__(128, kFaceMinBlocks) kb_face(const StepDev* __restrict__ evs,
                                                               const BItem* __restrict__ items,
                                                               bool predict) {
  const BItem it = items[blockIdx.x];
  const StepDev& A = evs[it.ev];
  const FaceBatch fb = face_batch(A.g, A.f.flist ? A.f.fcount + (predict ? 0 : 3) : nullptr);
  const int b = 6 * it.blk + blockIdx.y;
  if (b >= fb.blocks[0] + fb.blocks[1] + fb.blocks[2]) return;
  const Geo g = A.g;
  const EosDev E = A.eos;
  d_face<EK>(g, E, predict, fb, predict ? A.f.Q : A.f.Qh, A.f.m2, A.f.Fx, A.f.Fy, A.f.Fz,
             A.f.flist, A.clk, A.f.err, b);
}

template <bool PRED, int EK>
__global__ void __launch_bounds__(128, kUpdateMinBlocks) kb_update(const StepDev* __restrict__ evs,
                                                 const BItem* __restrict__ items) {
  VH_ITEM
  const EosDev E = A.eos;
  double* pB = PRED && A.viscous ? A.f.pBC : nullptr;
  double* pA = !PRED && A.viscous ? A.f.pA : nullptr;
  const int* ulist = A.f.ulist;
  const int n = ulist ? A.f.fcount[PRED ? 7 : 8] : (int)g.N;
  const long long idx = blk * blockDim.x + threadIdx.x;
  if (blk * blockDim.x >= n) return;
  d_update<PRED, EK>(g, E, A.f.Q, A.f.Qh, A.f.Qprev, A.f.Fx, A.f.Fy, A.f.Fz, A.f.fact, A.clk,
                     A.f.err, pB, pA, nullptr, A.f.pD, A.f.wet, A.f.fcount + 6,
                     idx >= n ? g.N : ulist ? ulist[idx] : idx);
}

template <bool HALF, bool FULL>
__global__ void kb_ghost(const StepDev* __restrict__ evs, const BItem* __restrict__ items) {
  VH_ITEM
  d_ghost<HALF, FULL>(g, A.f.gsrc, A.f, HALF && A.viscous ? A.f.wet : nullptr, FULL ? A.clk : nullptr,
                      blk);
}

template <int EK>
__global__ void __launch_bounds__(128, kPrimsMinBlocks) kb_visc_prims(const StepDev* __restrict__ evs,
                                                     const BItem* __restrict__ items) {
  VH_ITEM
  // a work item's 128 cells: two blocks (grid.y) of two threads a cell
  const int n = A.f.fcount[6], half = blockDim.x >> 1;
  const bool second = (int)threadIdx.x >= half;
  const long long first = (2 * blk + blockIdx.y) * half;
  const long long idx = first + (second ? threadIdx.x - half : threadIdx.x);
  if (first >= n) return;
  const EosDev E = A.eos;
  const TrDev tr = A.tr;
  d_visc_prims<EK, false>(g, E, tr, A.f.Q, A.f.Qprev, A.f.Qh, A.f.m2, A.f.pA, A.f.pD, A.f.pTh,
                   A.f.pBC, A.clk, A.f.active, A.f.nactive, nullptr,
                          nullptr, nullptr, idx < n ? A.f.wet[idx] : 0, idx < n, second);
}

__global__ void __launch_bounds__(kRelaxBlock, kRelaxMinBlocks) kb_is_relax(
    const StepDev* __restrict__ evs, const BItem* __restrict__ items) {
  VH_ITEM
  d_is_relax(g, A.f.pA, A.f.pD, A.f.pTh, A.f.pBC, A.f.pi, A.f.Pi, A.f.pi0, A.f.piH0, A.f.Pi0,
             A.f.PiH0, A.f.flux, A.clk, A.f.err, A.f.active, A.f.nactive, blk);
}

__global__ void __launch_bounds__(128) kb_is_advect(const StepDev* __restrict__ evs,
                                                    const BItem* __restrict__ items) {
  VH_ITEM
  d_is_advect(g, A.f.pA, A.f.pi0, A.f.piH0, A.f.Pi0, A.f.PiH0, A.f.pi, A.f.piH, A.f.Pi,
              A.f.PiH, A.f.vcc, A.f.flux, A.clk, A.f.active, A.f.nactive, blk);
}

__global__ void __launch_bounds__(128, 8) kb_visc_update(const StepDev* __restrict__ evs,
                                                      const BItem* __restrict__ items) {
  VH_ITEM
  d_visc_update(g, A.f.pA, A.f.piH, A.f.PiH, A.f.m2, A.f.flux, A.f.Q, A.clk, blk);
}
#undef VH_ITEM

__global__ void kb_clock_op(const StepDev* __restrict__ evs, int nev, int op,
                            const int* __restrict__ ns) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nev) return;
  double* clk = evs[e].clk;
  const int n = ns ? ns[e] : 1;
  if (op == 1)
    clk[1] = clk[1] / n;
  else
    clk[1] = clk[1] * n;
}

// launch_step_ek's stages in its order, over the work table
template <int EK>
static int launch_step_batched_ek(bool viscous, const StepDev* evs, int nev, const BItem* items,
                                  int nitems, cudaStream_t s) {
  const unsigned nb = (unsigned)nitems;
  int launches = 0;
  kb_update_m<<<nb, kBatchBlock, 0, s>>>(evs, items);
  launches++;
  const dim3 fgrid(nb, 6);
  kb_face_list<<<nb, kBatchBlock, 0, s>>>(evs, items, true);
  kb_face<EK><<<fgrid, kBatchBlock, 0, s>>>(evs, items, true);
  kb_update<true, EK><<<nb, kBatchBlock, 0, s>>>(evs, items);
  kb_face_list<<<nb, kBatchBlock, 0, s>>>(evs, items, false);
  kb_face<EK><<<fgrid, kBatchBlock, 0, s>>>(evs, items, false);
  kb_update<false, EK><<<nb, kBatchBlock, 0, s>>>(evs, items);
  launches += 6;
  if (!viscous) {
    kb_ghost<true, true><<<nb, kBatchBlock, 0, s>>>(evs, items);
    launches++;
  } else {
    kb_ghost<true, false><<<nb, kBatchBlock, 0, s>>>(evs, items);
    kb_visc_prims<EK><<<dim3(nb, 2), kBatchBlock, 0, s>>>(evs, items);
    kb_is_relax<<<nb, kRelaxBlock, kRelaxSmem, s>>>(evs, items);
    kb_is_advect<<<nb, kBatchBlock, 0, s>>>(evs, items);
    kb_visc_update<<<nb, kBatchBlock, 0, s>>>(evs, items);
    kb_ghost<false, true><<<nb, kBatchBlock, 0, s>>>(evs, items);
    launches += 6;
  }
  return launches;
}

int step_ek(const EosDev& E) {
  if (E.kind == 3) return EK_TABLE3;
  if (E.kind == 6) return EK_AZH;
  if (E.kind == 7) return EK_CMFE;
  const bool chiral = E.kind == 2;
  if (E.slope) return chiral ? EK_CHIRAL_SL : EK_TABLE_SL;
  return chiral ? EK_CHIRAL : EK_TABLE;
}

int launch_step_batched(int ek, bool viscous, const StepDev* evs, int nev, const BItem* items,
                        int nitems, cudaStream_t s) {
  switch (ek) {
    case EK_TABLE3: return launch_step_batched_ek<EK_TABLE3>(viscous, evs, nev, items, nitems, s);
    case EK_AZH: return launch_step_batched_ek<EK_AZH>(viscous, evs, nev, items, nitems, s);
    case EK_CMFE: return launch_step_batched_ek<EK_CMFE>(viscous, evs, nev, items, nitems, s);
    case EK_CHIRAL_SL:
      return launch_step_batched_ek<EK_CHIRAL_SL>(viscous, evs, nev, items, nitems, s);
    case EK_TABLE_SL:
      return launch_step_batched_ek<EK_TABLE_SL>(viscous, evs, nev, items, nitems, s);
    case EK_CHIRAL: return launch_step_batched_ek<EK_CHIRAL>(viscous, evs, nev, items, nitems, s);
    default: return launch_step_batched_ek<EK_TABLE>(viscous, evs, nev, items, nitems, s);
  }
}

void launch_clock_op_batched(const StepDev* evs, int nev, int op, const int* ns, cudaStream_t s) {
  kb_clock_op<<<nblk(nev, 128), 128, 0, s>>>(evs, nev, op, ns);
}

cudaError_t step_kernels_setup() {
  cudaError_t e = cudaFuncSetAttribute(k_is_relax, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kRelaxSmem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kb_is_relax, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kRelaxSmem);
}

void launch_clock_set(double* clk, double tau, double dt, cudaStream_t s) {
  k_clock_set<<<1, 1, 0, s>>>(clk, tau, dt);
}
void launch_clock_op(double* clk, int op, int n, cudaStream_t s) {
  k_clock_op<<<1, 1, 0, s>>>(clk, op, n);
}

// ------------------------------------------------------- small helpers
__global__ void k_fill(double* __restrict__ p, long long n, double v) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// Cell::setQ (src/cll.h:75-80): a row with Q_t < 0 becomes zero.
__global__ void k_zero_negative_rows(double* __restrict__ Q, long long N) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  if (Q[i] < 0.) {
#pragma unroll
    for (int k = 0; k < 7; k++) Q[k * N + i] = 0.;
  }
}

void launch_fill(double* p, long long n, double v, cudaStream_t s) {
  if (n > 0) k_fill<<<nblk(n, 256), 256, 0, s>>>(p, n, v);
}

void launch_zero_negative_rows(double* Q, long long N, cudaStream_t s) {
  if (N > 0) k_zero_negative_rows<<<nblk(N, 256), 256, 0, s>>>(Q, N);
}

// expandGrid2x decimation (src/main.cpp:259-266): new cell (ix, iy, iz) takes
// the old cell 2*(i - n/2) + n/2 in x and y, clamped like Fluid::getCell, and
// the same iz.  ncomp component planes of N cells each.
__global__ void k_resize_gather(Geo g, const double* __restrict__ src, double* __restrict__ dst,
                                int ncomp) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  int ix, iy, iz;
  coords(g, i, ix, iy, iz);
  int sx = 2 * (ix - g.nx / 2) + g.nx / 2, sy = 2 * (iy - g.ny / 2) + g.ny / 2;
  sx = sx > 0 ? sx : 0;
  sx = sx < g.nx ? sx : g.nx - 1;
  sy = sy > 0 ? sy : 0;
  sy = sy < g.ny ? sy : g.ny - 1;
  const long long j = cidx(g, sx, sy, iz);
  for (int k = 0; k < ncomp; k++) dst[k * g.N + i] = src[k * g.N + j];
}

void launch_resize_gather(const Geo& g, const double* src, double* dst, int ncomp,
                          cudaStream_t s) {
  if (g.N > 0) k_resize_gather<<<nblk(g.N, 256), 256, 0, s>>>(g, src, dst, ncomp);
}

// Planes z0 .. z0 + nz - 1 of every listed field to or from one contiguous
// buffer laid out [field][component][plane][nx*ny] (pack = 1: fields ->
// buffer).  A z-plane of a component is contiguous (x fastest, then y),
// so a thread moves one double and consecutive threads move consecutive
// doubles of one plane.
__global__ void k_planes(PlaneFields pf, long long N, long long nxy, int z0, int nz,
                         double* __restrict__ buf, int pack) {
  const long long per = (long long)nz * nxy;  // doubles per component
  const long long total = per * pf.ncomp_total;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    long long c = t / per;
    const long long r = t - c * per;
    int f = 0;
    while (c >= pf.ncomp[f]) c -= pf.ncomp[f++];
    double* p = pf.p[f] + c * N + (long long)z0 * nxy + r;
    if (pack)
      buf[t] = *p;
    else
      *p = buf[t];
  }
}

void launch_planes(const PlaneFields& pf, long long N, long long nxy, int z0, int nz,
                   double* buf, bool pack, cudaStream_t s) {
  const long long total = (long long)nz * nxy * pf.ncomp_total;
  if (total <= 0) return;
  const long long blocks = std::min<long long>((total + 255) / 256, 148LL * 16);
  k_planes<<<(unsigned)blocks, 256, 0, s>>>(pf, N, nxy, z0, nz, buf, pack ? 1 : 0);
}

}  // namespace vh
