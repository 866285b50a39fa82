// stage1d.cuh -- one SSP-RK3 stage of 1D grids for launches that leave the GPU mostly idle.
//
// The stage kernel (stage.cuh) gives a 1D tile of 256 cells one thread per face and per
// cell.  On small grids its time is one thread's dependent chain -- five reconstructions, a
// Riemann solve and con2prim, some 2700 instructions -- on a handful of SMs, and ncu shows
// what the chain waits for: instruction fetch (34 % of warp time: every instruction of two
// inlined reconstruction sides and two inlined Riemann sides is fetched for a few warps),
// dependent loads (24 %: block map, descriptor, clock, data, then face table, up and u where
// they are used) and the barriers between its phases.  Here a tile has S1_CELLS cells and
// the work is spread over a block's threads, one short item each, in phases through shared
// memory:
//   0  the grid's descriptor in one coalesced read; then, all in flight at once (cp.async),
//      the primitives with their halo, the face table, up, u and con2prim's metric fields
//   1  (face, variable): both interface states (reconstruct_1d_core)
//   2  (face, side): physical flux, conserved state and wave speeds (HLLE), or one thread
//      per face (HLLC); meanwhile the warps without a face evaluate the metric sources
//   3  (face, variable): the HLLE combination
//   4  (cell, variable): flux divergence, RK combination
//   5  cell: con2prim
// The expressions and their order are those of the other kernels, so FP64 results are the
// same to the bit.  So are those of the mixed policies, whose multiply-add pairs the compiler
// contracts: both states of a face are one thread's work and con2prim is the same inlined
// function, whose pairs come out alike (their FP64 primitives compared before they are stored in
// FP32: 409700 of 409700 equal, random states included); the HLLE combination and the RK stage
// spell their pairs out.  (tests/test_gpu_stage1d_forms.py.)  Measured: at STAGE1D_TILES_MAX in
// grhd2_gpu.cu.
#pragma once

#include "stage.cuh"

namespace grhd {

constexpr int S1_FACES = 64, S1_CELLS = S1_FACES - 1;  // whole warps of faces
constexpr int S1_BS = 320;                             // one thread per (face, variable)
constexpr int S1_BOX = S1_CELLS + 2 * STAGE_H;
constexpr int S1_META = 13;  // con2prim's metric: gamma_ij, gamma^ij, sqrt(gamma)
constexpr int S1_SIDE_WARPS = 2 * S1_FACES / 32;
// Resident blocks per SM (96 registers): 3 (64) was 8 % slower at one tile per SM, 1 equal with
// HLLE and 5 % faster with HLLC there but 60 % slower at two tiles per SM.
constexpr int S1_MIN_BLOCKS = 2;
static_assert(S1_BS == S1_FACES * NEQ && S1_BS / 32 >= S1_SIDE_WARPS + 2, "one (face, variable) per thread");

// shared memory of a block, in order (bytes rounded to 16)
template <class R>
struct S1Layout {
  static constexpr size_t desc = 0;
  static constexpr size_t up = stage_align(desc + sizeof(GridDev));
  static constexpr size_t u = up + stage_align(sizeof(double) * NEQ * S1_CELLS);
  static constexpr size_t meta = u + stage_align(sizeof(double) * NEQ * S1_CELLS);
  static constexpr size_t src = meta + stage_align(sizeof(double) * S1_META * S1_CELLS);
  static constexpr size_t cs = src + stage_align(sizeof(double) * NEQ * S1_CELLS);  // new state, then its carry
  static constexpr size_t box = cs + stage_align(sizeof(double) * 2 * NEQ * S1_CELLS);
  static constexpr size_t table = box + stage_align(sizeof(R) * NEQ * S1_BOX);
  static constexpr size_t q = table + stage_align(sizeof(R) * NFF * S1_FACES);
  static constexpr size_t fu = q + stage_align(sizeof(R) * 2 * NEQ * S1_FACES);  // per side: flux, state, min, max speed
  static constexpr size_t flux = fu + stage_align(sizeof(R) * 2 * 12 * S1_FACES);
  static constexpr size_t total = flux + stage_align(sizeof(R) * NEQ * S1_FACES);
};

// a table in shared memory as load_face_metric / load_face_frame read one (face f of n)
template <class R>
__device__ __forceinline__ FaceMetric<R> shared_face_metric(const R *T, int f) {
  FaceMetric<R> m;
  auto ld = [&](int fld) { return T[fld * S1_FACES + f]; };
  m.alpha = ld(FF_ALPHA); m.beta_n = ld(FF_BETA_N);
  m.g11 = ld(FF_G11); m.g12 = ld(FF_G12); m.g13 = ld(FF_G13);
  m.g22 = ld(FF_G22); m.g23 = ld(FF_G23); m.g33 = ld(FF_G33);
  m.sqg = ld(FF_SQG); m.gup = ld(FF_GUP);
  return m;
}
template <class R>
__device__ __forceinline__ FaceFrame<R> shared_face_frame(const R *T, int f) {
  FaceFrame<R> fr;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int i = 0; i < 3; ++i) fr.cof[a][i] = T[(FF_COF + 3 * a + i) * S1_FACES + f];
  fr.gup = T[FF_GUP * S1_FACES + f];
  fr.ok = T[FF_FRAME_OK * S1_FACES + f] != R(0);
  return fr;
}

// con2prim's metric of cell a from shared memory
struct S1Metric {
  const double *s;
  __device__ __forceinline__ double at(int k) const { return s[k * S1_CELLS]; }
  __device__ __forceinline__ double g11() const { return at(0); }
  __device__ __forceinline__ double g12() const { return at(1); }
  __device__ __forceinline__ double g13() const { return at(2); }
  __device__ __forceinline__ double g22() const { return at(3); }
  __device__ __forceinline__ double g23() const { return at(4); }
  __device__ __forceinline__ double g33() const { return at(5); }
  __device__ __forceinline__ double i11() const { return at(6); }
  __device__ __forceinline__ double i12() const { return at(7); }
  __device__ __forceinline__ double i13() const { return at(8); }
  __device__ __forceinline__ double i22() const { return at(9); }
  __device__ __forceinline__ double i23() const { return at(10); }
  __device__ __forceinline__ double i33() const { return at(11); }
  __device__ __forceinline__ double sqg() const { return at(12); }
};
static_assert(CF_I11 == CF_G11 + 6 && CF_SQG == CF_G11 + 12, "con2prim's fields are consecutive in the centre table");

// the seed of the mixed root finder (PrimSeed) reads the cell's primitives from the box
template <class R>
struct S1Prims {
  const R *p;
  __device__ __forceinline__ double prim(int v) const { return (double)p[v * S1_BOX]; }
};

template <int REC, int RS, class R, class PT>
__global__ void __launch_bounds__(S1_BS, S1_MIN_BLOCKS)
    k_stage1d(const GridDev *__restrict__ grids, const BlockMap *__restrict__ map, int mode, int advance) {
  extern __shared__ __align__(16) unsigned char s1[];
  using L = S1Layout<R>;
  double *s_up = (double *)(s1 + L::up), *s_u = (double *)(s1 + L::u), *s_meta = (double *)(s1 + L::meta);
  double *s_src = (double *)(s1 + L::src), *s_cs = (double *)(s1 + L::cs);
  R *s_p = (R *)(s1 + L::box), *s_t = (R *)(s1 + L::table), *s_q = (R *)(s1 + L::q), *s_fu = (R *)(s1 + L::fu);
  R *s_f = (R *)(s1 + L::flux);
  const int t = (int)threadIdx.x;
  const BlockMap bm = map[blockIdx.x];

  // ---- 0. descriptor, then everything the tile reads ----------------------------------------
  {
    constexpr int words = (int)(sizeof(GridDev) / sizeof(unsigned));
    static_assert(sizeof(GridDev) % sizeof(unsigned) == 0, "copied by words");
    const unsigned *src = (const unsigned *)&grids[bm.grid];
    for (int w = t; w < words; w += S1_BS) ((unsigned *)(s1 + L::desc))[w] = __ldg(&src[w]);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous launch is complete, its writes visible
  __syncthreads();
  const GridDev &G = *(const GridDev *)(s1 + L::desc);
  const GridClock ck = *G.clock;
  const Phys &P = G.phys;
  const int nx = G.nx, i0 = (bm.first / S1_BS) * S1_CELLS + 1;  // first cell of the tile (1-based)
  const int nc = min(S1_CELLS, nx - i0 + 1), nf = nc + 1;       // cells and faces of the tile
  const PT *Pin;
  PT *Pout;
  stage_buffers(G, mode, Pin, Pout);
  const long long pl = G.pplane;
  int lo, hi;
  stencil_range(REC, P.sensor, lo, hi);
  {
    const int ia = i0 - 3 + lo, ib = i0 + nc - 3 + hi;  // cells the faces read
    for (int pos = t; pos < NEQ * S1_BOX; pos += S1_BS) {
      const int v = pos / S1_BOX, i = i0 - STAGE_H + (pos - v * S1_BOX);
      if (i >= 1 && i <= nx && i >= ia && i <= ib) cp_async<sizeof(PT)>(&s_p[pos], &Pin[v * pl + (i - 1)]);
    }
    if (t < 2 * STAGE_H) {  // boundary fill of the cells outside the domain (coherent: Pin was written
                            // while this block was resident)
      const int i = t < STAGE_H ? i0 - STAGE_H + t : i0 + nc + (t - STAGE_H);
      if ((i < 1 || i > nx) && i >= ia && i <= ib) {
        double b[NEQ];
        load_cell<1, true>(Pin, G, i, 1, 1, b);
#pragma unroll
        for (int v = 0; v < NEQ; ++v) s_p[v * S1_BOX + (i - (i0 - STAGE_H))] = R(b[v]);
      }
    }
    const R *T = face_table<R>(G, 0);
    const long long ntab = G.nface[0];
    constexpr int nfld = RS == RS_HLLC ? NFF : FF_COF + 1;  // HLLE: the metric, and the flag in slot FF_COF
    for (int pos = t; pos < nfld * S1_FACES; pos += S1_BS) {
      const int k = pos / S1_FACES, f = pos - k * S1_FACES;
      const int fld = RS == RS_HLLC ? k : (k == FF_COF ? FF_ZERO : k);
      if (f < nf) cp_async<sizeof(R)>(&s_t[pos], &T[fld * ntab + (i0 - 1 + f)]);
    }
    for (int pos = t; pos < NEQ * S1_CELLS; pos += S1_BS) {
      const int v = pos / S1_CELLS, a = pos - v * S1_CELLS;
      if (a < nc) {
        cp_async<8>(&s_up[pos], &G.UP[v * pl + (i0 - 1 + a)]);
        if (mode >= 2) cp_async<8>(&s_u[pos], &G.U[v * pl + (i0 - 1 + a)]);
      }
    }
    for (int pos = t; pos < S1_META * S1_CELLS; pos += S1_BS) {
      const int k = pos / S1_CELLS, a = pos - k * S1_CELLS;
      if (a < nc) cp_async<8>(&s_meta[pos], &G.centre[(CF_G11 + k) * G.nij + (i0 - 1 + a)]);
    }
    cp_async_commit();
  }
  const bool skip = clock_skip(ck);  // the same for the whole block (one grid)
  const double dt = clock_dt(ck);
  cp_async_wait<0>();
  __syncthreads();
  if (skip) return;

  // ---- 1. interface states ---------------------------------------------------------------------
  unsigned clamps = 0;
  {
    const int v = t / S1_FACES, f = t - v * S1_FACES, face = i0 - 1 + f;
    if (f < nf) {
      int br = BR_GODUNOV;
      if (REC != REC_GODUNOV) {
        R rho[5], pr[5];
        const bool sensor = P.sensor != 0;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          rho[m] = sensor ? s_p[EQ_DE * S1_BOX + f + m] : R(0);
          pr[m] = sensor ? s_p[EQ_PR * S1_BOX + f + m] : R(0);
        }
        br = branch_of<REC>(P, rho, pr, face, nx, 1);
      }
      R s6[6], l, r;
#pragma unroll
      for (int m = 0; m < 6; ++m) s6[m] = (m >= lo && m <= hi) ? s_p[v * S1_BOX + f + m] : R(0);
      recon_one<REC>(br, P.lim, s6, l, r);
      if (v == EQ_DE || v == EQ_PR) {  // reconstruction.f90:647-655
        const R fl = v == EQ_DE ? R(P.rho_floor) : R(P.p_floor);
        if (f < S1_CELLS || face == nx)  // the tile that holds the upper cell counts
          clamps = (unsigned)!(l >= fl) + (unsigned)!(r >= fl);
        l = rmax(l, fl);
        r = rmax(r, fl);
      }
      s_q[v * S1_FACES + f] = l;
      s_q[(NEQ + v) * S1_FACES + f] = r;
    }
  }
  count_add(G.cnt, CNT_RECON_CLAMP, clamps);
  __syncthreads();

  // ---- 2. Riemann sides (or HLLC faces) and metric sources ---------------------------------------
  constexpr int face_threads = RS == RS_HLLC ? S1_FACES : 2 * S1_FACES;
  bool hll = true;  // HLLE combination wanted for this thread's face (HLLC: it fell back)
  if (t < face_threads) {
    const int side = t / S1_FACES, f = t - side * S1_FACES;
    if (f < nf) {
      const bool zero = s_t[(RS == RS_HLLC ? FF_ZERO : FF_COF) * S1_FACES + f] != R(0);  // evolution.f90:69-71
      const FaceMetric<R> m = shared_face_metric(s_t, f);
      if (RS == RS_HLLC) {
        R qL[NEQ], qR[NEQ], flux[NEQ] = {R(0), R(0), R(0), R(0), R(0)};
#pragma unroll
        for (int v = 0; v < NEQ; ++v) { qL[v] = s_q[v * S1_FACES + f]; qR[v] = s_q[(NEQ + v) * S1_FACES + f]; }
        hll = false;
        if (!zero) {
          hll = hllc_try(P, qL, qR, 1, m, shared_face_frame(s_t, f), flux);
          if (hll) hlle(P, qL, qR, 1, m, flux);
        }
#pragma unroll
        for (int v = 0; v < NEQ; ++v) s_f[v * S1_FACES + f] = flux[v];
        hll = hll && (f < S1_CELLS || i0 - 1 + f == nx);
      } else if (!zero) {
        R q[NEQ], ff[NEQ], uu[NEQ], wmin, wmax;
#pragma unroll
        for (int v = 0; v < NEQ; ++v) q[v] = s_q[(side * NEQ + v) * S1_FACES + f];
        flux_and_cons_bare(P, q, 1, m, ff, uu);
        wavespeeds(P, q, 1, m, wmin, wmax);
        R *o = s_fu + side * 12 * S1_FACES + f;
#pragma unroll
        for (int v = 0; v < NEQ; ++v) { o[v * S1_FACES] = ff[v]; o[(NEQ + v) * S1_FACES] = uu[v]; }
        o[10 * S1_FACES] = wmin;
        o[11 * S1_FACES] = wmax;
      }
    } else {
      hll = false;
    }
    if (RS == RS_HLLC) count_add(G.cnt, CNT_HLLC_FALLBACK, hll ? 1u : 0u);
  } else if (!P.srhd) {
    const int a = t - face_threads;
    if (a < nc) {
      const long long ij = i0 - 1 + a;
      double q[NEQ], src[NEQ];
#pragma unroll
      for (int v = 0; v < NEQ; ++v) q[v] = (double)s_p[v * S1_BOX + STAGE_H + a];
      const auto cr = global_col(centre_table<R>(G), G, ij);
      if constexpr (sizeof(R) == sizeof(float)) {
        sources<R>(P, cr, q, src, __ldg(&G.centre[CF_ALPHA * G.nij + ij]), s_meta[12 * S1_CELLS + a]);
      } else {
        sources<R>(P, cr, q, src, 0.0, 0.0);
      }
#pragma unroll
      for (int v = 0; v < NEQ; ++v) s_src[v * S1_CELLS + a] = src[v];
    }
  }
  __syncthreads();

  // From here on the next stage's blocks may take their places: they read map and descriptor,
  // which no kernel writes, and wait for this launch to complete.  At the kernel's entry instead
  // they would hold places, idle, that another stream's or group's stage could use: two batches of
  // 287 tiles on two streams 85 us (tubes, FP64), 155 (HLLC) and 77 (Michel) against 85, 134 and
  // 73 from here; two of 136 Michel tiles 51 against 44; a batch alone the same.
  asm volatile("griddepcontrol.launch_dependents;");

  // ---- 3. the HLLE flux of one variable -----------------------------------------------------------
  if (RS == RS_HLLE) {
    const int v = t / S1_FACES, f = t - v * S1_FACES;
    if (f < nf) {
      R flux = R(0);
      if (s_t[FF_COF * S1_FACES + f] == R(0)) {
        const R *l = s_fu + f, *r = s_fu + 12 * S1_FACES + f;
        const R ap = rmax(rmax(R(0), l[11 * S1_FACES]), r[11 * S1_FACES]);
        const R am = rmin(rmin(R(0), l[10 * S1_FACES]), r[10 * S1_FACES]);
        const R sqg = s_t[FF_SQG * S1_FACES + f];
        if (!(fabs(ap - am) < R(1.0e-14))) {
          const R inv = sizeof(R) == sizeof(float) ? R(1) / (ap - am) : R(0);
          flux = hlle_combine(ap, am, inv, sqg, l[v * S1_FACES], r[v * S1_FACES], l[(NEQ + v) * S1_FACES],
                              r[(NEQ + v) * S1_FACES]);
        }
      }
      s_f[v * S1_FACES + f] = flux;
    }
    __syncthreads();
  }

  // ---- 4. flux divergence and RK combination of one variable ---------------------------------------
  {
    const int v = t / S1_CELLS, a = t - v * S1_CELLS;
    if (v < NEQ && a < nc) {
      const R hiF = s_f[v * S1_FACES + a + 1], loF = s_f[v * S1_FACES + a];
      const double src = P.srhd ? 0.0 : s_src[v * S1_CELLS + a];
      const double rhs = (double)(div_pos(-(hiF - loF), R(G.dx)) + src);
      const double up = s_up[v * S1_CELLS + a];
      const long long k = v * pl + (i0 - 1 + a);
      double nv, low = 0.0;
      if (sizeof(PT) == sizeof(float) && G.carry != 0) {
        rk_compensated(G, k, mode, dt, up, mode >= 2 ? s_u[v * S1_CELLS + a] : 0.0, rhs, nv, low);
      } else if (mode == 1) {
        G.U[k] = up;  // u = up (grhd2.f90:232)
        nv = up + rhs * dt;
      } else if (mode == 2) {
        const double u = s_u[v * S1_CELLS + a], x = up + rhs * dt;
        // mixed: the multiply-add pair the compiler contracts in the other kernels, spelled out
        if (sizeof(PT) == sizeof(float)) nv = fma(0.75, u, 0.25 * x);
        else nv = 0.75 * u + 0.25 * x;
      } else {
        nv = (s_u[v * S1_CELLS + a] + 2.0 * (up + rhs * dt)) / 3.0;
      }
      s_cs[v * S1_CELLS + a] = nv;
      if (sizeof(PT) == sizeof(float)) s_cs[(NEQ + v) * S1_CELLS + a] = low;
    }
  }
  __syncthreads();

  if (advance && t == S1_BS - 1) advance_when_done(G.clock, (unsigned)((nx + S1_CELLS - 1) / S1_CELLS));

  // ---- 5. con2prim ---------------------------------------------------------------------------------
  if (t >= nc) return;
  const S1Metric cm{s_meta + t};
  double cs[NEQ], pr[NEQ];
#pragma unroll
  for (int v = 0; v < NEQ; ++v) cs[v] = s_cs[v * S1_CELLS + t];
  unsigned fl;
  if constexpr (sizeof(PT) == sizeof(float)) {
    const S1Prims<R> in{s_p + STAGE_H + t};
    fl = cons_to_prim(P, cm, cs, pr, PrimSeed<S1Prims<R>, S1Metric>{in, cm});
  } else {
    fl = cons_to_prim(P, cm, cs, pr);
  }
  const long long c = i0 - 1 + t;
#pragma unroll
  for (int v = 0; v < NEQ; ++v) {
    G.UP[v * pl + c] = cs[v];
    Pout[v * pl + c] = (PT)pr[v];
  }
  if (sizeof(PT) == sizeof(float) && G.carry != 0) {  // a value con2prim changed starts without a carry
#pragma unroll
    for (int v = 0; v < NEQ; ++v)
      store_carry(G, G.UPc, v * pl + c, cs[v] == s_cs[v * S1_CELLS + t] ? s_cs[(NEQ + v) * S1_CELLS + t] : 0.0);
  }
  c2p_count(G.cnt, fl);
}

}  // namespace grhd
