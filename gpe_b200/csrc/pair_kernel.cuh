// pair_kernel.cuh -- two Runge-Kutta stages per launch.
//
// A step of rk4 is two launches and a step of rk2 one (src/solve.f90:78-154):
// the first stage of a pair is evaluated on the tile and a ring of R = order/2
// sites around it, its result stays in shared memory, and the second stage
// takes its neighbours from there.  With d2 = dt/2 f(psi), d3 = dt/2 f(psi+d2),
// d4 = dt f(psi+d3) (the increment form of stage_kernel.cuh) the pairs are
//   PAIR_RK4_A: d2, d3 -> u3 = psi + d3 and acc = d2/3 + 2 d3/3
//   PAIR_RK4_B: d4 and f(psi + d4) -> psi' = psi + [dt/6 f + d4/3 + acc]
//   PAIR_RK2:   u = psi + dt/2 f(psi) -> psi' = psi + dt f(u)
// (psi' Kahan-compensated when KAHAN).  Fields moved per site: A reads psi and
// writes u3, acc; B reads u3, psi, acc (c) and writes psi' (c): 9 (7 without
// compensation) against 15 (13) with one stage per launch.  The operations on
// a site are those of stage_kernel.cuh in the same order, so the two forms of
// a step leave the same bits (u3 is the sum psi + d3 that the one-stage form
// adds as it reads).
//
// Tiling: a CTA owns 64 x TY sites in (x, y) and marches a chunk of z-planes.
// Interior warps own ROWS adjacent rows (two consecutive x sites per lane) in
// both stages; ring warps evaluate the first stage on the 2R rows above and
// below the tile and the one site pair left and right of each row (the star
// of the second stage needs no corners).  One more warp is the producer: it
// streams, per plane, one TMA box of the stencil field with a halo of 2R (and
// of psi with a halo of R, and the pointwise tiles) into a ring of S slots.
// The first stage of plane f = k - R runs when plane k has arrived, the second
// of plane z = f - R right after it: the planes above and below come from
// register queues in both.  The first stage's values pass through U_SLOTS
// (5) shared planes; a warp arrives on a barrier when its part of plane f is
// written and waits for the one of plane f - 1, so warps may be a plane apart
// (with R >= 1 the second stage reads plane f - R at the latest; the slot
// overwritten next, plane f - 4, was read by every warp before it arrived for
// plane f - 1).
//
// The kernel writes the interior; fill_ghosts_kernel then fills the ghosts,
// edges of the box included (with the ghost stores in its five-fold unrolled
// loop the kernel missed the instruction cache: 425 against 148 us at 256^3;
// the first stage
// is evaluated on ghost sites too, where it equals its image: the star's sums
// are symmetric, the per-axis tables hold the image's entries and the one
// antisymmetric term, the x gradient, takes the mirrored sign).  Equation 3's
// sphere mask has no pair kernel.
//
// What bounds it, at 512^3 in complex64, order 4, compensated: pair A (0.895 ms,
// 24 B/site: 0.55 of the copy rate) the L1 data pipe, 86% busy, with 1.33
// first-stage sites per site; pair B (1.44 ms, 48 B/site: 0.68) the latency of
// its planes, of which shared memory holds four, one in flight.  DRAM carries the
// bytes counted above and no more.  complex128 is bound by the registers: 12 warps
// of 168.  A step of rk4, one stage per launch -> in pairs, ghosts and norm
// included: 512^3 complex64 compensated order 4 2930 -> 2430 us; 256^3 the same
// 477 -> 351, at order 2 409 -> 278; 256^3 complex128 order 4 1163 -> 737, order 2
// 813 -> 454; 64^3 complex128 order 2 41 -> 30 (24 with overlapped launches).
#pragma once

#include "device_utils.cuh"
#include "rhs.cuh"
#include "stage_kernel.cuh"
#include "vec2.cuh"

namespace gpe {

enum : int { PAIR_RK4_A = 0, PAIR_RK4_B = 1, PAIR_RK2 = 2 };

constexpr int U_SLOTS = 5;   // planes of first-stage values in shared memory
constexpr int PT_SLOTS = 2;  // planes of pointwise tiles: one used, one in flight

// Rows of an interior warp, and the widths (sites) of the staged boxes: 72 and
// 68 are needed; the rows are widened so that the ring's column accesses, one
// row apart per lane, fall into different banks.
template <typename T>
struct PairTile;
template <>
struct PairTile<float> {
  static constexpr int ROWS = 1, BW = 74, UW = 70, TY_MAX = 16;
};
template <>
struct PairTile<double> {
  static constexpr int ROWS = 1, BW = 73, UW = 69, TY_MAX = 8;
};

// Ring positions in units of one row of 32 site pairs: R rows below, R above,
// and one unit for the pairs left and right of the tile's rows; two units per
// ring warp (at R = 2, with the producer, 20 warps of 96 registers in complex64
// and 12 of 168, three per scheduler, in complex128).
constexpr int RING_UNITS = 2;
__host__ __device__ constexpr int pair_ring_warps(int r) { return (2 * r + 1 + RING_UNITS - 1) / RING_UNITS; }
template <typename T>
__host__ __device__ constexpr int pair_warps(int r, int ty) {
  return ty / PairTile<T>::ROWS + pair_ring_warps(r);
}
template <typename T>
__host__ __device__ constexpr int pair_max_threads(int r) {
  return 32 * (pair_warps<T>(r, PairTile<T>::TY_MAX) + 1);
}

// Increments d of planes f - R .. f: in registers, or (complex64 at order 4,
// whose queues fill the registers) in shared memory, each lane its own.
template <typename T>
__host__ __device__ constexpr bool pair_d_in_smem(int r, int kind) {
  return sizeof(T) == 4 && r == 2 && kind != PAIR_RK2;
}

template <typename T>
struct PairParams {
  // maps: halo = stencil field (box BW x (TY+4R)), halo2 = psi with a halo of R
  // (UW x (TY+2R), PAIR_RK4_B), pt[0] = acc (PAIR_RK4_B), pt[1] = compensation
  RunDesc<T, T> run;         // single-run launch
  const RunDesc<T, T>* runs;  // batched launch: per-run descriptors
  const WorkItem* items;      // batched launch: the work list,
  const int* starts;          // and where in it each CTA's items start
  int nitems;
  int TY, stages;
  // bytes a box delivers, offsets in a slot, strides of the three rings
  // (stencil and psi planes, pointwise tiles, u planes) and their offsets
  unsigned s_bytes, base_bytes, pt_bytes;
  unsigned base_off, comp_off, slot_stride, pt_stride, u_stride;
  unsigned pt_ring, u_ring, d_ring;
  T a_r[2], a_i[2];  // the two stages' coefficient of K (carries dt)
  double* partials;  // 2 doubles per work item
  int* status;
  unsigned long long wait_limit_ns;
  int stall_plane;
};

template <typename T, int R, int KIND, bool KAHAN, int FORM, bool BATCH>
__device__ __forceinline__ void pair_body(const PairParams<T>& p) {
  using V = typename VT<T>::T;
  using RD = RunDesc<T, T>;
  using PT = PairTile<T>;
  constexpr bool FULL = FORM == FORM_FULL, TRAP = FORM == FORM_TRAP;
  constexpr int ROWS = PT::ROWS, BW = PT::BW, UW = PT::UW;
  constexpr int W = (int)(sizeof(T) / 4);  // 8-byte TMA units per complex
  constexpr int QN = 2 * R + 1;
  constexpr unsigned ES = 2 * sizeof(T);
  constexpr bool B4 = KIND == PAIR_RK4_B;
  constexpr bool NORM = KIND != PAIR_RK4_A;
  constexpr int NPT = (B4 ? 1 : 0) + (KAHAN ? 1 : 0);
  static_assert(!(KAHAN && KIND == PAIR_RK4_A), "the first pair of rk4 has no compensation");
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_abort, s_issued, s_pissued, s_stop;
  __shared__ double s_red[16];

  const int TY = p.TY, S = p.stages;
  const int NI = TY / ROWS;             // interior warps
  const int NC = NI + pair_ring_warps(R);  // + ring warps; warp NC produces
  const int lane = threadIdx.x, warp = threadIdx.y, tid = warp * 32 + lane;

  auto item_of = [&](int it) -> WorkItem {
    if (BATCH) return p.items[it];
    const int ntiles = p.run.ntx * p.run.nty;
    const int ch = it / ntiles;
    const int z0 = ch * p.run.zchunk;
    return WorkItem{0, it - ch * ntiles, z0, min(z0 + p.run.zchunk, p.run.nz)};
  };
  const int it0 = BATCH ? p.starts[blockIdx.x] : (int)blockIdx.x;
  const int it1 = BATCH ? p.starts[blockIdx.x + 1] : p.nitems;
  const int its = BATCH ? 1 : (int)gridDim.x;
  auto run_of = [&](const WorkItem& w) -> const RD& {
    if (BATCH) return p.runs[w.run];
    return p.run;
  };

  // shared memory: full[8], empty[8], ubar[2], pfull[2], pempty[2], then the
  // three rings
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + 8;
  uint64_t* ubar = empty + 8;
  uint64_t* pfull = ubar + 2;
  uint64_t* pempty = pfull + PT_SLOTS;
  unsigned char* sbase = smem + 256;

  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], (uint32_t)NC);
    }
    mbar_init(&ubar[0], (uint32_t)NC);
    mbar_init(&ubar[1], (uint32_t)NC);
    for (int s = 0; s < PT_SLOTS; s++) {
      mbar_init(&pfull[s], 1);
      mbar_init(&pempty[s], (uint32_t)NI);
    }
    fence_mbar_init();
    s_abort = 0;
    s_issued = 0;
    s_pissued = 0;
    s_stop = 0;
  }
  __syncthreads();
  after_previous();

  if (warp == NC) {
    // ---------------- producer warp: lane 0 streams the planes -------------
    if (lane == 0) {
      int slot = 0, issued = 0, pissued = 0;
      uint32_t cyc = 0;  // completed passes over the ring
      bool stop = false;
      for (int it = it0; it < it1 && !stop; it += its) {
        const WorkItem w = item_of(it);
        const RD& rd = run_of(w);
        const int tile_x = w.tile % rd.ntx, tile_y = w.tile / rd.ntx;
        const int niters = (w.z1 - w.z0) + 3 * R;
        prefetch_tmap(&rd.maps.halo);
        if (B4) {
          prefetch_tmap(&rd.maps.halo2);
          prefetch_tmap(&rd.maps.pt[0]);
        }
        if (KAHAN) prefetch_tmap(&rd.maps.pt[1]);
        for (int u = 0; u < niters; u++) {
          if (u == p.stall_plane) {  // failure-detection test: never loaded
            stop = true;
            break;
          }
          if (cyc > 0) {
            if (!mbar_wait_bounded(&empty[slot], (cyc - 1) & 1u, p.wait_limit_ns)) {
              s_abort = 1;
              atomicExch(p.status, 6);
              stop = true;
              break;
            }
            fence_proxy_async();
          }
          unsigned char* st = sbase + (size_t)slot * p.slot_stride;
          const bool with_base = B4 && u >= R;
          mbar_arrive_expect_tx(&full[slot], p.s_bytes + (with_base ? p.base_bytes : 0u));
          // stencil plane k = z0 - R + u, psi at f = k - R
          tma_load_3d(st, &rd.maps.halo, &full[slot], W * (tile_x * TX + GH - 4),
                      tile_y * TY + GH - 2 * R, w.z0 - R + u + GH);
          if (with_base)
            tma_load_3d(st + p.base_off, &rd.maps.halo2, &full[slot], W * (tile_x * TX + GH - 2),
                        tile_y * TY + GH - R, w.z0 - 2 * R + u + GH);
          if (NPT > 0 && u >= 3 * R) {
            // pointwise tiles of z = f - R, two planes deep
            const int ps = pissued % PT_SLOTS, pc = pissued / PT_SLOTS;
            if (pc > 0) {
              if (!mbar_wait_bounded(&pempty[ps], (pc - 1) & 1u, p.wait_limit_ns)) {
                s_abort = 1;
                atomicExch(p.status, 6);
                s_issued = ++issued;  // the plane's own loads are in flight
                stop = true;
                break;
              }
              fence_proxy_async();
            }
            unsigned char* pt = smem + p.pt_ring + (size_t)ps * p.pt_stride;
            mbar_arrive_expect_tx(&pfull[ps], NPT * p.pt_bytes);
            if (B4)
              tma_load_3d(pt, &rd.maps.pt[0], &pfull[ps], W * (tile_x * TX + GH), tile_y * TY + GH,
                          w.z0 - 3 * R + u + GH);
            if (KAHAN)
              tma_load_3d(pt + p.comp_off, &rd.maps.pt[1], &pfull[ps], W * (tile_x * TX + GH),
                          tile_y * TY + GH, w.z0 - 3 * R + u + GH);
            s_pissued = ++pissued;
          }
          s_issued = ++issued;
          if (++slot == S) {
            slot = 0;
            ++cyc;
          }
          if (*(volatile int*)&s_abort) {
            stop = true;
            break;
          }
        }
      }
    }
  } else {
    // ------------------------------ compute warps ------------------------------
    const bool interior = warp < NI;
    // the warp's units: ROWS rows of 32 site pairs (interior), or ring units
    constexpr int NU = RING_UNITS;
    static_assert(ROWS <= NU, "interior rows fit the unit arrays");
    // A complex128 pair is two 16-byte accesses 16 bytes apart, lanes 32 bytes
    // apart: in each group of eight lanes the upper four take their second site
    // first (sel = 1: e = 0 is site x + 1), so that the group covers all banks
    // (taken in order, half of them twice: 95% of the L1 data pipe's time).
    constexpr bool D = sizeof(T) == 8;
    int urow[NU], ucol[NU], sel[NU];
    bool act[NU];
#pragma unroll
    for (int rr = 0; rr < NU; rr++) {
      if (interior) {
        urow[rr] = warp * ROWS + (rr < ROWS ? rr : 0);
        ucol[rr] = 2 * lane;
        act[rr] = rr < ROWS;
        sel[rr] = D ? (lane >> 2) & 1 : 0;
      } else {
        const int q = (warp - NI) * NU + rr;
        ucol[rr] = 2 * lane;
        act[rr] = q <= 2 * R;
        sel[rr] = D && q < 2 * R ? (lane >> 2) & 1 : 0;
        if (q < R) {
          urow[rr] = -(q + 1);
        } else if (q < 2 * R) {
          urow[rr] = TY + (q - R);
        } else {  // the pairs left (lanes below TY) and right of the rows
          act[rr] = q == 2 * R && lane < 2 * TY;
          urow[rr] = act[rr] ? (lane < TY ? lane : lane - TY) : 0;
          ucol[rr] = act[rr] ? (lane < TY ? -2 : TX) : 0;
        }
      }
    }
    const V ar0 = vsplat(p.a_r[0]), ax0 = vpair(-p.a_i[0], p.a_i[0]);
    const V ar1 = vsplat(p.a_r[1]), ax1 = vpair(-p.a_i[1], p.a_i[1]);
    const V third = vsplat((T)(1.0 / 3.0)), twothird = vsplat((T)(2.0 / 3.0));
    const V mone = vsplat(T(-1));

    int slot = 0, cslot = 0;  // slots of planes k and f
    uint32_t phase = 0, g = 0;  // g: first-stage planes so far (all items)
    unsigned gp = 0;            // pointwise planes so far
    // shared-memory offsets of slots k and f and of u planes g and g - R
    const unsigned s_first = 256u;
    const unsigned u_end = p.u_ring + U_SLOTS * p.u_stride;
    unsigned so = s_first, fo = s_first, uo = p.u_ring,
             zo = p.u_ring + (U_SLOTS - R) * p.u_stride;

    for (int it = it0; it < it1; it += its) {
      const WorkItem w = item_of(it);
      const RD& rd = run_of(w);
      const int nx = rd.nx, ny = rd.ny, bcs = rd.bcs;
      const int tile_x = w.tile % rd.ntx, tile_y = w.tile / rd.ntx;
      const int z0 = w.z0;
      const int niters = (w.z1 - w.z0) + 3 * R;
      const size_t Nx = (size_t)rd.Nx, NxNy = (size_t)rd.Nx * (size_t)rd.Ny;
      const T c0s = rd.c0, cns = rd.cn, cVs = rd.cV;
      const FullTerms<T> ft = {rd.c0, rd.cV, rd.cn, rd.ar0, rd.ard, rd.ai, rd.gx1, rd.gx2};
      const int useV = rd.use_V, useD = rd.use_diss, useG = rd.use_grad;
      const LapCoef<V> lc = {vsplat(rd.cx1), vsplat(rd.cx2), vsplat(rd.cy1), vsplat(rd.cy2),
                             vsplat(rd.cz1), vsplat(rd.cz2), vsplat(rd.c0lap)};
      const V cLv = vsplat(rd.cL);
      // per-unit constants of this item
      T Vxy[NU][2], Dxy[NU][2], Us[NU][2];
#pragma unroll
      for (int rr = 0; rr < NU; rr++) {
        const int i = tile_x * TX + ucol[rr], j = tile_y * TY + urow[rr];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int ie = i + (e ^ sel[rr]);
          Vxy[rr][e] = Dxy[rr][e] = Us[rr][e] = T(0);
          if (TRAP || (FULL && useV)) Vxy[rr][e] = rd.tabV[0][ie] + rd.tabV[1][j];
          if (FULL && useD) Dxy[rr][e] = rd.tabD[0][ie] + rd.tabD[1][j];
          // beyond a mirror the gradient of the image has the other sign
          if (FULL) Us[rr][e] = (bcs == 2 && (ie < 0 || ie >= nx)) ? -rd.U : rd.U;
        }
      }

      // right-hand side of one site of unit rr in plane z
      auto rhs = [&](const Star<V>& st, int rr, int e, T Vz, T Dz) -> V {
        const V L = star_laplacian<R>(st, lc);
        if (!FULL)
          return rhs_plain<TRAP>(L, st.f0, TRAP ? Vxy[rr][e] + Vz : T(0), c0s, cVs, cns, cLv);
        return rhs_full<R>(st, L, cLv, ft, useV ? Vxy[rr][e] + Vz : T(0), useD != 0,
                           Dxy[rr][e] + Dz, useG != 0, Us[rr][e]);
      };
      // star of site e of a pair: c the pair, xa and xc the pairs left and right
      auto star = [&](int e, int sl, const CPair<T>& c, const CPair<T>& xa, const CPair<T>& xc,
                      const CPair<T>& ym1, const CPair<T>& yp1, const CPair<T>& ym2,
                      const CPair<T>& yp2, const CPair<T>& zm1, const CPair<T>& zp1,
                      const CPair<T>& zm2, const CPair<T>& zp2) -> Star<V> {
        Star<V> s;
        s.f0 = e ? c.b : c.a;
        if (D) {
          // all three pairs come in this lane's order (sel): the distance-2
          // neighbours are of the same e, one distance-1 neighbour is the
          // pair's other site and the other one is chosen by sel
          const V own = e ? c.a : c.b;
          const V far = e ? vsel(sl, xa.a, xc.a) : vsel(sl, xc.b, xa.b);
          const bool up = (e != 0) == (sl != 0);  // the other site is x + 1 of this one
          s.xp1 = FULL ? vsel(up, own, far) : own;
          s.xm1 = FULL ? vsel(up, far, own) : far;
          s.xm2 = e ? xa.b : xa.a;
          s.xp2 = e ? xc.b : xc.a;
        } else {
          s.xm1 = e ? c.a : xa.b;
          s.xp1 = e ? xc.a : c.b;
          s.xm2 = e ? xa.b : xa.a;
          s.xp2 = e ? xc.b : xc.a;
        }
        s.ym1 = e ? ym1.b : ym1.a;
        s.yp1 = e ? yp1.b : yp1.a;
        s.ym2 = e ? ym2.b : ym2.a;
        s.yp2 = e ? yp2.b : yp2.a;
        s.zm1 = e ? zm1.b : zm1.a;
        s.zp1 = e ? zp1.b : zp1.a;
        s.zm2 = e ? zm2.b : zm2.a;
        s.zp2 = e ? zp2.b : zp2.a;
        return s;
      };
      // a pair in shared memory: `a` points at the lane's first access, which
      // is its second site for sel = 1 (`o` the way to the other one)
      auto ld = [&](const unsigned char* a, int o) -> CPair<T> {
        if constexpr (D)
          return {*reinterpret_cast<const V*>(a), *reinterpret_cast<const V*>(a + o)};
        else
          return ld_cpair<T, T>(reinterpret_cast<const T*>(a));
      };
      auto st = [&](unsigned char* a, int o, V x, V y) {
        if constexpr (D) {
          *reinterpret_cast<V*>(a) = x;
          *reinterpret_cast<V*>(a + o) = y;
        } else {
          st_cpair<T, V>(reinterpret_cast<T*>(a), x, y);
        }
      };

      // z-queue of the stencil field, one per unit: push number c sits in
      // slot c % QN, and plane f + d in slot (KK + d + QN) % QN
      CPair<T> q[NU][QN];
#pragma unroll
      for (int rr = 0; rr < NU; rr++) {
        const int i = tile_x * TX + ucol[rr] + GH, j = tile_y * TY + urow[rr] + GH;
        const bool in = act[rr] && i + 1 < rd.Nx && j < rd.Ny;
#pragma unroll
        for (int c = 0; c < QN; c++) {
          CPair<T> v = {vsplat(T(0)), vsplat(T(0))};
          if (c < R && in) {
            v = ld_cpair<T, T>(rd.stencil +
                               2 * ((size_t)(z0 - 2 * R + c + GH) * NxNy + (size_t)j * Nx + (size_t)i));
            if (sel[rr]) v = {v.b, v.a};
          }
          q[rr][c] = v;
        }
      }
      int t = 0;
      double red0 = 0.0;
      bool aborted = false;

      // waits shared by both kinds of warp; false: the wait ran out
      auto wait_plane = [&]() -> bool {
        if (mbar_wait_bounded(&full[slot], phase, p.wait_limit_ns)) return true;
        s_abort = 1;
        atomicExch(p.status, 6);
        return false;
      };
      auto publish = [&]() {  // this warp's part of u plane g is written
        __syncwarp();
        if (lane == 0) mbar_arrive(&ubar[g & 1u]);
      };
      auto wait_u = [&]() -> bool {  // u plane g - 1 is whole
        if (g == 0) return true;
        if (mbar_wait_bounded(&ubar[(g - 1) & 1u], ((g - 1) >> 1) & 1u, p.wait_limit_ns))
          return true;
        s_abort = 1;
        atomicExch(p.status, 6);
        return false;
      };
      auto finish_plane = [&]() {
        if (t >= R) {  // plane f is no longer read by this warp
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[cslot]);
          fo += p.slot_stride;
          if (++cslot == S) {
            cslot = 0;
            fo = s_first;
          }
          ++g;
          uo += p.u_stride;
          if (uo == u_end) uo = p.u_ring;
          zo += p.u_stride;
          if (zo == u_end) zo = p.u_ring;
        }
        so += p.slot_stride;
        if (++slot == S) {
          slot = 0;
          so = s_first;
          phase ^= 1u;
        }
        ++t;
      };

      if (interior) {
        const int i0 = tile_x * TX + 2 * lane;
        const int j0 = tile_y * TY + warp * ROWS;
        const int sl = sel[0], oth = 16 - 32 * sl;  // bytes from the first access to the other
        const unsigned s_off = ES * (unsigned)((warp * ROWS + 2 * R) * BW + 2 * lane + 4 + sl);
        const unsigned u_off = ES * (unsigned)((warp * ROWS + R) * UW + 2 * lane + 2 + sl);
        const unsigned pt_off = ES * (unsigned)(warp * ROWS * TX + 2 * lane + sl);
        bool ok[ROWS][2];
        double Wxy[ROWS][2];
#pragma unroll
        for (int rr = 0; rr < ROWS; rr++) {
          const int j = j0 + rr;
          Wxy[rr][0] = Wxy[rr][1] = 0.0;
          if (NORM) {
            Wxy[rr][0] = rd.tabW[0][i0 + sl] * rd.tabW[1][j];
            Wxy[rr][1] = rd.tabW[0][i0 + (1 ^ sl)] * rd.tabW[1][j];
          }
          ok[rr][0] = i0 + sl < nx && j < ny;
          ok[rr][1] = i0 + (1 ^ sl) < nx && j < ny;
        }
        T* const out0 = rd.out[0];
        T* const out1 = rd.out[1];
        size_t base = (size_t)(z0 + GH) * NxNy + (size_t)(j0 + GH) * Nx + (size_t)(i0 + sl + GH);
        const int o1 = 2 * (1 - 2 * sl);  // scalars from site e = 0 to e = 1
        auto store = [&](T* o, const bool* okr, const V* r) {
          if constexpr (D) {
            if (okr[0]) st_c1<T>(o, r[0]);
            if (okr[1]) st_c1<T>(o + o1, r[1]);
          } else {
            if (okr[1]) st_cpair<T, V>(o, r[0], r[1]);
            else if (okr[0]) st_c1<T>(o, r[0]);
          }
        };
        // u queue: the plane pushed at iteration t sits in slot (t - R) % QN,
        // plane z + d in (KK - 2R + d + 4 QN) % QN; d queue shifts
        constexpr bool DS = pair_d_in_smem<T>(R, KIND);
        const unsigned d_plane = ES * (unsigned)(TY * TX);
        unsigned d_at = 0;  // d ring: plane g % (R + 1)
        CPair<T> uq[ROWS][QN], dq[ROWS][R + 1];
#pragma unroll
        for (int rr = 0; rr < ROWS; rr++) {
#pragma unroll
          for (int c = 0; c < QN; c++) uq[rr][c] = {vsplat(T(0)), vsplat(T(0))};
#pragma unroll
          for (int c = 0; c <= R; c++) dq[rr][c] = {vsplat(T(0)), vsplat(T(0))};
        }

        auto step = [&](auto kc) -> bool {
          constexpr int KK = decltype(kc)::value;
          if (t >= niters) return false;
          if (!wait_plane()) {
            aborted = true;
            return false;
          }
          const unsigned char* ss = smem + so;
          const unsigned char* fs = smem + fo;
          auto zq = [&](int rr, int d) -> const CPair<T>& { return q[rr][(KK + d + QN) % QN]; };
          auto zu = [&](int rr, int d) -> const CPair<T>& {
            return uq[rr][(KK - 2 * R + d + 4 * QN) % QN];
          };
#pragma unroll
          for (int rr = 0; rr < ROWS; rr++) q[rr][(R + KK) % QN] = ld(ss + s_off + ES * rr * BW, oth);
          if (t >= R) {
            // ---- first stage of plane f = z0 - 2R + t
            const int f = z0 - 2 * R + t;
            const unsigned char* hc = fs + s_off;
            CPair<T> ylo[R], yhi[R];
#pragma unroll
            for (int k = 0; k < R; k++) {
              ylo[k] = ld(hc + (int)ES * ((k - R) * BW), oth);
              yhi[k] = ld(hc + (int)ES * ((ROWS + k) * BW), oth);
            }
            auto yrow = [&](int dr) -> const CPair<T>& {
              return dr < 0 ? ylo[R + dr] : dr >= ROWS ? yhi[dr - ROWS] : zq(dr, 0);
            };
            const T Vz = (TRAP || (FULL && useV)) ? rd.tabV[2][f] : T(0);
            const T Dz = (FULL && useD) ? rd.tabD[2][f] : T(0);
            unsigned char* uw = smem + uo + u_off;
#pragma unroll
            for (int rr = 0; rr < ROWS; rr++) {
              const CPair<T> xa = ld(hc + (int)ES * (rr * BW - 2), oth);
              const CPair<T> xc = ld(hc + (int)ES * (rr * BW + 2), oth);
              CPair<T> bs = zq(rr, 0);
              if (B4) bs = ld(ss + p.base_off + u_off + ES * rr * UW, oth);
              CPair<T> d, u;
#pragma unroll
              for (int e = 0; e < 2; e++) {
                const Star<V> sv =
                    star(e, sl, zq(rr, 0), xa, xc, yrow(rr - 1), yrow(rr + 1),
                         yrow(R == 2 ? rr - 2 : rr - 1), yrow(R == 2 ? rr + 2 : rr + 1), zq(rr, -1),
                         zq(rr, 1), zq(rr, R == 2 ? -2 : -1), zq(rr, R == 2 ? 2 : 1));
                const V K = rhs(sv, rr, e, Vz, Dz);
                const V dv = vfma(ar0, K, vmul(ax0, vswap(K)));
                (e ? d.b : d.a) = dv;
                (e ? u.b : u.a) = vadd(e ? bs.b : bs.a, dv);
              }
              st(uw + ES * rr * UW, oth, u.a, u.b);
              uq[rr][(KK - R + 2 * QN) % QN] = u;
              if (DS) {
                st(smem + p.d_ring + d_at * d_plane + pt_off + ES * rr * TX, oth, d.a, d.b);
              } else if (KIND != PAIR_RK2) {
#pragma unroll
                for (int c = 0; c < R; c++) dq[rr][c] = dq[rr][c + 1];
                dq[rr][R] = d;
              }
            }
            publish();
            if (!wait_u()) {
              aborted = true;
              return false;
            }
          }
          if (t >= 3 * R) {
            // ---- second stage of plane z = f - R
            const int z = z0 + t - 3 * R;
            const unsigned char* hc = smem + zo + u_off;
            const unsigned char* pt = smem + p.pt_ring + (gp & 1u) * p.pt_stride + pt_off;
            if (NPT > 0 &&
                !mbar_wait_bounded(&pfull[gp & 1u], (gp >> 1) & 1u, p.wait_limit_ns)) {
              s_abort = 1;
              atomicExch(p.status, 6);
              aborted = true;
              return false;
            }
            CPair<T> ylo[R], yhi[R];
#pragma unroll
            for (int k = 0; k < R; k++) {
              ylo[k] = ld(hc + (int)ES * ((k - R) * UW), oth);
              yhi[k] = ld(hc + (int)ES * ((ROWS + k) * UW), oth);
            }
            auto yrow = [&](int dr) -> const CPair<T>& {
              return dr < 0 ? ylo[R + dr] : dr >= ROWS ? yhi[dr - ROWS] : zu(dr, 0);
            };
            const T Vz = (TRAP || (FULL && useV)) ? rd.tabV[2][z] : T(0);
            const T Dz = (FULL && useD) ? rd.tabD[2][z] : T(0);
            const double Wz = NORM ? rd.tabW[2][z] : 0.0;
#pragma unroll
            for (int rr = 0; rr < ROWS; rr++) {
              const CPair<T> xa = ld(hc + (int)ES * (rr * UW - 2), oth);
              const CPair<T> xc = ld(hc + (int)ES * (rr * UW + 2), oth);
              if (DS) {
                const unsigned at = d_at + 1 > (unsigned)R ? 0 : d_at + 1;  // plane f - R
                dq[rr][0] = ld(smem + p.d_ring + at * d_plane + pt_off + ES * rr * TX, oth);
              }
              CPair<T> psi = zq(rr, -R), acc = psi, cc = psi;
              if (B4) {
                psi = ld(fs + p.base_off + u_off + ES * rr * UW, oth);
                acc = ld(pt + ES * rr * TX, oth);
              }
              if (KAHAN) cc = ld(pt + p.comp_off + ES * rr * TX, oth);
              V r0[2], r1[2];
#pragma unroll
              for (int e = 0; e < 2; e++) {
                const Star<V> sv =
                    star(e, sl, zu(rr, 0), xa, xc, yrow(rr - 1), yrow(rr + 1),
                         yrow(R == 2 ? rr - 2 : rr - 1), yrow(R == 2 ? rr + 2 : rr + 1), zu(rr, -1),
                         zu(rr, 1), zu(rr, R == 2 ? -2 : -1), zu(rr, R == 2 ? 2 : 1));
                const V K = rhs(sv, rr, e, Vz, Dz);
                V v = vfma(ar1, K, vmul(ax1, vswap(K)));
                const V ps = e ? psi.b : psi.a;
                const V dz = e ? dq[rr][0].b : dq[rr][0].a;
                if (KIND == PAIR_RK4_A) {
                  r0[e] = vadd(ps, v);
                  r1[e] = vfma(twothird, v, vmul(third, dz));
                } else {
                  if (B4) v = vadd(vfma(third, dz, v), e ? acc.b : acc.a);
                  if (KAHAN) {
                    const V y = vfma(e ? cc.b : cc.a, mone, v);
                    const V tt = vadd(ps, y);
                    r1[e] = vfma(y, mone, vfma(ps, mone, tt));
                    r0[e] = tt;
                  } else {
                    r0[e] = vadd(v, ps);
                  }
                  if (ok[rr][e]) {
                    const double vr = (double)r0[e].x, vi = (double)r0[e].y;
                    red0 = fma(Wxy[rr][e] * Wz, fma(vr, vr, vi * vi), red0);
                  }
                }
              }
              const size_t at = base + rr * Nx;
              if (KIND == PAIR_RK4_A || KAHAN) store(out1 + 2 * at, ok[rr], r1);
              store(out0 + 2 * at, ok[rr], r0);
            }
            base += NxNy;
            if (NPT > 0) {
              __syncwarp();
              if (lane == 0) mbar_arrive(&pempty[gp & 1u]);
              ++gp;
            }
          }
          if (DS && t >= R) d_at = d_at + 1 > (unsigned)R ? 0 : d_at + 1;
          finish_plane();
          return true;
        };
        while (!*(volatile int*)&s_abort) {
          if (!step(IC<0>())) break;
          if (!step(IC<1>())) break;
          if (!step(IC<2>())) break;
          if constexpr (QN > 3) {
            if (!step(IC<3>())) break;
            if (!step(IC<4>())) break;
          }
        }
      } else {
        // ---- ring warp: the first stage around the tile
        unsigned s_off[NU], u_off[NU];
        int oth[NU];
#pragma unroll
        for (int rr = 0; rr < NU; rr++) {
          s_off[rr] = ES * (unsigned)((urow[rr] + 2 * R) * BW + ucol[rr] + 4 + sel[rr]);
          oth[rr] = 16 - 32 * sel[rr];
          u_off[rr] = ES * (unsigned)((urow[rr] + R) * UW + ucol[rr] + 2 + sel[rr]);
        }
        auto step = [&](auto kc) -> bool {
          constexpr int KK = decltype(kc)::value;
          if (t >= niters) return false;
          if (!wait_plane()) {
            aborted = true;
            return false;
          }
          const unsigned char* ss = smem + so;
          const unsigned char* fs = smem + fo;
          auto zq = [&](int rr, int d) -> const CPair<T>& { return q[rr][(KK + d + QN) % QN]; };
#pragma unroll
          for (int rr = 0; rr < NU; rr++)
            if (act[rr]) q[rr][(R + KK) % QN] = ld(ss + s_off[rr], oth[rr]);
          if (t >= R) {
            const int f = z0 - 2 * R + t;
            const T Vz = (TRAP || (FULL && useV)) ? rd.tabV[2][f] : T(0);
            const T Dz = (FULL && useD) ? rd.tabD[2][f] : T(0);
#pragma unroll
            for (int rr = 0; rr < NU; rr++) {
              if (!act[rr]) continue;
              const unsigned char* hc = fs + s_off[rr];
              const CPair<T> xa = ld(hc - (int)ES * 2, oth[rr]), xc = ld(hc + (int)ES * 2, oth[rr]);
              const CPair<T> ym1 = ld(hc - (int)ES * BW, oth[rr]), yp1 = ld(hc + (int)ES * BW, oth[rr]);
              CPair<T> ym2 = ym1, yp2 = yp1;
              if (R == 2) {
                ym2 = ld(hc - (int)ES * 2 * BW, oth[rr]);
                yp2 = ld(hc + (int)ES * 2 * BW, oth[rr]);
              }
              CPair<T> bs = zq(rr, 0);
              if (B4) bs = ld(ss + p.base_off + u_off[rr], oth[rr]);
              CPair<T> u;
#pragma unroll
              for (int e = 0; e < 2; e++) {
                const Star<V> sv =
                    star(e, sel[rr], zq(rr, 0), xa, xc, ym1, yp1, ym2, yp2, zq(rr, -1), zq(rr, 1),
                         zq(rr, R == 2 ? -2 : -1), zq(rr, R == 2 ? 2 : 1));
                const V K = rhs(sv, rr, e, Vz, Dz);
                (e ? u.b : u.a) = vadd(e ? bs.b : bs.a, vfma(ar0, K, vmul(ax0, vswap(K))));
              }
              st(smem + uo + u_off[rr], oth[rr], u.a, u.b);
            }
            publish();
            if (!wait_u()) {
              aborted = true;
              return false;
            }
          }
          finish_plane();
          return true;
        };
        while (!*(volatile int*)&s_abort) {
          if (!step(IC<0>())) break;
          if (!step(IC<1>())) break;
          if (!step(IC<2>())) break;
          if constexpr (QN > 3) {
            if (!step(IC<3>())) break;
            if (!step(IC<4>())) break;
          }
        }
      }
      aborted = aborted || t < niters;
      if (!aborted) {
        // hand back the item's last R planes, held for their x/y neighbours
#pragma unroll
        for (int k = 0; k < R; k++) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[cslot]);
          fo += p.slot_stride;
          if (++cslot == S) {
            cslot = 0;
            fo = s_first;
          }
        }
      }
      if (NORM && interior) {
        // per-item partials of the norm; every interior warp reaches both
        // barriers of every item it starts, an aborted one included, and all
        // leave the item loop on one decision (as in stage_kernel.cuh)
        red0 = warp_sum(red0);
        if (lane == 0) s_red[warp] = red0;
        named_barrier_sync(1, 32 * NI);
        if (tid == 0) {
          double a = 0.0;
          for (int w2 = 0; w2 < NI; w2++) a += s_red[w2];
          p.partials[2 * (size_t)it + 0] = a;
          p.partials[2 * (size_t)it + 1] = 0.0;
          s_stop = *(volatile int*)&s_abort;
        }
        named_barrier_sync(1, 32 * NI);
        if (*(volatile int*)&s_stop) break;
      } else if (aborted) {
        break;
      }
    }  // items
  }

  __syncthreads();
  // After a timed-out wait the copies in flight land (bounded) before the
  // CTA's shared memory is released (as in stage_kernel.cuh).
  if (s_abort && tid == 0) {
    const int issued = s_issued;
    const unsigned long long drain =
        p.wait_limit_ns > 2000000000ull ? p.wait_limit_ns : 2000000000ull;
    for (int u = max(0, issued - S); u < issued; u++)
      mbar_wait_bounded(&full[u % S], (uint32_t)((u / S) & 1), drain);
    const int pissued = s_pissued;
    for (int u = max(0, pissued - PT_SLOTS); u < pissued; u++)
      mbar_wait_bounded(&pfull[u % PT_SLOTS], (uint32_t)((u / PT_SLOTS) & 1), drain);
  }
}

template <typename T, int R, int KIND, bool KAHAN, int FORM, bool BATCH>
__global__ void __launch_bounds__(pair_max_threads<T>(R), 1)
    pair_kernel(const __grid_constant__ PairParams<T> p) {
  pair_body<T, R, KIND, KAHAN, FORM, BATCH>(p);
}

}  // namespace gpe
