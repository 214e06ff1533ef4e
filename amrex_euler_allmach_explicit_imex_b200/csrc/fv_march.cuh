// Default explicit step: warps march up column strips.  Included inside the
// arithmetic namespace of stencil.cuh, after fv_fast.cuh (the fast build's
// Newton-refined arithmetic and flux functions) or fv_exact.cuh (the exact
// build's, under the same names).
//
// A warp owns the 28 cells [c0, c0+28) of a row strip; lane l holds column
// c0 - 2 + l (lanes 0-1 and 30-31 carry the MUSCL halo).  It walks rows
// j0 .. j0+H-1:
//   * the y-slope of a row is computed once and reused by both y-faces;
//   * the y-face flux above row j becomes the flux below row j+1 without
//     leaving registers.
// Every face flux is evaluated once per warp strip (the x-face at a strip
// edge by both strips), with no block barrier in the loop.  Reductions (CFL
// rate, admissibility, degenerate count) accumulate in registers and are
// committed once per block.
// Two forms: rows through shared memory (march_strip_staged, the default), and
// rows j-1 .. j+2 in registers with the x-neighbours by warp shuffles
// (march_strip, the fast build's tile_y 2 and 3).  The HLLC-P flux takes the
// strips in the fast build only, too.
namespace march {

#ifdef ECG_FAST_KERNEL
constexpr bool kExact = false;
#else
constexpr bool kExact = true;
#endif
constexpr int kLanes = 32;
constexpr int kCells = 28;  // interior cells per warp strip

__device__ __forceinline__ double shup(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double shdn(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

template <int LIM>
__device__ __forceinline__ Prim slope3(const Prim& m, const Prim& c, const Prim& p, bool second)
{
  if (!second) return Prim{0.0, 0.0, 0.0, 0.0};
  return Prim{fast::slope_f(c.rho - m.rho, p.rho - c.rho, LIM), fast::slope_f(c.u - m.u, p.u - c.u, LIM),
              fast::slope_f(c.v - m.v, p.v - c.v, LIM), fast::slope_f(c.p - m.p, p.p - c.p, LIM)};
}

// (0.5 s is exact, so the fused form rounds like q + 0.5 s in either build)
__device__ __forceinline__ Prim plus_half(const Prim& q, const Prim& s)
{
  return Prim{fma(0.5, s.rho, q.rho), fma(0.5, s.u, q.u), fma(0.5, s.v, q.v), fma(0.5, s.p, q.p)};
}
__device__ __forceinline__ Prim minus_half(const Prim& q, const Prim& s)
{
  return Prim{fma(-0.5, s.rho, q.rho), fma(-0.5, s.u, q.u), fma(-0.5, s.v, q.v), fma(-0.5, s.p, q.p)};
}

// One face on its own, every branch taken (the y-face below the first row of a
// strip, and the faces the branch-free cores send back).  deg: HLLC fell back to
// Rusanov.  sensor: of the HLLC-P flux, h^3 of the five faces' ratios.
template <int RK>
__device__ __forceinline__ Cons face_one(Prim l, Prim r, int axis, double g, double inv_gm1, double sensor, bool& deg)
{
  deg = false;
#ifdef ECG_FAST_KERNEL
  if (RK == ECG_RIEMANN_XIE_AM_HLLC_P) return fast::xie_f(l, r, axis, g, inv_gm1, sensor, deg);
#endif
  if (RK == ECG_RIEMANN_RUSANOV) return fast::rusanov_f(l, r, axis, g, inv_gm1);
  if (RK == ECG_RIEMANN_LOWMACH_HLLC) fast::lowmach_f(l, r, g);
  return fast::hllc_f(l, r, axis, g, inv_gm1, deg);
}

// The face without branches; `b` marks one that face_one must evaluate instead.
template <int RK>
__device__ __forceinline__ Cons face_core(const Prim& l, const Prim& r, int axis, double g, double inv_gm1,
                                          double sensor, bool& b)
{
#ifdef ECG_FAST_KERNEL
  if (RK == ECG_RIEMANN_XIE_AM_HLLC_P) return fast::xie_core(l, r, axis, g, inv_gm1, sensor, b);
#endif
  if (RK == ECG_RIEMANN_RUSANOV) return fast::rusanov_core(l, r, axis, g, inv_gm1, b);
  return fast::hllc_core<RK == ECG_RIEMANN_LOWMACH_HLLC>(l, r, axis, g, inv_gm1, b);
}

// One face, repaired after a vote of its own.
template <int RK>
__device__ __forceinline__ Cons face_voted(const Prim& l, const Prim& r, int axis, double g, double inv_gm1,
                                           double sensor, bool& deg)
{
  bool b;
  Cons f = face_core<RK>(l, r, axis, g, inv_gm1, sensor, b);
  deg = false;
  if (__any_sync(0xffffffffu, b)) {
    if (b) f = face_one<RK>(l, r, axis, g, inv_gm1, sensor, deg);
  }
  return f;
}

// Reductions of one warp strip over the new state.
struct MarchAcc {
  unsigned long long kmax, krho, kp;
  int nonfinite, degenerate;
  __device__ __forceinline__ void init()
  {
    kmax = okey(kLowest);
    krho = okey(kMax);
    kp = okey(kMax);
    nonfinite = degenerate = 0;
  }
};

#ifdef ECG_FAST_KERNEL
struct Lane {
  Prim q[4];  // rows j-1, j, j+1, j+2 of this lane's column
};

// The x-face and the y-face of a row, evaluated back to back on the fast
// path (independent instruction streams the scheduler can interleave); faces
// that need the reference path (degenerate HLLC star state, sound speed off
// the rsqrt path) are recomputed after one warp vote.  deg_*: HLLC fell back
// to Rusanov on that face.  Returns whether the vote fired (the same on every
// lane): deg_* can only be set then.
template <int RK>
__device__ __forceinline__ bool face_pair(const Prim& xl, const Prim& xr, const Prim& yl, const Prim& yr, double g,
                                          double inv_gm1, Cons& fx, Cons& fy, bool& deg_x, bool& deg_y)
{
  bool bx, by;
  fx = face_core<RK>(xl, xr, 0, g, inv_gm1, 0.0, bx);
  fy = face_core<RK>(yl, yr, 1, g, inv_gm1, 0.0, by);
  deg_x = deg_y = false;
  if (__any_sync(0xffffffffu, bx || by)) {
    if (bx) fx = face_one<RK>(xl, xr, 0, g, inv_gm1, 0.0, deg_x);
    if (by) fy = face_one<RK>(yl, yr, 1, g, inv_gm1, 0.0, deg_y);
    return true;
  }
  return false;
}

// Advances the strip of 28 cells starting at column c0 over rows
// [j0, min(j0 + H, ny)) from u into out.  Called by all 32 lanes of a warp
// (the flux helpers vote across the warp).
template <int RK, int LIM, bool PAIR>
__device__ __forceinline__ void march_strip(const EcgFvParams& P, const double* __restrict__ u,
                                            double* __restrict__ out, int c0, int j0, int H, double dt,
                                            bool count_deg, MarchAcc& acc)
{
  const int lane = threadIdx.x & 31;
  const int x = c0 - 2 + lane;
  const int nx = P.g.nx, ny = P.g.ny;
  const double g = P.gamma, inv_gm1 = fast::frcp(g - 1.0);
  const double idx = P.g.inv_dx, idy = P.g.inv_dy;
  const bool second = P.order > 1;
  const bool inner = lane >= 2 && lane < 2 + kCells;   // owns a cell of the strip
  const bool cell_ok = inner && x < nx;                 // that cell is in the domain
  const bool xface = lane >= 2 && lane <= 2 + kCells;   // its x-face on the left belongs to the strip
  const int xs = x < 0 ? 0 : (x < nx ? x : nx - 1);     // in-bounds column for the old-state reload
  const int rhi = P.row_hi > 0 && P.row_hi < ny ? P.row_hi : ny;  // end of the band of rows being updated
  const int jend = j0 + H < rhi ? j0 + H : rhi;

  // ---- prologue: rows j0-2 .. j0+1, y-slopes of rows j0-1 and j0, the y-face below row j0 ----
  Prim q_m2 = fast::to_prim_f(load_cell(P, u, x, j0 - 2), g);
  Lane L;
  L.q[1] = fast::to_prim_f(load_cell(P, u, x, j0 - 1), g);
  L.q[2] = fast::to_prim_f(load_cell(P, u, x, j0), g);
  L.q[3] = fast::to_prim_f(load_cell(P, u, x, j0 + 1), g);
  const Prim sy_m1 = slope3<LIM>(q_m2, L.q[1], L.q[2], second);
  Prim sy_cur = slope3<LIM>(L.q[1], L.q[2], L.q[3], second);
  Cons gb;
  {
    bool deg;
    gb = face_one<RK>(plus_half(L.q[1], sy_m1), minus_half(L.q[2], sy_cur), 1, g, inv_gm1, 0.0, deg);
    if (count_deg && deg && cell_ok && j0 < ny) acc.degenerate += 1;
  }
  for (int j = j0; j < jend; ++j) {
    // window rows j-1 .. j+2
    L.q[0] = L.q[1];
    L.q[1] = L.q[2];
    L.q[2] = L.q[3];
    L.q[3] = fast::to_prim_f(load_cell(P, u, x, j + 2), g);
    const Prim& qc = L.q[1];
    // slopes: y of row j+1 (for the y-face above row j), x of this lane's cell
    const Prim sy_next = slope3<LIM>(L.q[1], L.q[2], L.q[3], second);
    const Prim ql{shup(qc.rho), shup(qc.u), shup(qc.v), shup(qc.p)};
    const Prim qr{shdn(qc.rho), shdn(qc.u), shdn(qc.v), shdn(qc.p)};
    const Prim sx = slope3<LIM>(ql, qc, qr, second);
    const Prim sxl{shup(sx.rho), shup(sx.u), shup(sx.v), shup(sx.p)};
    // the x-face on this lane's left and the y-face above row j; every lane
    // evaluates both (lanes 0, 1 and 31 cost nothing extra in lockstep), only
    // lanes 2..30 use or count their x-face
    Cons fl, gt;
    bool deg_x, deg_y, voted = true;
    if (PAIR) {
      voted = face_pair<RK>(plus_half(ql, sxl), minus_half(qc, sx), plus_half(qc, sy_cur), minus_half(L.q[2], sy_next),
                            g, inv_gm1, fl, gt, deg_x, deg_y);
    } else {
      gt = face_voted<RK>(plus_half(qc, sy_cur), minus_half(L.q[2], sy_next), 1, g, inv_gm1, 0.0, deg_y);
      fl = face_voted<RK>(plus_half(ql, sxl), minus_half(qc, sx), 0, g, inv_gm1, 0.0, deg_x);
    }
    const Cons fr{shdn(fl.rho), shdn(fl.mx), shdn(fl.my), shdn(fl.E)};
    if (count_deg && voted) {
      // each face counts once per adjacent cell of this strip in the domain
      // (count_hllc_degenerate_star_states, explicit_update.hpp:2-56)
      const bool left_ok = lane >= 3 && lane <= 2 + kCells && x - 1 < nx;
      if (deg_x && xface) acc.degenerate += (left_ok ? 1 : 0) + (cell_ok ? 1 : 0);
      if (deg_y && cell_ok) acc.degenerate += 1 + (j + 1 < jend ? 1 : 0);
    }
    // update (explicit_update.hpp:92-95) and the reductions of the new state;
    // all lanes compute, lanes outside the strip or the domain neither store
    // nor reduce
    const long long o = static_cast<long long>(j) * P.g.pitch + xs;
    const long long pl = P.g.plane;
    Cons n;
    n.rho = load_coherent(u + o) - dt * ((fr.rho - fl.rho) * idx + (gt.rho - gb.rho) * idy);
    n.mx = load_coherent(u + o + pl) - dt * ((fr.mx - fl.mx) * idx + (gt.mx - gb.mx) * idy);
    n.my = load_coherent(u + o + 2 * pl) - dt * ((fr.my - fl.my) * idx + (gt.my - gb.my) * idy);
    n.E = load_coherent(u + o + 3 * pl) - dt * ((fr.E - fl.E) * idx + (gt.E - gb.E) * idy);
    const Prim q = fast::to_prim_f(n, g);
    const double cs = fast::fsound_w(q.rho, q.p, g);
    if (cell_ok) {
      out[o] = n.rho;
      out[o + pl] = n.mx;
      out[o + 2 * pl] = n.my;
      out[o + 3 * pl] = n.E;
      const double rate = (fabs(q.u) + cs) * idx + (fabs(q.v) + cs) * idy;
      if (!isnan(rate)) acc.kmax = umax64(acc.kmax, okey(rate));
      const bool bad = !isfinite(q.rho) || !isfinite(q.u) || !isfinite(q.v) || !isfinite(q.p) || !isfinite(n.E);
      acc.krho = umin64(acc.krho, okey(bad ? -kInf : q.rho));
      acc.kp = umin64(acc.kp, okey(bad ? -kInf : q.p));
      acc.nonfinite += bad ? 1 : 0;
    }
    gb = gt;
    sy_cur = sy_next;
  }
}
#endif  // ECG_FAST_KERNEL

// ---- the staged march: rows live in shared memory --------------------------
//
// Each warp keeps the conserved values of the rows it is about to use in a
// ring of kRing rows in shared memory (slot = row mod kRing, component planes
// of 32 lanes).  A lane requests the cell of its column kAhead rows ahead of
// the one being converted with cp.async (8 bytes per component, straight
// from the state, the exact-Dirichlet ring or a slab halo, whichever the
// ghost policy names); constant ghost states are stored directly.  The load
// latency of a row is thus hidden behind kAhead rows of flux work, and the
// old state of the updated row is read back from the ring.
// A row that has landed is converted once; its velocities and pressure go to a
// second ring of kPrim rows (the density is the conserved one), from which the
// lanes read their own column's rows j .. j+2 for the y-slope and their
// neighbours' row j for the x-slope.  Between rows a lane carries only the
// y-face below it and the upper face state of its cell.
constexpr int kRing = 8;
constexpr int kAhead = 4;
constexpr int kPrim = 4;
static_assert(kAhead + 4 <= kRing, "rows j-1 .. j+2+kAhead are in the ring");

struct StageRing {
  double v[kRing][4][kLanes];
  double q[kPrim][3][kLanes];  // u, v, p
};

__device__ __forceinline__ void cp_async8(unsigned dst, const double* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

#ifdef ECG_FAST_KERNEL
// The multiface sensor's pressure ratio (xie_pressure_ratio_from_states,
// reconstruction_fluxes.hpp:390-397) of the x-face on this lane's left in a
// row of which this lane holds the pressure pc: the face pressures of the
// MUSCL states, as the tile kernel forms them.
template <int LIM>
__device__ __forceinline__ double xface_ratio(double pc, bool second)
{
  const double pl = shup(pc), pr = shdn(pc);
  const double s = second ? fast::slope_f(pc - pl, pr - pc, LIM) : 0.0;
  return fast::pratio_f(fma(0.5, shup(s), pl), fma(-0.5, s, pc));
}

__device__ __forceinline__ double sensor_of(double ratio)
{
  const double h = clamp01(ratio);
  return h * h * h;
}
#endif

// Advances the strip as march_strip does.  The x- and the y-face of a row are
// evaluated back to back on the branch-free cores; faces those send back are
// recomputed after one warp vote, their states rebuilt from the rings, so that
// the common path keeps no face state alive for the repair.
// RK = xie_am_hllc_p: each face with its 5-face sensor.  The pressure ratios
// it needs come along the march: the y-faces' below and above row j (carried,
// and this row's), and the x-faces' of rows j and j+1 (row j+1's from the
// pressure of the window's next row, carried on).
// control(dt) gives the step's dt, or false to stop, after the first rows have
// been requested: its chain of loads and divisions runs beside theirs.  Returns
// what it returned.
template <int RK, int LIM, class Control>
__device__ __forceinline__ bool march_strip_staged(const EcgFvParams& P, const double* __restrict__ u,
                                                   double* __restrict__ out, int c0, int j0, int H, Control control,
                                                   bool count_deg, MarchAcc& acc, StageRing& ring)
{
  const int lane = threadIdx.x & 31;
  const int x = c0 - 2 + lane;
  const int nx = P.g.nx, ny = P.g.ny;
  const double g = P.gamma, inv_gm1 = fast::frcp(g - 1.0);
  const bool second = P.order > 1;
  const bool inner = lane >= 2 && lane < 2 + kCells;
  const bool cell_ok = inner && x < nx;
  const int rhi = P.row_hi > 0 && P.row_hi < ny ? P.row_hi : ny;
  const int jend = j0 + H < rhi ? j0 + H : rhi;
  const int jlast = jend + 1;  // the last row the strip reads

  double* const col = &ring.v[0][0][lane];
  double* const qcol = &ring.q[0][0][lane];
  const unsigned col_s = static_cast<unsigned>(__cvta_generic_to_shared(col));
  const int left = lane > 0 ? -1 : 0, right = lane < 31 ? 1 : 0;  // neighbour columns (the end lanes' own)
  unsigned flips = 0;  // bit (row mod kRing): that staged row is a mirror image (my to negate)
  // Where this lane's column comes from in rows of the domain does not depend
  // on the row (the state, a wrapped or clamped column of it, the ghost ring, a
  // slab halo, or the constant state when null): found once, then a pointer
  // that moves one row a request (the rows are requested in order).  Only the
  // rows above and below the domain go through the ghost policy again; with
  // the whole policy per cell, the strips on an x boundary ran 12 % longer than
  // the others and held the launch up.
  const CellSrc colsrc = cell_src(P, u, x, 0);
  const long long cpl = colsrc.pl;
  const long long cpitch = colsrc.p && ny > 1 ? cell_src(P, u, x, 1).p - colsrc.p : 0;
  const long long pl = P.g.plane;
  const double* rowp = colsrc.p + static_cast<long long>(j0 - 2) * cpitch;  // dereferenced only when in the domain
  // request row jr of this lane's column (an empty group past the strip's rows)
  auto put = [&](int jr) {
    if (jr <= jlast) {
      const int sl = jr & (kRing - 1);
      CellSrc c{rowp, cpl, false};
      if (static_cast<unsigned>(jr) >= static_cast<unsigned>(ny)) {
        if (P.bc.ring) {
          c = cell_src(P, u, x, jr);
        } else {
          const int jj = ghost_row(P, jr, c.flip);
          c.p = jj < 0 ? nullptr : colsrc.p + static_cast<long long>(jj) * cpitch;
        }
      }
      if (!colsrc.p) c = CellSrc{nullptr, 0, false};
      flips = c.flip ? (flips | (1u << sl)) : (flips & ~(1u << sl));
      if (c.p) {
        const unsigned d = col_s + static_cast<unsigned>(sl * 4 * kLanes * 8);
        cp_async8(d, c.p);
        cp_async8(d + kLanes * 8, c.p + c.pl);
        cp_async8(d + 2 * kLanes * 8, c.p + 2 * c.pl);
        cp_async8(d + 3 * kLanes * 8, c.p + 3 * c.pl);
      } else {
        double* d = col + sl * 4 * kLanes;
        d[0] = P.bc.cst[0];
        d[kLanes] = P.bc.cst[1];
        d[2 * kLanes] = P.bc.cst[2];
        d[3 * kLanes] = P.bc.cst[3];
      }
    }
    rowp += cpitch;
    cp_async_commit();
  };
  auto conserved = [&](int jr) {
    const double* d = col + (jr & (kRing - 1)) * 4 * kLanes;
    return Cons{d[0], d[kLanes], d[2 * kLanes], d[3 * kLanes]};
  };
  // primitives of row jr of this lane's column, into the second ring
  auto convert = [&](int jr) {
    Cons c = conserved(jr);
    if ((flips >> (jr & (kRing - 1))) & 1u) c.my = -c.my;
    const Prim q = fast::to_prim_f(c, g);
    double* d = qcol + (jr & (kPrim - 1)) * 3 * kLanes;
    d[0] = q.u;
    d[kLanes] = q.v;
    d[2 * kLanes] = q.p;
    return q;
  };
  // row jr of the column `dl` lanes over
  auto prim = [&](int jr, int dl) {
    const double* d = qcol + (jr & (kPrim - 1)) * 3 * kLanes + dl;
    return Prim{col[(jr & (kRing - 1)) * 4 * kLanes + dl], d[0], d[kLanes], d[2 * kLanes]};
  };
  // The two states of the x-face on this lane's left in row j, and of the
  // y-face above it, from the rings (the repair of a face).
  auto xstates = [&](int j, Prim& l, Prim& r) {
    const Prim a = prim(j, lane > 1 ? -2 : left), b = prim(j, left), c = prim(j, 0), d = prim(j, right);
    l = plus_half(b, slope3<LIM>(a, b, c, second));
    r = minus_half(c, slope3<LIM>(b, c, d, second));
  };
  auto ystates = [&](int j, Prim& l, Prim& r) {
    const Prim a = prim(j - 1, 0), b = prim(j, 0), c = prim(j + 1, 0), d = prim(j + 2, 0);
    l = plus_half(b, slope3<LIM>(a, b, c, second));
    r = minus_half(c, slope3<LIM>(b, c, d, second));
  };

  // ---- prologue: stage rows j0-2 .. j0+1+kAhead; rows j0-2 .. j0+1 first ----
#pragma unroll
  for (int r = -2; r <= 1 + kAhead; ++r) put(j0 + r);
  double dt;
  if (!control(dt)) {
    cp_async_wait<0>();
    return false;
  }
  const double dtx = dt * P.g.inv_dx, dty = dt * P.g.inv_dy;
  cp_async_wait<kAhead>();
  Prim yp;  // row j's state at its upper y-face
  Cons gb;  // the y-face below row j
  double yr_prev = 0.0, xr_cur = 0.0;  // HLLC-P: pressure ratios of the y-face below row j, the x-face left of row j
  {
    const Prim q_m2 = convert(j0 - 2), q_m1 = convert(j0 - 1), qa = convert(j0), qb = convert(j0 + 1);
    const Prim sy_m1 = slope3<LIM>(q_m2, q_m1, qa, second);
    const Prim s0 = slope3<LIM>(q_m1, qa, qb, second);
    const Prim yl = plus_half(q_m1, sy_m1), yr = minus_half(qa, s0);
    yp = plus_half(qa, s0);
    bool deg;
#ifdef ECG_FAST_KERNEL
    if constexpr (RK == ECG_RIEMANN_XIE_AM_HLLC_P) {
      yr_prev = fast::pratio_f(yl.p, yr.p);
      const double xm1 = xface_ratio<LIM>(q_m1.p, second);
      xr_cur = xface_ratio<LIM>(qa.p, second);
      const double m = smin(smin(smin(smin(yr_prev, xm1), shdn(xm1)), xr_cur), shdn(xr_cur));
      gb = face_voted<RK>(yl, yr, 1, g, inv_gm1, sensor_of(m), deg);
    } else
#endif
      gb = face_one<RK>(yl, yr, 1, g, inv_gm1, 0.0, deg);
    if (count_deg && deg && cell_ok && j0 < ny) acc.degenerate += 1;
  }
  double* o = out + static_cast<long long>(j0) * P.g.pitch + (x < 0 ? 0 : (x < nx ? x : nx - 1));
  double rate_max = kLowest, rho_min = kMax, p_min = kMax;

  for (int j = j0; j < jend; ++j) {
    put(j + 2 + kAhead);
    cp_async_wait<kAhead>();  // row j + 2 has landed
    const Prim q2 = convert(j + 2);
    __syncwarp();  // every lane's row j + 2 is in the rings
    bool bx, by;
    Cons gt, fl;
    double mx = 0.0, my = 0.0;  // HLLC-P: the sensors of the two faces
    {
      const Prim q1 = prim(j + 1, 0);
      const Prim sn = slope3<LIM>(prim(j, 0), q1, q2, second);
      const Prim yr = minus_half(q1, sn);
#ifdef ECG_FAST_KERNEL
      if constexpr (RK == ECG_RIEMANN_XIE_AM_HLLC_P) {
        // sensors: the y-face above, from its own ratio and the x-faces' left
        // and right of cell i in rows j and j+1; the x-face on the left, from
        // its own ratio and the y-faces' below and above cells i-1 and i
        const double yr_cur = fast::pratio_f(yp.p, yr.p);
        const double xr_next = xface_ratio<LIM>(q1.p, second);
        my = smin(smin(yr_cur, xr_cur), shdn(xr_cur));
        my = smin(smin(my, xr_next), shdn(xr_next));
        mx = smin(smin(xr_cur, shup(yr_prev)), shup(yr_cur));
        mx = smin(smin(mx, yr_prev), yr_cur);
        my = clamp01(my);
        mx = clamp01(mx);
        yr_prev = yr_cur;
        xr_cur = xr_next;
      }
#endif
      gt = face_core<RK>(yp, yr, 1, g, inv_gm1, my * my * my, by);
      yp = plus_half(q1, sn);
    }
    {
      const Prim q0 = prim(j, 0);
      const Prim sx = slope3<LIM>(prim(j, left), q0, prim(j, right), second);
      const Prim xp = plus_half(q0, sx), xr = minus_half(q0, sx);
      const Prim xl{shup(xp.rho), shup(xp.u), shup(xp.v), shup(xp.p)};
      fl = face_core<RK>(xl, xr, 0, g, inv_gm1, mx * mx * mx, bx);
    }
    if (__any_sync(0xffffffffu, bx || by)) {
      Prim l, r;
      bool deg_x = false, deg_y = false;
      if (bx) {
        xstates(j, l, r);
        fl = face_one<RK>(l, r, 0, g, inv_gm1, mx * mx * mx, deg_x);
      }
      if (by) {
        ystates(j, l, r);
        gt = face_one<RK>(l, r, 1, g, inv_gm1, my * my * my, deg_y);
      }
      if (count_deg) {
        // each face counts once per adjacent cell of this strip in the domain
        // (count_hllc_degenerate_star_states, explicit_update.hpp:2-56); a
        // face is degenerate only where the warp's fallback vote fired
        const bool xface = lane >= 2 && lane <= 2 + kCells;
        const bool left_ok = lane >= 3 && lane <= 2 + kCells && x - 1 < nx;
        if (deg_x && xface) acc.degenerate += (left_ok ? 1 : 0) + (cell_ok ? 1 : 0);
        if (deg_y && cell_ok) acc.degenerate += 1 + (j + 1 < jend ? 1 : 0);
      }
    }
    // update (explicit_update.hpp:92-95) from the staged old state of row j, rounded
    // once at its magnitude
    const Cons fr{shdn(fl.rho), shdn(fl.mx), shdn(fl.my), shdn(fl.E)};
    const Cons old = conserved(j);
    Cons n;
    if constexpr (kExact) {
      const double idx = P.g.inv_dx, idy = P.g.inv_dy;
      n.rho = old.rho - dt * ((fr.rho - fl.rho) * idx + (gt.rho - gb.rho) * idy);
      n.mx = old.mx - dt * ((fr.mx - fl.mx) * idx + (gt.mx - gb.mx) * idy);
      n.my = old.my - dt * ((fr.my - fl.my) * idx + (gt.my - gb.my) * idy);
      n.E = old.E - dt * ((fr.E - fl.E) * idx + (gt.E - gb.E) * idy);
    } else {
      n.rho = old.rho - fma(dtx, fr.rho - fl.rho, dty * (gt.rho - gb.rho));
      n.mx = old.mx - fma(dtx, fr.mx - fl.mx, dty * (gt.mx - gb.mx));
      n.my = old.my - fma(dtx, fr.my - fl.my, dty * (gt.my - gb.my));
      n.E = old.E - fma(dtx, fr.E - fl.E, dty * (gt.E - gb.E));
    }
    gb = gt;
    const Prim q = fast::to_prim_f(n, g);
    const double cs = fast::fsound_w(q.rho, q.p, g);
    if (cell_ok) {
      o[0] = n.rho;
      o[pl] = n.mx;
      o[2 * pl] = n.my;
      o[3 * pl] = n.E;
      // running extrema as doubles: the comparisons skip a NaN as the keys'
      // NaN test does, and a strip with a bad cell takes the floor at its end
      const double rate = kExact ? (fabs(q.u) + cs) / P.g.dx + (fabs(q.v) + cs) / P.g.dy
                                 : (fabs(q.u) + cs) * P.g.inv_dx + (fabs(q.v) + cs) * P.g.inv_dy;
      rate_max = rate > rate_max ? rate : rate_max;
      rho_min = q.rho < rho_min ? q.rho : rho_min;
      p_min = q.p < p_min ? q.p : p_min;
      // a nonfinite component (or velocity) makes the pressure nonfinite
      if (!isfinite(q.p)) acc.nonfinite += 1;
    }
    o += P.g.pitch;
  }
  cp_async_wait<0>();  // no request outlives the strip
  __syncwarp();        // nor a neighbour's read of this lane's rows the next strip's requests
  if (acc.nonfinite > 0) rho_min = p_min = -kInf;
  acc.kmax = umax64(acc.kmax, okey(rate_max));
  acc.krho = umin64(acc.krho, okey(rho_min));
  acc.kp = umin64(acc.kp, okey(p_min));
  return true;
}

// Resident warps per SM the staged strips are compiled for.  They need 146 to
// 150 registers unconstrained (the XIE flux 168 and some spill): 16 warps at 128
// registers, without a spill, beat 12 for the HLLC fluxes on large grids
// (2048x2048 132 against 137 us, 2560x640 equal), 20 at 96 registers spill and
// lose (164 us, 70 us); the XIE flux (2560x640: 104 us at 12, 116 at 16) and
// Rusanov, which spills at 128, stay at 12, as does the exact build, whose IEEE
// divisions and square roots spill at 128 (1280x320 33.4 us at 16, 31.9 at 12).
template <int RK>
constexpr int kStagedWarps = !kExact && (RK == ECG_RIEMANN_HLLC || RK == ECG_RIEMANN_LOWMACH_HLLC) ? 16 : 12;

// The register-loaded strips take at most 128 registers a thread (16 warps
// per SM), measured faster than the 166-register schedule the paired faces get
// unbounded.
// How the rows come and the faces are evaluated: through the shared-memory rings,
// the two faces of a row together (march_strip_staged); straight from global
// memory into registers (march_strip), the faces together or one after the other.
enum class Form { kStaged, kPaired, kSingle };

template <int RK, int LIM, int WPB, Form FORM>
__global__ void __launch_bounds__(WPB * 32, (FORM == Form::kStaged ? kStagedWarps<RK> : 16) / WPB)
fv_march_kernel(const EcgFvParams P, const double* __restrict__ u, double* __restrict__ out,
                EcgStepStats* __restrict__ stats, const EcgDtCtl ctl, const int H)
{
  __shared__ BlockRed<WPB * 32> red;
  __shared__ StageRing ring[FORM == Form::kStaged ? WPB : 1];
  const int strip = blockIdx.x * WPB + (threadIdx.x >> 5);
  const int c0 = strip * kCells;
  const int j0 = (P.row_hi > 0 ? P.row_lo : 0) + blockIdx.y * H;

  loop_wait();
  auto control = [&](double& dt) { return step_control(stats, ctl, dt); };

  MarchAcc acc;
  acc.init();
  double dt;
  if constexpr (FORM == Form::kStaged) {
    // (a stop is the same for every warp of the launch)
    const bool go = c0 < P.g.nx ? march_strip_staged<RK, LIM>(P, u, out, c0, j0, H, control, ctl.count_degenerate != 0,
                                                              acc, ring[threadIdx.x >> 5])
                                : control(dt);
    if (!go) return;
  }
#ifdef ECG_FAST_KERNEL
  if constexpr (FORM != Form::kStaged) {
    if (!control(dt)) return;
    if (c0 < P.g.nx)
      march_strip<RK, LIM, FORM == Form::kPaired>(P, u, out, c0, j0, H, dt, ctl.count_degenerate != 0, acc);
  }
#endif
  loop_ready();
  block_commit<WPB * 32>(red, acc.kmax, acc.krho, acc.kp, acc.nonfinite, acc.degenerate, &stats[ctl.acc_slot]);
}

// Rows per warp: the count H with the least
//   (H + 3) ((w + ceil w) / 2 + 0.15),   w = blocks(H) / resident blocks,
// where 3 rows stand for a strip's prologue, and the mean of w and ceil w for
// a last wave that is partly filled (its blocks run somewhat faster, and blocks
// of the waves before it drift apart).  Fits the measured times of 15 grids
// from 256x256 to 2048x2048 and H from 1 to 86 within 10 %; taking the rows
// that give one wave of warps instead put 470 blocks on 444 slots at
// 1021x509 (37 us a step, 27.5 with 12 rows) and ran 2048x2048 as a single
// wave of 86 rows (219 us, 157 with 24).
inline int rows_per_warp(int rows, int blocks_x, long long slots)
{
  const int lo = (rows + 65534) / 65535;  // blocks along y
  int best = lo;
  double least = 1.0e300;
  for (int H = lo; H <= 96 && H <= rows; ++H) {
    const double w = static_cast<double>(blocks_x) * ((rows + H - 1) / H) / static_cast<double>(slots);
    const double c = (H + 3) * (0.5 * (w + ceil(w)) + 0.15);
    if (c < least) {
      least = c;
      best = H;
    }
  }
  return best;
}

// Two warps a block: the strips of a row of blocks overhang the grid by at
// most one (four a block: 2 % to 8 % of the warps idle on odd widths).
template <int RK, int LIM, Form FORM>
cudaError_t launch_lim(const EcgFvParams& p, const double* in, double* out, EcgStepStats* stats, const EcgDtCtl& ctl,
                       cudaStream_t s)
{
  constexpr int WPB = 2;
  const int strips = (p.g.nx + kCells - 1) / kCells;
  // a band of rows (the pipelined host step) or the whole grid
  const int rlo = p.row_hi > 0 ? p.row_lo : 0;
  const int rhi = p.row_hi > 0 && p.row_hi < p.g.ny ? p.row_hi : p.g.ny;
  const int rows = rhi - rlo;
  if (rows <= 0) return cudaSuccess;
  const int bx = (strips + WPB - 1) / WPB;
  int H = p.march_rows;
  if (H <= 0) {
    static int blocks_per_sm = 0;
    if (blocks_per_sm == 0) {
      int b = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fv_march_kernel<RK, LIM, WPB, FORM>, WPB * 32, 0) !=
              cudaSuccess ||
          b < 1)
        b = 1;
      blocks_per_sm = b;
    }
    H = rows_per_warp(rows, bx, static_cast<long long>(p.sm_count > 0 ? p.sm_count : 148) * blocks_per_sm);
  }
  const dim3 grid(bx, (rows + H - 1) / H);
  return launch_loop(ctl.device_dt != 0, fv_march_kernel<RK, LIM, WPB, FORM>, grid, WPB * 32, 0, s, p, in, out,
                     stats, ctl, H);
}

template <int RK, Form FORM>
cudaError_t launch_rk(const EcgFvParams& p, const double* in, double* out, EcgStepStats* stats, const EcgDtCtl& ctl,
                      cudaStream_t s)
{
  switch (p.limiter) {
    case ECG_LIMITER_MC: return launch_lim<RK, ECG_LIMITER_MC, FORM>(p, in, out, stats, ctl, s);
    case ECG_LIMITER_VANLEER: return launch_lim<RK, ECG_LIMITER_VANLEER, FORM>(p, in, out, stats, ctl, s);
    default: return launch_lim<RK, ECG_LIMITER_MINMOD, FORM>(p, in, out, stats, ctl, s);
  }
}

#ifndef ECG_FAST_KERNEL
// Exact build, every flux but XIE (launch_fv_step): 1280x320 HLLC 31.9 us
// against 42.8 on the 32x16 tiles, 2560x640 105 against 165, 128x128 7.1
// against 14.7.
inline cudaError_t launch(const EcgFvParams& p, const double* in, double* out, EcgStepStats* stats,
                          const EcgDtCtl& ctl, cudaStream_t s)
{
  switch (p.riemann) {
    case ECG_RIEMANN_RUSANOV: return launch_rk<ECG_RIEMANN_RUSANOV, Form::kStaged>(p, in, out, stats, ctl, s);
    case ECG_RIEMANN_LOWMACH_HLLC: return launch_rk<ECG_RIEMANN_LOWMACH_HLLC, Form::kStaged>(p, in, out, stats, ctl, s);
    default: return launch_rk<ECG_RIEMANN_HLLC, Form::kStaged>(p, in, out, stats, ctl, s);
  }
}
#else
template <int RK>
cudaError_t launch_form(const EcgFvParams& p, const double* in, double* out, EcgStepStats* stats, const EcgDtCtl& ctl,
                        cudaStream_t s, Form form)
{
  switch (form) {
    case Form::kStaged: return launch_rk<RK, Form::kStaged>(p, in, out, stats, ctl, s);
    case Form::kPaired: return launch_rk<RK, Form::kPaired>(p, in, out, stats, ctl, s);
    default: return launch_rk<RK, Form::kSingle>(p, in, out, stats, ctl, s);
  }
}

inline cudaError_t launch(const EcgFvParams& p, const double* in, double* out, EcgStepStats* stats,
                          const EcgDtCtl& ctl, cudaStream_t s, Form form)
{
  switch (p.riemann) {
    case ECG_RIEMANN_RUSANOV: return launch_form<ECG_RIEMANN_RUSANOV>(p, in, out, stats, ctl, s, form);
    case ECG_RIEMANN_LOWMACH_HLLC: return launch_form<ECG_RIEMANN_LOWMACH_HLLC>(p, in, out, stats, ctl, s, form);
    case ECG_RIEMANN_XIE_AM_HLLC_P: {
      // Staged strips carry the 5-face sensor along (2560x640 104 us against
      // the tile kernel's 150, 512x512 22.5 against 28.0, 128x128 7.2 against
      // 8.9); on grids of one to three 16x16 tiles an SM, where the strips
      // are too few and short and the tiles run as one wave, the tile kernel is
      // the faster (256x256 10.4 against 11.2, 333x331 12.8 against 14.0;
      // 512x256, 512 tiles, 18.1 against 14.2).  A band of rows (the pipelined
      // host step) takes the strips: the tile kernel steps whole grids only.
      const long long tiles = static_cast<long long>((p.g.nx + 15) / 16) * ((p.g.ny + 15) / 16);
      const long long sms = p.sm_count > 0 ? p.sm_count : 148;
      if (form == Form::kStaged && (p.row_hi > 0 || tiles <= sms || tiles > 3 * sms))
        return launch_rk<ECG_RIEMANN_XIE_AM_HLLC_P, Form::kStaged>(p, in, out, stats, ctl, s);
      return fast::launch(p, in, out, stats, ctl, s);
    }
    default: return launch_form<ECG_RIEMANN_HLLC>(p, in, out, stats, ctl, s, form);
  }
}

#endif

}  // namespace march
