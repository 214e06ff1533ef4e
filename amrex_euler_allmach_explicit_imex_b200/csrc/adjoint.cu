// Adjoint of the explicit step: ecg_explicit_step_device (the forward on
// caller arrays) and ecg_explicit_step_vjp_device (include/ecg.h).
//
// U1 = U0 - dt [ (F_{i+1/2} - F_{i-1/2}) / dx + (G_{j+1/2} - G_{j-1/2}) / dy ]
// (numerics/explicit_update.hpp:58-102) with dt held fixed, so
//   gU0 = gU1 + (dq/dU)^T gq,   gq = sum over faces f of (dF_f/dq)^T gF_f,
//   gF_{i+1/2} = dt/dx (gU1_{i+1} - gU1_i)   (and the same along y).
// One kernel does the whole transposed step on tiles of cells, gathering: it
// stages the primitives and the cotangent of a tile and its halo in shared
// memory, applies the transposed flux Jacobian of every face the tile's cells
// depend on (reverse mode, adjoint.cuh), and every cell collects the
// cotangents of its two faces and of the limited slopes it enters on each
// axis.  Cells that ghost cells copy collect those ghosts' cotangents too (the
// boundary policy transposed: outflow copies add to their source cell, the
// bubble wall mirror flips the v component, constant inflow states receive
// nothing; periodic axes wrap the tile instead).  No atomics: the result does
// not vary from run to run.
#include <cuda_runtime.h>

#include <cstring>

#include "ctx.h"
#include "ecg.h"

#include "adjoint.cuh"

namespace {

struct Src {
  int i, j;
  bool valid, flip;
};

__device__ __forceinline__ int wrapi(int i, int n)
{
  int r = i % n;
  return r < 0 ? r + n : r;
}

// Source cell of (i, j) under the ghost policy: the map of load_cell
// (problems/boundary_conditions.hpp:2-73) for the policies without a ring.
__device__ Src source_of(const EcgFvParams& P, int i, int j)
{
  const int nx = P.g.nx, ny = P.g.ny;
  Src s{i, j, true, false};
  if (i < 0) {
    if (P.bc.x_lo == BC_CONST) return Src{0, 0, false, false};
    s.i = P.bc.x_lo == BC_PERIODIC ? wrapi(i, nx) : 0;
  } else if (i >= nx) {
    if (P.bc.x_hi == BC_CONST) return Src{0, 0, false, false};
    s.i = P.bc.x_hi == BC_PERIODIC ? wrapi(i, nx) : nx - 1;
  }
  if (j < 0) {
    if (P.bc.y_lo == BC_CONST) return Src{0, 0, false, false};
    if (P.bc.y_lo == BC_PERIODIC) {
      s.j = wrapi(j, ny);
    } else if (P.bc.y_lo == BC_REFLECT) {
      s.j = -j - 1 > ny - 1 ? ny - 1 : -j - 1;
      s.flip = true;
    } else {
      s.j = 0;
    }
  } else if (j >= ny) {
    if (P.bc.y_hi == BC_CONST) return Src{0, 0, false, false};
    if (P.bc.y_hi == BC_PERIODIC) {
      s.j = wrapi(j, ny);
    } else if (P.bc.y_hi == BC_REFLECT) {
      s.j = 2 * ny - 1 - j < 0 ? 0 : 2 * ny - 1 - j;
      s.flip = true;
    } else {
      s.j = ny - 1;
    }
  }
  return s;
}

// Tiles of at most TX x TY cells, of equal sizes up to one (so a tile on a wall
// has both rows the wall mirrors, unless the grid has one row).  Staged per
// tile: primitives of the cells within 3 of it (the faces one beyond its own
// on each side and the slopes of their cells), cotangents within 2, and the
// two state cotangents of each face -1 .. w+1 of its rows and -1 .. h+1 of its
// columns.  632 faces over 320 threads: two a thread.
//
// Reverse mode costs about three flux evaluations a face where 16 forward
// directional derivatives, one per primitive of the 4-cell stencil, cost some
// thirty; with the gather in shared memory the 32 atomics a face and the
// separate pass over the cells are gone too: one VJP at 256x256 325 us (158 +
// 160 + 6 in three launches) -> 14.5 us (1024x1024: 178 us).
constexpr int TX = 32, TY = 8, NT = 320;
constexpr int PW = TX + 6, PH = TY + 6, PN = PW * PH;        // primitives, cells -3 .. T+2
constexpr int GW = TX + 4, GH = TY + 4, GN = GW * GH;        // cotangents, cells -2 .. T+1
constexpr int FXW = TX + 3, FYH = TY + 3;                    // faces -1 .. T+1
constexpr int FX = FXW * TY, FY = TX * FYH, FN = FX + FY;
constexpr size_t kSmem = sizeof(double) * (4 * PN + 4 * GN + 8 * FN);

template <int RK>
__global__ void __launch_bounds__(NT, 2)
step_vjp_kernel(const EcgFvParams P, const double* __restrict__ u0, const double* __restrict__ gu1, double dt,
                double* __restrict__ gu0, int tiles_x, int tiles_y)
{
  extern __shared__ double sh[];
  double* const prim = sh;           // 4 planes of PN: rho, u, v, p
  double* const gu = prim + 4 * PN;  // 4 planes of GN
  double* const gl = gu + 4 * GN;    // 4 planes of FN: cotangents of the faces' left / lower states
  double* const gr = gl + 4 * FN;    // and of their right / upper states
  const int nx = P.g.nx, ny = P.g.ny;
  const long long n = static_cast<long long>(nx) * ny;
  const int bx = static_cast<int>(blockIdx.x) % tiles_x, by = static_cast<int>(blockIdx.x) / tiles_x;
  auto cut = [](int cells, int k, int tiles) { return static_cast<int>(static_cast<long long>(cells) * k / tiles); };
  const int i0 = cut(nx, bx, tiles_x), w = cut(nx, bx + 1, tiles_x) - i0;
  const int j0 = cut(ny, by, tiles_y), h = cut(ny, by + 1, tiles_y) - j0;
  const bool per_x = P.bc.x_lo == BC_PERIODIC, per_y = P.bc.y_lo == BC_PERIODIC;
  const bool second = P.order > 1;
  const double g = P.gamma, inv_gm1 = 1.0 / (g - 1.0);
  const int tid = threadIdx.x;

  // ---- primitives (ghosts included: to_primitive, core/state_primitives.hpp:103-111) and cotangents ----
  for (int e = tid; e < PN; e += NT) {
    const int x = e % PW - 3, y = e / PW - 3;
    const Src s = source_of(P, i0 + x, j0 + y);
    double rho = P.bc.cst[0], mx = P.bc.cst[1], my = P.bc.cst[2], E = P.bc.cst[3];
    if (s.valid) {
      const long long o = static_cast<long long>(s.j) * nx + s.i;
      rho = u0[o];
      mx = u0[o + n];
      my = s.flip ? -u0[o + 2 * n] : u0[o + 2 * n];
      E = u0[o + 3 * n];
    }
    const double inv_rho = 1.0 / rho;
    const double uu = mx * inv_rho, vv = my * inv_rho;
    prim[e] = rho;
    prim[e + PN] = uu;
    prim[e + 2 * PN] = vv;
    prim[e + 3 * PN] = (g - 1.0) * (E - 0.5 * rho * (uu * uu + vv * vv));
  }
  for (int e = tid; e < GN; e += NT) {
    int i = i0 + e % GW - 2, j = j0 + e / GW - 2;
    if (per_x) i = wrapi(i, nx);
    if (per_y) j = wrapi(j, ny);
    const bool in = i >= 0 && i < nx && j >= 0 && j < ny;
    const long long o = static_cast<long long>(j) * nx + i;
#pragma unroll
    for (int m = 0; m < 4; ++m) gu[e + m * GN] = in ? gu1[o + m * n] : 0.0;
  }
  __syncthreads();

  // ---- faces: cotangents of the two states of each ----
  for (int e = tid; e < FN; e += NT) {
    const bool xf = e < FX;
    const int k = xf ? e : e - FX;
    // the cell on the face's right / upper side, and the step to its neighbour
    const int x = xf ? k % FXW - 1 : k % TX, y = xf ? k / FXW : k / TX - 1;
    const bool used = xf ? (x <= w + 1 && y < h) : (x < w && y <= h + 1);
    const int st = xf ? 1 : PW, gst = xf ? 1 : GW;
    const int c = (y + 3) * PW + x + 3, gc = (y + 2) * GW + x + 2;
    const double coef = dt * (xf ? P.g.inv_dx : P.g.inv_dy);
    double wf[4];
    bool any = false;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      wf[m] = used ? coef * (gu[gc + m * GN] - gu[gc - gst + m * GN]) : 0.0;
      any = any || wf[m] != 0.0;
    }
    ecg_adj::State dl{0.0, 0.0, 0.0, 0.0}, dr{0.0, 0.0, 0.0, 0.0};
    if (any) {
      double ql[4], qr[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const double* q = prim + m * PN + c;
        const double a = q[-2 * st], b = q[-st], d = q[0], f = q[st];
        ql[m] = second ? b + 0.5 * ecg_adj::limited(b - a, d - b, P.limiter).s : b;
        qr[m] = second ? d - 0.5 * ecg_adj::limited(d - b, f - d, P.limiter).s : d;
      }
      const ecg_adj::State l{ql[0], xf ? ql[1] : ql[2], xf ? ql[2] : ql[1], ql[3]};
      const ecg_adj::State r{qr[0], xf ? qr[1] : qr[2], xf ? qr[2] : qr[1], qr[3]};
      const ecg_adj::Flux wn{wf[0], xf ? wf[1] : wf[2], xf ? wf[2] : wf[1], wf[3]};
      ecg_adj::reverse_face<RK>(l, r, g, inv_gm1, wn, dl, dr);
    }
    gl[e] = dl.rho;
    gl[e + FN] = xf ? dl.un : dl.ut;
    gl[e + 2 * FN] = xf ? dl.ut : dl.un;
    gl[e + 3 * FN] = dl.p;
    gr[e] = dr.rho;
    gr[e + FN] = xf ? dr.un : dr.ut;
    gr[e + 2 * FN] = xf ? dr.ut : dr.un;
    gr[e + 3 * FN] = dr.p;
  }
  __syncthreads();

  // ---- cells: gather the primitive cotangent, then (dq/dU)^T ----
  for (int e = tid; e < TX * TY; e += NT) {
    const int x = e % TX, y = e / TX;
    if (x >= w || y >= h) continue;
    const int c = (y + 3) * PW + x + 3;
    double gq[4] = {0.0, 0.0, 0.0, 0.0};
    // The cotangent of cell k of this cell's row (AXIS 0) or column, one axis'
    // share: its two face states, and the slopes of cells k-1, k, k+1.  Faces
    // outside -1 .. T+1 have no cotangent; a slope without one is not evaluated.
    auto collect = [&](bool xa, int k, bool flip) {
      const int fbase = xa ? y * FXW + 1 : FX + TX + x, fst = xa ? 1 : TX;
      const int last = xa ? w + 1 : h + 1;
      const int pbase = xa ? c - x : c - y * PW, pst = xa ? 1 : PW;
      auto face = [&](const double* t, int f) { return f >= -1 && f <= last ? t[fbase + f * fst] : 0.0; };
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const double* L = gl + m * FN;
        const double* R = gr + m * FN;
        double v = face(L, k + 1) + face(R, k);
        if (second) {
          const double* q = prim + m * PN + pbase;
#pragma unroll
          for (int s = -1; s <= 1; ++s) {
            const int kk = k + s;
            const double gs = 0.5 * (face(L, kk + 1) - face(R, kk));
            if (gs != 0.0) {
              const double q0 = q[kk * pst];
              const ecg_adj::Slope sl = ecg_adj::limited(q0 - q[(kk - 1) * pst], q[(kk + 1) * pst] - q0, P.limiter);
              if (s == -1) v += gs * sl.db;
              else if (s == 0) v += gs * (sl.da - sl.db);
              else v -= gs * sl.da;
            }
          }
        }
        gq[m] += flip && m == 2 ? -v : v;
      }
    };
    collect(true, x, false);
    collect(false, y, false);
    const int gi = i0 + x, gj = j0 + y;
    if (!per_x) {
      // ghost columns copy the edge column (a constant inflow none)
      if (gi == 0 && P.bc.x_lo != BC_CONST) {
        collect(true, -1, false);
        collect(true, -2, false);
      }
      if (gi == nx - 1 && P.bc.x_hi != BC_CONST) {
        collect(true, w, false);
        collect(true, w + 1, false);
      }
    }
    if (!per_y && (gj < 2 || gj >= ny - 2)) {
      for (int t = 0; t < 4; ++t) {
        const int ghost = t < 2 ? -1 - t : ny + t - 2;
        const Src s = source_of(P, gi, ghost);
        if (s.valid && s.j == gj) collect(false, ghost - j0, s.flip);
      }
    }
    const double rho = prim[c], uu = prim[c + PN], vv = prim[c + 2 * PN];
    const double inv_rho = 1.0 / rho, gm1 = g - 1.0;
    const long long o = static_cast<long long>(gj) * nx + gi;
    const double* gc = gu + (y + 2) * GW + x + 2;
    gu0[o] = gc[0] + gq[0] - (gq[1] * uu + gq[2] * vv) * inv_rho + gq[3] * gm1 * 0.5 * (uu * uu + vv * vv);
    gu0[o + n] = gc[GN] + gq[1] * inv_rho - gq[3] * gm1 * uu;
    gu0[o + 2 * n] = gc[2 * GN] + gq[2] * inv_rho - gq[3] * gm1 * vv;
    gu0[o + 3 * n] = gc[3 * GN] + gq[3] * gm1;
  }
}

template <int RK>
cudaError_t launch_vjp(const EcgFvParams& p, const double* u0, const double* gu1, double dt, double* gu0,
                       cudaStream_t s)
{
  const cudaError_t e =
      cudaFuncSetAttribute(step_vjp_kernel<RK>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem));
  if (e != cudaSuccess) return e;
  const int tiles_x = (p.g.nx + TX - 1) / TX, tiles_y = (p.g.ny + TY - 1) / TY;
  step_vjp_kernel<RK><<<tiles_x * tiles_y, NT, kSmem, s>>>(p, u0, gu1, dt, gu0, tiles_x, tiles_y);
  return cudaGetLastError();
}

// Compact planes (i fastest, no padding) of the context's grid.
EcgFvParams compact_params(ecg_ctx* c)
{
  EcgFvParams p = ecgi::fv_params(c, false);
  p.g.pitch = c->grid.nx;
  p.g.plane = static_cast<long long>(c->grid.nx) * c->grid.ny;
  return p;
}

// The record the forward step reduces into; nothing reads it, so it is
// initialised once and left to accumulate.
bool ensure_stats(ecg_ctx* c)
{
  if (c->adj_stats) return true;
  return ecgi::cuda_ok(c, cudaMalloc(&c->adj_stats, sizeof(EcgStepStats)), "alloc adjoint stats") &&
         ecgi::cuda_ok(c, c->ops->init_stats(c->adj_stats, 1, 0.0, c->stream), "init stats");
}

// Whether two arrays of n doubles share a byte.
bool overlap(const double* a, const double* b, long long n)
{
  return a < b + n && b < a + n;
}

}  // namespace

extern "C" {

ecg_status ecg_explicit_step_device(ecg_ctx* c, const double* u0, double dt, double* u1)
{
  if (!c || !u0 || !u1 || u0 == u1) return ECG_ERR_BAD_ARG;
  const EcgFvParams p = compact_params(c);
  if (p.bc.ring) {
    c->err = "exact-Dirichlet ghost rings are not supported on caller arrays";
    return ECG_ERR_UNSUPPORTED;
  }
  if (!ensure_stats(c)) return ECG_ERR_CUDA;
  EcgDtCtl ctl;
  std::memset(&ctl, 0, sizeof(ctl));
  ctl.dt = dt;
  ctl.count_degenerate = c->cfg.riemann != ECG_RIEMANN_RUSANOV;
  ctl.read_slot = 0;
  ctl.acc_slot = 0;
  ctl.reset_slot = -1;
  if (!ecgi::cuda_ok(c, c->ops->fv_step(p, u0, u1, c->adj_stats, ctl, c->tile_y, c->stream), "fv_step"))
    return ECG_ERR_CUDA;
  return ECG_OK;
}

ecg_status ecg_explicit_step_vjp_device(ecg_ctx* c, const double* u0, double dt, const double* g_u1, double* g_u0)
{
  if (!c || !u0 || !g_u1 || !g_u0 || g_u1 == g_u0) return ECG_ERR_BAD_ARG;
  const EcgFvParams p = compact_params(c);
  if (p.bc.ring) {
    c->err = "exact-Dirichlet ghost rings are not supported by the adjoint";
    return ECG_ERR_UNSUPPORTED;
  }
  if (c->cfg.riemann == ECG_RIEMANN_XIE_AM_HLLC_P) {
    c->err = "the adjoint covers rusanov, hllc and lowmach_hllc";
    return ECG_ERR_UNSUPPORTED;
  }
  const long long n = 4LL * c->grid.nx * c->grid.ny;
  // Tiles read u0 and g_u1 around the cells other tiles write: a result that
  // lies on either of them goes through the context's scratch.
  const bool scratch = overlap(g_u0, u0, n) || overlap(g_u0, g_u1, n);
  if (scratch && !c->adj_gq &&
      !ecgi::cuda_ok(c, cudaMalloc(&c->adj_gq, sizeof(double) * n), "alloc adjoint"))
    return ECG_ERR_CUDA;
  double* out = scratch ? c->adj_gq : g_u0;
  cudaError_t e;
  switch (c->cfg.riemann) {
    case ECG_RIEMANN_RUSANOV: e = launch_vjp<ECG_RIEMANN_RUSANOV>(p, u0, g_u1, dt, out, c->stream); break;
    case ECG_RIEMANN_LOWMACH_HLLC: e = launch_vjp<ECG_RIEMANN_LOWMACH_HLLC>(p, u0, g_u1, dt, out, c->stream); break;
    default: e = launch_vjp<ECG_RIEMANN_HLLC>(p, u0, g_u1, dt, out, c->stream); break;
  }
  if (!ecgi::cuda_ok(c, e, "step vjp")) return ECG_ERR_CUDA;
  if (scratch && !ecgi::cuda_ok(c, cudaMemcpyAsync(g_u0, out, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream),
                                "copy vjp"))
    return ECG_ERR_CUDA;
  return ECG_OK;
}

}  // extern "C"
