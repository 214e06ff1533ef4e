// The arithmetic of the column strips (fv_march.cuh) in the exact build: the
// names the fast build defines in fv_fast.cuh, with the reference's IEEE
// expressions (ecg_device.cuh), for the fluxes the exact build's strips
// evaluate (HLLC-P stays on the tiles).  Included inside the ecg_exact namespace
// of stencil.cuh.  A face flux takes its branches as it goes; `fallback` then
// only reports a degenerate star state, whose face the strip evaluates once
// more for its count.
namespace fast {

__device__ __forceinline__ double frcp(double b) { return 1.0 / b; }
__device__ __forceinline__ Prim to_prim_f(const Cons& c, double g) { return to_prim(c, g); }
__device__ __forceinline__ double slope_f(double bk, double fw, int lim) { return limited_slope(bk, fw, lim); }
__device__ __forceinline__ double fsound_w(double rho, double p, double g) { return sqrt(g * p / rho); }

__device__ __forceinline__ Cons rusanov_f(const Prim& l, const Prim& r, int axis, double g, double)
{
  return rusanov_flux(l, r, axis, g);
}
__device__ __forceinline__ Cons rusanov_core(const Prim& l, const Prim& r, int axis, double g, double, bool& fallback)
{
  fallback = false;
  return rusanov_flux(l, r, axis, g);
}
__device__ __forceinline__ void lowmach_f(Prim& l, Prim& r, double g) { lowmach_correct(l, r, g); }
__device__ __forceinline__ Cons hllc_f(const Prim& l, const Prim& r, int axis, double g, double, bool& deg)
{
  return hllc_flux(l, r, axis, g, deg);
}
template <bool LM>
__device__ __forceinline__ Cons hllc_core(Prim l, Prim r, int axis, double g, double, bool& fallback)
{
  if (LM) lowmach_correct(l, r, g);
  return hllc_flux(l, r, axis, g, fallback);
}

}  // namespace fast
