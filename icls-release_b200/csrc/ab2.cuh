// ab2.cuh — the AB2 predictor (ab2.f90:21-138 with mom_main's RHS,
// mom.f90:13-301) as a kernel template.  k_navier.cu instantiates it for the
// plain FP64 path, compiled with -fmad=false so every expression keeps the
// reference's evaluation order; k_ab2_f32.cu instantiates the FP32 form,
// compiled with multiply-add contraction (that form is held to tolerances,
// not to the reference's rounding).  The device code sits in each file's
// own anonymous namespace.
#pragma once

#include <type_traits>

#include "batch.cuh"

namespace icls {

// the fields of the predictor, type-erased: all but rho_avr hold the form's
// field type (FP64, or FP32 in the precision form)
struct MomArgs {
  const double *u, *v, *w, *miu, *rho_u, *rho_v, *rho_w;
  const double *duold, *dvold, *dwold;
  const double *pnew, *pold, *px, *py, *pz, *pxold, *pyold, *pzold;
  const double* rho_avr;
  // far rows (k_ab2): one byte per tile and row, and nonzero where a pressure is not finite
  const uint8_t* near;
  const int* p_bad;
};

namespace {

// T is the form's field type (double, or float in the precision form);
// TC(x) is the constant x in T
#define TC(x) static_cast<T>(x)

// ---- RHS of mom_main for one component ----------------------------------
// U(di,dj,dk) returns u at (i+di, j+dj, k+dk), likewise V, W and M (miu):
// the same expressions serve the shared-memory march of k_ab2 and the
// global-memory k_mom_main.  T is the form's field type; TC(x) the
// constant x in T.  by_rho(x) is x over the component's face density.
template <typename T, int PW = -1, class FU, class FV, class FW, class FM, class FD>
__device__ __forceinline__ T rhs_u(const Params& p, const FU& U, const FV& V, const FW& W, const FM& M,
                                   const FD& by_rho, T rho_avr) {
  T RCu = TC(0.);
  if (!p.TwoD) {
    T uuip = TC(0.25) * (U(1, 0, 0) + U(0, 0, 0)) * (U(1, 0, 0) + U(0, 0, 0));
    T uuim = TC(0.25) * (U(-1, 0, 0) + U(0, 0, 0)) * (U(-1, 0, 0) + U(0, 0, 0));
    T uvjp = TC(0.25) * (U(0, 1, 0) + U(0, 0, 0)) * (V(1, 0, 0) + V(0, 0, 0));
    T uvjm = TC(0.25) * (U(0, -1, 0) + U(0, 0, 0)) * (V(1, -1, 0) + V(0, -1, 0));
    T uwkp = TC(0.25) * (U(0, 0, 1) + U(0, 0, 0)) * (W(1, 0, 0) + W(0, 0, 0));
    T uwkm = TC(0.25) * (U(0, 0, -1) + U(0, 0, 0)) * (W(1, 0, -1) + W(0, 0, -1));
    RCu = (divx<PW>(p, (-uuip + uuim)) + divy<PW>(p, (-uvjp + uvjm))) + divz<PW>(p, (-uwkp + uwkm));
  }
  T RDu = TC(0.);
  if (!p.TwoD) {
    T dudxp = divx<PW>(p, (U(1, 0, 0) - U(0, 0, 0)));
    T dudxm = divx<PW>(p, (U(0, 0, 0) - U(-1, 0, 0)));
    T dudyp = divy<PW>(p, (U(0, 1, 0) - U(0, 0, 0)));
    T dudym = divy<PW>(p, (U(0, 0, 0) - U(0, -1, 0)));
    T dvdxp = divx<PW>(p, (V(1, 0, 0) - V(0, 0, 0)));
    T dvdxm = divx<PW>(p, (V(1, -1, 0) - V(0, -1, 0)));
    T dudzp = divz<PW>(p, (U(0, 0, 1) - U(0, 0, 0)));
    T dudzm = divz<PW>(p, (U(0, 0, 0) - U(0, 0, -1)));
    T dwdxp = divx<PW>(p, (W(1, 0, 0) - W(0, 0, 0)));
    T dwdxm = divx<PW>(p, (W(1, 0, -1) - W(0, 0, -1)));
    T ma1 = TC(0.25) * (((M(0, 0, 0) + M(0, -1, 0)) + M(1, -1, 0)) + M(1, 0, 0));
    T ma2 = TC(0.25) * (((M(0, 0, 0) + M(0, 1, 0)) + M(1, 1, 0)) + M(1, 0, 0));
    T ma3 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, -1)) + M(1, 0, -1)) + M(1, 0, 0));
    T ma4 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, 1)) + M(1, 0, 1)) + M(1, 0, 0));
    T RD1 = divx<PW>(p, TC(2.) * (dudxp * M(1, 0, 0) - dudxm * M(0, 0, 0)));
    T RD2 = divy<PW>(p, (dudyp * ma2 - dudym * ma1));
    T RD3 = divy<PW>(p, (dvdxp * ma2 - dvdxm * ma1));
    T RD4 = divz<PW>(p, (dudzp * ma4 - dudzm * ma3));
    T RD5 = divz<PW>(p, (dwdxp * ma4 - dwdxm * ma3));
    RDu = by_rho((((RD1 + RD2) + RD3) + RD4) + RD5);
  }
  // buoyancy iFr (1 - rho_avr/rho) g: skipped (with its divide) where iFr or
  // this component of g is zero; the term is then an exact +-0, which
  // changes the sum at most in the sign of an exactly zero result
  if (p.TwoD || p.iFr == 0. || p.g1 == 0.) return RCu + RDu * TC(p.visc);
  T RGu = TC(p.iFr) * (TC(1.) - by_rho(rho_avr)) * TC(p.g1);
  return (RCu + RDu * TC(p.visc)) + RGu;
}

template <typename T, int PW = -1, class FU, class FV, class FW, class FM, class FD>
__device__ __forceinline__ T rhs_v(const Params& p, const FU& U, const FV& V, const FW& W, const FM& M,
                                   const FD& by_rho, T rho_avr) {
  T uvip = TC(0.25) * (U(0, 0, 0) + U(0, 1, 0)) * (V(0, 0, 0) + V(1, 0, 0));
  T uvim = TC(0.25) * (U(-1, 0, 0) + U(-1, 1, 0)) * (V(0, 0, 0) + V(-1, 0, 0));
  T vvjp = TC(0.25) * (V(0, 0, 0) + V(0, 1, 0)) * (V(0, 0, 0) + V(0, 1, 0));
  T vvjm = TC(0.25) * (V(0, 0, 0) + V(0, -1, 0)) * (V(0, 0, 0) + V(0, -1, 0));
  T wvkp = TC(0.25) * (W(0, 0, 0) + W(0, 1, 0)) * (V(0, 0, 1) + V(0, 0, 0));
  T wvkm = TC(0.25) * (W(0, 0, -1) + W(0, 1, -1)) * (V(0, 0, -1) + V(0, 0, 0));
  T RCv = (divx<PW>(p, (-uvip + uvim)) + divy<PW>(p, (-vvjp + vvjm))) + divz<PW>(p, (-wvkp + wvkm));
  T dvdxp = divx<PW>(p, (V(1, 0, 0) - V(0, 0, 0)));
  T dvdxm = divx<PW>(p, (V(0, 0, 0) - V(-1, 0, 0)));
  T dudyp = divy<PW>(p, (U(0, 1, 0) - U(0, 0, 0)));
  T dudym = divy<PW>(p, (U(-1, 1, 0) - U(-1, 0, 0)));
  T dvdyp = divy<PW>(p, (V(0, 1, 0) - V(0, 0, 0)));
  T dvdym = divy<PW>(p, (V(0, 0, 0) - V(0, -1, 0)));
  T dvdzp = divz<PW>(p, (V(0, 0, 1) - V(0, 0, 0)));
  T dvdzm = divz<PW>(p, (V(0, 0, 0) - V(0, 0, -1)));
  T dwdyp = divy<PW>(p, (W(0, 1, 0) - W(0, 0, 0)));
  T dwdym = divy<PW>(p, (W(0, 1, -1) - W(0, 0, -1)));
  T ma2 = TC(0.25) * (((M(0, 0, 0) + M(0, 1, 0)) + M(1, 1, 0)) + M(1, 0, 0));
  T ma5 = TC(0.25) * (((M(0, 0, 0) + M(0, 1, 0)) + M(-1, 1, 0)) + M(-1, 0, 0));
  T ma6 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, -1)) + M(0, 1, -1)) + M(0, 1, 0));
  T ma7 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, 1)) + M(0, 1, 1)) + M(0, 1, 0));
  T RD1 = divx<PW>(p, (dvdxp * ma2 - dvdxm * ma5));
  T RD2 = divx<PW>(p, (dudyp * ma2 - dudym * ma5));
  T RD3 = divy<PW>(p, TC(2.) * (dvdyp * M(0, 1, 0) - dvdym * M(0, 0, 0)));
  T RD4 = divz<PW>(p, (dvdzp * ma7 - dvdzm * ma6));
  T RD5 = divz<PW>(p, (dwdyp * ma7 - dwdym * ma6));
  T RDv = by_rho((((RD1 + RD2) + RD3) + RD4) + RD5);
  if (p.iFr == 0. || p.g2 == 0.) return RCv + RDv * TC(p.visc);  // buoyancy as in rhs_u
  T RGv = TC(p.iFr) * (TC(1.) - by_rho(rho_avr)) * TC(p.g2);
  return (RCv + RDv * TC(p.visc)) + RGv;
}

template <typename T, int PW = -1, class FU, class FV, class FW, class FM, class FD>
__device__ __forceinline__ T rhs_w(const Params& p, const FU& U, const FV& V, const FW& W, const FM& M,
                                   const FD& by_rho, T rho_avr) {
  T uwip = TC(0.25) * (W(0, 0, 0) + W(1, 0, 0)) * (U(0, 0, 0) + U(0, 0, 1));
  T uwim = TC(0.25) * (W(0, 0, 0) + W(-1, 0, 0)) * (U(-1, 0, 0) + U(-1, 0, 1));
  T vwjp = TC(0.25) * (W(0, 0, 0) + W(0, 1, 0)) * (V(0, 0, 0) + V(0, 0, 1));
  T vwjm = TC(0.25) * (W(0, 0, 0) + W(0, -1, 0)) * (V(0, -1, 0) + V(0, -1, 1));
  T wwkp = TC(0.25) * (W(0, 0, 0) + W(0, 0, 1)) * (W(0, 0, 0) + W(0, 0, 1));
  T wwkm = TC(0.25) * (W(0, 0, 0) + W(0, 0, -1)) * (W(0, 0, 0) + W(0, 0, -1));
  T RCw = (divx<PW>(p, (-uwip + uwim)) + divy<PW>(p, (-vwjp + vwjm))) + divz<PW>(p, (-wwkp + wwkm));
  T dwdxp = divx<PW>(p, (W(1, 0, 0) - W(0, 0, 0)));
  T dwdxm = divx<PW>(p, (W(0, 0, 0) - W(-1, 0, 0)));
  T dudzp = divz<PW>(p, (U(0, 0, 1) - U(0, 0, 0)));
  T dudzm = divz<PW>(p, (U(-1, 0, 1) - U(-1, 0, 0)));
  T dwdyp = divy<PW>(p, (W(0, 1, 0) - W(0, 0, 0)));
  T dwdym = divy<PW>(p, (W(0, 0, 0) - W(0, -1, 0)));
  T dvdzp = divz<PW>(p, (V(0, 0, 1) - V(0, 0, 0)));
  T dvdzm = divz<PW>(p, (V(0, -1, 1) - V(0, -1, 0)));
  T dwdzp = divz<PW>(p, (W(0, 0, 1) - W(0, 0, 0)));
  T dwdzm = divz<PW>(p, (W(0, 0, 0) - W(0, 0, -1)));
  T ma4 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, 1)) + M(1, 0, 1)) + M(1, 0, 0));
  T ma8 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, 1)) + M(-1, 0, 1)) + M(-1, 0, 0));
  T ma7 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, 1)) + M(0, 1, 1)) + M(0, 1, 0));
  T ma9 = TC(0.25) * (((M(0, 0, 0) + M(0, 0, 1)) + M(0, -1, 1)) + M(0, -1, 0));
  T RD1 = divx<PW>(p, (dwdxp * ma4 - dwdxm * ma8));
  T RD2 = divx<PW>(p, (dudzp * ma4 - dudzm * ma8));
  T RD3 = divy<PW>(p, (dwdyp * ma7 - dwdym * ma9));
  T RD4 = divy<PW>(p, (dvdzp * ma7 - dvdzm * ma9));
  T RD5 = divz<PW>(p, TC(2.) * (dwdzp * M(0, 0, 1) - dwdzm * M(0, 0, 0)));
  T RDw = by_rho((((RD1 + RD2) + RD3) + RD4) + RD5);
  if (p.iFr == 0. || p.g3 == 0.) return RCw + RDw * TC(p.visc);  // buoyancy as in rhs_u
  T RGw = TC(p.iFr) * (TC(1.) - by_rho(rho_avr)) * TC(p.g3);
  return (RCw + RDw * TC(p.visc)) + RGw;
}

// ---- the ab2 update of one component (ab2.f90:51-61, 79-129) -------------
// u0 = u at the cell, R = its mom_main RHS, rold the previous RHS, irf one
// over its face density, dhi the 1/dx of the component's axis; the pressure-split
// term is formed in FP64 (the pressures are FP64 fields) from: ph_p / ph_0 the
// extrapolated pressures 2 pnew - pold at the + neighbour and the cell,
// pjh the extrapolated pressure gradient 2 p_x - p_x,old
// PT is the pressure term's arithmetic: FP64 in the plain path; in the FP32
// form, whose pressures are stored in FP32, the term is formed in FP32 too
// (it is part of the momentum predictor, which that form computes in FP32)
template <typename T, typename PT>
__device__ __forceinline__ T ab2_update_v(const Params& p, T u0, T R, T rold, PT irf, PT ph_p, PT ph_0, PT pjh,
                                          double dhi) {
  T d = u0 + TC(p.dt) * (TC(1.5) * R - TC(0.5) * rold);
  const PT dn = -((irf - (PT)p.rrho0) * (PT)dhi * ((ph_p - pjh) - ph_0));
  return d + TC((PT)p.dt * dn);
}

// element copies global -> shared that complete asynchronously (waited for
// with cp_async_wait_all before the block's barrier)
template <typename T>
__device__ __forceinline__ void cp_async_el(T* dst, const T* src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
// two consecutive elements (8 bytes in FP32, 16 in FP64); both addresses
// aligned to the pair's size
template <typename T>
__device__ __forceinline__ void cp_async_pair(T* dst, const T* src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ab2 over shape C with bounduvw(dudt,dvdt,dwdt) (bound.f90:36-75) in-kernel.
// A block is a 32 x 8 column tile marching up a chunk of interior rows.
// u, v, w, miu (tile plus one halo column each side) and pnew, pold (tile
// plus the + neighbours in x and y) pass through a four-plane shared-memory
// ring filled by asynchronous copies: at row k the block issues row k+1's
// planes and this cell's own operands together, then waits once, so one
// memory latency is exposed per row and the ring needs one barrier per row
// (the slot a row's copies fill is not one any thread can still be reading).
// A thread writes its column's periodic halo images and, at k = 1 and
// k = kmax, the wall rows k = 0 and k = k1.  Every plane row starts at
// column i0 - 1 (even).  Indices are 32-bit: an array has less than 2^30
// elements.
//
// FAR: rows that a byte per tile and row (k_ab2_near) says have no drop next
// to them.  There the viscosity and the face densities are the carrier's and
// the face jumps zero, so these ten of the 24 fields are not read, and the row
// runs the same expressions with one viscosity and one density: the same
// bits.  Where the carrier is the lighter phase the pressure-split factor
// 1/rho1 - 1/rho0 is exactly zero too, and while every pressure is finite
// (p_bad) its product is: the two pressures are not read either.  Three
// quarters of the rows are far at 256^3 with 48 drops.  FAR false: the fields
// were written by a caller, every row is general.
// The planes arrive one row ahead of their use, and so do the AB2 history
// values; a near row's other operands are read at the row.  (Waiting for a
// row's planes right after issuing them, the long-scoreboard and barrier
// stalls were a third of the FP64 form's issue slots.)
//
// 256^3 with 48 drops, k_ab2_near (0.013 ms) included: FP64 0.843 -> 0.626 ms,
// FP32 0.489 -> 0.357 ms; every row general: 256^3 FP64 0.865 -> 0.788 ms, 384 x
// 192 x 150 FP32 0.305 -> 0.283 ms.  The general FP32 row issues in 76 % of the
// cycles and waits two more per issue on global loads, the nine operands that
// are read at the row.  FP64
// takes two blocks per SM at 128 registers (three at 80: 0.660 and 0.808 ms),
// FP32 four.  Two cells per thread (adjacent in y, sharing their stencil) were
// slower in both forms (FP64 0.743, FP32 0.396): the registers they take cost
// more warps than the shared loads save.
constexpr int MX = kAb2X, MY = kAb2Y, MSX = MX + 2, MSY = MY + 2, MPY = MY + 1, MRING = 4;
static_assert(MX == kSeg, "a tile is one segment wide");
template <typename T>
constexpr int ab2_smem() {
  return (int)(4 * MRING * MSY * MSX * sizeof(T) + 2 * MRING * MPY * MSX * sizeof(T));
}
template <typename T, int PW, int MB, bool FAR>
__global__ void __launch_bounds__(MX * MY, MB)
    k_ab2(Params p, MomArgs a, T* __restrict__ dudt, T* __restrict__ dvdt, T* __restrict__ dwdt,
          T* __restrict__ duold_out, T* __restrict__ dvold_out, T* __restrict__ dwold_out, int kc) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char ab2_dyn[];
  typedef T PT;  // the pressure term's arithmetic
  typedef T Plane[MSY][MSX];
  typedef T PPlane[MPY][MSX];  // pnew, pold (columns i0-1.., rows j0..) in the form's field type
  constexpr int NTH = MX * MY;
  Plane* ring = reinterpret_cast<Plane*>(ab2_dyn);  // [field * MRING + slot]
  PPlane* pring = reinterpret_cast<PPlane*>(ab2_dyn + 4 * MRING * sizeof(Plane));
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + MX * ty;
  const int i0 = 1 + MX * (int)blockIdx.x, j0 = 1 + MY * (int)blockIdx.y;
  const int ka = 1 + (int)blockIdx.z * kc, kb = blockIdx.z == gridDim.z - 1 ? p.kmax : ka + kc - 1;
  const int i = i0 + tx, j = j0 + ty;
  const bool ok = i <= p.imax && j <= p.jmax;
  // imax is even (every FFT length validate() admits is), so the rows of
  // shape C have an even length and each plane row's first element (column
  // i0-1, even) sits at an even index: pair copies (8 bytes in FP32, 16 in
  // FP64) are aligned.
  // This thread's copy slots, the same for every row: slot r is the pair
  // tid + r 256 of a plane, at plane offset gi + nCx gj of storage row 0 (row
  // kk is kk nCx nCy further), -1 where it lies outside the grid.
  constexpr int RW = MSX / 2;  // copies per plane row
  constexpr int NS = (RW * MSY + NTH - 1) / NTH;
  int ro[NS], po[NS];
#pragma unroll
  for (int r = 0; r < NS; ++r) {
    const int e = tid + r * NTH;
    const int sy = e / RW, gi = i0 - 1 + 2 * (e - sy * RW);
    // gi even: gi + 1 <= imax + 1
    ro[r] = (e < RW * MSY && gi <= p.imax && j0 - 1 + sy <= p.jmax + 1) ? gi + p.nCx * (j0 - 1 + sy) : -1;
    // pnew, pold rows start at j0
    po[r] = (e < RW * MPY && gi <= p.imax && j0 + sy <= p.jmax + 1) ? gi + p.nCx * (j0 + sy) : -1;
  }
  const int psz = p.nCx * p.nCy;
  const T* __restrict__ fu = cT<T>(a.u);
  const T* __restrict__ fv = cT<T>(a.v);
  const T* __restrict__ fw = cT<T>(a.w);
  auto issue_uvw = [&](int kk) {
    const int s = kk & (MRING - 1), o = kk * psz;
#pragma unroll
    for (int r = 0; r < NS; ++r)
      if (ro[r] >= 0) {
        const int g = o + ro[r], e = 2 * (tid + r * NTH);
        cp_async_pair(&ring[0 * MRING + s][0][0] + e, fu + g);
        cp_async_pair(&ring[1 * MRING + s][0][0] + e, fv + g);
        cp_async_pair(&ring[2 * MRING + s][0][0] + e, fw + g);
      }
  };
  auto issue_miu = [&](int kk) {
    const int s = kk & (MRING - 1), o = kk * psz;
#pragma unroll
    for (int r = 0; r < NS; ++r)
      if (ro[r] >= 0) cp_async_pair(&ring[3 * MRING + s][0][0] + 2 * (tid + r * NTH), cT<T>(a.miu) + (o + ro[r]));
  };
  auto issue_p = [&](int kk) {
    const int s = kk & (MRING - 1), o = kk * psz;
#pragma unroll
    for (int r = 0; r < NS; ++r)
      if (po[r] >= 0) {
        const int g = o + po[r], e = 2 * (tid + r * NTH);
        cp_async_pair(&pring[s][0][0] + e, cT<T>(a.pnew) + g);
        cp_async_pair(&pring[MRING + s][0][0] + e, cT<T>(a.pold) + g);
      }
  };
  const T rho1 = TC(p.rho1), miu1 = TC(p.miu1), rrho1 = TC(p.rrho1);
  const PT irho1 = PT(1.) / (PT)rho1;
  __shared__ uint8_t near_row[kAb2Rows + 2];  // [1 + r] row ka + r; 0 before the first and after the last
  bool noP = false;
  if constexpr (FAR) {
    noP = *a.p_bad == 0 && irho1 - (PT)p.rrho0 == PT(0.);
    const uint8_t* near = a.near + ((long long)blockIdx.x + (long long)gridDim.x * blockIdx.y) * p.nCz + ka;
    if (tid < kAb2Rows + 2) near_row[tid] = (tid >= 1 && tid <= kb - ka + 1) ? near[tid - 1] : 0;
  }
  // row kk of the viscosity is read by the near rows among kk-1..kk+1, of
  // the pressures by rows kk-1 and kk
  auto near_at = [&](int k) -> bool { return !FAR || near_row[1 + k - ka]; };
  auto issue_rest = [&](int kk) {
    const bool lo = kk > ka && near_at(kk - 1), at = kk >= ka && kk <= kb && near_at(kk);
    if (lo || at || (kk < kb && near_at(kk + 1))) issue_miu(kk);
    if (!noP || lo || at) issue_p(kk);
  };
  issue_uvw(ka - 1);
  issue_uvw(ka);
  issue_uvw(ka + 1);
  if constexpr (FAR) __syncthreads();
  issue_rest(ka - 1);
  issue_rest(ka);
  issue_rest(ka + 1);
  const T rho_avr = TC(*a.rho_avr);
  // the thread's column in the arrays, and its periodic images
  const int cc0 = i + p.nCx * j, q0 = (i - 1) + p.imax * (j - 1), szI = p.imax * p.jmax;
  const int di = i == 1 ? p.imax : (i == p.imax ? -p.imax : 0);
  const int dj = j == 1 ? p.nCx * p.jmax : (j == p.jmax ? -p.nCx * p.jmax : 0);
  auto put = [&](T* __restrict__ f, int c, T v) {
    f[c] = v;
    if (di) f[c + di] = v;
    if (dj) {
      f[c + dj] = v;
      if (di) f[c + di + dj] = v;
    }
  };
  T dw_km1 = TC(0.), ou = TC(0.), ov = TC(0.), ow = TC(0.);
  auto history = [&](int k) {
    if (!ok) return;
    const int q = q0 + (k - 1) * szI;
    ou = cT<T>(a.duold)[q];
    ov = cT<T>(a.dvold)[q];
    ow = cT<T>(a.dwold)[q];
  };
  history(ka);
  for (int k = ka; k <= kb; ++k) {
    const bool near = near_at(k);
    const int c = cc0 + k * psz, q = q0 + (k - 1) * szI;
    T ru = rho1, rv = rho1, rw = rho1;
    PT jx = PT(0.), jy = PT(0.), jz = PT(0.);
    if (near && ok) {  // the near row's own operands
      ru = cT<T>(a.rho_u)[q]; rv = cT<T>(a.rho_v)[q]; rw = cT<T>(a.rho_w)[q];
      jx = PT(2.) * cT<T>(a.px)[c] - cT<T>(a.pxold)[c];
      jy = PT(2.) * cT<T>(a.py)[c] - cT<T>(a.pyold)[c];
      jz = PT(2.) * cT<T>(a.pz)[c] - cT<T>(a.pzold)[c];
    }
    cp_async_wait_all();  // row k+1's planes, issued a row ago
    __syncthreads();      // everyone's; and everyone is done with the slot of row k-2
    if (k < kb) {
      issue_uvw(k + 2);
      issue_rest(k + 2);
    }
    const int s_m = (k - 1) & (MRING - 1), s_0 = k & (MRING - 1), s_p = (k + 1) & (MRING - 1);
    auto sl = [&](int dk) { return dk < 0 ? s_m : (dk > 0 ? s_p : s_0); };
    auto U = [&](int di, int dj, int dk) { return ring[0 * MRING + sl(dk)][ty + 1 + dj][tx + 1 + di]; };
    auto V = [&](int di, int dj, int dk) { return ring[1 * MRING + sl(dk)][ty + 1 + dj][tx + 1 + di]; };
    auto W = [&](int di, int dj, int dk) { return ring[2 * MRING + sl(dk)][ty + 1 + dj][tx + 1 + di]; };
    auto M = [&](int di, int dj, int dk) { return ring[3 * MRING + sl(dk)][ty + 1 + dj][tx + 1 + di]; };
    auto PH = [&](int di, int dj, int dk) {
      return PT(2.) * (PT)pring[sl(dk)][ty + dj][tx + 1 + di] - (PT)pring[MRING + sl(dk)][ty + dj][tx + 1 + di];
    };
    T Ru, Rv, Rw, du, dv, dw;
    if (near) {
      Ru = rhs_u<T, PW>(p, U, V, W, M, [&](T x) { return x / ru; }, rho_avr);
      Rv = rhs_v<T, PW>(p, U, V, W, M, [&](T x) { return x / rv; }, rho_avr);
      Rw = rhs_w<T, PW>(p, U, V, W, M, [&](T x) { return x / rw; }, rho_avr);
    } else {
      auto M1 = [&](int, int, int) { return miu1; };
      // a power-of-two density: the product by its reciprocal is the quotient
      auto by_rho = [&](T x) { return p.rho1_pow2 ? x * rrho1 : x / rho1; };
      Ru = rhs_u<T, PW>(p, U, V, W, M1, by_rho, rho_avr);
      Rv = rhs_v<T, PW>(p, U, V, W, M1, by_rho, rho_avr);
      Rw = rhs_w<T, PW>(p, U, V, W, M1, by_rho, rho_avr);
    }
    if (near || !noP) {
      const PT ph0 = PH(0, 0, 0);
      const PT iu = near ? PT(1.) / (PT)ru : irho1, iv = near ? PT(1.) / (PT)rv : irho1,
               iw = near ? PT(1.) / (PT)rw : irho1;
      du = ab2_update_v<T, PT>(p, U(0, 0, 0), Ru, ou, iu, PH(1, 0, 0), ph0, jx, p.dxi);
      dv = ab2_update_v<T, PT>(p, V(0, 0, 0), Rv, ov, iv, PH(0, 1, 0), ph0, jy, p.dyi);
      dw = ab2_update_v<T, PT>(p, W(0, 0, 0), Rw, ow, iw, PH(0, 0, 1), ph0, jz, p.dzi);
    } else {
      du = U(0, 0, 0) + TC(p.dt) * (TC(1.5) * Ru - TC(0.5) * ou);
      dv = V(0, 0, 0) + TC(p.dt) * (TC(1.5) * Rv - TC(0.5) * ov);
      dw = W(0, 0, 0) + TC(p.dt) * (TC(1.5) * Rw - TC(0.5) * ow);
    }
    if (p.forceytot != 0.) dv = dv - TC(p.forceytot * p.dt) / rv;  // constPoi driving (exact zero otherwise)
    if (k < kb) history(k + 1);
    if (!ok) continue;
    duold_out[q] = Ru;
    dvold_out[q] = Rv;
    dwold_out[q] = Rw;
    if (k == p.kmax - 1) dw_km1 = dw;
    if (k == p.kmax) dw = TC(0.);
    put(dudt, c, du);
    put(dvdt, c, dv);
    put(dwdt, c, dw);
    if (k == 1) {
      put(dudt, c - psz, -du);
      put(dvdt, c - psz, TC(2. * p.v_lower) - dv);
      put(dwdt, c - psz, TC(0.));
    }
    if (k == p.kmax) {
      put(dudt, c + psz, -du);
      put(dvdt, c + psz, TC(2. * p.v_upper) - dv);
      put(dwdt, c + psz, dw_km1);
    }
  }
}

template <typename T>
T* ab2_ptr(double* q) { return reinterpret_cast<T*>(q); }

template <typename T, int PW, int MB, bool FAR>
void ab2_launch_far(Ctx& c, const MomArgs& a, int o) {
  int kc;
  const dim3 grid = ab2_grid(c.P, sizeof(T) == 8, kc);
  static unsigned attr = 0;  // devices this instance's shared-memory limit is raised on
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr & (1u << (dev & 31)))) {
    cudaFuncSetAttribute(k_ab2<T, PW, MB, FAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, ab2_smem<T>());
    attr |= 1u << (dev & 31);
  }
  pdl(k_ab2<T, PW, MB, FAR>, grid, dim3(MX, MY, 1), ab2_smem<T>(), c.s)(
      c.P, a, ab2_ptr<T>(c.dudt), ab2_ptr<T>(c.dvdt), ab2_ptr<T>(c.dwdt), ab2_ptr<T>(c.duold[o]),
      ab2_ptr<T>(c.dvold[o]), ab2_ptr<T>(c.dwold[o]), kc);
}
template <typename T, int PW, int MB>
void ab2_launch_pw(Ctx& c, const MomArgs& a, int o) {
  if (a.near) ab2_launch_far<T, PW, MB, true>(c, a, o);
  else ab2_launch_far<T, PW, MB, false>(c, a, o);
}
// one instance per spacing case: with power-of-two spacings every a/dx is
// the product, so neither the test nor the division is in the kernel.  The
// FP32 form, held to tolerances rather than to the reference's rounding,
// always takes the product by the reciprocal (within an ulp of the quotient).
// The instance's blocks per SM as measured (k_ab2).
template <typename T>
void ab2_launch(Ctx& c, const MomArgs& a, int o) {
  if constexpr (sizeof(T) == 8) {
    if (c.P.pow2) ab2_launch_pw<T, 1, 2>(c, a, o);
    else ab2_launch_pw<T, 0, 2>(c, a, o);
  } else {
    ab2_launch_pw<T, 1, 4>(c, a, o);
  }
}

#undef TC
}  // namespace

// the FP32 form's instance (k_ab2_f32.cu)
void ab2_launch_f32(Ctx& c, const MomArgs& a, int o);
// the TMA-fed FP64 predictor (k_ab2_tma.cu); false when it does not apply
bool ab2_tma_launch(Ctx& c, const MomArgs& a, int o);

}  // namespace icls
