// k_levelset.cu — level-set kernels of the ICLS hot path (FP64, -fmad=false).
//
//   tube_construction  levelset.f90:87-197
//   HOUC5_nb/WENO5_nb  hyperPDE.f90:397-800, fused with RK_nb
//                      levelset.f90:342-367 and boundsls bound.f90:386-483
//   ls_reinit          levelset.f90:619-882 with WENO5_reinit/WENO5_deri
//                      hyperPDE.f90:2646-2746, 2932-3197
//   inflation          levelset.f90:407-582
//   update_materials   misc.f90:79-290 with Heaviside 'trig' misc.f90:297-464
//
// Halo handling: instead of a separate boundsls pass, a thread computes an
// interior column and writes it together with its periodic halo images;
// the wall rows k=0 and k=k1 are the linear extrapolation of the two
// interior values next to them, evaluated by the thread that computes
// those.  This reproduces boundsls (z-extrapolation, then periodic x, then
// periodic y) exactly, because the inputs satisfy the periodic halo
// invariant.
//
// Sweep regions: after tube_construction clips the level set to +-6dz,
// every cell outside a drop's band holds the same far-field value, and
// every kernel maps a uniform neighbourhood to a uniform value (the
// stencils of a constant field are exactly zero).  Each per-drop kernel
// therefore sweeps only a region around the band (periodic column spans in
// x and y, rows in z) and writes the far-field value, replayed on the host
// with the same arithmetic, into a 3-cell apron around it; reads never
// leave the region plus apron.  All drops of a step go through one launch
// per stage (batch.cuh).
//
// In-place stages: the last RK stage may write the array it takes as its
// pointwise base (phi0): a thread reads phi0 only in its own column, and
// it writes a wall row only after it has computed the rows it extrapolates.
#include <algorithm>
#include <climits>

#include "batch.cuh"

namespace icls {

namespace {

constexpr int NT = TBX * TBY;
const dim3 kTile(TBX, TBY, 1);
const dim3 kBlock(BX, BY, 1);

// T is the type the level-set fields are stored and computed in: double
// for the reference form, float for the precision form.  TC(x) is the
// constant x in T.
#define TC(x) static_cast<T>(x)

template <typename T>
__device__ __forceinline__ T clipNB(T x, T NB) {
  return x > NB ? NB : (x < -NB ? -NB : x);
}
__device__ __forceinline__ bool interior(const Params& p, int i, int j, int k) {
  return i >= 1 && i <= p.imax && j >= 1 && j <= p.jmax && k >= 1 && k <= p.kmax;
}

// ---------------------------------------------------------------- band extents
// The band box a tube_construction sweep of the whole array would measure
// (the cells of rows -2..k1+2 whose clipped value differs from +NB, rows 0
// and k1 by the wall extrapolation), in the same two frames per periodic
// axis, without writing anything: one thread per (i,j) column.
template <typename T>
__global__ void __launch_bounds__(NT) k_band_extents(Params p, const T* __restrict__ phi, int l,
                                                     int* __restrict__ bbox_lo, int* __restrict__ bbox_hi) {
  pdl_wait();
  const long long q = blockIdx.x * (long long)NT + threadIdx.x;
  int lo[5] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX, INT_MAX};
  int hi[5] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN, INT_MIN};
  if (q < (long long)p.imax * p.jmax) {
    const int i = (int)(q % p.imax) + 1, j = (int)(q / p.imax) + 1;
    const int hx = p.imax / 2, hy = p.jmax / 2;
    const int ib = i + hx > p.imax ? i + hx - p.imax : i + hx;
    const int jb = j + hy > p.jmax ? j + hy - p.jmax : j + hy;
    const T NB = TC(p.NB);
    const long long sz = (long long)p.nLx * p.nLy, c0 = idxL(p, i, j, 0);
    for (int k = -2; k <= p.k1 + 2; ++k) {
      T val;
      if (k == 0)
        val = TC(2.) * clipNB(phi[c0 + sz], NB) - clipNB(phi[c0 + 2 * sz], NB);
      else if (k == p.k1)
        val = TC(2.) * clipNB(phi[c0 + p.kmax * sz], NB) - clipNB(phi[c0 + (p.kmax - 1) * sz], NB);
      else
        val = clipNB(phi[c0 + k * sz], NB);
      if (val != NB) {
        lo[0] = min(lo[0], i); hi[0] = max(hi[0], i);
        lo[1] = min(lo[1], ib); hi[1] = max(hi[1], ib);
        lo[2] = min(lo[2], j); hi[2] = max(hi[2], j);
        lo[3] = min(lo[3], jb); hi[3] = max(hi[3], jb);
        lo[4] = min(lo[4], k); hi[4] = max(hi[4], k);
      }
    }
  }
  for (int a = 0; a < 5; ++a) {
    int lv = lo[a], h = hi[a];
    for (int o = 16; o > 0; o >>= 1) {
      lv = min(lv, __shfl_down_sync(0xffffffffu, lv, o));
      h = max(h, __shfl_down_sync(0xffffffffu, h, o));
    }
    if ((threadIdx.x & 31) == 0 && lv != INT_MAX) {
      atomicMin(&bbox_lo[5 * l + a], lv);
      atomicMax(&bbox_hi[5 * l + a], h);
    }
  }
}

// ---------------------------------------------------------------- tube
// A band cell of a batch: (i-1) | (j-1) << 12 | task << 24, and k.
struct BandCell {
  unsigned ijt;
  int k;
};

// Appends the cells that the block's threads marked (bit r of rows: row ka + r
// of the thread's column) to the list (null: counts only): one addition to the
// counter per block; within a warp the rows in order, lanes (x fastest) within
// a row.  Returns the block's number of cells (in thread 0).
__device__ __forceinline__ int append_cells(unsigned rows, int ka, unsigned ijt, BandCell* __restrict__ list,
                                            int* __restrict__ count) {
  __shared__ int wsum[NT / 32], base_sh;
  const int lane = flat_tid() & 31, warp = flat_tid() >> 5;
  const unsigned any = __reduce_or_sync(0xffffffffu, rows);
  int n = 0, tot = 0;
  for (unsigned r = any; r; r &= r - 1) n += __popc(__ballot_sync(0xffffffffu, rows >> (__ffs(r) - 1) & 1u));
  if (lane == 0) wsum[warp] = n;
  __syncthreads();
  if (flat_tid() == 0) {
    for (int w = 0; w < NT / 32; ++w) {
      const int v = wsum[w];
      wsum[w] = tot;
      tot += v;
    }
    base_sh = (tot && list) ? atomicAdd(count, tot) : 0;
  }
  __syncthreads();
  if (list && n) {
    int at = base_sh + wsum[warp];
    for (unsigned r = any; r; r &= r - 1) {
      const int row = __ffs(r) - 1;
      const unsigned m = __ballot_sync(0xffffffffu, rows >> row & 1u);
      if (rows >> row & 1u) list[at + __popc(m & ((1u << lane) - 1u))] = BandCell{ijt, ka + row};
      at += __popc(m);
    }
  }
  return tot;
}

// Clip to +-NB (levelset.f90:120-128) and the band mask (130-160) over the
// tasks' regions.  phi0 holds valid data on vin's written cells, bgin
// (rows 0..k1) or bggin (ghost rows) elsewhere.  Counts the band per drop
// and records the extent of the cells whose clipped value is not +NB:
// bbox_lo[5 l + a], bbox_hi[5 l + a] for a = x, x shifted by imax/2, y, y
// shifted by jmax/2, z.  A far-field cell is outside the band only if all
// 15 axial neighbours clip to +-NB, so the test stops at the first that
// does not (the reference's sums of |clip|-NB <= 0 are zero exactly then).
//
// With a list, the band cells of the batch are also appended to it for the
// advection stages (k_adv_band), and the clipped values go to out2 and out3
// as well, where those stages read neighbours that they do not write.
//
// A thread marches one column of a flat tile up a chunk of at most 31 rows.
// It reads its own column once (a register window of five rows) and the
// eight x and y neighbours within two cells; each neighbouring column is
// either held by the input region or far field throughout.  Bound by
// instruction issue: the version before staged 2-D tiles of flags in shared
// memory with a barrier per row and 64-bit index products per store, 580
// instructions a warp row.  With the list and the two more copies a sweep
// takes 0.244 ms instead of 0.203 (256^3 x 48, FP64; FP32 0.136 instead of
// 0.140), and the three stages 0.34 instead of 0.67 ms (FP32 0.19 instead of
// 0.31).  Chunks of 8 rows (16: 0.254 and 0.161 ms, one drop at 64^3 28 instead
// of 22 us).
constexpr int kTubeRows = 8;
template <typename T>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 5 : 4)) k_tube(Params p, const __grid_constant__ LsBatch B,
                                             long long* __restrict__ cnt, int* __restrict__ bbox_lo,
                                             int* __restrict__ bbox_hi, BandCell* __restrict__ list,
                                             int* __restrict__ count) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  const T NB = TC(p.NB);
  const T bgin = TC(t.bgin), bggin = TC(t.bggin);
  const int sy = p.nLx, sz = p.nLx * p.nLy, szI = p.imax * p.jmax;
  const int i = c.i, j = c.j;
  unsigned rows = 0;  // bit r: row ka + r is a band cell
  int kmin = INT_MAX, kmax = INT_MIN;
  if (c.ok) {
    const int col = (int)idxL(p, i, j, 0);
    const T* __restrict__ in = cT<T>(t.phi0) + col;
    T* const out = mT<T>(t.out);
    T* const out2 = list ? mT<T>(t.out2) : nullptr;
    T* const out3 = list ? mT<T>(t.out3) : nullptr;
    // the column's storage and that of its periodic images
    const int ii = image_of<3>(i, p.imax), jj = image_of<3>(j, p.jmax);
    const int o1 = ii != INT_MIN ? (int)idxL(p, ii, j, 0) : -1;
    const int o2 = jj != INT_MIN ? (int)idxL(p, i, jj, 0) : -1;
    const int o3 = (ii != INT_MIN && jj != INT_MIN) ? (int)idxL(p, ii, jj, 0) : -1;
    auto store = [&](T* a, int o, T v) {
      a[col + o] = v;
      if (o1 >= 0) a[o1 + o] = v;
      if (o2 >= 0) {
        a[o2 + o] = v;
        if (o3 >= 0) a[o3 + o] = v;
      }
    };
    // columns that the input region holds: x offsets -2..2 (bits 0..4, bit 2
    // this column), y offsets -2..2 (bits 5..9)
    unsigned held = 0;
    {
      const bool yh = span_has(t.vin.ya, t.vin.yn, p.jmax, j), xh = span_has(t.vin.xa, t.vin.xn, p.imax, i);
#pragma unroll
      for (int d = -2; d <= 2; ++d) {
        if (yh && span_has(t.vin.xa, t.vin.xn, p.imax, wrapx(p, i + d))) held |= 1u << (d + 2);
        if (xh && span_has(t.vin.ya, t.vin.yn, p.jmax, wrapy(p, j + d))) held |= 1u << (d + 7);
      }
    }
    auto far = [&](int k) { return (k < 0 || k > p.k1) ? bggin : bgin; };
    auto own = [&](int k) -> T {
      return ((held & 4u) && k >= t.vin.z0 && k <= t.vin.z1) ? in[k * sz] : far(k);
    };
    // |clip(v)| != NB (true for NaN)
    auto in_band = [&](T v) { return !(fabs(v) >= NB); };
    // own column, rows k-2 .. k+2
    T a0 = own(c.ka - 2), a1 = own(c.ka - 1), a2 = own(c.ka), a3 = own(c.ka + 1), a4 = own(c.ka + 2);
    for (int k = c.ka; k <= c.kb; ++k) {
      const T nxt = own(k + 3);
      const int o = k * sz;
      T val;
      if (!computed(c, t.r, k)) {
        val = clipNB(far(k), NB);
      } else {
        if (k == 0) val = TC(2.) * clipNB(a3, NB) - clipNB(a4, NB);
        else if (k == p.k1) val = TC(2.) * clipNB(a1, NB) - clipNB(a0, NB);
        else val = clipNB(a2, NB);
        if (k >= 1 && k <= p.kmax) {
          bool m = in_band(a0) | in_band(a1) | in_band(a2) | in_band(a3) | in_band(a4);
          if (!m && held == 0x3FFu && k >= t.vin.z0 && k <= t.vin.z1) {  // every neighbour is stored
            m = in_band(in[o - 2]) | in_band(in[o - 1]) | in_band(in[o + 1]) | in_band(in[o + 2]) |
                in_band(in[o - 2 * sy]) | in_band(in[o - sy]) | in_band(in[o + sy]) | in_band(in[o + 2 * sy]);
          } else if (!m) {
            const T fk = far(k);
            const bool kin = k >= t.vin.z0 && k <= t.vin.z1;
#pragma unroll
            for (int d = -2; d <= 2; ++d) {
              if (d == 0) continue;
              const T vx = (kin && (held >> (d + 2) & 1u)) ? in[o + d] : fk;
              const T vy = (kin && (held >> (d + 7) & 1u)) ? in[o + d * sy] : fk;
              m = m | in_band(vx) | in_band(vy);
            }
          }
          t.mask[(i - 1) + p.imax * (j - 1) + szI * (k - 1)] = m ? 1 : 0;
          if (m) rows |= 1u << (k - c.ka);
        }
        if (val != NB) {
          kmin = min(kmin, k);
          kmax = k;
        }
      }
      store(out, o, val);
      if (list) {
        store(out2, o, val);
        store(out3, o, val);
      }
      a0 = a1; a1 = a2; a2 = a3; a3 = a4; a4 = nxt;
    }
  }
  const int lane = flat_tid() & 31;
  const unsigned ijt = (unsigned)(i - 1) | ((unsigned)(j - 1) << 12) | ((unsigned)ti << 24);
  const int tot = append_cells(rows, c.ka, ijt, list, count);
  if (flat_tid() == 0 && tot) atomicAdd((unsigned long long*)(cnt + t.l), (unsigned long long)tot);
  int lo[5] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX, INT_MAX};
  int hi[5] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN, INT_MIN};
  if (kmin != INT_MAX) {
    const int hx = p.imax / 2, hy = p.jmax / 2;
    lo[0] = hi[0] = i;
    lo[1] = hi[1] = i + hx > p.imax ? i + hx - p.imax : i + hx;
    lo[2] = hi[2] = j;
    lo[3] = hi[3] = j + hy > p.jmax ? j + hy - p.jmax : j + hy;
    lo[4] = kmin;
    hi[4] = kmax;
  }
  if (__any_sync(0xffffffffu, kmin != INT_MAX)) {
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      const int l = __reduce_min_sync(0xffffffffu, lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
      if (lane == 0) {
        atomicMin(&bbox_lo[5 * t.l + a], l);
        atomicMax(&bbox_hi[5 * t.l + a], h);
      }
    }
  }
}

// ------------------------------------------------------- advection RHS
// The 19 values of the axial stencil of a cell (the centre and offsets
// -3..3 along each axis).
template <typename T>
struct Axial19 {
  T c, x[7], y[7], z[7];  // x[d + 3] = phi at offset d along x (x[3] == c), likewise y, z
};

// dfdt of HOUC5_nb (hyperPDE.f90:397-495) or WENO5_nb (503-800) at row k
// from its axial stencil S
template <int SCHEME, int PW = -1, typename T>
__device__ __forceinline__ T adv_rhs(const Params& p, const Axial19<T>& S, T vu, T vv, T vw, int k) {
#define PX(d) S.x[(d) + 3]
#define PY(d) S.y[(d) + 3]
#define PZ(d) S.z[(d) + 3]
  T udfdx, vdfdy, wdfdz, dfx, dfy, dfz;
  if (SCHEME == ICLS_HOUC5) {
    if (p.TwoD) {
      udfdx = TC(0.);
    } else {
      if (vu >= TC(0.))
        dfx = houc5_pos(PX(-3), PX(-2), PX(-1), PX(0), PX(1), PX(2));
      else
        dfx = houc5_neg(PX(3), PX(2), PX(1), PX(0), PX(-1), PX(-2));
      udfdx = -divx<PW>(p, vu * dfx);
    }
    if (vv >= TC(0.))
      dfy = houc5_pos(PY(-3), PY(-2), PY(-1), PY(0), PY(1), PY(2));
    else
      dfy = houc5_neg(PY(3), PY(2), PY(1), PY(0), PY(-1), PY(-2));
    vdfdy = -divy<PW>(p, vv * dfy);
  } else {
    if (p.TwoD) {
      udfdx = TC(0.);
    } else {
      if (vu >= TC(0.))
        dfx = weno5(divx<PW>(p, PX(-2) - PX(-3)), divx<PW>(p, PX(-1) - PX(-2)), divx<PW>(p, PX(0) - PX(-1)),
                    divx<PW>(p, PX(1) - PX(0)), divx<PW>(p, PX(2) - PX(1)));
      else
        dfx = weno5(divx<PW>(p, PX(3) - PX(2)), divx<PW>(p, PX(2) - PX(1)), divx<PW>(p, PX(1) - PX(0)),
                    divx<PW>(p, PX(0) - PX(-1)), divx<PW>(p, PX(-1) - PX(-2)));
      udfdx = -(vu * dfx);
    }
    // y uses dx, as in the reference (hyperPDE.f90:622-626)
    if (vv >= TC(0.))
      dfy = weno5(divx<PW>(p, PY(-2) - PY(-3)), divx<PW>(p, PY(-1) - PY(-2)), divx<PW>(p, PY(0) - PY(-1)),
                  divx<PW>(p, PY(1) - PY(0)), divx<PW>(p, PY(2) - PY(1)));
    else
      dfy = weno5(divx<PW>(p, PY(3) - PY(2)), divx<PW>(p, PY(2) - PY(1)), divx<PW>(p, PY(1) - PY(0)),
                  divx<PW>(p, PY(0) - PY(-1)), divx<PW>(p, PY(-1) - PY(-2)));
    vdfdy = -(vv * dfy);
  }
  if (k > 2 && k < p.kmax - 1) {
    if (SCHEME == ICLS_HOUC5) {
      if (vw >= TC(0.))
        dfz = houc5_pos(PZ(-3), PZ(-2), PZ(-1), PZ(0), PZ(1), PZ(2));
      else
        dfz = houc5_neg(PZ(3), PZ(2), PZ(1), PZ(0), PZ(-1), PZ(-2));
      wdfdz = -divz<PW>(p, vw * dfz);
    } else {
      if (vw >= TC(0.))
        dfz = weno5(divz<PW>(p, PZ(-2) - PZ(-3)), divz<PW>(p, PZ(-1) - PZ(-2)), divz<PW>(p, PZ(0) - PZ(-1)),
                    divz<PW>(p, PZ(1) - PZ(0)), divz<PW>(p, PZ(2) - PZ(1)));
      else
        dfz = weno5(divz<PW>(p, PZ(3) - PZ(2)), divz<PW>(p, PZ(2) - PZ(1)), divz<PW>(p, PZ(1) - PZ(0)),
                    divz<PW>(p, PZ(0) - PZ(-1)), divz<PW>(p, PZ(-1) - PZ(-2)));
      wdfdz = -(vw * dfz);
    }
  } else if (k == 2 || k == p.kmax - 1) {  // HOUC3 near the walls
    if (vw >= TC(0.))
      dfz = ((TC(1. / 6.) * PZ(-2) - PZ(-1)) + TC(1. / 2.) * PZ(0)) + TC(1. / 3.) * PZ(1);
    else
      dfz = ((-(TC(1. / 6.) * PZ(2)) + PZ(1)) - TC(1. / 2.) * PZ(0)) - TC(1. / 3.) * PZ(-1);
    wdfdz = -divz<PW>(p, vw * dfz);
  } else {  // first-order upwinding at k=1,kmax
    if (vw >= TC(0.)) dfz = PZ(0) - PZ(-1);
    else dfz = PZ(1) - PZ(0);
    wdfdz = -divz<PW>(p, vw * dfz);
  }
#undef PX
#undef PY
#undef PZ
  return (udfdx + vdfdy) + wdfdz;
}
// u_lc, v_lc, w_lc of levelset.f90:527-548, with u_l,v_l,w_l of 530-532
// after bounduvw evaluated on the fly
template <typename T>
__device__ __forceinline__ T infl_face(const Params& p, const T* __restrict__ dheav, T temp, int axis, int i, int j,
                                       int k) {
  const long long n = idxC(p, i, j, k);
  if (axis == 0) return -divx(p, temp * (dheav[n + 1] - dheav[n]));
  if (axis == 1) return -divy(p, temp * (dheav[n + p.nCx] - dheav[n]));
  return -divz(p, temp * (dheav[n + (long long)p.nCx * p.nCy] - dheav[n]));
}
// v_l(i,0,k) and v_l(i,jmax,k) with the y walls of boundp(dheav) and
// bounduvw(u_l,v_l,w_l) (levelset.f90:466-478, bound.f90:81-282) for
// BC_in_y = Walls, InOut, OutOut: v_l = 0 on a wall, v_inflow at the inlet,
// the OutOut extrapolation at y = 0, and dheav(i,j1,k) = -dheav(i,jmax,k) at
// an outflow end
template <typename T>
__device__ __forceinline__ T infl_v_front(const Params& p, const T* __restrict__ dheav, T temp, int i, int k,
                                          const double* __restrict__ vin) {
  if (p.bcy == ICLS_BCY_WALLS) return TC(0.);
  if (p.bcy == ICLS_BCY_INOUT) return TC(vin[i + (long long)(p.i1 + 1) * k]);
  const T wl_1 = (k == p.kmax) ? TC(0.) : infl_face(p, dheav, temp, 2, i, 1, k);
  const T wl_0 = (k == 1) ? TC(0.) : infl_face(p, dheav, temp, 2, i, 1, k - 1);
  return infl_face(p, dheav, temp, 1, i, 1, k) + TC(p.dy / p.dz) * (wl_1 - wl_0);
}
template <typename T>
__device__ __forceinline__ T infl_v_back(const Params& p, const T* __restrict__ dheav, T temp, int i, int k) {
  if (p.bcy == ICLS_BCY_WALLS) return TC(0.);
  const T h = dheav[idxC(p, i, p.jmax, k)];
  return -divy(p, temp * (-h - h));
}
// H is not uniform around an interior cell (where it is, the velocity of a
// finite temp is +-0 and moves nothing)
template <typename T>
__device__ __forceinline__ bool infl_moves(const Params& p, const T* __restrict__ dheav, T temp, int i, int j, int k) {
  const long long n = idxC(p, i, j, k), sy = p.nCx, sz = (long long)p.nCx * p.nCy;
  const T h0 = dheav[n];
  return !((p.bcy == ICLS_BCY_PERIODIC || (j != 1 && j != p.jmax)) && isfinite(temp) && dheav[n + 1] == h0 &&
           dheav[n - 1] == h0 && dheav[n + sy] == h0 && dheav[n - sy] == h0 && dheav[n + sz] == h0 &&
           dheav[n - sz] == h0);
}
// (a, b, c) = u_lc, v_lc, w_lc at an interior cell
template <typename T>
__device__ __forceinline__ void infl_velocity(const Params& p, const T* __restrict__ dheav,
                                              const T* __restrict__ kappa, T temp, int i, int j, int k,
                                              const double* __restrict__ vin, T& a, T& b, T& cc) {
  const long long n = idxC(p, i, j, k);
  const bool inner_y = p.bcy == ICLS_BCY_PERIODIC || (j != 1 && j != p.jmax);
  const T ul_m = infl_face(p, dheav, temp, 0, wrapx(p, i - 1), j, k);
  const T ul_0 = infl_face(p, dheav, temp, 0, i, j, k);
  T vl_m, vl_0;
  if (inner_y) {
    vl_m = infl_face(p, dheav, temp, 1, i, wrapy(p, j - 1), k);
    vl_0 = infl_face(p, dheav, temp, 1, i, j, k);
  } else {
    vl_m = j == 1 ? infl_v_front(p, dheav, temp, i, k, vin) : infl_face(p, dheav, temp, 1, i, j - 1, k);
    vl_0 = j == p.jmax ? infl_v_back(p, dheav, temp, i, k) : infl_face(p, dheav, temp, 1, i, j, k);
  }
  const T wl_m = (k == 1) ? TC(0.) : infl_face(p, dheav, temp, 2, i, j, k - 1);
  const T wl_0 = (k == p.kmax) ? TC(0.) : infl_face(p, dheav, temp, 2, i, j, k);
  a = (ul_m + ul_0) / TC(2.);
  b = (vl_m + vl_0) / TC(2.);
  cc = (wl_m + wl_0) / TC(2.);
  if (p.ispeed_curv) {
    const T kp = kappa[n];
    a = a * kp;
    b = b * kp;
    cc = cc * kp;
  }
}

template <int SCHEME, typename T, int PW>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 5 : 4)) k_adv_stage(Params p, const __grid_constant__ LsBatch B, int stage1,
                                                     double a_, double bb_, double fdt_, const T* __restrict__ vu,
                                                     const T* __restrict__ vv, const T* __restrict__ vw) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  if (!c.ok) return;
  const T a = TC(a_), bb = TC(bb_), fdt = TC(fdt_);
  const int i = c.i, j = c.j;
  // This column's storage, and that of its periodic images in out, from
  // row 0; row k is `k * sz` further (32-bit offsets within one array).
  const int sy = p.nLx, sz = p.nLx * p.nLy, szI = p.imax * p.jmax;
  const long long col = idxL(p, i, j, 0);
  const T* f0c = cT<T>(t.phi0) + col;
  const T* fsc = cT<T>(t.phis) + col;
  T* out = mT<T>(t.out);
  T* const o0 = out + col;
  const int ii = image_of<3>(i, p.imax), jj = image_of<3>(j, p.jmax);
  T* const o1 = ii != INT_MIN ? out + idxL(p, ii, j, 0) : nullptr;
  T* const o2 = jj != INT_MIN ? out + idxL(p, i, jj, 0) : nullptr;
  T* const o3 = (ii != INT_MIN && jj != INT_MIN) ? out + idxL(p, ii, jj, 0) : nullptr;
  const long long qc = idxI(p, i, j, 1);  // row k at qc + (k - 1) * szI
  auto put = [&](int k, T v) {
    const int o = k * sz;
    o0[o] = v;
    if (o1) o1[o] = v;
    if (o2) o2[o] = v;
    if (o3) o3[o] = v;
  };
  T v1 = TC(0.), v2 = TC(0.), vkm = TC(0.), vk = TC(0.);
  bool wall0 = false;
  for (int k = c.ka; k <= c.kb; ++k) {
    if (!computed(c, t.r, k)) {
      put(k, (k < 0 || k > p.k1) ? TC(t.bgg) : TC(t.bg));
      continue;
    }
    if (k == 0) {  // written once rows 1 and 2 are known
      wall0 = true;
      continue;
    }
    T val;
    if (k == p.k1) {
      val = TC(2.) * vk - vkm;
    } else {
      // every operand (phi0, phis' axial stencil, the band flag and the
      // velocities) is read first, so one memory latency is exposed per row;
      // the stencil result is used on band cells only
      const int o = k * sz;
      const T f0 = f0c[o];
      if (!(k >= 1 && k <= p.kmax)) {
        val = stage1 ? f0 : a * f0 + bb * fsc[o];
      } else {
        const long long q = qc + (long long)(k - 1) * szI;
        const uint8_t m = t.mask[q];
        const T u = vu[q], v = vv[q], w = vw[q];
        const T* f = fsc + o;
        Axial19<T> S;
        S.c = f[0];
#pragma unroll
        for (int d = -3; d <= 3; ++d) {
          if (d == 0) continue;
          S.x[d + 3] = f[d];
          S.y[d + 3] = f[d * sy];
          S.z[d + 3] = f[d * sz];
        }
        S.x[3] = S.y[3] = S.z[3] = S.c;
        val = stage1 ? f0 : a * f0 + bb * S.c;
        if (m) val = val + fdt * adv_rhs<SCHEME, PW>(p, S, u, v, w, k);
      }
      if (k == 1) v1 = val;
      if (k == 2) v2 = val;
      if (k == p.kmax - 1) vkm = val;
      if (k == p.kmax) vk = val;
    }
    put(k, val);
    if (k == 2 && wall0) put(0, TC(2.) * v1 - v2);
  }
}

// ------------------------------------------------- band-list advection
// One RK stage over the batch's list of band cells (k_tube), one thread per
// cell, the arithmetic of k_adv_stage.  Cells outside the band are exactly
// +-NB: the first two stages leave them, and the tube wrote them to every
// buffer the stages read; the last one rounds a/3 + 2a/3, which returns NB
// where the spacing is a power of two and is applied by k_adv_rest where it
// does not.  Rows outside 1..kmax of drops next to a wall follow in
// k_adv_ghosts.
// Bound by the latency of the 19 stencil loads (a quarter of the box's cells
// are band cells; the column stage loads all of them and walks every row):
// 256^3 x 48, FP64 0.223 -> 0.112 ms, FP32 0.104 -> 0.063 ms per stage.
// INFL: a stage of the mass correction over its list of moving cells
// (k_inflate_base), the velocity u_lc, v_lc, w_lc formed at the cell.
template <int SCHEME, typename T, int PW, bool INFL>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 5 : 4))
    k_adv_band(Params p, const __grid_constant__ LsBatch B, const BandCell* __restrict__ list,
               const int* __restrict__ count, int stage1, double a_, double bb_, double fdt_,
               const T* __restrict__ vu, const T* __restrict__ vv, const T* __restrict__ vw,
               const InflateState* __restrict__ inf, const double* __restrict__ vin) {
  pdl_wait();
  const int total = *count, stride = (int)gridDim.x * NT;
  const T a = TC(a_), bb = TC(bb_), fdt = TC(fdt_);
  const int sy = p.nLx, sz = p.nLx * p.nLy;
  // the tasks' arrays, where a lane finds its cell's without a walk through
  // the launch parameters
  __shared__ const T *sf0[kTasks], *sfs[kTasks];
  __shared__ T* so[kTasks];
  for (int q = flat_tid(); q < B.n; q += NT) {
    sf0[q] = cT<T>(B.t[q].phi0);
    sfs[q] = cT<T>(B.t[q].phis);
    so[q] = mT<T>(B.t[q].out);
  }
  __syncthreads();
  int n = (int)(blockIdx.x * NT) + flat_tid();
  BandCell next = n < total ? list[n] : BandCell{0u, 1};
  for (; n < total; n += stride) {
    const BandCell bc = next;
    if (n + stride < total) next = list[n + stride];
    const int i = (int)(bc.ijt & 0xFFFu) + 1, j = (int)((bc.ijt >> 12) & 0xFFFu) + 1, k = bc.k;
    const int ti = (int)(bc.ijt >> 24);
    const int o = (i + 2) + sy * (j + 2) + sz * (k + 2);
    const T* f = sfs[ti] + o;
    const T f0 = sf0[ti][o];
    T u, v, w;
    if constexpr (INFL) {
      const LsTask& t = B.t[ti];
      u = v = w = TC(0.);
      infl_velocity(p, cT<T>(t.aux), cT<T>(t.orig), TC(inf[t.l].temp), i, j, k, vin, u, v, w);
    } else {
      const int q = (i - 1) + p.imax * ((j - 1) + p.jmax * (k - 1));
      u = vu[q];
      v = vv[q];
      w = vw[q];
    }
    Axial19<T> S;
    S.c = f[0];
#pragma unroll
    for (int d = -3; d <= 3; ++d) {
      if (d == 0) continue;
      S.x[d + 3] = f[d];
      S.y[d + 3] = f[d * sy];
      S.z[d + 3] = f[d * sz];
    }
    S.x[3] = S.y[3] = S.z[3] = S.c;
    const T val = (stage1 ? f0 : a * f0 + bb * S.c) + fdt * adv_rhs<SCHEME, PW>(p, S, u, v, w, k);
    T* const out = so[ti];
    out[o] = val;
    if (i <= 3 || i > p.imax - 3 || j <= 3 || j > p.jmax - 3) putL(p, out, i, j, k, val);
  }
}

// After a band stage, the rows outside 1..kmax of the tasks whose computed
// part holds them: the ghost rows by the stage's combination, the wall rows
// from the two rows next to them
template <typename T>
__global__ void __launch_bounds__(NT) k_adv_ghosts(Params p, const __grid_constant__ LsBatch B, int stage1, double a_,
                                                   double bb_) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  if (!c.ok || !c.cxy || t.r.cz0 > -2) return;
  const T a = TC(a_), bb = TC(bb_);
  const T* f0 = cT<T>(t.phi0);
  const T* fs = cT<T>(t.phis);
  T* out = mT<T>(t.out);
  auto at = [&](int k) { return idxL(p, c.i, c.j, k); };
  for (int k : {-2, -1, p.k1 + 1, p.k1 + 2}) {
    const T v = f0[at(k)];
    putL(p, out, c.i, c.j, k, stage1 ? v : a * v + bb * fs[at(k)]);
  }
  putL(p, out, c.i, c.j, 0, TC(2.) * out[at(1)] - out[at(2)]);
  putL(p, out, c.i, c.j, p.k1, TC(2.) * out[at(p.kmax)] - out[at(p.kmax - 1)]);
}

// After the last band stage, where its combination rounds NB: the interior
// rows' cells outside the band in place (the RK3 combinations of a value that
// no stage moves), and the far-field value on the aprons
template <typename T>
__global__ void __launch_bounds__(NT) k_adv_rest(Params p, const __grid_constant__ LsBatch B) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  if (!c.ok) return;
  T* out = mT<T>(t.out);
  for (int k = c.ka; k <= c.kb; ++k) {
    if (!computed(c, t.r, k)) {
      putL(p, out, c.i, c.j, k, (k < 0 || k > p.k1) ? TC(t.bgg) : TC(t.bg));
      continue;
    }
    if (k < 1 || k > p.kmax || t.mask[idxI(p, c.i, c.j, k)]) continue;
    const T x = out[idxL(p, c.i, c.j, k)];
    const T y = TC(3. / 4.) * x + TC(1. / 4.) * x;
    putL(p, out, c.i, c.j, k, TC(1. / 3.) * x + TC(2. / 3.) * y);
  }
}

// ------------------------------------------------------------ reinit
// sgn(phi_0) of ls_reinit (levelset.f90:668-678)
template <typename T>
__device__ __forceinline__ T reinit_sgn(const Params& p, T p0) {
  const T dz = TC(p.dz);
  if (p0 < -dz) return TC(-1.);
  if (p0 > dz) return TC(1.);
  return p0 / sqrt(p0 * p0 + dz * dz);
}

// RHS of WENO5_reinit at an interior cell (hyperPDE.f90:2646-2746); c its
// index in shape L, s = sgn(phi_0) there.  An axis along which the seven
// values are equal (next to the far field) has derivatives of exactly +0
// either way, without the WENO5 evaluations.
template <int PW, typename T>
__device__ __forceinline__ T reinit_rhs(const Params& p, const T* __restrict__ phi, T s, int c, int k) {
  const int sx = 1, sy = p.nLx, sz = p.nLx * p.nLy;
#define PH(o) phi[c + (o)]
  T A = TC(0.), B = TC(0.), C = TC(0.), D = TC(0.), E = TC(0.), F = TC(0.);
  const T f0 = PH(0);
  if (!p.TwoD) {
    const T m3 = PH(-3 * sx), m2 = PH(-2 * sx), m1 = PH(-sx), p1 = PH(sx), p2 = PH(2 * sx), p3 = PH(3 * sx);
    if (!(m3 == f0 & m2 == f0 & m1 == f0 & p1 == f0 & p2 == f0 & p3 == f0)) {
      const T d1 = divx<PW>(p, m2 - m3), d2 = divx<PW>(p, m1 - m2), d3 = divx<PW>(p, f0 - m1),
              d4 = divx<PW>(p, p1 - f0), d5 = divx<PW>(p, p2 - p1), d6 = divx<PW>(p, p3 - p2);
      A = weno5(d1, d2, d3, d4, d5);
      B = weno5(d6, d5, d4, d3, d2);
    }
  }
  {
    const T m3 = PH(-3 * sy), m2 = PH(-2 * sy), m1 = PH(-sy), p1 = PH(sy), p2 = PH(2 * sy), p3 = PH(3 * sy);
    if (!(m3 == f0 & m2 == f0 & m1 == f0 & p1 == f0 & p2 == f0 & p3 == f0)) {
      const T d1 = divx<PW>(p, m2 - m3), d2 = divx<PW>(p, m1 - m2), d3 = divx<PW>(p, f0 - m1),
              d4 = divx<PW>(p, p1 - f0), d5 = divx<PW>(p, p2 - p1), d6 = divx<PW>(p, p3 - p2);
      C = weno5(d1, d2, d3, d4, d5);
      D = weno5(d6, d5, d4, d3, d2);
    }
  }
  if (k >= 3 && k <= p.kmax - 2) {
    const T m3 = PH(-3 * sz), m2 = PH(-2 * sz), m1 = PH(-sz), p1 = PH(sz), p2 = PH(2 * sz), p3 = PH(3 * sz);
    if (!(m3 == f0 & m2 == f0 & m1 == f0 & p1 == f0 & p2 == f0 & p3 == f0)) {
      const T d1 = divz<PW>(p, m2 - m3), d2 = divz<PW>(p, m1 - m2), d3 = divz<PW>(p, f0 - m1),
              d4 = divz<PW>(p, p1 - f0), d5 = divz<PW>(p, p2 - p1), d6 = divz<PW>(p, p3 - p2);
      E = weno5(d1, d2, d3, d4, d5);
      F = weno5(d6, d5, d4, d3, d2);
    }
  } else {
    E = divz<PW>(p, f0 - PH(-sz));
    F = divz<PW>(p, PH(sz) - f0);
  }
#undef PH
  T dydx, dydy, dydz;
  if (p.TwoD) {
    dydx = TC(0.);
  } else {
    if ((B * s < TC(0.)) && ((A + B) * s < TC(0.))) dydx = B;
    else if ((A * s > TC(0.)) && ((A + B) * s > TC(0.))) dydx = A;
    else dydx = TC(0.5) * (A + B);
  }
  if ((D * s < TC(0.)) && ((C + D) * s < TC(0.))) dydy = D;
  else if ((C * s > TC(0.)) && ((C + D) * s > TC(0.))) dydy = C;
  else dydy = TC(0.5) * (C + D);
  if ((F * s < TC(0.)) && ((E + F) * s < TC(0.))) dydz = F;
  else if ((E * s > TC(0.)) && ((E + F) * s > TC(0.))) dydz = E;
  else dydz = TC(0.5) * (E + F);
  return s * (TC(1.) - sqrt((dydx * dydx + dydy * dydy) + dydz * dydz));
}

// one SSP-RK3 stage value of ls_reinit (levelset.f90:800-810)
template <typename T>
__device__ __forceinline__ T reinit_val(int stage, T f0, T fs, T dtau, T rhs) {
  if (stage == 1) return f0 + dtau * rhs;
  if (stage == 2) return TC(3. / 4.) * f0 + TC(1. / 4.) * (fs + dtau * rhs);
  return TC(1. / 3.) * f0 + TC(2. / 3.) * (fs + dtau * rhs);
}

// One SSP-RK3 stage of ls_reinit over the tasks' regions; stage 3 folds
// max|phi_new - phi_0| into the drop's residual.  out may equal phi0.
//
// Two passes over a block's 256 columns x one chunk of rows.  First every
// thread marches its column and finishes the cells whose right-hand side
// needs no derivative: outside |phi| < NB + dz it is 0, and where the three
// axial neighbours each way all equal the cell (most of a drop's region is
// clipped far field) every difference is exactly +0 and it is sgn.  The
// others go to a queue in shared memory, which the block then works off with
// full warps.  Bound by the FP64 units: a cell is six WENO5 derivatives of
// six IEEE divisions each, and only a third of a box's cells need them;
// evaluated where they occurred 21 of 32 lanes took part (256^3 x 48 FP64
// 1.11 -> 0.78 ms, FP32 0.44 -> 0.38 ms per stage; 96 x 192 x 100 with ten
// drops, FP64 and a spacing that divides, 0.37 -> 0.21 ms).
template <typename T, int PW>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 4 : 3)) k_reinit_stage(Params p, const __grid_constant__ LsBatch B, int stage,
                                                        double dtau_, ReinitState* __restrict__ rs) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  const T* phi0 = cT<T>(t.phi0);
  T* out = mT<T>(t.out);
  if (rs[t.l].done) {
    // an iteration after convergence is the identity (levelset.f90:833-835)
    if (stage == 3 && c.ok && t.out != t.phi0)
      for (int k = c.ka; k <= c.kb; ++k) putL(p, out, c.i, c.j, k, phi0[idxL(p, c.i, c.j, k)]);
    return;
  }
  __shared__ CellQueue queue;
  queue_init(queue, c);
  const T dtau = TC(dtau_);
  const T* phis = cT<T>(t.phis);
  const T* orig = cT<T>(t.orig);
  const int sy = p.nLx, sz = p.nLx * p.nLy;
  const int col = (int)idxL(p, c.ok ? c.i : 1, c.ok ? c.j : 1, 0);
  const T lim = TC(p.NB + p.dz);
  double r = 0.;
  for (int k = c.ka; k <= c.kb; ++k) {
    bool heavy = false;
    if (c.ok) {
      const int n = col + k * sz;
      if (!computed(c, t.r, k)) {
        putL(p, out, c.i, c.j, k, (k < 0 || k > p.k1) ? TC(t.bgg) : TC(t.bg));
      } else if (k != 0 && k != p.k1) {
        const T fs = phis[n];
        T rhs = TC(0.);
        if (k >= 1 && k <= p.kmax && fabs(fs) < lim) {
          heavy = true;
          bool uni = true;
#pragma unroll
          for (int d = 1; d <= 3; ++d)
            uni = uni & (phis[n + d] == fs) & (phis[n - d] == fs) & (phis[n + d * sy] == fs) &
                  (phis[n - d * sy] == fs) & (phis[n + d * sz] == fs) & (phis[n - d * sz] == fs);
          if (uni) {
            heavy = false;
            rhs = reinit_sgn(p, orig[n]);
          }
        }
        if (!heavy) {
          const T f0 = phi0[n];
          const T val = reinit_val(stage, f0, fs, dtau, rhs);
          if (stage == 3) r = fmax(r, (double)fabs(val - f0));
          putL(p, out, c.i, c.j, k, val);
        }
      }
    }
    queue_push(queue, heavy, k - c.ka);
  }
  __syncthreads();
  for (int e = flat_tid(); e < queue.n; e += NT) {
    int i, j, k;
    queue_cell(queue, e, c.ka, i, j, k);
    const int n = (int)idxL(p, i, j, k);
    const T f0 = phi0[n];
    const T rhs = reinit_rhs<PW>(p, phis, reinit_sgn(p, orig[n]), n, k);
    const T val = reinit_val(stage, f0, phis[n], dtau, rhs);
    if (stage == 3) r = fmax(r, (double)fabs(val - f0));
    putL(p, out, i, j, k, val);
  }
  if (t.r.cz0 <= 0 || t.r.cz1 >= p.k1) {
    // the wall rows, from the finished rows next to them (in this chunk)
    __syncthreads();
    if (c.ok) {
      for (int h = 0; h < 2; ++h) {
        const int k = h ? p.k1 : 0;
        if (k < c.ka || k > c.kb || !computed(c, t.r, k)) continue;
        const int n = col + k * sz, d = h ? -sz : sz;
        const T f0 = phi0[n];
        const T val = TC(2.) * out[n + d] - out[n + 2 * d];
        if (stage == 3) r = fmax(r, (double)fabs(val - f0));
        putL(p, out, c.i, c.j, k, val);
      }
    }
  }
  if (stage == 3) {
    const double bm = block_max<double, NT>(r);
    if (flat_tid() == 0) atomic_max_nonneg(&rs[t.l].residual, bm);
  }
}

__global__ void k_reinit_reset(const __grid_constant__ LsBatch B, int maxiter, ReinitState* __restrict__ rs) {
  pdl_wait();
  for (int q = threadIdx.x; q < B.n; q += blockDim.x) {
    ReinitState& s = rs[B.t[q].l];
    s.residual = 0.;
    s.last = 0.;
    s.done = 0;
    s.iters = maxiter;
  }
}
// end of iteration `it`: far is the change of the far-field cells outside
// the drop's region (0 when none); the last drop's state is also published
// as the scalars of the last ls_reinit call
__global__ void k_reinit_check(const __grid_constant__ LsBatch B, int it, int maxiter, double thr,
                               ReinitState* __restrict__ rs, DevScalars* __restrict__ dsc, int last_drop) {
  pdl_wait();
  for (int q = threadIdx.x; q < B.n; q += blockDim.x) {
    const int l = B.t[q].l;
    ReinitState& s = rs[l];
    if (!s.done) {
      double r = s.residual;
      if (B.t[q].far > r) r = B.t[q].far;
      s.last = r;
      s.residual = 0.;
      if (r < thr) {
        s.done = 1;
        s.iters = it;
      } else {
        s.iters = maxiter;
      }
    }
    if (l == last_drop) {
      dsc->residual = s.last;
      dsc->reinit_iters = s.iters;
      dsc->reinit_done = s.done;
    }
  }
}

// --------------------------------------------------------- Heaviside
template <typename T>
__device__ __forceinline__ T heav_trig(const Params& p, T phi, T eps) {
  if (phi < -eps) return TC(0.);
  if (phi < eps) return (TC(.5) + TC(.5) * phi / eps) + TC(.5) / TC(p.pi) * sin(TC(p.pi) * phi / eps);
  return TC(1.);
}
template <typename T>
__device__ __forceinline__ T dirac_trig(const Params& p, T phi, T eps) {
  if (phi < -eps) return TC(0.);
  if (phi < eps) return TC(.5) / eps + TC(.5) / eps * cos(TC(p.pi) * phi / eps);
  return TC(0.);
}

// disp_cg and disp_speed (write_vtk.f90:438-566) of one drop: over the
// interior cells with phi <= 1.5 dz, the count, the sums of the cell-centre
// coordinates (i - 1/2)/dxi, ... and of ucc dx dy dz (1 - H), ... (H the
// 'trig' Heaviside of the drop).  Warp w of the grid takes the rows (j,k)
// w, w + W, ...; per-block partials part[7 * block + q] in a fixed order.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_disp(Params p, const T* __restrict__ phi,
                                                      const T* __restrict__ ucc, const T* __restrict__ vcc,
                                                      const T* __restrict__ wcc, double* __restrict__ part) {
  pdl_wait();
  double s[7] = {0., 0., 0., 0., 0., 0., 0.};
  const int rows = p.jmax * p.kmax;
  const int W = (int)((gridDim.x * kRedThreads) >> 5);
  const int lane = threadIdx.x & 31;
  const T lim = TC(1.5 * p.dz), eps = TC(1.5 * p.dz);
  for (int r = (int)((blockIdx.x * kRedThreads + threadIdx.x) >> 5); r < rows; r += W) {
    const int j = 1 + r % p.jmax, k = 1 + r / p.jmax;
    const double cy = (j - 0.5) / p.dyi, cz = (k - 0.5) / p.dzi;
    for (int i = 1 + lane; i <= p.imax; i += 32) {
      const T f = phi[idxL(p, i, j, k)];
      if (f <= lim) {
        const long long q = idxI(p, i, j, k);
        const double g = 1. - (double)heav_trig(p, f, eps);
        s[0] += 1.;
        s[1] += (i - 0.5) / p.dxi;
        s[2] += cy;
        s[3] += cz;
        s[4] += ((((double)ucc[q] * p.dx) * p.dy) * p.dz) * g;
        s[5] += ((((double)vcc[q] * p.dx) * p.dy) * p.dz) * g;
        s[6] += ((((double)wcc[q] * p.dx) * p.dy) * p.dz) * g;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    const double b = block_sum<double, kRedThreads>(s[q]);
    if (threadIdx.x == 0) part[7 * blockIdx.x + q] = b;
  }
}
__global__ void __launch_bounds__(kRedThreads) k_disp_final(const double* __restrict__ part, int nblk,
                                                            double* __restrict__ out) {
  pdl_wait();
#pragma unroll 1
  for (int q = 0; q < 7; ++q) {
    double s = 0.;
    for (int b = threadIdx.x; b < nblk; b += kRedThreads) s += part[7 * b + q];
    s = block_sum<double, kRedThreads>(s);
    if (threadIdx.x == 0) out[q] = s;
  }
}

// jiemian = min(jiemian, H_l) over the tasks' computed cells (shape-C
// regions) and exact sums of H_l over their interior cells (misc.f90:110-141),
// one per column tile and z chunk: part[l*cap + tile + tiles*chunk].  jiemian
// starts at 1, the far-field value of H, so only cells with H < 1 are touched;
// min is order-free, so drops may share cells.
// For v >= +0 the signed-integer order of the bit patterns is the numeric
// order against every non-negative value, and every negative value (sign
// bit set) compares below it, as it does numerically: one atomicMin that
// returns nothing (the thread does not wait for it).  A negative v (H is
// negative only by rounding, ~1e-17) takes the compare-and-swap loop.
__device__ __forceinline__ void min_into(double* a, double v) {
  if (!(v < 0.)) {
    atomicMin(reinterpret_cast<long long*>(a), __double_as_longlong(v));
    return;
  }
  unsigned long long* q = reinterpret_cast<unsigned long long*>(a);
  unsigned long long old = *q;
  while (v < __longlong_as_double((long long)old)) {
    const unsigned long long prev = atomicCAS(q, old, (unsigned long long)__double_as_longlong(v));
    if (prev == old) break;
    old = prev;
  }
}
__device__ __forceinline__ void min_into(float* a, float v) {
  if (!(v < 0.f)) {
    atomicMin(reinterpret_cast<int*>(a), __float_as_int(v));
    return;
  }
  unsigned int* q = reinterpret_cast<unsigned int*>(a);
  unsigned int old = *q;
  while (v < __uint_as_float(old)) {
    const unsigned int prev = atomicCAS(q, old, __float_as_uint(v));
    if (prev == old) break;
    old = prev;
  }
}
// a Heaviside value into an exact sum: the zeros add nothing and the ones
// (most cells of a box) are counted, so only interface cells pay the limb
// arithmetic
template <typename T>
__device__ __forceinline__ void heav_add(XSum& s, int& ones, T H) {
  if (H == TC(1.)) ++ones;
  else if (H != TC(0.)) xs_add(s, (double)H);
}

template <typename T>
__global__ void __launch_bounds__(NT, 4) k_heaviside(Params p, const __grid_constant__ LsBatch B,
                                                  T* __restrict__ jiemian, uint8_t* __restrict__ seg,
                                                  XSum* __restrict__ part, int cap) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  const T eps = TC(1.5 * p.dz);
  const T* __restrict__ phi = cT<T>(t.phi0);
  XSum s;
  xs_zero(s);
  int ones = 0;
  if (c.ok && c.cxy) {
    const int i = c.i, j = c.j;
    const int ii = image_of<1>(i, p.imax), jj = image_of<1>(j, p.jmax);
    const int ka = max(c.ka, t.r.cz0), kb = min(c.kb, t.r.cz1);
    const long long sz = (long long)p.nLx * p.nLy;
    // eight rows' phi in flight before their minima and sums (same order)
    for (int k0 = ka; k0 <= kb; k0 += 8) {
      T f[8];
      const long long c0 = idxL(p, i, j, k0);
#pragma unroll
      for (int u = 0; u < 8; ++u) f[u] = (k0 + u <= kb) ? phi[c0 + u * sz] : TC(1.);
#pragma unroll
      for (int u = 0; u < 8; ++u) {  // rows past kb skipped without a break, so f stays in registers
        const int k = k0 + u;
        if (k <= kb) {
          const T H = heav_trig(p, f[u], eps);
          if (H < TC(1.)) {
            seg[seg_of(p, i, j, k)] = 1;
            min_into(jiemian + idxC(p, i, j, k), H);
            if (ii != INT_MIN) min_into(jiemian + idxC(p, ii, j, k), H);
            if (jj != INT_MIN) {
              min_into(jiemian + idxC(p, i, jj, k), H);
              if (ii != INT_MIN) min_into(jiemian + idxC(p, ii, jj, k), H);
            }
          }
          if (k >= 1 && k <= p.kmax) heav_add(s, ones, H);
        }
      }
    }
  }
  xs_add_count(s, ones);
  const XSum bs = block_xsum<NT>(s);
  // one partial per (column tile, z chunk) of the task
  if (flat_tid() == 0) part[(long long)t.l * cap + c.tile + (long long)t.tx * c.ch] = bs;
}

// volume(l) and rho_avr from the per-(tile, chunk) sums (misc.f90:139-173) of
// drops l0 .. l0 + nl - 1: n[l - l0] partials each, and v[l - l0] interior
// cells in the drop's far field, where H = 1.  The counts travel as a kernel
// parameter, so a launch takes up to kMaxDropsParam drops; launches of more
// drops follow one another, and the last one, which sees every volume, sums
// them in order.
struct PerDrop {
  double v[kMaxDropsParam];
  int n[kMaxDropsParam];
};
// One warp per drop: its lanes merge every 32nd partial, the lanes' sums
// (limbs below 2^48 after each merge) add limb by limb across the warp
// (below 2^53), and lane 0 rounds the exact total once.
// (and into pinned memory for the host, with the band extents where asked:
// copies and small memsets between the step's kernels left the GPU idle for
// their length and broke the overlapped launches; without two copies and eight
// memsets one drop at 64^3 takes 334 instead of 370 us)
__global__ void k_volumes(Params p, const XSum* __restrict__ part, int cap, PerDrop pd, int l0, int nl,
                          double* __restrict__ vol, DevScalars* __restrict__ dsc, double* __restrict__ h_vol,
                          const int* __restrict__ bbox, int* __restrict__ h_bbox) {
  pdl_wait();
  const bool last = l0 + nl == p.L;
  if (bbox && last)
    for (int t = threadIdx.x; t < 10 * p.L; t += blockDim.x) h_bbox[t] = bbox[t];
  const double N = (1. * p.imax * p.jmax) * p.kmax;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int q = warp; q < nl; q += nw) {
    const int l = l0 + q, nb = pd.n[q];
    XSum s;
    xs_zero(s);
    for (int b = lane; b < nb; b += 32) xs_merge(s, part[(long long)l * cap + b]);
#pragma unroll
    for (int m = 0; m < 4; ++m)
      for (int d = 16; d > 0; d >>= 1) s.L[m] += __shfl_down_sync(0xffffffffu, s.L[m], d);
    if (lane == 0) {
      xs_norm(s);
      xs_add_count(s, (long long)pd.v[q]);
      vol[l] = 1. - xs_value(s) / N;
      h_vol[l] = vol[l];
    }
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    double sv = 0.;
    for (int l = 0; l < p.L; ++l) sv += vol[l];
    dsc->rho_avr = p.rho1 * (1. - sv) + p.rho2 * sv;
  }
}

template <typename T>
__global__ void __launch_bounds__(NT) k_fill(T* __restrict__ a, long long n, double v) {
  pdl_wait();
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    a[q] = TC(v);
}

// miu, rho (shape C) and the face densities (misc.f90:121-172)
template <typename T>
__global__ void __launch_bounds__(NT) k_materials_final(Params p, const T* __restrict__ jiemian, T* __restrict__ miu,
                                                        T* __restrict__ rho, T* __restrict__ rho_u,
                                                        T* __restrict__ rho_v, T* __restrict__ rho_w) {
  pdl_wait();
  const int r0[3] = {0, 0, 0}, r1[3] = {p.i1, p.j1, p.k1};
  int i, j, k;
  if (!cell3(r0, r1, i, j, k)) return;
  const long long n = idxC(p, i, j, k);
  const T rho1 = TC(p.rho1), rho2 = TC(p.rho2);
  const T J0 = jiemian[n];
  miu[n] = TC(p.miu1) * J0 + TC(p.miu2) * (TC(1.) - J0);
  const T r0v = rho1 * J0 + rho2 * (TC(1.) - J0);
  rho[n] = r0v;
  if (interior(p, i, j, k)) {
    const long long q = idxI(p, i, j, k);
    if (p.rho1 == p.rho2) {
      rho_u[q] = rho1; rho_v[q] = rho1; rho_w[q] = rho1;
    } else {
      const T Jx = jiemian[n + 1], Jy = jiemian[n + p.nCx], Jz = jiemian[n + (long long)p.nCx * p.nCy];
      const T rx = rho1 * Jx + rho2 * (TC(1.) - Jx);
      const T ry = rho1 * Jy + rho2 * (TC(1.) - Jy);
      const T rz = rho1 * Jz + rho2 * (TC(1.) - Jz);
      rho_u[q] = (r0v + rx) / TC(2.);
      rho_v[q] = (r0v + ry) / TC(2.);
      rho_w[q] = (r0v + rz) / TC(2.);
    }
  }
}

// One warp per 32 segments: the lanes read the segments' bytes, then the
// warp takes the set ones in turn, a lane per cell.  bytes(q, sx, j, k): what
// segment q is to be visited for (0: not), and f(sx, j, k, that) visits it.
template <class Bytes, class F>
__device__ __forceinline__ void for_segments(const Params& p, int per, const Bytes& bytes, const F& f) {
  const int nsx = seg_row(p);
  const long long ns = seg_count(p), lane = threadIdx.x & 31;
  const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long W = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long g = w0; g * per < ns; g += W) {
    const long long q = g * per + lane;
    int sx = 0, j = 0, k = 0;
    int on = 0;
    if (lane < per && q < ns) {
      const long long r = q / nsx;
      sx = (int)(q - r * nsx);
      k = (int)(r / p.jmax);
      j = (int)(r - (long long)k * p.jmax) + 1;
      on = bytes(q, sx, j, k);
    }
    unsigned m = __ballot_sync(0xffffffffu, on != 0);
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      f(__shfl_sync(0xffffffffu, sx, b), __shfl_sync(0xffffffffu, j, b), __shfl_sync(0xffffffffu, k, b),
        __shfl_sync(0xffffffffu, on, b));
    }
  }
}

// jiemian = 1 in the segments of a map (with the periodic images), and the
// next map zero
template <typename T>
__global__ void __launch_bounds__(NT) k_seg_reset(Params p, int per, const uint8_t* __restrict__ seg,
                                                  uint8_t* __restrict__ next, T* __restrict__ jiemian) {
  pdl_wait();
  for_segments(
      p, per,
      [&](long long q, int, int, int) {
        next[q] = 0;
        return (int)seg[q];
      },
      [&](int sx, int j, int k, int) {
        const int i = 1 + kSeg * sx + (int)(threadIdx.x & 31);
        if (i <= p.imax) putC(p, jiemian, i, j, k, TC(1.));
      });
}
// p_x, p_y, p_z = 0 in the segments of `faces`, p_jump = 0 in those of `lap`
// (interior cells: gfm4p writes no others); then faces and the row map are
// zero, for the jumps that follow
template <typename T>
__global__ void __launch_bounds__(NT) k_seg_clear_jumps(Params p, int per, uint8_t* faces,
                                                        const uint8_t* __restrict__ lap, uint8_t* __restrict__ row,
                                                        T* __restrict__ px, T* __restrict__ py, T* __restrict__ pz,
                                                        double* __restrict__ pjump) {
  pdl_wait();
  for (long long q = blockIdx.x * (long long)NT + threadIdx.x; q < (long long)p.jmax * p.nCz; q += (long long)gridDim.x * NT)
    row[q] = 0;
  for_segments(
      p, per,
      [&](long long q, int, int, int) {
        const int on = (faces[q] ? 1 : 0) | (lap[q] ? 2 : 0);
        if (on & 1) faces[q] = 0;
        return on;
      },
      [&](int sx, int j, int k, int on) {
        const int i = 1 + kSeg * sx + (int)(threadIdx.x & 31);
        if (i > p.imax || k < 1 || k > p.kmax) return;
        const long long n = idxC(p, i, j, k);
        if (on & 1) px[n] = py[n] = pz[n] = TC(0.);
        if (on & 2) pjump[n] = 0.;
      });
}
// k_materials_final's fields where they can have changed: a segment whose
// own cells, or the + neighbours that its face densities read, are or were
// (prev) set; everywhere else they hold the carrier's values already.
// Bound by the set segments' stores: six arrays over about 12 % of the
// domain at 256^3 x 48, where the whole sweep wrote all of them (FP64
// 0.19 -> 0.05 ms, FP32 0.13 -> 0.05 ms with the reset of jiemian).
template <typename T>
__global__ void __launch_bounds__(NT) k_materials_seg(Params p, int per, const uint8_t* __restrict__ cur,
                                                      const uint8_t* __restrict__ prev, const T* __restrict__ jiemian,
                                                      T* __restrict__ miu, T* __restrict__ rho, T* __restrict__ rho_u,
                                                      T* __restrict__ rho_v, T* __restrict__ rho_w) {
  pdl_wait();
  const int nsx = seg_row(p);
  const T rho1 = TC(p.rho1), rho2 = TC(p.rho2);
  const long long sz = (long long)p.nCx * p.nCy;
  for_segments(
      p, per,
      [&](long long q, int sx, int j, int k) {
        const long long qx = sx + 1 < nsx ? q + 1 : q - sx;
        const long long qy = j < p.jmax ? q + nsx : q - (long long)nsx * (p.jmax - 1);
        const long long qz = k < p.k1 ? q + (long long)nsx * p.jmax : q;
        return cur[q] | cur[qx] | cur[qy] | cur[qz] | prev[q] | prev[qx] | prev[qy] | prev[qz];
      },
      [&](int sx, int j, int k, int) {
        const int i = 1 + kSeg * sx + (int)(threadIdx.x & 31);
        if (i > p.imax) return;
        const long long n = idxC(p, i, j, k);
        const T J0 = jiemian[n];
        const bool in = k >= 1 && k <= p.kmax;
        T Jx = TC(0.), Jy = TC(0.), Jz = TC(0.);
        if (in) {
          Jx = jiemian[n + 1];
          Jy = jiemian[n + p.nCx];
          Jz = jiemian[n + sz];
        }
        putC(p, miu, i, j, k, TC(p.miu1) * J0 + TC(p.miu2) * (TC(1.) - J0));
        const T r0v = rho1 * J0 + rho2 * (TC(1.) - J0);
        putC(p, rho, i, j, k, r0v);
        if (!in) return;
        const long long q = idxI(p, i, j, k);
        if (p.rho1 == p.rho2) {
          rho_u[q] = rho1; rho_v[q] = rho1; rho_w[q] = rho1;
        } else {
          const T rx = rho1 * Jx + rho2 * (TC(1.) - Jx);
          const T ry = rho1 * Jy + rho2 * (TC(1.) - Jy);
          const T rz = rho1 * Jz + rho2 * (TC(1.) - Jz);
          rho_u[q] = (r0v + rx) / TC(2.);
          rho_v[q] = (r0v + ry) / TC(2.);
          rho_w[q] = (r0v + rz) / TC(2.);
        }
      });
}

// ------------------------------------------------------------ inflation
// dheav with boundp semantics over the tasks' shape-C regions (aux: the
// drop's |grad phi|, orig: its curvature; out: dheav), the far-field value 1
// on their aprons, and per-(tile, chunk) area and volume sums (FP64) over the
// interior computed cells (levelset.f90:493-507, 525)
template <typename T>
__global__ void __launch_bounds__(NT) k_inflate_sums(Params p, const __grid_constant__ LsBatch B,
                                                     double* __restrict__ part_area,
                                                     XSum* __restrict__ part_heav, int cap) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  const T s1 = TC(1.5 * p.dz);
  const T* phi = cT<T>(t.phi0);
  const T* __restrict__ kappa = cT<T>(t.orig);
  const T* __restrict__ nrm_m = cT<T>(t.aux);
  T* dheav = mT<T>(t.out);
  double sa = 0.;
  XSum sh;
  xs_zero(sh);
  int ones = 0;
  if (c.ok) {
    const int i = c.i, j = c.j;
    for (int k = c.ka; k <= c.kb; ++k) {
      if (!computed(c, t.r, k)) {
        putC(p, dheav, i, j, k, TC(1.));
        continue;
      }
      const int K = k == 0 ? 1 : (k == p.k1 ? p.kmax : k);
      const T ph = phi[idxL(p, i, j, K)];
      const T H = heav_trig(p, ph, s1);
      putC(p, dheav, i, j, k, H);
      if (k >= 1 && k <= p.kmax) {
        heav_add(sh, ones, H);
        const T del = dirac_trig(p, ph, s1);
        if (del != TC(0.)) {
          const T m = nrm_m[idxI(p, i, j, k)];
          sa += (double)(p.ispeed_curv ? (del * kappa[idxC(p, i, j, k)]) * m : del * m);
        }
      }
    }
  }
  xs_add_count(sh, ones);
  const double ba = block_sum<double, NT>(sa);
  const XSum bh = block_xsum<NT>(sh);
  if (flat_tid() == 0) {
    const long long at = (long long)t.l * cap + c.tile + (long long)t.tx * c.ch;
    part_area[at] = ba;
    part_heav[at] = bh;
  }
}

// the partials of one task (block blockIdx.x), added in a fixed order: every
// thread's strided share, then a fixed tree
constexpr int kFinalThreads = 256;
__device__ __forceinline__ XSum task_heav(const LsTask& t, const XSum* __restrict__ part, int cap) {
  XSum hs;
  xs_zero(hs);
  const int n = t.tx * t.nch;
  for (int b = threadIdx.x; b < n; b += kFinalThreads) xs_merge(hs, part[(long long)t.l * cap + b]);
  hs = block_xsum<kFinalThreads>(hs);
  xs_add_count(hs, (long long)t.far);
  return hs;
}
__global__ void __launch_bounds__(kFinalThreads)
    k_inflate_final(Params p, const __grid_constant__ LsBatch B, const double* __restrict__ part_area,
                    const XSum* __restrict__ part_heav, int cap, double istep_dt, double* __restrict__ vol,
                    const double* __restrict__ vol0, double* __restrict__ maxchk, InflateState* __restrict__ inf) {
  pdl_wait();
  const LsTask& t = B.t[blockIdx.x];
  const int l = t.l, n = t.tx * t.nch;
  double sa = 0.;
  for (int b = threadIdx.x; b < n; b += kFinalThreads) sa += part_area[(long long)l * cap + b];
  sa = block_sum<double, kFinalThreads>(sa);
  const XSum hs = task_heav(t, part_heav, cap);
  if (threadIdx.x != 0) return;
  double area = sa * p.dx * p.dy * p.dz;
  if (p.TwoD) area = area / p.lx;
  const double volume = 1. - xs_value(hs) / ((1. * p.imax * p.jmax) * p.kmax);
  vol[l] = volume;
  double loss_rate = p.lx * p.ly * p.lz * (volume - vol0[l]) / istep_dt;
  if (p.TwoD) loss_rate = loss_rate / p.lx;
  const double temp = loss_rate / area;
  inf[l].temp = temp;
  maxchk[l] = temp / (1.5 * p.dz);
}

// ------------------------------------------------ gain-one mass correction
// icls_config.mass_gain_one (no counterpart in the reference).  The
// reference's inflation moves the interface by about K/inflate_step times
// the volume error it measured (K ~ 0.66/s1 in grid units), so with the
// option the inflated level set phi1 is blended with the one before it,
// phi = phi0 + g (phi1 - phi0), g = (V0 - V)/(V1 - V) from the exact
// volumes before (V) and after (V1) the inflation: the blend removes the
// measured error to first order in the (small) displacement.

// The start of the mass correction's RK3 over the tasks' written cells: phi0
// into the buffers that the stages read around the cells they move (out, out2
// and, where set, out3), its RK3 combinations into phis, the last stage's
// output (which may be phi0 itself), and the list of the band's moving cells
// (infl_moves): about a twelfth of a box, which the column stages walked
// three times to find (256^3 x 48 after a reinitialisation, three stages FP64
// 1.20 -> 0.54 ms with this sweep, FP32 0.78 -> 0.39 ms).
template <typename T>
__global__ void __launch_bounds__(NT) k_inflate_base(Params p, const __grid_constant__ LsBatch B,
                                                     const InflateState* __restrict__ inf,
                                                     BandCell* __restrict__ list, int* __restrict__ count) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  unsigned rows = 0;
  if (c.ok) {
    const T* src = cT<T>(t.phi0);
    T* fin = const_cast<T*>(cT<T>(t.phis));
    const T temp = TC(inf[t.l].temp);
    for (int k = c.ka; k <= c.kb; ++k) {
      const T x = src[idxL(p, c.i, c.j, k)];
      const bool in = computed(c, t.r, k);
      const T y = TC(3. / 4.) * x + TC(1. / 4.) * x;
      putL(p, mT<T>(t.out), c.i, c.j, k, x);
      putL(p, mT<T>(t.out2), c.i, c.j, k, x);
      if (t.out3) putL(p, mT<T>(t.out3), c.i, c.j, k, x);
      putL(p, fin, c.i, c.j, k,
           in ? TC(1. / 3.) * x + TC(2. / 3.) * y : ((k < 0 || k > p.k1) ? TC(t.bgg) : TC(t.bg)));
      if (in && k >= 1 && k <= p.kmax && t.mask[idxI(p, c.i, c.j, k)] &&
          infl_moves(p, cT<T>(t.aux), temp, c.i, c.j, k))
        rows |= 1u << (k - c.ka);
    }
  }
  append_cells(rows, c.ka, (unsigned)(c.i - 1) | ((unsigned)(c.j - 1) << 12) | ((unsigned)ti << 24), list, count);
}

// per-(tile, chunk) exact sums of H(phi0) over the tasks' computed interior cells
template <typename T>
__global__ void __launch_bounds__(NT) k_region_heav(Params p, const __grid_constant__ LsBatch B,
                                                    XSum* __restrict__ part, int cap) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  const T s1 = TC(1.5 * p.dz);
  const T* __restrict__ phi = cT<T>(t.phi0);
  XSum sh;
  xs_zero(sh);
  int ones = 0;
  if (c.ok)
    for (int k = max(c.ka, 1); k <= min(c.kb, p.kmax); ++k)
      if (computed(c, t.r, k)) heav_add(sh, ones, heav_trig(p, phi[idxL(p, c.i, c.j, k)], s1));
  xs_add_count(sh, ones);
  const XSum bh = block_xsum<NT>(sh);
  if (flat_tid() == 0) part[(long long)t.l * cap + c.tile + (long long)t.tx * c.ch] = bh;
}

// g = (V0 - V)/(V1 - V) of each task's drop, V1 from the partials and the far-field count
__global__ void __launch_bounds__(kFinalThreads)
    k_gain_final(Params p, const __grid_constant__ LsBatch B, const XSum* __restrict__ part, int cap,
                 const double* __restrict__ vol, const double* __restrict__ vol0, InflateState* __restrict__ inf) {
  pdl_wait();
  const LsTask& t = B.t[blockIdx.x];
  const XSum hs = task_heav(t, part, cap);
  if (threadIdx.x != 0) return;
  const int l = t.l;
  const double v1 = 1. - xs_value(hs) / ((1. * p.imax * p.jmax) * p.kmax);
  const double d = v1 - vol[l];
  inf[l].gain = d != 0. ? (vol0[l] - vol[l]) / d : 0.;
}

// the volume of each task's drop now
__global__ void __launch_bounds__(kFinalThreads)
    k_volume_now(Params p, const __grid_constant__ LsBatch B, const XSum* __restrict__ part, int cap,
                 double* __restrict__ vnow) {
  pdl_wait();
  const LsTask& t = B.t[blockIdx.x];
  const XSum hs = task_heav(t, part, cap);
  if (threadIdx.x == 0) vnow[t.l] = 1. - xs_value(hs) / ((1. * p.imax * p.jmax) * p.kmax);
}

// out (the level set before the correction) += g (phi0 - out), phi0 the
// inflated one, on the written cells
template <typename T>
__global__ void __launch_bounds__(NT) k_region_blend(Params p, const __grid_constant__ LsBatch B,
                                                     const InflateState* __restrict__ inf) {
  pdl_wait();
  const int ti = task_of(B);
  const LsTask& t = B.t[ti];
  const Col c = col_of(p, t, (int)blockIdx.x - B.start[ti]);
  if (!c.ok) return;
  const double g = inf[t.l].gain;
  const T* __restrict__ p1 = cT<T>(t.phi0);
  T* __restrict__ p0 = mT<T>(t.out);
  for (int k = c.ka; k <= c.kb; ++k) {
    const long long n = idxL(p, c.i, c.j, k);
    const double a0 = (double)p0[n];
    putL(p, p0, c.i, c.j, k, TC(a0 + g * ((double)p1[n] - a0)));
  }
}

// boundmls, extrap='line' (bound.f90:518-~657): three wall layers by
// repeated linear extrapolation from the interior column, then the periodic
// copies.  Reads only interior cells, writes only the others.
template <typename T>
__global__ void __launch_bounds__(NT) k_boundmls(Params p, T* __restrict__ y) {
  pdl_wait();
  const int r0[3] = {-2, -2, -2}, r1[3] = {p.i1 + 2, p.j1 + 2, p.k1 + 2};
  int i, j, k;
  if (!cell3(r0, r1, i, j, k)) return;
  const long long n = idxL(p, i, j, k);
  const int I = wrapx(p, i), J = wrapy(p, j);
  if (k >= 1 && k <= p.kmax) {
    if (I != i || J != j) y[n] = y[idxL(p, I, J, k)];
    return;
  }
  if (k <= 0) {
    const T y1 = y[idxL(p, I, J, 1)], y2 = y[idxL(p, I, J, 2)];
    const T y0 = TC(2.) * y1 - y2;
    const T ym1 = TC(2.) * y0 - y1;
    const T ym2 = TC(2.) * ym1 - y0;
    y[n] = (k == 0) ? y0 : (k == -1 ? ym1 : ym2);
  } else {
    const T yk = y[idxL(p, I, J, p.kmax)], ykm = y[idxL(p, I, J, p.kmax - 1)];
    const T y0 = TC(2.) * yk - ykm;
    const T yp1 = TC(2.) * y0 - yk;
    const T yp2 = TC(2.) * yp1 - y0;
    y[n] = (k == p.k1) ? y0 : (k == p.k1 + 1 ? yp1 : yp2);
  }
}

// far-field value into every cell outside the written cells of r (makes a
// drop's stored array valid everywhere, e.g. before a download)
template <typename T>
__global__ void __launch_bounds__(NT) k_materialize(Params p, Region r, double bg, double bgg, T* __restrict__ y) {
  pdl_wait();
  const int r0[3] = {-2, -2, -2}, r1[3] = {p.i1 + 2, p.j1 + 2, p.k1 + 2};
  int i, j, k;
  if (!cell3(r0, r1, i, j, k)) return;
  if (!in_written(p, r, i, j, k)) y[idxL(p, i, j, k)] = (k < 0 || k > p.k1) ? TC(bgg) : TC(bg);
}

// field conversions of the precision form (upload / download)
__global__ void k_to_float(float* __restrict__ dst, const double* __restrict__ src, long long n) {
  pdl_wait();
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    dst[q] = (float)src[q];
}
__global__ void k_to_double(double* __restrict__ dst, const float* __restrict__ src, long long n) {
  pdl_wait();
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    dst[q] = (double)src[q];
}

#undef TC

}  // namespace

dim3 grid_of(const int* r0, const int* r1) {
  const int nx = r1[0] - r0[0] + 1, ny = r1[1] - r0[1] + 1, nz = r1[2] - r0[2] + 1;
  return dim3((unsigned)((nx + BX - 1) / BX), (unsigned)((ny + BY - 1) / BY), (unsigned)nz);
}

namespace {
int wrap1(int v, int n) {
  v = (v - 1) % n;
  if (v < 0) v += n;
  return v + 1;
}
}  // namespace

Region full_region(const Params& P) {
  Region r;
  r.xa = 1; r.xn = P.imax; r.cx0 = 0; r.cx1 = P.imax - 1;
  r.ya = 1; r.yn = P.jmax; r.cy0 = 0; r.cy1 = P.jmax - 1;
  r.z0 = r.cz0 = -2;
  r.z1 = r.cz1 = P.k1 + 2;
  return r;
}

bool region_full(const Params& P, const Region& r) {
  return r.xn == P.imax && r.cx0 == 0 && r.cx1 == P.imax - 1 && r.yn == P.jmax && r.cy0 == 0 &&
         r.cy1 == P.jmax - 1 && r.cz0 <= -2 && r.cz1 >= P.k1 + 2;
}

// the shape-C region of a level-set region: the same computed columns with
// an apron of `ap` columns; full z becomes rows 0..k1
Region c_region(const Params& P, const Region& r, int ap) {
  Region q;
  auto axis = [&](int xa, int xn, int c0, int c1, int n, int& qa, int& qn, int& q0, int& q1) {
    if (xn == n && c0 == 0 && c1 == n - 1) {
      qa = 1; qn = n; q0 = 0; q1 = n - 1;
      return;
    }
    const int a = wrap1(xa + c0, n), len = c1 - c0 + 1;
    qa = wrap1(a - ap, n);
    qn = len + 2 * ap;
    q0 = ap;
    q1 = ap + len - 1;
  };
  axis(r.xa, r.xn, r.cx0, r.cx1, P.imax, q.xa, q.xn, q.cx0, q.cx1);
  axis(r.ya, r.yn, r.cy0, r.cy1, P.jmax, q.ya, q.yn, q.cy0, q.cy1);
  if (r.cz0 <= -2 && r.cz1 >= P.k1 + 2) {
    q.z0 = q.cz0 = 0;
    q.z1 = q.cz1 = P.k1;
  } else {
    q.cz0 = r.cz0;
    q.cz1 = r.cz1;
    q.z0 = std::max(0, r.cz0 - ap);
    q.z1 = std::min(P.k1, r.cz1 + ap);
  }
  return q;
}

// tiles of 256 consecutive columns (col_of), z chunks (kc rows each, the last
// one longer; kc <= 0: one chunk) and block offsets of a batch
void set_tiles(LsBatch& b, int kc) {
  int s = 0;
  for (int q = 0; q < b.n; ++q) {
    LsTask& t = b.t[q];
    t.tx = (t.r.xn * t.r.yn + TBX * TBY - 1) / (TBX * TBY);
    const int nz = t.r.z1 - t.r.z0 + 1;
    t.head = 0;
    if (kc <= 0 || kc >= nz) {
      t.nch = 1;
      t.kc = nz;
    } else {
      t.nch = nz / kc;
      t.kc = kc;
    }
    b.start[q] = s;
    s += t.tx * t.nch;
  }
  b.start[b.n] = s;
}

// Tiles with chunks of kc rows, halved down to kmin while the batch has
// fewer than `blocks` blocks: few drops leave SMs idle, and the cells of a
// chunk are worked off one after the other.  The chunks at a wall are
// lengthened to the five rows -2..2 or k1-2..k1+2.  Lines and minima are set
// where each sweep is launched, from microseconds per call at 8 / 4 / 2 rows (drops,
// grid, blocks at 8 rows):
//                         reinit stage   Heaviside     curvature     jumps
//   one, 64^3 (128)       48 / 31 / 25   17 / 13 / 11  27 / 21 / 18  24 / 17 / 15
//   one, 128^2 x 256 (385) 45 / 34 / 31   18 / 14 / 18  27 / 21 / 21  22 / 18 / 18
//   10, 96 x 192 x 100 (3000) 210 / 212 / 245  40 / 52 / 85
//   24, 256^3 (600)                                    65 / 53 / 51  34 / 27 / 30
//   48, 256^3 (3000-7000) 775 / 868 / 1066  79 / 107 / 178  172 / 185 / 218  110 / 122 / 156
void size_tiles(const Params& p, LsBatch& b, int kc, int kmin, int blocks) {
  for (;; kc /= 2) {
    int s = 0;
    for (int q = 0; q < b.n; ++q) {
      LsTask& t = b.t[q];
      t.tx = (t.r.xn * t.r.yn + TBX * TBY - 1) / (TBX * TBY);
      const int nz = t.r.z1 - t.r.z0 + 1, more = std::max(0, 5 - kc);
      t.kc = kc;
      t.head = t.r.z0 <= 0 ? more : 0;
      t.nch = (nz - t.head - (t.r.z1 >= p.k1 ? more : 0)) / kc;
      if (t.nch < 1) {
        t.nch = 1;
        t.kc = nz;
        t.head = 0;
      }
      b.start[q] = s;
      s += t.tx * t.nch;
    }
    b.start[b.n] = s;
    if (s >= blocks || kc / 2 < kmin) return;
  }
}

// ================================================================ launchers
// Each launcher picks the field type of the context's form.
#define BY_FORM(c, call_f32, call_f64) \
  do {                                  \
    if ((c).P.f32) {                    \
      call_f32;                         \
    } else {                            \
      call_f64;                         \
    }                                   \
  } while (0)

// the band counts, extents and list length before the tubes of a step
__global__ void k_band_begin(int L, long long* __restrict__ nbcnt, int* __restrict__ bbox, int* __restrict__ count) {
  pdl_wait();
  for (int t = threadIdx.x; t < 10 * L; t += blockDim.x) {
    bbox[t] = t < 5 * L ? 0x7F7F7F7F : (int)0x80808080;
    if (t < L) nbcnt[t] = 0;
  }
  if (threadIdx.x == 0) *count = 0;
}
void launch_band_begin(Ctx& c) {
  Scope sc_(c.prof, c.s, "band_begin", 1);
  pdl(k_band_begin, 1, 256, 0, c.s)(c.P.L, c.d_nbcnt, c.d_bbox, c.band_count);
}
void launch_tube(Ctx& c, LsBatch& b, bool list, bool fresh) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "tube", 1);
  // the register window along z is filled once per chunk (one drop at 64^3:
  // 8 rows 21.0 us, 4 rows 19.1, 2 rows 23.2)
  size_tiles(c.P, b, kTubeRows, 4, 4 * 148);
  int* lo = c.d_bbox;
  int* hi = c.d_bbox + 5 * c.P.L;
  if (list && !fresh) cudaMemsetAsync(c.band_count, 0, sizeof(int), c.s);
  BandCell* l = list ? reinterpret_cast<BandCell*>(c.band_list) : nullptr;
  BY_FORM(c, (pdl(k_tube<float>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.d_nbcnt, lo, hi, l, c.band_count)),
          (pdl(k_tube<double>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.d_nbcnt, lo, hi, l, c.band_count)));
}

void launch_band_extents(Ctx& c, int l) {
  Scope sc_(c.prof, c.s, "band_extents", 1);
  int* lo = c.d_bbox;
  int* hi = c.d_bbox + 5 * c.P.L;
  const unsigned g = (unsigned)(((long long)c.P.imax * c.P.jmax + NT - 1) / NT);
  BY_FORM(c, (pdl(k_band_extents<float>, g, NT, 0, c.s)(c.P, reinterpret_cast<const float*>(c.lv[l]), l, lo, hi)),
          (pdl(k_band_extents<double>, g, NT, 0, c.s)(c.P, c.lv[l], l, lo, hi)));
}

template <typename T>
void adv_launch(Ctx& c, const LsBatch& b, int scheme, int stage1, double a, double bb, double fdt, const double* vu,
                const double* vv, const double* vw) {
  const T* u = reinterpret_cast<const T*>(vu);
  const T* v = reinterpret_cast<const T*>(vv);
  const T* w = reinterpret_cast<const T*>(vw);
  // one instance per scheme and spacing case (PW: every a/dx a product;
  // the FP32 form always takes the product by the reciprocal)
  const unsigned g = b.start[b.n];
  const bool pw = c.P.pow2 || sizeof(T) == 4;
  auto go = [&](auto kernel) { pdl(kernel, g, kTile, 0, c.s)(c.P, b, stage1, a, bb, fdt, u, v, w); };
  if (scheme == ICLS_HOUC5) {
    if (pw) go(k_adv_stage<ICLS_HOUC5, T, 1>);
    else go(k_adv_stage<ICLS_HOUC5, T, 0>);
  } else {
    if (pw) go(k_adv_stage<ICLS_WENO5, T, 1>);
    else go(k_adv_stage<ICLS_WENO5, T, 0>);
  }
}
// one RK stage over the batch from the list of its tube sweep; need = the
// upper bound of its length that the caller checked against c.band_cap
template <typename T, bool INFL>
void adv_band_launch(Ctx& c, const LsBatch& b, int scheme, int stage1, double a, double bb, double fdt,
                     const double* vu, const double* vv, const double* vw, long long need, bool rest, bool walls) {
  const T* u = reinterpret_cast<const T*>(vu);
  const T* v = reinterpret_cast<const T*>(vv);
  const T* w = reinterpret_cast<const T*>(vw);
  const BandCell* list = reinterpret_cast<const BandCell*>(c.band_list);
  const unsigned nb = (unsigned)std::min<long long>((need + NT - 1) / NT, 8 * 148);
  const bool pw = c.P.pow2 || sizeof(T) == 4;
  auto go = [&](auto kernel) { pdl(kernel, nb, NT, 0, c.s)(c.P, b, list, c.band_count, stage1, a, bb, fdt, u, v, w, c.dinf, c.vin); };
  if (nb > 0) {
    if (scheme == ICLS_HOUC5) {
      if (pw) go(k_adv_band<ICLS_HOUC5, T, 1, INFL>);
      else go(k_adv_band<ICLS_HOUC5, T, 0, INFL>);
    } else {
      if (pw) go(k_adv_band<ICLS_WENO5, T, 1, INFL>);
      else go(k_adv_band<ICLS_WENO5, T, 0, INFL>);
    }
  }
  if (rest) pdl(k_adv_rest<T>, b.start[b.n], kTile, 0, c.s)(c.P, b);
  if (walls) {
    LsBatch w1 = b;
    set_tiles(w1, 0);
    pdl(k_adv_ghosts<T>, w1.start[w1.n], kTile, 0, c.s)(c.P, w1, stage1, a, bb);
  }
}
bool holds_walls(const LsBatch& b) {
  for (int q = 0; q < b.n; ++q)
    if (b.t[q].r.cz0 <= -2) return true;
  return false;
}
void launch_adv_band(Ctx& c, const LsBatch& b, int scheme, int stage1, double a, double bb, double fdt,
                     const double* vu, const double* vv, const double* vw, long long need, bool rest) {
  if (b.n == 0) return;
  const bool walls = holds_walls(b);
  Scope sc_(c.prof, c.s, "adv_stage", 1 + (walls ? 1 : 0) + (rest ? 1 : 0));
  BY_FORM(c, (adv_band_launch<float, false>(c, b, scheme, stage1, a, bb, fdt, vu, vv, vw, need, rest, walls)),
          (adv_band_launch<double, false>(c, b, scheme, stage1, a, bb, fdt, vu, vv, vw, need, rest, walls)));
}
// the mass correction's stages: its buffers and list, then one stage over the list
void launch_inflate_base(Ctx& c, const LsBatch& b) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "inflate_stage", 1);
  cudaMemsetAsync(c.band_count, 0, sizeof(int), c.s);
  BandCell* l = reinterpret_cast<BandCell*>(c.band_list);
  BY_FORM(c, (pdl(k_inflate_base<float>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.dinf, l, c.band_count)),
          (pdl(k_inflate_base<double>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.dinf, l, c.band_count)));
}
void launch_inflate_stage(Ctx& c, const LsBatch& b, int scheme, int stage1, double a, double bb, double fdt,
                          long long need) {
  if (b.n == 0) return;
  const bool walls = holds_walls(b);
  Scope sc_(c.prof, c.s, "inflate_stage", 1 + (walls ? 1 : 0));
  BY_FORM(c, (adv_band_launch<float, true>(c, b, scheme, stage1, a, bb, fdt, nullptr, nullptr, nullptr, need, false, walls)),
          (adv_band_launch<double, true>(c, b, scheme, stage1, a, bb, fdt, nullptr, nullptr, nullptr, need, false, walls)));
}

void launch_adv_stage(Ctx& c, const LsBatch& b, int scheme, int stage1, double a, double bb, double fdt,
                      const double* vu, const double* vv, const double* vw) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "adv_stage", 1);
  BY_FORM(c, adv_launch<float>(c, b, scheme, stage1, a, bb, fdt, vu, vv, vw),
          adv_launch<double>(c, b, scheme, stage1, a, bb, fdt, vu, vv, vw));
}

void launch_reinit_stage(Ctx& c, const LsBatch& b, int stage, double dtau) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "reinit_stage", 1);
  const unsigned g = b.start[b.n];
  // the FP32 form takes the product by the reciprocal at any spacing
  if (c.P.f32) pdl(k_reinit_stage<float, 1>, g, kTile, 0, c.s)(c.P, b, stage, dtau, c.drs);
  else if (c.P.pow2) pdl(k_reinit_stage<double, 1>, g, kTile, 0, c.s)(c.P, b, stage, dtau, c.drs);
  else pdl(k_reinit_stage<double, 0>, g, kTile, 0, c.s)(c.P, b, stage, dtau, c.drs);
}
void launch_reinit_reset(Ctx& c, const LsBatch& b, int maxiter) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "reinit_reset", 1);
  pdl(k_reinit_reset, 1, 64, 0, c.s)(b, maxiter, c.drs);
}
void launch_reinit_check(Ctx& c, const LsBatch& b, int it, int maxiter, double thr) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "reinit_check", 1);
  pdl(k_reinit_check, 1, 64, 0, c.s)(b, it, maxiter, thr, c.drs, c.dsc, c.P.L - 1);
}

// the per-(tile, chunk) exact sums of H: hcap per drop (4 words each)
XSum* hparts(Ctx& c) { return reinterpret_cast<XSum*>(c.hpart); }

void launch_heaviside(Ctx& c, const LsBatch& b) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "heaviside", 1);
  BY_FORM(c,
          (pdl(k_heaviside<float>, b.start[b.n], kTile, 0, c.s)(c.P, b, reinterpret_cast<float*>(c.jiemian),
                                                                c.seg_mat[c.mat_cur], hparts(c), c.hcap)),
          (pdl(k_heaviside<double>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.jiemian, c.seg_mat[c.mat_cur], hparts(c),
                                                                 c.hcap)));
}

// n elements of a; tfield: a holds the form's field type (else FP64)
void launch_fill(Ctx& c, double* a, long long n, double v, bool tfield) {
  Scope sc_(c.prof, c.s, "fill", 1);
  if (tfield && c.P.f32)
    pdl(k_fill<float>, 1184, NT, 0, c.s)(reinterpret_cast<float*>(a), n, v);
  else
    pdl(k_fill<double>, 1184, NT, 0, c.s)(a, n, v);
}

void launch_disp(Ctx& c, int l) {
  Scope sc_(c.prof, c.s, "disp", 2);
  BY_FORM(c, (pdl(k_disp<float>, kRedBlocks, kRedThreads, 0, c.s)(c.P, reinterpret_cast<const float*>(c.lv[l]),
                                                                  reinterpret_cast<const float*>(c.ucc),
                                                                  reinterpret_cast<const float*>(c.vcc),
                                                                  reinterpret_cast<const float*>(c.wcc), c.diag)),
          (pdl(k_disp<double>, kRedBlocks, kRedThreads, 0, c.s)(c.P, c.lv[l], c.ucc, c.vcc, c.wcc, c.diag)));
  pdl(k_disp_final, 1, kRedThreads, 0, c.s)(c.diag, kRedBlocks, c.diag + 7 * kRedBlocks);
}

// outside, ntiles: each drop's far-field cells and its partials
void launch_volumes(Ctx& c, const double* outside, const int* ntiles, bool extents) {
  const int L = c.P.L;
  Scope sc_(c.prof, c.s, "volumes", (L + kMaxDropsParam - 1) / kMaxDropsParam);
  for (int l0 = 0; l0 < L; l0 += kMaxDropsParam) {
    const int nl = std::min(kMaxDropsParam, L - l0);
    PerDrop o = {};
    std::copy(outside + l0, outside + l0 + nl, o.v);
    std::copy(ntiles + l0, ntiles + l0 + nl, o.n);
    pdl(k_volumes, 1, 1024, 0, c.s)(c.P, hparts(c), c.hcap, o, l0, nl, c.dvol, c.dsc, c.h_vol,
                                  extents ? c.d_bbox : nullptr, c.h_bbox);
  }
}
// the warps of a sweep over the segments: enough for one group of 32 each, at
// most eight blocks per SM
// map bytes per warp (for_segments), 32 halved down to 2 while the warps are
// fewer than 2^14: a warp takes its set segments one after the other
// (k_materials_seg with 32 / 8 / 4 / 2: 64^3 22.8 / 10.6 / 9.6 / 8.4 us,
// 128^2 x 256 21.0 / 12.6 / 14.6 / 20.5 us; 256^3 x 48, 16 instead of 32: 35.0
// for 37.3 us, but the jumps' clearing 20.2 for 18.0)
int seg_per_warp(const Params& p) {
  int per = 32;
  while (per > 2 && seg_count(p) < ((long long)per << 14)) per /= 2;
  return per;
}
unsigned seg_blocks(const Params& p) {
  const int n = seg_per_warp(p) * (NT / 32);
  return (unsigned)std::min<long long>((seg_count(p) + n - 1) / n, kRedBlocks);
}
void launch_seg_reset(Ctx& c, const uint8_t* seg, uint8_t* next) {
  Scope sc_(c.prof, c.s, "fill", 1);
  const int per = seg_per_warp(c.P);
  BY_FORM(c,
          (pdl(k_seg_reset<float>, seg_blocks(c.P), NT, 0, c.s)(c.P, per, seg, next, reinterpret_cast<float*>(c.jiemian))),
          (pdl(k_seg_reset<double>, seg_blocks(c.P), NT, 0, c.s)(c.P, per, seg, next, c.jiemian)));
}
void launch_seg_clear_jumps(Ctx& c, uint8_t* faces, const uint8_t* lap) {
  Scope sc_(c.prof, c.s, "clear_jumps", 1);
  const int per = seg_per_warp(c.P);
  auto f = [](double* q) { return reinterpret_cast<float*>(q); };
  BY_FORM(c,
          (pdl(k_seg_clear_jumps<float>, seg_blocks(c.P), NT, 0, c.s)(c.P, per, faces, lap, c.row_jmp, f(c.px), f(c.py),
                                                                      f(c.pz), c.pjump)),
          (pdl(k_seg_clear_jumps<double>, seg_blocks(c.P), NT, 0, c.s)(c.P, per, faces, lap, c.row_jmp, c.px, c.py, c.pz,
                                                                       c.pjump)));
}
// miu, rho and the face densities; cur and prev: the maps of jiemian (null:
// one thread per cell of the whole arrays, ICLS_MATERIALS=rows1)
void launch_materials(Ctx& c, const uint8_t* cur, const uint8_t* prev) {
  Scope sc_(c.prof, c.s, "materials_final", 1);
  auto go = [&](auto zero, auto view) {
    using T = decltype(zero);
    if (cur) {
      pdl(k_materials_seg<T>, seg_blocks(c.P), NT, 0, c.s)(c.P, seg_per_warp(c.P), cur, prev, view(c.jiemian), view(c.miu), view(c.rho),
                                                          view(c.rho_u), view(c.rho_v), view(c.rho_w));
      return;
    }
    const int r0[3] = {0, 0, 0}, r1[3] = {c.P.i1, c.P.j1, c.P.k1};
    pdl(k_materials_final<T>, grid_of(r0, r1), kBlock, 0, c.s)(c.P, view(c.jiemian), view(c.miu), view(c.rho),
                                                              view(c.rho_u), view(c.rho_v), view(c.rho_w));
  };
  BY_FORM(c, go(0.f, [](double* q) { return reinterpret_cast<float*>(q); }), go(0., [](double* q) { return q; }));
}

// the area sums behind the exact sums
double* aparts(Ctx& c) { return c.hpart + (size_t)4 * c.P.L * c.hcap; }
// tasks: the drops' shape-C regions, apron 1, in z chunks of kStageRows (at
// most hcap partials per drop), phi0 = their level sets, far = the interior
// cells outside them
void launch_inflate_sums(Ctx& c, const LsBatch& b) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "inflate_sums", 2);
  BY_FORM(c, (pdl(k_inflate_sums<float>, b.start[b.n], kTile, 0, c.s)(c.P, b, aparts(c), hparts(c), c.hcap)),
          (pdl(k_inflate_sums<double>, b.start[b.n], kTile, 0, c.s)(c.P, b, aparts(c), hparts(c), c.hcap)));
  pdl(k_inflate_final, b.n, kFinalThreads, 0, c.s)(c.P, b, aparts(c), hparts(c), c.hcap,
                                                  (double)c.cfg.inflate_step * c.dt, c.dvol, c.dvol0, c.dmaxchk,
                                                  c.dinf);
}
// gain-one inflation: the volume after it, and the blend
void launch_region_heav(Ctx& c, const LsBatch& b) {
  BY_FORM(c, (pdl(k_region_heav<float>, b.start[b.n], kTile, 0, c.s)(c.P, b, hparts(c), c.hcap)),
          (pdl(k_region_heav<double>, b.start[b.n], kTile, 0, c.s)(c.P, b, hparts(c), c.hcap)));
}
void launch_gain(Ctx& c, const LsBatch& b) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "gain_one", 2);
  launch_region_heav(c, b);
  pdl(k_gain_final, b.n, kFinalThreads, 0, c.s)(c.P, b, hparts(c), c.hcap, c.dvol, c.dvol0, c.dinf);
}
void launch_volume_now(Ctx& c, const LsBatch& b) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "gain_one", 2);
  launch_region_heav(c, b);
  pdl(k_volume_now, b.n, kFinalThreads, 0, c.s)(c.P, b, hparts(c), c.hcap, c.dvolnow);
}
void launch_region_blend(Ctx& c, const LsBatch& b) {
  if (b.n == 0) return;
  Scope sc_(c.prof, c.s, "gain_one", 1);
  BY_FORM(c, (pdl(k_region_blend<float>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.dinf)),
          (pdl(k_region_blend<double>, b.start[b.n], kTile, 0, c.s)(c.P, b, c.dinf)));
}

void launch_boundmls(Ctx& c, double* phi) {
  Scope sc_(c.prof, c.s, "boundmls", 1);
  const int r0[3] = {-2, -2, -2}, r1[3] = {c.P.i1 + 2, c.P.j1 + 2, c.P.k1 + 2};
  BY_FORM(c, (pdl(k_boundmls<float>, grid_of(r0, r1), kBlock, 0, c.s)(c.P, reinterpret_cast<float*>(phi))),
          (pdl(k_boundmls<double>, grid_of(r0, r1), kBlock, 0, c.s)(c.P, phi)));
}

void launch_materialize(Ctx& c, const Region& r, double bg, double bgg, double* phi) {
  Scope sc_(c.prof, c.s, "materialize", 1);
  const int r0[3] = {-2, -2, -2}, r1[3] = {c.P.i1 + 2, c.P.j1 + 2, c.P.k1 + 2};
  BY_FORM(c,
          (pdl(k_materialize<float>, grid_of(r0, r1), kBlock, 0, c.s)(c.P, r, bg, bgg, reinterpret_cast<float*>(phi))),
          (pdl(k_materialize<double>, grid_of(r0, r1), kBlock, 0, c.s)(c.P, r, bg, bgg, phi)));
}

void launch_to_float(Ctx& c, double* dst_f32, const double* src, long long n) {
  pdl(k_to_float, 1184, 256, 0, c.s)(reinterpret_cast<float*>(dst_f32), src, n);
}
void launch_to_double(Ctx& c, double* dst, const double* src_f32, long long n) {
  pdl(k_to_double, 1184, 256, 0, c.s)(dst, reinterpret_cast<const float*>(src_f32), n);
}

}  // namespace icls
