// k_navier.cu — momentum, projection and check kernels (FP64, -fmad=false).
//
//   mom_main       mom.f90:13-62 (CNTR2_conv 67-130, delta_diff 134-273,
//                  NS_grav 277-301)
//   ab2            ab2.f90:21-138 with momxp/yp/zp mom.f90:779-851
//   fillps         fillps.f90:13-57
//   correc         correc.f90:15-44
//   bounduvw/boundp bound.f90:15-287
//   pressure update main.f90:164-185
//   averages       misc.f90:587-655;  chkdiv chkdiv.f90:10-90;
//   chkdt          chkdt.f90:11-105
//
// Boundary rows and periodic halos are produced in the kernel that computes
// the field: a halo or wall cell evaluates the interior value(s) it copies
// or extrapolates from (bound.f90:36-75), so no separate boundary pass runs.
#include <algorithm>

#include "ab2.cuh"
#include "batch.cuh"

namespace icls {

namespace {

constexpr int NT = 256;
// T is the form's field type (double, or float in the precision form);
// TC(x) is the constant x in T
#define TC(x) static_cast<T>(x)
inline unsigned nblocks(long long n, int nt = NT) { return (unsigned)((n + nt - 1) / nt); }

__device__ __forceinline__ void decodeI(const Params& p, int q, int& i, int& j, int& k) {
  i = q % p.imax + 1;
  const int r = q / p.imax;
  j = r % p.jmax + 1;
  k = r / p.jmax + 1;
}

__constant__ int kC0[3] = {0, 0, 0};
__constant__ int kI0[3] = {1, 1, 1};
struct I3 {
  int v[3];
};
__device__ __forceinline__ I3 cC1(const Params& p) { return I3{{p.i1, p.j1, p.k1}}; }
__device__ __forceinline__ I3 cI1(const Params& p) { return I3{{p.imax, p.jmax, p.kmax}}; }
const dim3 kBlock(BX, BY, 1);
inline dim3 gridC(const Params& p) {
  return dim3((unsigned)((p.nCx + BX - 1) / BX), (unsigned)((p.nCy + BY - 1) / BY), (unsigned)p.nCz);
}
inline dim3 gridI(const Params& p) {
  return dim3((unsigned)((p.imax + BX - 1) / BX), (unsigned)((p.jmax + BY - 1) / BY), (unsigned)p.kmax);
}


// mom_main alone (init.f90:90): RHS into shape-I arrays
template <typename T>
__global__ void __launch_bounds__(NT) k_mom_main(Params p, MomArgs a, T* __restrict__ ru, T* __restrict__ rv,
                                                 T* __restrict__ rw) {
  pdl_wait();
  int i, j, k;
  if (!cell3(kI0, cI1(p).v, i, j, k)) return;
  const long long q = idxI(p, i, j, k);
  const long long c = idxC(p, i, j, k);
  const long long sy = p.nCx, sz = (long long)p.nCx * p.nCy;
  const T rho_avr = TC(*a.rho_avr);
  const T *u = cT<T>(a.u), *v = cT<T>(a.v), *w = cT<T>(a.w), *miu = cT<T>(a.miu);
  auto U = [&](int di, int dj, int dk) { return u[c + di + dj * sy + dk * sz]; };
  auto V = [&](int di, int dj, int dk) { return v[c + di + dj * sy + dk * sz]; };
  auto W = [&](int di, int dj, int dk) { return w[c + di + dj * sy + dk * sz]; };
  auto M = [&](int di, int dj, int dk) { return miu[c + di + dj * sy + dk * sz]; };
  ru[q] = rhs_u<T>(p, U, V, W, M, [&](T x) { return x / cT<T>(a.rho_u)[q]; }, rho_avr);
  rv[q] = rhs_v<T>(p, U, V, W, M, [&](T x) { return x / cT<T>(a.rho_v)[q]; }, rho_avr);
  rw[q] = rhs_w<T>(p, U, V, W, M, [&](T x) { return x / cT<T>(a.rho_w)[q]; }, rho_avr);
}

// The predictor's near rows: a tile (32 x 8 columns) and row whose cells, or
// the neighbours that its stencil reads, lie in a set segment of the
// materials, or whose own cells lie in one of the face jumps' (now or old).
// One thread per four segments; few are set, and those mark the tiles around
// them (near starts at 0).
__global__ void __launch_bounds__(NT) k_ab2_near(Params p, const uint8_t* __restrict__ mat,
                                                 const uint8_t* __restrict__ jmp, const uint8_t* __restrict__ jmpold,
                                                 uint8_t* __restrict__ near) {
  pdl_wait();
  const long long w = blockIdx.x * (long long)NT + threadIdx.x;
  if (4 * w >= seg_count(p)) return;
  // (the maps are padded with zeros to a multiple of four)
  const unsigned m4 = reinterpret_cast<const unsigned*>(mat)[w];
  const unsigned j4 = reinterpret_cast<const unsigned*>(jmp)[w] | reinterpret_cast<const unsigned*>(jmpold)[w];
  if (!(m4 | j4)) return;
  const int nsx = seg_row(p);
  for (int b = 0; b < 4; ++b) {
    const bool m = (m4 >> 8 * b) & 0xFFu, jj = (j4 >> 8 * b) & 0xFFu;
    if (!m && !jj) continue;
    const long long q = 4 * w + b, r = q / nsx;
    const int sx = (int)(q - r * nsx), k = (int)(r / p.jmax), j = (int)(r - (long long)k * p.jmax) + 1;
    auto set = [&](int s, int y, int kk) { near[((long long)s + (long long)nsx * ((y - 1) / kAb2Y)) * p.nCz + kk] = 1; };
    if (!m) {
      set(sx, j, k);
      continue;
    }
    const int xm = sx ? sx - 1 : nsx - 1, xp = sx + 1 < nsx ? sx + 1 : 0;
    const int ym = wrapy(p, j - 1), yp = wrapy(p, j + 1);
    for (int kk = max(k - 1, 1); kk <= min(k + 1, p.kmax); ++kk)
      for (int s : {xm, sx, xp}) {
        set(s, ym, kk);
        set(s, j, kk);
        set(s, yp, kk);
      }
  }
}

// fillps (fillps.f90:36-53), optionally followed by p = p + p_jump
template <typename T>
__global__ void __launch_bounds__(NT) k_fillps(Params p, const T* __restrict__ dudt, const T* __restrict__ dvdt,
                                               const T* __restrict__ dwdt, const double* __restrict__ pjump, int add,
                                               double* __restrict__ out) {
  pdl_wait();
  int i, j, k;
  if (!cell3(kI0, cI1(p).v, i, j, k)) return;
  const long long q = idxI(p, i, j, k);
  const long long c = idxC(p, i, j, k);
  const double coef = p.rho0 / p.dt;
  const double vel_x = ((double)dudt[c] - (double)dudt[c - 1]) * p.dxi;
  const double vel_y = ((double)dvdt[c] - (double)dvdt[c - p.nCx]) * p.dyi;
  const double vel_z = ((double)dwdt[c] - (double)dwdt[c - (long long)p.nCx * p.nCy]) * p.dzi;
  double v = coef * ((vel_x + vel_y) + vel_z);
  if (add) v = v + pjump[c];
  out[c] = v;
}

__global__ void __launch_bounds__(NT) k_add(Params p, double* __restrict__ a, const double* __restrict__ b) {
  pdl_wait();
  const long long n = blockIdx.x * (long long)NT + threadIdx.x;
  if (n < p.nC) a[n] = a[n] + b[n];
}

// correc of one component (correc.f90:27-39)
// (the pressure gradient in FP64, the result in the form's type T)
template <typename T>
__device__ __forceinline__ T corr_u(const Params& p, const T* dudt, const double* pp, const T* px, int i, int j,
                                    int k) {
  const long long c = idxC(p, i, j, k);
  if (sizeof(T) == sizeof(double)) return (T)(dudt[c] - div_rho0(p, p.dt * p.dxi * ((pp[c + 1] - pp[c]) - (double)px[c])));
  return dudt[c] - (T)(div_rho0(p, p.dt * p.dxi * ((pp[c + 1] - pp[c]) - (double)px[c])));
}
template <typename T>
__device__ __forceinline__ T corr_v(const Params& p, const T* dvdt, const double* pp, const T* py, int i, int j,
                                    int k) {
  const long long c = idxC(p, i, j, k);
  if (sizeof(T) == sizeof(double)) return (T)(dvdt[c] - div_rho0(p, p.dt * p.dyi * ((pp[c + p.nCx] - pp[c]) - (double)py[c])));
  return dvdt[c] - (T)(div_rho0(p, p.dt * p.dyi * ((pp[c + p.nCx] - pp[c]) - (double)py[c])));
}
template <typename T>
__device__ __forceinline__ T corr_w(const Params& p, const T* dwdt, const double* pp, const T* pz, int i, int j,
                                    int k) {
  const long long c = idxC(p, i, j, k);
  const long long sz = (long long)p.nCx * p.nCy;
  if (sizeof(T) == sizeof(double)) return (T)(dwdt[c] - div_rho0(p, p.dt * p.dzi * ((pp[c + sz] - pp[c]) - (double)pz[c])));
  return dwdt[c] - (T)(div_rho0(p, p.dt * p.dzi * ((pp[c + sz] - pp[c]) - (double)pz[c])));
}

struct CorrArgs {
  const double *dudt, *dvdt, *dwdt, *p, *px, *py, *pz;
  double *u, *v, *w, *ucc, *vcc, *wcc;
  DevScalars* dsc;
  const uint8_t* seg;  // segment map of px, py, pz
};

// correc + bounduvw(unew,vnew,wnew) + average_vel_at_center + NaN probe
// (main.f90:159-160,190,207) over shape C
template <typename T>
__global__ void __launch_bounds__(NT) k_correc_fused(Params p, CorrArgs a) {
  pdl_wait();
  int i, j, k;
  if (!cell3(kC0, cC1(p).v, i, j, k)) return;
  const long long n = idxC(p, i, j, k);
  const int I = wrapx(p, i), J = wrapy(p, j);
  const T *du = cT<T>(a.dudt), *dv = cT<T>(a.dvdt), *dw = cT<T>(a.dwdt);
  T uu, vv, ww;
  if (k >= 1 && k <= p.kmax) {
    uu = corr_u(p, du, a.p, cT<T>(a.px), I, J, k);
    vv = corr_v(p, dv, a.p, cT<T>(a.py), I, J, k);
    ww = (k == p.kmax) ? TC(0.) : corr_w(p, dw, a.p, cT<T>(a.pz), I, J, k);
  } else if (k == 0) {
    uu = -corr_u(p, du, a.p, cT<T>(a.px), I, J, 1);
    vv = TC(2. * p.v_lower) - corr_v(p, dv, a.p, cT<T>(a.py), I, J, 1);
    ww = TC(0.);
  } else {
    uu = -corr_u(p, du, a.p, cT<T>(a.px), I, J, p.kmax);
    vv = TC(2. * p.v_upper) - corr_v(p, dv, a.p, cT<T>(a.py), I, J, p.kmax);
    ww = corr_w(p, dw, a.p, cT<T>(a.pz), I, J, p.kmax - 1);
  }
  mT<T>(a.u)[n] = uu;
  mT<T>(a.v)[n] = vv;
  mT<T>(a.w)[n] = ww;
  if (i == I && j == J && k >= 1 && k <= p.kmax) {
    const long long q = idxI(p, i, j, k);
    const T um = corr_u(p, du, a.p, cT<T>(a.px), wrapx(p, i - 1), j, k);
    const T vm = corr_v(p, dv, a.p, cT<T>(a.py), i, wrapy(p, j - 1), k);
    const T wm = (k == 1) ? TC(0.) : corr_w(p, dw, a.p, cT<T>(a.pz), i, j, k - 1);
    mT<T>(a.ucc)[q] = (um + uu) / TC(2.);
    mT<T>(a.vcc)[q] = (vm + vv) / TC(2.);
    mT<T>(a.wcc)[q] = (wm + ww) / TC(2.);
    if (i == 1 && j == 1 && k == 1 && isnan(vv)) a.dsc->nan_flag = 1;
  }
}

// One correc value (correc.f90:27-39), d - dt dhi ((p+ - p) - jump) / rho0:
// the expression of corr_u/v/w with cd = dt dhi (the reference's first
// product) and the division by rho0 chosen at compile time (RP 1: rho0 a power
// of two, the product by its exact reciprocal)
template <typename T, int RP>
__device__ __forceinline__ T corr_val(const Params& p, T d, double pp, double p0, T jump, double cd) {
  const double a = cd * ((pp - p0) - (double)jump);
  const double g = RP == 1 ? a * p.rrho0 : a / p.rho0;
  if (sizeof(T) == sizeof(double)) return (T)((double)d - g);
  return d - (T)g;
}

// k_correc_fused's fields with one thread per interior cell: the thread
// writes its cell's u, v, w with their periodic images, at k = 1 and
// k = kmax the wall rows k = 0 and k1 with theirs, and the cell-centre
// velocities.  The halo and wall cells are the images k_correc_fused
// computes from the same source cells, so the fields are the same bits;
// every warp is a full row segment and no thread recomputes a source
// column's corrections for a halo cell.  The face jumps are read where the
// segment map says that they can be nonzero (a warp is one segment of a row);
// at 256^3 with 48 drops that leaves 10 of the 13 fields.  The pressure of the
// cell serves its west, south and lower neighbours' corrections (its images
// are the same value).  Instruction issue bounds the FP32 form (77 % busy), so
// indices are 32-bit (an array has less than 2^30 elements) and the images'
// tests are made once per thread: with the map, FP64 0.373 -> 0.293 ms and
// FP32 0.257 -> 0.232 ms; 128 x 128 x 256 FP64 with a rho0 that divides 0.126 ->
// 0.093 ms.
// A thread takes `rows` rows upwards, whose lower neighbours' corrections and
// own pressures it then has in registers: one row per thread read the p planes
// three times through L2 (256^3: FP64 0.293 -> 0.266 ms, FP32 0.232 -> 0.167).
// Rows and blocks per SM: FP64 4 and 4 (8 and 5: 0.273 ms), FP32 8 and 8 (4
// and 6: 0.179 ms).
template <typename T>
constexpr int kCorRows = sizeof(T) == 4 ? 8 : 4;
template <typename T, int RP>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 8 : 4)) k_correc_own(Params p, CorrArgs a, int rows) {
  pdl_wait();
  const int i = 1 + BX * (int)blockIdx.x + (int)threadIdx.x, j = 1 + BY * (int)blockIdx.y + (int)threadIdx.y;
  const int ka = 1 + rows * (int)blockIdx.z, kb = min(ka + rows - 1, p.kmax);
  if (i > p.imax || j > p.jmax) return;
  const int sy = p.nCx, sz = p.nCx * p.nCy;
  int c = i + sy * j + sz * ka;
  const int ox = i > 1 ? -1 : p.imax - 1, oy = j > 1 ? -sy : sy * (p.jmax - 1);
  const T* __restrict__ du = cT<T>(a.dudt);
  const T* __restrict__ dv = cT<T>(a.dvdt);
  const T* __restrict__ dw = cT<T>(a.dwdt);
  const double* __restrict__ pp = a.p;
  const int nsx = seg_row(p), sp = nsx * p.jmax;
  const uint8_t* __restrict__ seg = a.seg + ((int)blockIdx.x + nsx * (j - 1) + sp * ka);
  const int ow = blockIdx.x ? -1 : nsx - 1, os = j > 1 ? -nsx : sp - nsx;
  T* __restrict__ u = mT<T>(a.u);
  T* __restrict__ v = mT<T>(a.v);
  T* __restrict__ w = mT<T>(a.w);
  T* __restrict__ uc = mT<T>(a.ucc);
  T* __restrict__ vc = mT<T>(a.vcc);
  T* __restrict__ wc = mT<T>(a.wcc);
  int q = (i - 1) + p.imax * ((j - 1) + p.jmax * (ka - 1));
  const bool ex = i == 1 || i == p.imax, ey = j == 1 || j == p.jmax;
  double p0 = pp[c];
  // the correction of the row below, or the wall's
  T wl = corr_val<T, RP>(p, dw[c - sz], p0, pp[c - sz], seg[-sp] ? cT<T>(a.pz)[c - sz] : TC(0.), p.cdz);
  for (int k = ka; k <= kb; ++k) {
    const uint8_t own = seg[0], west = seg[ow], south = seg[os];
    const double pe = pp[c + 1], pn = pp[c + sy], pu = pp[c + sz], pw = pp[c + ox], ps = pp[c + oy];
    const T d0 = du[c], d1 = dv[c], d2 = dw[c], e0 = du[c + ox], e1 = dv[c + oy];
    T qx = TC(0.), qy = TC(0.), qz = TC(0.), qxm = TC(0.), qym = TC(0.);
    if (own) {
      qx = cT<T>(a.px)[c];
      qy = cT<T>(a.py)[c];
      qz = cT<T>(a.pz)[c];
    }
    if (own | west) qxm = cT<T>(a.px)[c + ox];
    if (south) qym = cT<T>(a.py)[c + oy];
    const T uu = corr_val<T, RP>(p, d0, pe, p0, qx, p.cdx);
    const T vv = corr_val<T, RP>(p, d1, pn, p0, qy, p.cdy);
    const T ww = (k == p.kmax) ? TC(0.) : corr_val<T, RP>(p, d2, pu, p0, qz, p.cdz);
    // the cell-centre average's (i-1) and (j-1) corrections
    const T um = corr_val<T, RP>(p, e0, p0, pw, qxm, p.cdx);
    const T vm = corr_val<T, RP>(p, e1, p0, ps, qym, p.cdy);
    u[c] = uu;
    v[c] = vv;
    w[c] = ww;
    uc[q] = (um + uu) / TC(2.);
    vc[q] = (vm + vv) / TC(2.);
    wc[q] = (((k == 1) ? TC(0.) : wl) + ww) / TC(2.);
    if (ex | ey | (k == 1) | (k == p.kmax)) {  // images and wall rows
      const int di = ex ? (i == 1 ? p.imax : -p.imax) : 0, dj = ey ? sy * (j == 1 ? p.jmax : -p.jmax) : 0;
      auto put = [&](T* __restrict__ f, int n, T x) {
        f[n] = x;
        if (di) f[n + di] = x;
        if (dj) {
          f[n + dj] = x;
          if (di) f[n + di + dj] = x;
        }
      };
      put(u, c, uu);
      put(v, c, vv);
      put(w, c, ww);
      if (k == 1) {
        put(u, c - sz, -uu);
        put(v, c - sz, TC(2. * p.v_lower) - vv);
        put(w, c - sz, TC(0.));
      }
      if (k == p.kmax) {
        put(u, c + sz, -uu);
        put(v, c + sz, TC(2. * p.v_upper) - vv);
        put(w, c + sz, wl);
      }
      if (i == 1 && j == 1 && k == 1 && isnan(vv)) a.dsc->nan_flag = 1;
    }
    wl = ww;
    p0 = pu;
    c += sz;
    q += p.imax * p.jmax;
    seg += sp;
  }
}

// correc over the interior only (the separate reference call): rows upwards
// and the face jumps where the map has them, as above (with
// every jump read, against one row per thread: 256^3
// FP64 0.256 -> 0.209 ms)
template <typename T, int RP>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 8 : 6)) k_correc_interior(Params p, CorrArgs a, int rows) {
  pdl_wait();
  const int i = 1 + BX * (int)blockIdx.x + (int)threadIdx.x, j = 1 + BY * (int)blockIdx.y + (int)threadIdx.y;
  const int ka = 1 + rows * (int)blockIdx.z, kb = min(ka + rows - 1, p.kmax);
  if (i > p.imax || j > p.jmax) return;
  const int sy = p.nCx, sz = p.nCx * p.nCy, sp = seg_row(p) * p.jmax;
  int c = i + sy * j + sz * ka;
  const double* __restrict__ pp = a.p;
  const uint8_t* __restrict__ seg = a.seg + ((int)blockIdx.x + seg_row(p) * (j - 1) + sp * ka);
  double p0 = pp[c];
  for (int k = ka; k <= kb; ++k) {
    const double pe = pp[c + 1], pn = pp[c + sy], pu = pp[c + sz];
    const T d0 = cT<T>(a.dudt)[c], d1 = cT<T>(a.dvdt)[c], d2 = cT<T>(a.dwdt)[c];
    T qx = TC(0.), qy = TC(0.), qz = TC(0.);
    if (*seg) {
      qx = cT<T>(a.px)[c];
      qy = cT<T>(a.py)[c];
      qz = cT<T>(a.pz)[c];
    }
    mT<T>(a.u)[c] = corr_val<T, RP>(p, d0, pe, p0, qx, p.cdx);
    mT<T>(a.v)[c] = corr_val<T, RP>(p, d1, pn, p0, qy, p.cdy);
    mT<T>(a.w)[c] = corr_val<T, RP>(p, d2, pu, p0, qz, p.cdz);
    p0 = pu;
    c += sz;
    seg += sp;
  }
}

// The halo cells of shape C by number: the planes k = 0 and k = k1, then the
// x faces (i = 0, i1 of every row, side fastest: the end of a row and the
// start of the next share a sector), then the y faces, both for k = 1..kmax.
// One thread per halo cell: a sweep of the whole array to find them read
// nothing but launched 64x the threads (256^3 FP64: boundp 48 -> 11 us,
// bounduvw 74 -> 15 us).
__host__ __device__ __forceinline__ int halo_plane_cells(const Params& p) { return p.nCx * p.nCy; }
inline int halo_cells(const Params& p) {
  return 2 * halo_plane_cells(p) + 2 * p.nCy * p.kmax + 2 * p.imax * p.kmax;
}
__device__ __forceinline__ bool halo_cell(const Params& p, int q, int& i, int& j, int& k) {
  const int np = halo_plane_cells(p);
  if (q < 2 * np) {
    k = q < np ? 0 : p.k1;
    if (q >= np) q -= np;
    j = q / p.nCx;
    i = q - j * p.nCx;
    return true;
  }
  q -= 2 * np;
  if (q < 2 * p.nCy * p.kmax) {
    i = (q & 1) ? p.i1 : 0;
    q >>= 1;
    k = q / p.nCy;
    j = q - k * p.nCy;
    ++k;
    return true;
  }
  q -= 2 * p.nCy * p.kmax;
  if (q >= 2 * p.imax * p.kmax) return false;
  const int r = q / p.imax;
  i = q - r * p.imax + 1;
  j = (r & 1) ? p.j1 : 0;
  k = (r >> 1) + 1;
  return true;
}

// bounduvw (bound.f90:15-177, Dirichl z, periodic x,y) on an existing
// triple: the halo cells, and w = 0 on the whole plane k = kmax (numbered
// after them)
template <typename T>
__global__ void __launch_bounds__(NT) k_bounduvw(Params p, T* __restrict__ u, T* __restrict__ v, T* __restrict__ w,
                                                 int halo) {
  pdl_wait();
  const int q = (int)(blockIdx.x * NT + threadIdx.x);
  if (q >= halo) {
    const int e = q - halo;
    if (e < halo_plane_cells(p)) w[idxC(p, 0, 0, p.kmax) + e] = TC(0.);
    return;
  }
  int i, j, k;
  if (!halo_cell(p, q, i, j, k)) return;
  const long long n = idxC(p, i, j, k);
  const int I = wrapx(p, i), J = wrapy(p, j);
  if (k == 0) {
    u[n] = -u[idxC(p, I, J, 1)];
    v[n] = TC(2. * p.v_lower) - v[idxC(p, I, J, 1)];
    w[n] = TC(0.);
  } else if (k == p.k1) {
    u[n] = -u[idxC(p, I, J, p.kmax)];
    v[n] = TC(2. * p.v_upper) - v[idxC(p, I, J, p.kmax)];
    w[n] = w[idxC(p, I, J, p.kmax - 1)];
  } else {
    u[n] = u[idxC(p, I, J, k)];
    v[n] = v[idxC(p, I, J, k)];
    if (k != p.kmax) w[n] = w[idxC(p, I, J, k)];
  }
}

// boundp (bound.f90:182-287, BC_in_y='Periodic')
template <typename T>
__global__ void __launch_bounds__(NT) k_boundp(Params p, T* __restrict__ a, int halo) {
  pdl_wait();
  const int q = (int)(blockIdx.x * NT + threadIdx.x);
  int i, j, k;
  if (q >= halo || !halo_cell(p, q, i, j, k)) return;
  const int I = wrapx(p, i), J = wrapy(p, j);
  const int K = k == 0 ? 1 : (k == p.k1 ? p.kmax : k);
  a[idxC(p, i, j, k)] = a[idxC(p, I, J, K)];
}

// the y boundaries of bounduvw for BC_in_y = Walls, InOut, OutOut
// (bound.f90:81-172), over i = 1..imax, k = 1..kmax once the periodic halos
// are in place: a thread does its (i,k) front row, then its back row
template <typename T>
__global__ void __launch_bounds__(NT) k_ywalls_uvw(Params p, T* __restrict__ u, T* __restrict__ v,
                                                   T* __restrict__ w, const double* __restrict__ vin) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
  if (i > p.imax) return;
  const long long f0 = idxC(p, i, 0, k), f1 = idxC(p, i, 1, k);
  if (p.bcy == ICLS_BCY_WALLS || p.bcy == ICLS_BCY_INOUT) {
    u[f0] = -u[f1];
    w[f0] = -w[f1];
    v[f0] = p.bcy == ICLS_BCY_WALLS ? TC(0.) : TC(vin[i + (long long)(p.i1 + 1) * k]);
  } else {
    u[f0] = u[f1];
    w[f0] = w[f1];
    v[f0] = v[f1] + TC(p.dy / p.dz) * (w[f1] - w[idxC(p, i, 1, k - 1)]);
  }
  const long long bj = idxC(p, i, p.jmax, k), b1 = idxC(p, i, p.j1, k);
  if (p.bcy == ICLS_BCY_WALLS) {
    u[b1] = -u[bj];
    v[bj] = TC(0.);
    v[b1] = v[bj];
    w[b1] = -w[bj];
  } else {
    u[b1] = u[bj];
    v[b1] = TC(2.) * v[bj] - v[idxC(p, i, p.jmax - 1, k)];
    w[b1] = w[bj];
  }
}
// the y boundaries of boundp (bound.f90:207-282): zero Neumann, or zero
// Dirichlet at an outflow end
template <typename T>
__global__ void __launch_bounds__(NT) k_ywalls_p(Params p, T* __restrict__ a) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
  if (i > p.imax) return;
  const T f = a[idxC(p, i, 1, k)], b = a[idxC(p, i, p.jmax, k)];
  a[idxC(p, i, 0, k)] = p.bcy == ICLS_BCY_OUTOUT ? -f : f;
  a[idxC(p, i, p.j1, k)] = p.bcy == ICLS_BCY_WALLS ? b : -b;
}
// isnan(vnew(1,1,1)) (main.f90:207)
template <typename T>
__global__ void k_nan_probe(Params p, const T* __restrict__ v, DevScalars* __restrict__ dsc) {
  pdl_wait();
  if (isnan(v[idxC(p, 1, 1, 1)])) dsc->nan_flag = 1;
}

// the plane i = const of an array with extents nx x ny x nz: dst(j,k) =
// src(ioff + nx j + nx ny k), j < n1, k < n2, converted to FP64
template <typename T>
__global__ void __launch_bounds__(NT) k_gather_plane_x(const T* __restrict__ src, long long nx, long long nxy, long long ioff,
                                                       int n1, int n2, double* __restrict__ dst) {
  pdl_wait();
  const long long q = blockIdx.x * (long long)NT + threadIdx.x;
  if (q >= (long long)n1 * n2) return;
  const long long j = q % n1, k = q / n1;
  dst[q] = (double)src[ioff + nx * j + nxy * k];
}

// average_vel_at_center (misc.f90:587-604)
template <typename T>
__global__ void __launch_bounds__(NT) k_average_vel(Params p, const T* __restrict__ u, const T* __restrict__ v,
                                                    const T* __restrict__ w, T* __restrict__ ucc, T* __restrict__ vcc,
                                                    T* __restrict__ wcc) {
  pdl_wait();
  int i, j, k;
  if (!cell3(kI0, cI1(p).v, i, j, k)) return;
  const long long q = idxI(p, i, j, k);
  const long long c = idxC(p, i, j, k);
  ucc[q] = (u[c - 1] + u[c]) / TC(2.);
  vcc[q] = (v[c - p.nCx] + v[c]) / TC(2.);
  wcc[q] = (w[c - (long long)p.nCx * p.nCy] + w[c]) / TC(2.);
}

// ---- pressure update (main.f90:164-185) ----------------------------------
// norm = sum(sum(pnew(:,:,1),2),1) in the Fortran order: for each i the
// sum over j, then the sum of those over i.
// the mean of p over the k = 1 plane, halo included (main.f90:173-175), by
// one block: the plane's (i, j) cells in a fixed strided order per thread,
// then a fixed tree
constexpr int kNormThreads = 1024;
__global__ void __launch_bounds__(kNormThreads) k_plane_norm(Params p, const double* __restrict__ pp,
                                                             DevScalars* __restrict__ dsc) {
  pdl_wait();
  const long long n = (long long)p.nCx * p.nCy, base = idxC(p, 0, 0, 1);
  double s = 0.;
  // eight loads under way, added in the same order (one at a time 11 us at 256^2;
  // the 128 x 90 x 75 projection 90 -> 86 us)
  for (long long e = threadIdx.x; e < n; e += 8 * kNormThreads) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = e + u * kNormThreads < n ? pp[base + e + u * kNormThreads] : 0.;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (e + u * kNormThreads < n) s += v[u];
  }
  s = block_sum<double, kNormThreads>(s);
  if (threadIdx.x == 0) {
    dsc->p_bad = 0;  // k_pupdate's, which follows
    dsc->norm_old = dsc->norm;
    dsc->norm = s / (1. * (p.imax) * p.jmax);
  }
}
// pnew and pold in the form's field type T (the arithmetic in FP64), two
// consecutive cells per thread through vector loads and stores (the
// buffers are 256-byte aligned and n is even); the same expressions per cell
template <typename T>
struct Vec2;
template <>
struct Vec2<float> {
  typedef float2 type;
};
template <>
struct Vec2<double> {
  typedef double2 type;
};
template <typename T>
__device__ __forceinline__ void pupdate_pair(double p0, double p1, T o0, T o1, T& n0, T& n1, T& d0, T& d1,
                                             int first, int normalise, double norm, double norm_old) {
  if (!normalise) {
    d0 = o0; d1 = o1;
    n0 = TC(p0); n1 = TC(p1);
    return;
  }
  const double a = (double)o0, b = (double)o1;
  d0 = TC(first ? a - norm : (a + norm_old) - norm);
  d1 = TC(first ? b - norm : (b + norm_old) - norm);
  n0 = TC(p0 - norm);
  n1 = TC(p1 - norm);
}
template <typename T>
__global__ void __launch_bounds__(NT) k_pupdate(Params p, const double* __restrict__ pp,
                                                T* __restrict__ pnew, T* __restrict__ pold, int first,
                                                int normalise, DevScalars* __restrict__ dsc) {
  pdl_wait();
  typedef typename Vec2<T>::type T2;
  const long long n = 2 * (blockIdx.x * (long long)NT + threadIdx.x);
  if (n >= p.nC) return;
  const double norm = normalise ? dsc->norm : 0., norm_old = normalise ? dsc->norm_old : 0.;
  if (n + 1 < p.nC) {
    const double2 pv = *reinterpret_cast<const double2*>(pp + n);
    const T2 ov = *reinterpret_cast<const T2*>(pnew + n);
    T2 nv, dv;
    pupdate_pair<T>(pv.x, pv.y, ov.x, ov.y, nv.x, nv.y, dv.x, dv.y, first, normalise, norm, norm_old);
    *reinterpret_cast<T2*>(pold + n) = dv;
    *reinterpret_cast<T2*>(pnew + n) = nv;
    if (!(isfinite(dv.x) && isfinite(dv.y) && isfinite(nv.x) && isfinite(nv.y))) dsc->p_bad = 1;
  } else {  // an odd last cell
    T n0, n1, d0, d1;
    pupdate_pair<T>(pp[n], 0., pnew[n], TC(0.), n0, n1, d0, d1, first, normalise, norm, norm_old);
    pold[n] = d0;
    pnew[n] = n0;
    if (!(isfinite(d0) && isfinite(n0))) dsc->p_bad = 1;
  }
}

// ---- reductions ------------------------------------------------------------
// sum over the interior: warp w of the grid takes rows (j,k) w, w + W, ...
// (W warps), its lanes the i of a row, eight loads in flight per lane
// before the adds (fixed grid, fixed order)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_sum_interior(Params p, const T* __restrict__ a,
                                                              double* __restrict__ partial) {
  pdl_wait();
  const int rows = p.jmax * p.kmax;
  const int W = (int)((gridDim.x * kRedThreads) >> 5);
  const int lane = threadIdx.x & 31;
  double acc[8] = {0., 0., 0., 0., 0., 0., 0., 0.};
  for (int r = (int)((blockIdx.x * kRedThreads + threadIdx.x) >> 5); r < rows; r += W) {
    const T* __restrict__ row = a + idxC(p, 1, 1 + r % p.jmax, 1 + r / p.jmax);
    for (int i0 = lane; i0 < p.imax; i0 += 256) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = (i0 + 32 * u < p.imax) ? (double)row[i0 + 32 * u] : 0.;
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] += v[u];
    }
  }
  const double s = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
  double b = block_sum<double, kRedThreads>(s);
  if (threadIdx.x == 0) partial[blockIdx.x] = b;
}
__global__ void __launch_bounds__(kRedThreads) k_stream_final(Params p, const double* __restrict__ partial, int nblk,
                                                              DevScalars* __restrict__ dsc) {
  pdl_wait();
  double s = 0.;
  for (int b = threadIdx.x; b < nblk; b += kRedThreads) s += partial[b];
  s = block_sum<double, kRedThreads>(s);
  if (threadIdx.x == 0) dsc->v_bulk = s / (double)((long long)p.imax * p.jmax * p.kmax);
}

// chkdiv: sum of div and max|div| with its first column-major location
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_chkdiv(Params p, const T* __restrict__ u, const T* __restrict__ v,
                                                        const T* __restrict__ w,
                                                        double* __restrict__ part_sum, double* __restrict__ part_max,
                                                        long long* __restrict__ part_loc) {
  pdl_wait();
  double s = 0., m = 0.;
  long long loc = -1;
  for (int q = blockIdx.x * kRedThreads + threadIdx.x; q < (int)p.nI; q += gridDim.x * kRedThreads) {
    int i, j, k;
    decodeI(p, q, i, j, k);
    const long long c = idxC(p, i, j, k);
    const double wc = w[c], wm = w[c - (long long)p.nCx * p.nCy], vc = v[c], vm = v[c - p.nCx];
    const double uc = u[c], um = u[c - 1];
    double div = ((wc - wm) * p.dzi + (vc - vm) * p.dyi) + (uc - um) * p.dxi;
    s += div;
    div = fabs(div);
    if (div > m) { m = div; loc = (long long)q; }
  }
  __shared__ double sm[kRedThreads];
  __shared__ long long sl[kRedThreads];
  double b = block_sum<double, kRedThreads>(s);
  sm[threadIdx.x] = m;
  sl[threadIdx.x] = loc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double bm = 0.;
    long long bl = -1;
    for (int t = 0; t < kRedThreads; ++t) {
      if (sm[t] > bm || (sm[t] == bm && sm[t] > 0. && sl[t] < bl)) { bm = sm[t]; bl = sl[t]; }
    }
    part_sum[blockIdx.x] = b;
    part_max[blockIdx.x] = bm;
    part_loc[blockIdx.x] = bl;
  }
}
__global__ void k_chkdiv_final(const double* __restrict__ part_sum, const double* __restrict__ part_max,
                               const long long* __restrict__ part_loc, int nblk, DevScalars* __restrict__ dsc) {
  pdl_wait();
  if (threadIdx.x) return;
  double s = 0., m = 0.;
  long long l = -1;
  for (int b = 0; b < nblk; ++b) {
    s += part_sum[b];
    if (part_max[b] > m || (part_max[b] == m && part_max[b] > 0. && part_loc[b] < l)) { m = part_max[b]; l = part_loc[b]; }
  }
  dsc->divtot = s;
  dsc->divmax = m;
  dsc->divloc = l;
}

// chkdt maxima (chkdt.f90:31-52) and max_vel_at_center (misc.f90:619-633)
template <typename T>
__global__ void __launch_bounds__(NT) k_chkdt(Params p, const T* __restrict__ u, const T* __restrict__ v,
                                              const T* __restrict__ w, DevScalars* __restrict__ dsc) {
  pdl_wait();
  double a = 0., b = 0., c = 0.;
  int i, j, k;
  const I3 hi = cC1(p);
  if (cell3(kI0, hi.v, i, j, k)) {
    const long long cc = idxC(p, i, j, k);
    a = fabs(((double)u[cc] + (double)u[cc - 1]) / 2.);
    b = fabs(((double)v[cc] + (double)v[cc - p.nCx]) / 2.);
    c = fabs(((double)w[cc] + (double)w[cc - (long long)p.nCx * p.nCy]) / 2.);
  }
  a = block_max<double, NT>(a);
  b = block_max<double, NT>(b);
  c = block_max<double, NT>(c);
  if (flat_tid() == 0) {
    atomic_max_nonneg(&dsc->umax, a);
    atomic_max_nonneg(&dsc->vmax, b);
    atomic_max_nonneg(&dsc->wmax, c);
  }
}
template <typename T>
__global__ void __launch_bounds__(NT) k_maxvel(Params p, const T* __restrict__ ucc, const T* __restrict__ vcc,
                                               const T* __restrict__ wcc, DevScalars* __restrict__ dsc) {
  pdl_wait();
  const long long q = blockIdx.x * (long long)NT + threadIdx.x;
  double m = 0.;
  if (q < p.nI) {
    const double a = ucc[q], b = vcc[q], cc = wcc[q];
    m = sqrt((a * a + b * b) + cc * cc);
  }
  m = block_max<double, NT>(m);
  if (threadIdx.x == 0) atomic_max_nonneg(&dsc->velmax, m);
}

MomArgs mom_args(Ctx& c) {
  MomArgs a;
  a.u = c.u; a.v = c.v; a.w = c.w; a.miu = c.miu;
  a.rho_u = c.rho_u; a.rho_v = c.rho_v; a.rho_w = c.rho_w;
  a.duold = c.duold[c.hist]; a.dvold = c.dvold[c.hist]; a.dwold = c.dwold[c.hist];
  a.pnew = c.pnew; a.pold = c.pold;
  a.px = c.px; a.py = c.py; a.pz = c.pz; a.pxold = c.pxold; a.pyold = c.pyold; a.pzold = c.pzold;
  a.rho_avr = &c.dsc->rho_avr;
  a.near = nullptr; a.p_bad = &c.dsc->p_bad;
  return a;
}
CorrArgs corr_args(Ctx& c) {
  CorrArgs a;
  a.dudt = c.dudt; a.dvdt = c.dvdt; a.dwdt = c.dwdt; a.p = c.p; a.px = c.px; a.py = c.py; a.pz = c.pz;
  a.u = c.u; a.v = c.v; a.w = c.w; a.ucc = c.ucc; a.vcc = c.vcc; a.wcc = c.wcc; a.dsc = c.dsc;
  a.seg = c.seg_jmp[0];
  return a;
}

#undef TC
}  // namespace

// ================================================================ launchers
template <typename T>
T* fp(double* q) { return reinterpret_cast<T*>(q); }

void launch_ab2(Ctx& c) {
  // the segment maps hold unless a caller wrote the fields they describe
  const bool far = (c.P.f32 || c.ab2_ring) && !c.mat_dirty && !c.jmp_dirty[0] && !c.jmp_dirty[1];
  MomArgs a = mom_args(c);
  if (far) {
    Scope sc_(c.prof, c.s, "ab2_near", 1);
    cudaMemsetAsync(c.ab2_near, 0, (size_t)seg_row(c.P) * ((c.P.jmax + kAb2Y - 1) / kAb2Y) * c.P.nCz, c.s);
    pdl(k_ab2_near, nblocks((seg_count(c.P) + 3) / 4), NT, 0, c.s)(c.P, c.seg_mat[c.mat_cur], c.seg_jmp[0],
                                                                  c.seg_jmp[1], c.ab2_near);
    a.near = c.ab2_near;
    if (c.p_dirty) cudaMemsetAsync(&c.dsc->p_bad, 1, sizeof(int), c.s);  // unknown: nonzero
  }
  const int o = c.hist ^ 1;
  {
    Scope sc_(c.prof, c.s, "ab2", 1);
    if (c.P.f32) {
      ab2_launch_f32(c, a, o);  // k_ab2_f32.cu
    } else if (!ab2_tma_launch(c, a, o)) {  // k_ab2_tma.cu when chosen, else the ring
      ab2_launch<double>(c, a, o);
    }
  }
  launch_ywalls_uvw(c, c.dudt, c.dvdt, c.dwdt);  // the y walls of bounduvw(dudt,dvdt,dwdt)
  c.hist = o;
}
void launch_mom_main(Ctx& c, double* du, double* dv, double* dw) {
  Scope sc_(c.prof, c.s, "mom_main", 1);
  MomArgs a = mom_args(c);
  if (c.P.f32)
    pdl(k_mom_main<float>, gridI(c.P), kBlock, 0, c.s)(c.P, a, fp<float>(du), fp<float>(dv), fp<float>(dw));
  else
    pdl(k_mom_main<double>, gridI(c.P), kBlock, 0, c.s)(c.P, a, du, dv, dw);
}
void launch_fillps(Ctx& c, int add_pjump) {
  Scope sc_(c.prof, c.s, "fillps", 1);
  if (c.P.f32)
    pdl(k_fillps<float>, gridI(c.P), kBlock, 0, c.s)(c.P, fp<float>(c.dudt), fp<float>(c.dvdt), fp<float>(c.dwdt),
                                                     c.pjump, add_pjump, c.p);
  else
    pdl(k_fillps<double>, gridI(c.P), kBlock, 0, c.s)(c.P, c.dudt, c.dvdt, c.dwdt, c.pjump, add_pjump, c.p);
}
void launch_add_pjump(Ctx& c) {
  Scope sc_(c.prof, c.s, "add_pjump", 1); pdl(k_add, nblocks(c.P.nC), NT, 0, c.s)(c.P, c.p, c.pjump); }
void launch_correc(Ctx& c, int fused_bc) {
  Scope sc_(c.prof, c.s, "correc", 1);
  CorrArgs a = corr_args(c);
  // one thread per shape-C cell (ICLS_CORREC=shapec)
  if (fused_bc && c.correc_shapec) {
    if (c.P.f32) pdl(k_correc_fused<float>, gridC(c.P), kBlock, 0, c.s)(c.P, a);
    else pdl(k_correc_fused<double>, gridC(c.P), kBlock, 0, c.s)(c.P, a);
    return;
  }
  // one thread per interior column, which in the fused form writes the halo
  // and wall images too; several rows per thread while the blocks still fill
  // every SM
  dim3 g = gridI(c.P);
  int rows = c.P.f32 ? kCorRows<float> : kCorRows<double>;
  while (rows > 1 && (long long)g.x * g.y * ((g.z + rows - 1) / rows) < 8 * 148) rows /= 2;
  g.z = (g.z + rows - 1) / rows;
  auto go = [&](auto kernel) { pdl(kernel, g, kBlock, 0, c.s)(c.P, a, rows); };
  const bool rp = c.P.rho0_pow2 != 0;
  if (c.P.f32) {
    if (fused_bc) rp ? go(k_correc_own<float, 1>) : go(k_correc_own<float, 0>);
    else rp ? go(k_correc_interior<float, 1>) : go(k_correc_interior<float, 0>);
  } else {
    if (fused_bc) rp ? go(k_correc_own<double, 1>) : go(k_correc_own<double, 0>);
    else rp ? go(k_correc_interior<double, 1>) : go(k_correc_interior<double, 0>);
  }
}
void launch_bounduvw(Ctx& c, double* u, double* v, double* w) {
  const int halo = halo_cells(c.P);
  const unsigned g = nblocks(halo + halo_plane_cells(c.P));
  {
    Scope sc_(c.prof, c.s, "bounduvw", 1);
    if (c.P.f32) pdl(k_bounduvw<float>, g, NT, 0, c.s)(c.P, fp<float>(u), fp<float>(v), fp<float>(w), halo);
    else pdl(k_bounduvw<double>, g, NT, 0, c.s)(c.P, u, v, w, halo);
  }
  launch_ywalls_uvw(c, u, v, w);
}
inline dim3 grid_ik(const Params& p) { return dim3((unsigned)((p.imax + NT - 1) / NT), (unsigned)p.kmax, 1); }
void launch_boundp(Ctx& c, double* pp, bool tfield) {
  const int halo = halo_cells(c.P);
  {
    Scope sc_(c.prof, c.s, "boundp", 1);
    if (tfield && c.P.f32) pdl(k_boundp<float>, nblocks(halo), NT, 0, c.s)(c.P, fp<float>(pp), halo);
    else pdl(k_boundp<double>, nblocks(halo), NT, 0, c.s)(c.P, pp, halo);
  }
  launch_ywalls_p(c, pp, tfield);
}
void launch_ywalls_uvw(Ctx& c, double* u, double* v, double* w) {
  if (c.P.bcy == ICLS_BCY_PERIODIC) return;
  Scope sc_(c.prof, c.s, "ywalls", 1);
  if (c.P.f32)
    pdl(k_ywalls_uvw<float>, grid_ik(c.P), NT, 0, c.s)(c.P, fp<float>(u), fp<float>(v), fp<float>(w), c.vin);
  else
    pdl(k_ywalls_uvw<double>, grid_ik(c.P), NT, 0, c.s)(c.P, u, v, w, c.vin);
}
void launch_ywalls_p(Ctx& c, double* pp, bool tfield) {
  if (c.P.bcy == ICLS_BCY_PERIODIC) return;
  Scope sc_(c.prof, c.s, "ywalls", 1);
  if (tfield && c.P.f32) pdl(k_ywalls_p<float>, grid_ik(c.P), NT, 0, c.s)(c.P, fp<float>(pp));
  else pdl(k_ywalls_p<double>, grid_ik(c.P), NT, 0, c.s)(c.P, pp);
}
void launch_gather_plane_x(Ctx& c, const double* d, bool f32, long long nx, long long ny, long long ioff, int n1,
                           int n2, double* dst) {
  const unsigned g = nblocks((long long)n1 * n2);
  if (f32) pdl(k_gather_plane_x<float>, g, NT, 0, c.s)(reinterpret_cast<const float*>(d), nx, nx * ny, ioff, n1, n2, dst);
  else pdl(k_gather_plane_x<double>, g, NT, 0, c.s)(d, nx, nx * ny, ioff, n1, n2, dst);
}
void launch_nan_probe(Ctx& c) {
  Scope sc_(c.prof, c.s, "nan_probe", 1);
  if (c.P.f32) pdl(k_nan_probe<float>, 1, 1, 0, c.s)(c.P, fp<float>(c.v), c.dsc);
  else pdl(k_nan_probe<double>, 1, 1, 0, c.s)(c.P, c.v, c.dsc);
}
void launch_average_vel(Ctx& c) {
  Scope sc_(c.prof, c.s, "average_vel", 1);
  if (c.P.f32)
    pdl(k_average_vel<float>, gridI(c.P), kBlock, 0, c.s)(c.P, fp<float>(c.u), fp<float>(c.v), fp<float>(c.w),
                                                          fp<float>(c.ucc), fp<float>(c.vcc), fp<float>(c.wcc));
  else
    pdl(k_average_vel<double>, gridI(c.P), kBlock, 0, c.s)(c.P, c.u, c.v, c.w, c.ucc, c.vcc, c.wcc);
}
void launch_pressure_update(Ctx& c, int first) {
  Scope sc_(c.prof, c.s, "pressure_update", 2);
  // the plane-1 normalisation runs for BC_in_y Periodic and Walls only
  // (main.f90:169-185); otherwise pold = pnew, pnew = p
  const int norm = c.P.bcy == ICLS_BCY_PERIODIC || c.P.bcy == ICLS_BCY_WALLS;
  c.p_dirty = false;
  if (!norm) cudaMemsetAsync(&c.dsc->p_bad, 0, sizeof(int), c.s);  // else k_plane_norm
  if (norm) pdl(k_plane_norm, 1, kNormThreads, 0, c.s)(c.P, c.p, c.dsc);
  if (c.P.f32)
    pdl(k_pupdate<float>, nblocks((c.P.nC + 1) / 2), NT, 0, c.s)(c.P, c.p, fp<float>(c.pnew), fp<float>(c.pold), first, norm,
                                                       c.dsc);
  else
    pdl(k_pupdate<double>, nblocks((c.P.nC + 1) / 2), NT, 0, c.s)(c.P, c.p, c.pnew, c.pold, first, norm, c.dsc);
}
void launch_stream_vel(Ctx& c) {
  Scope sc_(c.prof, c.s, "stream_vel", 2);
  if (c.P.f32) pdl(k_sum_interior<float>, kRedBlocks, kRedThreads, 0, c.s)(c.P, fp<float>(c.v), c.partials);
  else pdl(k_sum_interior<double>, kRedBlocks, kRedThreads, 0, c.s)(c.P, c.v, c.partials);
  pdl(k_stream_final, 1, kRedThreads, 0, c.s)(c.P, c.partials, kRedBlocks, c.dsc);
}
void launch_chkdiv(Ctx& c) {
  Scope sc_(c.prof, c.s, "chkdiv", 2);
  double* ps = c.partials;
  double* pm = c.partials + kRedBlocks;
  if (c.P.f32)
    pdl(k_chkdiv<float>, kRedBlocks, kRedThreads, 0, c.s)(c.P, fp<float>(c.u), fp<float>(c.v), fp<float>(c.w), ps, pm,
                                                          c.lpartials);
  else
    pdl(k_chkdiv<double>, kRedBlocks, kRedThreads, 0, c.s)(c.P, c.u, c.v, c.w, ps, pm, c.lpartials);
  pdl(k_chkdiv_final, 1, 32, 0, c.s)(ps, pm, c.lpartials, kRedBlocks, c.dsc);
}
void launch_chkdt(Ctx& c) {
  Scope sc_(c.prof, c.s, "chkdt", 1);
  cudaMemsetAsync(&c.dsc->umax, 0, 3 * sizeof(double), c.s);
  if (c.P.f32) pdl(k_chkdt<float>, gridC(c.P), kBlock, 0, c.s)(c.P, fp<float>(c.u), fp<float>(c.v), fp<float>(c.w), c.dsc);
  else pdl(k_chkdt<double>, gridC(c.P), kBlock, 0, c.s)(c.P, c.u, c.v, c.w, c.dsc);
}
void launch_maxvel(Ctx& c) {
  Scope sc_(c.prof, c.s, "maxvel", 1);
  cudaMemsetAsync(&c.dsc->velmax, 0, sizeof(double), c.s);
  if (c.P.f32)
    pdl(k_maxvel<float>, nblocks(c.P.nI), NT, 0, c.s)(c.P, fp<float>(c.ucc), fp<float>(c.vcc), fp<float>(c.wcc), c.dsc);
  else
    pdl(k_maxvel<double>, nblocks(c.P.nI), NT, 0, c.s)(c.P, c.ucc, c.vcc, c.wcc, c.dsc);
}

}  // namespace icls
