// dynamics.cu -- the acoustic RK short step prog_wrtv_rk and its glue on the
// device (omodel/prog_wrtv_rk.f90:36-488, omodel/timestep.f90:430-612).
//
// Kernel per reference routine, each over the reference's loop table:
//   k_damp_first, k_damp_lap  divh_damp and vort_damp          (vort_div_damp.f90:1-445):
//                           the two first passes in one launch, the two
//                           Laplacians of a step in one
//   k_vtend                 the V points' set-up and Rayleigh terms with both dampings
//                           (prog_wrtv_rk.f90:166-303)
//   k_setup_w               the W columns' set-up (same lines); on the lean path
//                           k_wrt_begs forms it on the first stage
//   k_grad_upv4             fluxes_wrtv for thil, vxe, vye, vze (:950-1129), the four
//                           fields of one stage in one launch: the gradients
//                           and the V-face values in one pass over the W
//                           cells, with vmca of the stage and its share of
//                           vmasc (:320-368); on the last stage the fields
//                           with ithil_monot / iwind_monot > 0 take
//                           dynamics_monot.cu's values
//   k_vmca                  vmca / vmasc on a rank with a halo, or beside border columns
//   k_upw4                  the vertical face values where the column kernel does not
//                           form them (eddy, Rayleigh or flux-corrected terms)
//   k_wrt_begs              prog_wrt_begs (:494-884): lanes over levels for the explicit
//                           terms and for the tridiagonal solve (tridiffo,
//                           tridiag_lib.f90:10-36, by parallel cyclic
//                           reduction), one or two warps per column
//   k_prog_v                prog_v_begs (:888-946)
//   k_vel_t3d               vel_t3d_hex (vel_t3d.f90:39-108)
// With eddy diffusion registered, dynamics_eddy.cu's k_eddy_w follows
// k_setup_w (the vertical and horizontal eddy terms of :214-251).
// Precision as declared by OLAM: rho, press and the implicit weights are
// double; every other field is float.  Device level kd = Fortran k - 1.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "recip.cuh"
#include "transport_kernels.cuh"

namespace olamgpu {

struct DynK {
  int mza, mwa, mva, mma;
  const int* __restrict__ npoly;
  // read by no kernel here: without these three the compiler spills 28 bytes
  // of the column kernel's registers instead of 4 (373 us a stage against 326
  // at NXP=100, 60 levels)
  const int* __restrict__ w_nb;
  const int* __restrict__ w_ev;
  const float* __restrict__ w_dirv;
  const int* __restrict__ v_iw;
  const int* __restrict__ v_im;
  const int* __restrict__ m_iv;
  const int* __restrict__ m_im;
  const int* __restrict__ lpw;
  const int* __restrict__ lpv;
  const int* __restrict__ lpm;
  const float* __restrict__ volti;
  const float* __restrict__ a_w;
  const int4* __restrict__ edge;    // EDGE_W words per edge, 7 edges per W column
  // flat: lpw = lpv = 2 everywhere (device level 1), no table read needed;
  // off_*: the loop table is the contiguous run off, off + 1, ... (a
  // global domain), no table read needed; -1 otherwise
  int flat, off_w, off_vp, off_va;
};

// lowest device level of a W / V point; a loop table's j-th entry
#define LPW(i) (g.flat ? 1 : g.lpw[i])
#define LPV(i) (g.flat ? 1 : g.lpv[i])
#define WTAB(j) (g.off_w >= 0 ? g.off_w + (j) : prog[j])
#define VPTAB(j) (g.off_vp >= 0 ? g.off_vp + (j) : vprog[j])
#define VATAB(j) (g.off_va >= 0 ? g.off_va + (j) : vadj[j])

static DynK dynk(const DevGrid& d) {
  DynK k;
  k.mza = d.mza; k.mwa = d.mwa; k.mva = d.mva; k.mma = d.mma;
  k.npoly = d.npoly.p; k.w_nb = d.w_nb.p; k.w_ev = d.w_ev.p; k.w_dirv = d.w_dirv.p;
  k.v_iw = d.v_iw.p; k.v_im = d.v_im.p; k.m_iv = d.m_iv.p; k.m_im = d.m_im.p;
  k.lpw = d.lpw.p; k.lpv = d.lpv.p; k.lpm = d.lpm.p; k.volti = d.volti.p; k.a_w = d.a_w.p;
  k.edge = reinterpret_cast<const int4*>(d.edge.p);
  k.flat = ctx().tp.flat ? 1 : 0;
  k.off_w = d.off_wprog; k.off_vp = d.off_vprog; k.off_va = d.off_vwadj;
  return k;
}

// The edge records of the column 2048 on, which a later wave of warps runs,
// into L2 now: they are the first thing a warp waits for (NXP=100, 60 levels:
// faces 222 -> 209 us, velocities 80 -> 74; 1024 or 4096 columns the same).
// The column kernel and the dampings gain nothing by it.
#define EDGES_AHEAD 2048
__device__ __forceinline__ void edges_ahead(const DynK& g, const int4* E, int iw) {
  const int lane = threadIdx.x & 31;
  if (lane < 2 && iw + EDGES_AHEAD < g.mwa)
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(E + (size_t)EDGES_AHEAD * (7 * EDGE_W / 4) + 7 * lane));
}

// thread per (table entry j, level kd); n * mza < 2^31 (dyn_setup checks)
#define PK(j, kd, n)                                               \
  const unsigned i_ = blockIdx.x * blockDim.x + threadIdx.x;       \
  if (i_ >= (unsigned)(n) * (unsigned)g.mza) return;               \
  const int j = (int)(i_ / (unsigned)g.mza), kd = (int)(i_ - (unsigned)j * (unsigned)g.mza);

// ---- column set-up (prog_wrtv_rk.f90:166-253) --------------------------------
struct SetupW {
  const double* rho; const float* thil; const float* wmc;
  const float* thilt; const float* vmxet; const float* vmyet; const float* vmzet;
  const double* volt;
  double* rho0; double* rth0; float* wmc0;
  float* sh_th; float* sh_vx; float* sh_vy; float* sh_vz;
  const float* rayf_cof; const float* dn01d; const float* th01d; int krayf_bot;
};

__global__ void k_setup_w(DynK g, const int* __restrict__ prog, int nprog, SetupW a) {
  PK(j, kd, nprog);
  const int iw = WTAB(j);
  if (kd < LPW(iw)) return;
  const size_t x = (size_t)iw * g.mza + kd;
  const float v4 = (float)a.volt[x];
  a.rth0[x] = (double)a.thil[x] * a.rho[x];
  a.rho0[x] = a.rho[x];
  a.wmc0[x] = a.wmc[x];
  float th = a.thilt[x] * v4;
  if (a.rayf_cof && kd >= a.krayf_bot - 1)
    th = th + a.rayf_cof[kd] * a.dn01d[kd] * (a.th01d[kd] - a.thil[x]) * v4;
  a.sh_th[x] = th;
  a.sh_vx[x] = a.vmxet[x] * v4;
  a.sh_vy[x] = a.vmyet[x] * v4;
  a.sh_vz[x] = a.vmzet[x] * v4;
}

// ---- divh_damp ----------------------------------------------------------------
__global__ void k_div_fdivh(DynK g, const int* __restrict__ vprog, int nv, const float* __restrict__ arw0,
                            const float* __restrict__ dniv, const float* __restrict__ zfacit,
                            const float* __restrict__ dzit, const double* __restrict__ volt, double facth,
                            int level, float fact2, float* __restrict__ fdivh) {
  PK(j, kd, nv);
  const int iv = VPTAB(j);
  if (kd < LPV(iv)) return;
  const int iw1 = g.v_iw[iv * 2], iw2 = g.v_iw[iv * 2 + 1];
  const double vmin = fmin(volt[(size_t)iw1 * g.mza + kd], volt[(size_t)iw2 * g.mza + kd]);
  double v;
  if (level > 1) {
    const float amin = fminf(arw0[iw1], arw0[iw2]);
    float pw = 1.f;
    for (int i = 0; i < level - 1; ++i) pw = pw * amin;
    const double factb = facth * (double)pw;
    v = factb * (double)dniv[iv] * (double)zfacit[kd] * (double)dzit[kd] * vmin * 1.0;
  } else {
    v = (double)fact2 * (double)dniv[iv] * (double)zfacit[kd] * (double)dzit[kd] * vmin;
  }
  fdivh[(size_t)iv * g.mza + kd] = (float)v;
}

// ---- vort_damp ----------------------------------------------------------------
__global__ void k_vort_first_m(DynK g, const int* __restrict__ mprog, int nm, const float* __restrict__ dnv,
                               const float* __restrict__ arm0, float* __restrict__ vfact) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nm) return;
  const int im = mprog[j];
  for (int jv = 0; jv < 3; ++jv) {
    const int iv = g.m_iv[im * 3 + jv];
    const float v = dnv[iv] / arm0[im];
    vfact[im * 3 + jv] = (g.v_im[iv * 2 + 1] == im) ? v : -v;
  }
}

__global__ void k_vort_first_v(DynK g, const int* __restrict__ vprog, int nv, const float* __restrict__ dniu,
                               const float* __restrict__ arm0, float dtm_f, float fact, int level,
                               float* __restrict__ fvorth, float* __restrict__ fvortl) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nv) return;
  const int iv = VPTAB(j);
  const int im1 = g.v_im[iv * 2], im2 = g.v_im[iv * 2 + 1];
  const float a = -fact * fminf(arm0[im1], arm0[im2]);
  float ph = 1.f, pl = 1.f;
  for (int i = 0; i < level; ++i) ph = ph * a;
  for (int i = 0; i < level - 1; ++i) pl = pl * a;
  fvorth[iv] = 0.50f * dniu[iv] / dtm_f * ph;
  fvortl[iv] = (level > 2) ? 0.50f * dniu[iv] / dtm_f * pl : 0.f;
}

// The per-point kernels below give a warp to a point and R = 1, 2 or 4 levels
// (mza up to 32, 64, 128) to a lane: the point's table entries are one uniform
// read a warp, and every load of the R levels is issued before any is used.
// A thread per (point, level) over the flat range, its neighbours read in
// turn, left each warp waiting on one or two loads at a time; with one level
// a lane the table reads weigh as much as the data (NXP=100, 60 levels, one
// level against two: first planes 174 / 135 us, a Laplacian step 124 / 87,
// velocities 123 / 78).
#define WARP_POINT(n, first)                                                  \
  const int lane = threadIdx.x & 31;                                          \
  const unsigned w_ = (blockIdx.x - (first)) * 8u + (threadIdx.x >> 5);       \
  if (w_ >= (unsigned)(n)) return;

struct DampArgs {
  const int* wprog; int nw;           // divergence of the W columns
  const int* mprog; int nm, off_m;    // vorticity at the M points (off_m: the table is off_m, off_m + 1, ..., or -1)
  unsigned mblock;                    // first block of the M part
  const float* arv; const float* vmc; const float* vc;
  const float* xx_yy; const float* xx_yy_m; const float* vfact;
  const float* wsrc; float* wdst;     // planes of the Laplacian step
  const float* msrc; float* mdst;
};

// First planes of divh_damp and vort_damp (vort_div_damp.f90:126-148,
// 296-330), the W columns and the M points side by side in one launch.
// The saved div2d is not cleared: plane 1 accumulates onto what the previous
// call left there, as the Fortran does (vort_div_damp.f90:136-148).
template <int R>
__global__ void __launch_bounds__(256) k_damp_first(DynK g, DampArgs A) {
  const int mza = g.mza;
  if (blockIdx.x < A.mblock) {
    WARP_POINT(A.nw, 0u);
    const int* prog = A.wprog;
    const int iw = WTAB((int)w_), np = g.npoly[iw], kb = LPW(iw);
    const size_t cb = (size_t)iw * mza;
    const int4* E = g.edge + (size_t)iw * (7 * EDGE_W / 4);
    int4 e[6];
#pragma unroll
    for (int n = 0; n < 6; ++n) e[n] = __ldg(E + 2 * n);
    grid_wait();
    float d[R], vt[R], ar[R][6], vm[R][6];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      d[r] = vt[r] = 0.f;
      if (kd < mza) { d[r] = A.wdst[cb + kd]; vt[r] = g.volti[cb + kd]; }
#pragma unroll
      for (int n = 0; n < 6; ++n) {
        ar[r][n] = vm[r][n] = 0.f;
        if (kd < mza && kd >= e[n].z) {
          const size_t xv = (size_t)(e[n].y & 0x7fffffff) * mza + kd;
          ar[r][n] = A.arv[xv];
          vm[r][n] = A.vmc[xv];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      if (kd >= mza) continue;
#pragma unroll
      for (int n = 0; n < 6; ++n) d[r] = d[r] - ar[r][n] * __int_as_float(e[n].w) * vm[r][n];
      if (np > 6) {
        const int4 q = __ldg(E + 12);
        const size_t xv = (size_t)(q.y & 0x7fffffff) * mza + kd;
        if (kd >= q.z) d[r] = d[r] - A.arv[xv] * __int_as_float(q.w) * A.vmc[xv];
      }
      if (kd >= kb) d[r] = d[r] * vt[r];
      A.wdst[cb + kd] = d[r];
    }
  } else {
    WARP_POINT(A.nm, A.mblock);
    const int im = A.off_m >= 0 ? A.off_m + (int)w_ : A.mprog[w_];
    int iv[3], lv[3];
    float f[3], x[R][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) { iv[q] = g.m_iv[im * 3 + q]; f[q] = A.vfact[im * 3 + q]; }
#pragma unroll
    for (int q = 0; q < 3; ++q) lv[q] = LPV(iv[q]);
    grid_wait();
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int kd = lane + 32 * r;
        x[r][q] = 0.f;
        if (kd < mza && kd >= lv[q]) x[r][q] = A.vc[(size_t)iv[q] * mza + kd];
      }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      float v = 0.f;
#pragma unroll
      for (int q = 0; q < 3; ++q) v = v + x[r][q] * f[q];
      if (kd < mza) A.mdst[(size_t)im * mza + kd] = v;
    }
  }
}

// laplacian2d (grad_lib.f90:494-524) of the divergence plane and laplacian_m
// (:531-559) of the vorticity plane
template <int R>
__global__ void __launch_bounds__(256) k_damp_lap(DynK g, DampArgs A) {
  const int mza = g.mza;
  if (blockIdx.x < A.mblock) {
    WARP_POINT(A.nw, 0u);
    const int* prog = A.wprog;
    const int iw = WTAB((int)w_), np = g.npoly[iw];
    const size_t cb = (size_t)iw * mza;
    const int4* E = g.edge + (size_t)iw * (7 * EDGE_W / 4);
    int4 e[6];
    float c[6];
#pragma unroll
    for (int n = 0; n < 6; ++n) { e[n] = __ldg(E + 2 * n); c[n] = A.xx_yy[iw * 7 + n]; }
    grid_wait();
    float s[R], x[R][6];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      s[r] = kd < mza ? A.wsrc[cb + kd] : 0.f;
#pragma unroll
      for (int n = 0; n < 6; ++n) {
        x[r][n] = 0.f;
        if (kd < mza && kd >= e[n].z) x[r][n] = A.wsrc[(size_t)e[n].x * mza + kd];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      if (kd >= mza) continue;
      float d = 0.f;
#pragma unroll
      for (int n = 0; n < 6; ++n) if (kd >= e[n].z) d = d + (x[r][n] - s[r]) * c[n];
      if (np > 6) {
        const int4 q = __ldg(E + 12);
        if (kd >= q.z) d = d + (A.wsrc[(size_t)q.x * mza + kd] - s[r]) * A.xx_yy[iw * 7 + 6];
      }
      A.wdst[cb + kd] = d;
    }
  } else {
    WARP_POINT(A.nm, A.mblock);
    const int im = A.off_m >= 0 ? A.off_m + (int)w_ : A.mprog[w_];
    const size_t cb = (size_t)im * mza;
    int nb[3], lv[3];
    float c[3], s[R], x[R][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      nb[q] = g.m_im[im * 3 + q];
      c[q] = A.xx_yy_m[im * 3 + q];
      lv[q] = LPV(g.m_iv[im * 3 + q]);
    }
    grid_wait();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      s[r] = kd < mza ? A.msrc[cb + kd] : 0.f;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        x[r][q] = 0.f;
        if (kd < mza && kd >= lv[q]) x[r][q] = A.msrc[(size_t)nb[q] * mza + kd];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kd = lane + 32 * r;
      float d = 0.f;
#pragma unroll
      for (int q = 0; q < 3; ++q) if (kd >= lv[q]) d = d + (x[r][q] - s[r]) * c[q];
      if (kd < mza) A.mdst[cb + kd] = d;
    }
  }
}

// V tendency of the step: the long-step tendency, the Rayleigh term
// (prog_wrtv_rk.f90:289-303) and both dampings (vort_div_damp.f90:208-230,
// 400-445), each left out where its switch is off; with vmc0 the start
// momentum is kept too (prog_wrtv_rk.f90:289)
struct VtendArgs {
  const int* vprog; int nv;
  const float* src; float* dst;       // tendency in and out (may be one array)
  const float* vmc; float* vmc0;      // NULL vmc0: not kept
  const float* rayf_cof; const float* vc03d; const float* vc; int krayf_bot;
  const double* rho;
  const float* fdivh; const float* dh;             // NULL dh: no divergence damping
  const float* fvorth; const float* fvortl;        // NULL fvorth: no vorticity damping
  const float* vl; const float* vh;
  int lpm;                            // the second-order plane below the M points' floors (level 3)
};

// A warp to 32 levels of a V point: here two levels a lane cost more in
// registers (half the warps) than they save in table reads (203 us against
// 160 at NXP=100, 60 levels).
__global__ void __launch_bounds__(256) k_vtend(DynK g, VtendArgs A) {
  const int mza = g.mza;
  const unsigned nch = ((unsigned)mza + 31u) / 32u, q = blockIdx.x * 8u + (threadIdx.x >> 5), j = q / nch;
  if (j >= (unsigned)A.nv) return;
  const int kd = (int)((q - j * nch) * 32u + (threadIdx.x & 31u));
  if (kd >= mza) return;
  const int* vprog = A.vprog;
  const int iv = VPTAB((int)j), kv = LPV(iv);
  const int2 iw = *reinterpret_cast<const int2*>(g.v_iw + iv * 2), im = *reinterpret_cast<const int2*>(g.v_im + iv * 2);
  const size_t x = (size_t)iv * mza + kd;
  grid_wait();
  const bool open = kd >= kv, div = A.dh && open, vor = A.fvorth && open;
  const bool ray = A.rayf_cof && kd >= A.krayf_bot - 1;
  float t = A.src[x], v0 = 0.f, fd = 0.f, d1 = 0.f, d2 = 0.f, v1 = 0.f, v2 = 0.f, fv = 0.f;
  double r1 = 0.0, r2 = 0.0;
  if (A.vmc0) v0 = A.vmc[x];
  if (div) {
    fd = A.fdivh[x];
    d1 = A.dh[(size_t)iw.x * mza + kd];
    d2 = A.dh[(size_t)iw.y * mza + kd];
  }
  if (vor || ray) {
    r1 = A.rho[(size_t)iw.x * mza + kd];
    r2 = A.rho[(size_t)iw.y * mza + kd];
  }
  if (vor) {
    // below ka the level-3 damping takes the second-order plane
    const int ka = A.lpm ? max(g.lpm[im.x], g.lpm[im.y]) : kv;
    const float* p = kd < ka ? A.vl : A.vh;
    fv = kd < ka ? A.fvortl[iv] : A.fvorth[iv];
    v1 = p[(size_t)im.x * mza + kd];
    v2 = p[(size_t)im.y * mza + kd];
  }
  if (ray) {
    const double w = (double)(A.rayf_cof[kd] * 0.5f) * (r1 + r2) * (double)(A.vc03d[x] - A.vc[x]);
    t = (float)((double)t + w);
  }
  if (div) t = t + fd * (d2 - d1);
  if (vor) t = t + fv * (v2 - v1) * (float)(r1 + r2);
  A.dst[x] = t;
  if (A.vmc0) A.vmc0[x] = v0;
}

// ---- stage kernels ----------------------------------------------------------------
__global__ void k_vmca(DynK g, const int* __restrict__ vadj, int nv, const float* __restrict__ vmc,
                       const float* __restrict__ arv, float* __restrict__ vmca, float* __restrict__ vmasc,
                       int last) {
  PK(j, kd, nv);
  const int iv = VATAB(j);
  if (kd < LPV(iv)) return;
  const size_t x = (size_t)iv * g.mza + kd;
  const float v = vmc[x] * arv[x];
  vmca[x] = v;
  if (last) vmasc[x] = vmasc[x] + v;
}

struct Four { const float* f[4]; };

struct VSide { const float* dxps; const float* dyps; const float* xx0_v; const float* xy0_v; const float* yy0_v; };

// The horizontal face values of fluxes_wrtv (prog_wrtv_rk.f90:973-1075) in
// one pass over the W cells: grad_t2d (ORD 2) or grad_t2d_quadratic with
// bounded=.false. (ORD 3) of the fields in gmask, kept in registers, then
// scalar_v_column for the faces this cell is upwind of -- side 1 of the
// face unless vmc < 0 -- each face being written by exactly one of its two
// cells: S(k,iw) + dxps dS/dx + dyps dS/dy (+ the quadratic terms at ORD 3)
// for the fields in gmask, S(k,iw) alone for those in pmask.  No gradient
// planes go through memory.  The four values of a face and level are one
// 16-byte element of upv.  With vmca the cell also writes the mass flux
// vmc arv of its faces, and with vmasc adds it there (the last stage).
// A warp per column and 32 levels; the neighbours' values of all four fields
// are loaded before any is used.
struct FaceFlux { const float* arv; float* vmca; float* vmasc; };

// ALL: gmask holds the four fields.  Three edges a batch keep it at 64
// registers, 32 warps an SM: six at a time took 85 registers and 16 warps
// (316 us at NXP=100, 60 levels, against 208).
template <int ORD, bool ALL>
__global__ void __launch_bounds__(256, ORD == 2 ? 4 : 2)
k_grad_upv4(DynK g, const int* __restrict__ prog, int nprog, int nch, Four s, unsigned gmask_,
                            unsigned pmask, const float* __restrict__ xy_hu, VSide c, const float* vmc,
                            float4* upv, FaceFlux ff) {
  constexpr int NPL = ORD == 2 ? 2 : 5;
  const unsigned gmask = ALL ? 0xFu : gmask_;
  const unsigned w_ = blockIdx.x * 8u + (threadIdx.x >> 5);
  const unsigned j = w_ / (unsigned)nch;
  if (j >= (unsigned)nprog) return;
  const int mza = g.mza, kd = (int)((w_ - j * (unsigned)nch) * 32u + (threadIdx.x & 31u));
  if (kd >= mza) return;
  const int iw = WTAB((int)j), np = g.npoly[iw];
  const unsigned x = (unsigned)iw * (unsigned)mza + kd;
  const int4* E = g.edge + (size_t)iw * (7 * EDGE_W / 4);
  edges_ahead(g, E, iw);
  grid_wait();
  float c0[4], a[4][NPL];
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    c0[f] = (((gmask | pmask) >> f) & 1u) ? s.f[f][x] : 0.f;
#pragma unroll
    for (int m = 0; m < NPL; ++m) a[f][m] = 0.f;
  }
  auto gradient = [&](auto cnt, int n0) {
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    float q[N][4];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));
#pragma unroll
    for (int i = 0; i < N; ++i) {
#pragma unroll
      for (int f = 0; f < 4; ++f) q[i][f] = c0[f];
      if (kd >= e[i].z) {
        const unsigned xn = (unsigned)e[i].x * (unsigned)mza + kd;
#pragma unroll
        for (int f = 0; f < 4; ++f) if ((gmask >> f) & 1u) q[i][f] = s.f[f][xn];
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float w[NPL];
      if (ORD == 2) {
        const int4 b = __ldg(E + 2 * (n0 + i) + 1);
        w[0] = __int_as_float(b.x);
        w[1] = __int_as_float(b.y);
      } else {
#pragma unroll
        for (int m = 0; m < NPL; ++m) w[m] = n0 + i < np ? xy_hu[((size_t)iw * 7 + n0 + i) * 5 + m] : 0.f;
      }
      // a closed edge adds nothing: q = c0
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const float d = q[i][f] - c0[f];
#pragma unroll
        for (int m = 0; m < NPL; ++m) a[f][m] = a[f][m] + w[m] * d;
      }
    }
  };
  gradient(std::integral_constant<int, 3>(), 0);
  gradient(std::integral_constant<int, 3>(), 3);
  if (np > 6) gradient(std::integral_constant<int, 1>(), 6);
  auto faces = [&](auto cnt, int n0) {
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    float vm[N], ar[N], vs[N];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      vm[i] = ar[i] = vs[i] = 0.f;
      if (kd >= e[i].z) {
        const unsigned xv = (unsigned)(e[i].y & 0x7fffffff) * (unsigned)mza + kd;
        vm[i] = vmc[xv];
        if (ff.vmca) ar[i] = ff.arv[xv];
        if (ff.vmasc) vs[i] = ff.vmasc[xv];
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int side = e[i].y < 0 ? 1 : 0;
      if (kd < e[i].z || (vm[i] < 0.f) != (side == 1)) continue;   // closed, or the other cell is upwind
      const int iv = e[i].y & 0x7fffffff;
      const unsigned xv = (unsigned)iv * (unsigned)mza + kd;
      if (ff.vmca) {
        const float v = vm[i] * ar[i];
        ff.vmca[xv] = v;
        if (ff.vmasc) ff.vmasc[xv] = vs[i] + v;
      }
      float dx, dy, xx = 0.f, xy = 0.f, yy = 0.f;
      if (ORD == 2) {
        const int4 b = __ldg(E + 2 * (n0 + i) + 1);
        dx = __int_as_float(b.z);
        dy = __int_as_float(b.w);
      } else {
        dx = c.dxps[iv * 2 + side]; dy = c.dyps[iv * 2 + side];
        xx = c.xx0_v[iv * 2 + side]; xy = c.xy0_v[iv * 2 + side]; yy = c.yy0_v[iv * 2 + side];
      }
      float o[4];
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        float v = c0[f];
        if ((gmask >> f) & 1u) {
          v = v + dx * a[f][0] + dy * a[f][1];
          if (ORD == 3) v = v + xx * a[f][2] + xy * a[f][3] + yy * a[f][4];
        }
        o[f] = v;
      }
      if (ALL || (gmask | pmask) == 0xFu) upv[xv] = make_float4(o[0], o[1], o[2], o[3]);
      else {
        float* p = reinterpret_cast<float*>(upv + xv);
#pragma unroll
        for (int f = 0; f < 4; ++f) if (((gmask | pmask) >> f) & 1u) p[f] = o[f];
      }
    }
  };
  faces(std::integral_constant<int, 6>(), 0);
  if (np > 6) faces(std::integral_constant<int, 1>(), 6);
}

// vertical upwind face values of the four fields (scalar_w_column of
// fluxes_wrtv, prog_wrtv_rk.f90:1085-1126): thread per (column, face kd)
__global__ void k_upw4(DynK g, const int* __restrict__ prog, int nprog, Four s, const float* __restrict__ wmc,
                       float* __restrict__ upw) {
  PK(j, kd, nprog);
  const int iw = WTAB(j);
  const int kb = LPW(iw);
  const int mza = g.mza;
  if (kd < kb - 1) return;
  const size_t plane = (size_t)g.mwa * mza;
  const size_t cb = (size_t)iw * mza;
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const float* S = s.f[f] + cb;
    float v;
    if (kd == kb - 1) v = S[kb];
    else if (kd == mza - 1) v = S[mza - 1];
    else {
      const bool down = wmc[cb + kd] < 0.f;
      const int lev = down ? kd + 1 : kd;
      const float b = S[lev];
      const float dsk = (lev <= mza - 2) ? S[lev + 1] - b : 0.f;
      const float dskm1 = (lev >= kb + 1) ? b - S[lev - 1] : 0.f;
      const float c1 = g.a_w[lev + (down ? 0 : 2 * mza)];
      const float c2 = g.a_w[lev + (down ? mza : 3 * mza)];
      v = b + dsk * c1 + dskm1 * c2;
    }
    upw[(size_t)f * plane + cb + kd] = v;
  }
}

// ---- prog_wrt_begs ------------------------------------------
struct WrtArgs {
  int istage, nrk;
  double dt8;
  float dts, fcoriol, c8, c9, rocv;
  double pc2, pc3, fr;
  const int* prog; int nprog;
  const float* vmca; const float4* upv;                     // face mass flux, the four face values
  const float* upw;                                         // 4-field array (not LEAN)
  // *_rk at stage start: *_short, or the long-step tendencies (LEAN)
  const float* sh_th; const float* sh_vx; const float* sh_vy; const float* sh_vz;
  float* rk_vx; float* rk_vy; float* rk_vz;
  double* rho; double* press; double* rho0; double* rth0;
  float* thil; float* wc; float* wmc; float* wmc0; const float* vxe; const float* vye; const float* vze;
  float* wmasc;
  const float* alpha_press; const float* pwfac;
  const double* volt; const float* volwi; const float* arw; const float* wn;
  const double* gdz_wgtm8; const double* gdz_wgtp8; const float* gdz_wgtm; const float* gdz_wgtp;
  const double* zwgt_bot8; const double* zwgt_top8; const float* b20;
};

// warps per SM the column kernel is compiled for: 72 registers (at NXP=100, 60
// levels 326 us; 24 warps and 80 registers 363, 32 warps and 64 registers 349)
#define WRT_OCC 28
// columns per block: four one-warp columns, else one
#define WRT_COLS(NW) ((NW) == 1 ? 4 : 1)

// the lanes of a column meet
template <int NW>
__device__ __forceinline__ void column_sync() {
  if constexpr (NW == 1) __syncwarp();
  else __syncthreads();
}

// The W system of prog_wrt_begs, b31(k) x(k-1) + b32(k) x(k) + b33(k) x(k+1)
// = dwm(k) for n levels k, row i of which lane i of the column holds; the
// reference solves it with the Thomas algorithm (tridiffo,
// outils/tridiag_lib.f90:10-36).  The equations are FP64 (the inputs and the
// result are the reference's real(4)): w is a small residual of large terms,
// and FP64 keeps it nearer the exact solve than a real(4) sweep.
//
// n <= 64 (one or two warps a column): one step of cyclic reduction
// eliminates the even rows, which leaves at most 32 odd rows to the lanes of
// the first warp, and parallel cyclic reduction solves those: in a step of
// stride s every row, scaled to a unit diagonal, eliminates its couplings to
// rows m - s and m + s, whose coefficients come by shuffles (rows outside the
// system couple with 0).  The even rows follow by substitution.  All rows in
// parallel cyclic reduction through shared memory took 42 % of the kernel's
// shared-memory and 30 % of its issue slots.  P: seven arrays of 32 doubles.
// The solution goes to x[0 .. n) of shared memory.
template <int NW>
__device__ __forceinline__ void column_solve(double* P, int n, int i, double ra, double rb, double rc, double rd,
                                             float* x) {
  const int m = i >> 1;
  if (i & 1) {
    if (i < n) { P[96 + m] = ra; P[128 + m] = rb; P[160 + m] = rc; P[192 + m] = rd; }
  } else if (i < n) {
    const double r = recip(rb);
    P[m] = ra * r; P[32 + m] = rc * r; P[64 + m] = rd * r;
  }
  column_sync<NW>();
  if (i < 32) {
    const bool even = 2 * i < n, odd = 2 * i + 1 < n, next = 2 * i + 2 < n;
    const double ae = even ? P[i] : 0.0, ce = even ? P[32 + i] : 0.0, de = even ? P[64 + i] : 0.0;
    double a = 0.0, c = 0.0, d = 0.0;
    if (odd) {
      const double oa = P[96 + i], ob = P[128 + i], oc = P[160 + i], od = P[192 + i];
      const double an = next ? P[i + 1] : 0.0, cn = next ? P[33 + i] : 0.0, dn = next ? P[65 + i] : 0.0;
      const double r = recip(ob - oa * ce - oc * an);
      a = -oa * ae * r;
      c = -oc * cn * r;
      d = (od - oa * de - oc * dn) * r;
    }
    const int no = n >> 1;   // odd rows
    for (int s = 1; s < no; s <<= 1) {
      const double am = __shfl_up_sync(0xffffffffu, a, s), cm = __shfl_up_sync(0xffffffffu, c, s),
                   dm = __shfl_up_sync(0xffffffffu, d, s);
      const double ap = __shfl_down_sync(0xffffffffu, a, s), cp = __shfl_down_sync(0xffffffffu, c, s),
                   dp = __shfl_down_sync(0xffffffffu, d, s);
      const double r = recip(1.0 - a * cm - c * ap);
      d = (d - a * dm - c * dp) * r;
      a = -a * am * r;
      c = -c * cp * r;
    }
    const double below = __shfl_up_sync(0xffffffffu, d, 1);   // row 2 i - 1
    if (even) x[2 * i] = (float)(de - (i > 0 ? ae * below : 0.0) - ce * d);
    if (odd) x[2 * i + 1] = (float)d;
  }
  column_sync<NW>();
}

// n up to 128 (four warps a column): parallel cyclic reduction of all rows,
// each publishing a, c, d and 1 / b per step.  P: four arrays of 128 doubles.
template <>
__device__ __forceinline__ void column_solve<4>(double* P, int n, int i, double ra, double rb, double rc, double rd,
                                                float* x) {
  double* A = P;
  double* RB = P + 128;                             // 1 / b
  double* Cc = P + 256;
  double* D = P + 384;
  for (int s = 1; s < n; s <<= 1) {
    if (i < n) { A[i] = ra; RB[i] = recip(rb); Cc[i] = rc; D[i] = rd; }
    column_sync<4>();
    if (i < n) {
      const int im = i - s, ip = i + s;
      double al = 0.0, ga = 0.0, am = 0.0, cm = 0.0, dm = 0.0, ap = 0.0, cp = 0.0, dp = 0.0;
      if (im >= 0) { al = -ra * RB[im]; am = A[im]; cm = Cc[im]; dm = D[im]; }
      if (ip < n) { ga = -rc * RB[ip]; ap = A[ip]; cp = Cc[ip]; dp = D[ip]; }
      rb = rb + al * cm + ga * ap;
      rd = rd + al * dm + ga * dp;
      ra = al * am;
      rc = ga * cp;
    }
    column_sync<4>();
  }
  if (i < n) x[i] = (float)(rd * recip(rb));
  column_sync<4>();
}

// NW = 1, 2 or 4 warps per column (mza up to 32, 64, 128), a level per lane
// from the first phase to the last: what only the same level reads later
// stays in registers, what the levels above and below read goes through
// shared memory (64 B a level: the two halves of the explicit terms, then the
// solve's rows; the four fields, then w and rho; the four fields' W-face
// values).  Every load of a level is issued before the first is used: with a
// warp per column and two levels a lane in turn, a warp went to memory four
// times one after the other.
// LEAN: no eddy, Rayleigh or flux-corrected terms -- the tendencies are
// formed here from the long-step ones, the first stage keeps the start
// values, and the W-face values (scalar_w_column of fluxes_wrtv,
// prog_wrtv_rk.f90:1085-1126) are formed from the column's own rows, so that
// the set-up pass and the W-face pass are not run.
template <int NW, bool LEAN>
__global__ void __launch_bounds__(32 * NW * WRT_COLS(NW), WRT_OCC / (NW * WRT_COLS(NW))) k_wrt_begs(DynK g, WrtArgs A) {
  extern __shared__ double wsm[];
  constexpr int LANES = 32 * NW;
  const int grp = threadIdx.x / LANES, i = threadIdx.x - grp * LANES;   // the column of the block, the lane of the column
  const int j = blockIdx.x * WRT_COLS(NW) + grp;
  if (j >= A.nprog) return;                                             // whole columns
  const int mza = g.mza;
  // the solve's rows share the first half with the explicit terms
  constexpr int half = NW == 1 ? 224 : 4 * LANES;   // doubles: at least 4 mza and the solve's arrays
  double* base = wsm + (size_t)grp * (half + 4 * mza);
  double* PEX = base;
  double* REX = base + mza;
  float* B15 = reinterpret_cast<float*>(base + 2 * mza);
  float* RKX = B15 + mza;
  float* RKY = B15 + 2 * mza;
  float* RKZ = B15 + 3 * mza;
  float* S = reinterpret_cast<float*>(base + half);         // thil, vxe, vye, vze
  float* WMF = S;
  double* RHON = base + half + mza;
  float* U = reinterpret_cast<float*>(base + half + 2 * mza);   // their W-face values

  const int* prog = A.prog;
  const int iw = WTAB(j);
  const int kb = LPW(iw);
  const int np = g.npoly[iw];
  const size_t cb = (size_t)iw * mza;
  const int4* E = g.edge + (size_t)iw * (7 * EDGE_W / 4);
  const bool first = A.istage == 1;
  const bool in = kb + i < mza;
  const int kd = min(kb + i, mza - 1);   // lanes past the top repeat it and store nothing
  const size_t x = cb + kd;

  // phase 1: horizontal sums, Coriolis and explicit density / rho*thil terms
  int4 e[6];
#pragma unroll
  for (int n = 0; n < 6; ++n) e[n] = __ldg(E + 2 * n);
  grid_wait();
  float th = A.sh_th[x], vx = A.sh_vx[x], vy = A.sh_vy[x], vz = A.sh_vz[x];
  const double rho = A.rho[x], volt = A.volt[x];
  const float thil = A.thil[x], vye = A.vye[x], vxe = A.vxe[x], alpha = A.alpha_press[x];
  const float vti = g.volti[x];
  const float vze = LEAN ? A.vze[x] : 0.f, wms = LEAN ? A.wmc[x] : 0.f;
  float wm0 = wms;
  double rho0 = rho, t0 = 0.0;
  if (!(LEAN && first)) { wm0 = A.wmc0[x]; rho0 = A.rho0[x]; }
  if (!first) t0 = A.rth0[x];
  const int up = kd < mza - 1 ? 1 : 0;
  const float arwm = A.arw[x - 1], arw0 = A.arw[x], arwp = A.arw[x + up];
  const float wcm = A.wc[x - 1], wcp = A.wc[x + up];
  const float vwi = A.volwi[x], pwf = A.pwfac[x], vtp = g.volti[x + up];
  float vm[6];
  float4 fu[6];
#pragma unroll
  for (int n = 0; n < 6; ++n) {
    vm[n] = 0.f;
    fu[n] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kd >= e[n].z) {
      const size_t xv = (size_t)(e[n].y & 0x7fffffff) * mza + kd;
      vm[n] = A.vmca[xv];
      fu[n] = A.upv[xv];
    }
  }
  if (LEAN) {
    const float v4 = (float)volt;
    th = __fmul_rn(th, v4); vx = __fmul_rn(vx, v4); vy = __fmul_rn(vy, v4); vz = __fmul_rn(vz, v4);
  }
  double hf = 0.0;
  auto add = [&](const int4& q, float m, const float4& v) {
    if (__int_as_float(q.w) > 0.f) {
      hf = hf + (double)m;
      th = th + m * v.x;
      vx = vx + m * v.y;
      vy = vy + m * v.z;
      vz = vz + m * v.w;
    } else {
      hf = hf - (double)m;
      th = th - m * v.x;
      vx = vx - m * v.y;
      vy = vy - m * v.z;
      vz = vz - m * v.w;
    }
  };
#pragma unroll
  for (int n = 0; n < 6; ++n) add(e[n], vm[n], fu[n]);
  if (np > 6) {
    const int4 q = __ldg(E + 12);
    if (kd >= q.z) {
      const size_t xv = (size_t)(q.y & 0x7fffffff) * mza + kd;
      add(q, A.vmca[xv], A.upv[xv]);
    }
  }
  const float mass = (float)(rho * volt);
  vx = vx + mass * A.fcoriol * vye;
  vy = vy - mass * A.fcoriol * vxe;
  const double rt = rho * (double)thil;
  const double b10 = A.dt8 * (double)vti;
  const double b5 = (double)(alpha * powf((float)rt, A.rocv));
  double drho = b10 * hf;
  double drt = b10 * (double)th;
  if (!first) {
    drho = drho + rho0 - rho;
    drt = drt + t0 - rt;
  }
  if (in) {
    PEX[kd] = b5 * (rt + A.pc2 * drt);
    REX[kd] = rho + A.fr * drho;
    B15[kd] = (float)(b10 * b5);
    RKX[kd] = vx; RKY[kd] = vy; RKZ[kd] = vz;
    if (LEAN) {
      S[kd] = thil; S[mza + kd] = vxe; S[2 * mza + kd] = vye; S[3 * mza + kd] = vze;
      if (first) { A.rho0[x] = rho; A.rth0[x] = rt; A.wmc0[x] = wms; }
    }
  }
  column_sync<NW>();
  // the W-face values of the lane's level, and below the floor
  float u[4];
  if (LEAN) {
    const bool top = kd == mza - 1, down = wms < 0.f;
    const int lev = !top && down ? kd + 1 : kd;
    const float c1 = g.a_w[lev + (down ? 0 : 2 * mza)];
    const float c2 = g.a_w[lev + (down ? mza : 3 * mza)];
    const int lu = min(lev + 1, mza - 1), ld = max(lev - 1, kb);
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const float b = S[f * mza + lev];
      const float dsk = (lev <= mza - 2) ? S[f * mza + lu] - b : 0.f;
      const float dskm1 = (lev >= kb + 1) ? b - S[f * mza + ld] : 0.f;
      u[f] = top ? b : b + dsk * c1 + dskm1 * c2;
    }
  } else {
#pragma unroll
    for (int f = 0; f < 4; ++f) u[f] = A.upw[(size_t)f * g.mwa * mza + x];
  }
  if (in) {
#pragma unroll
    for (int f = 0; f < 4; ++f) U[f * mza + kd] = u[f];
  }
  if (i < 4) U[i * mza + kb - 1] = LEAN ? S[i * mza + kb] : A.upw[(size_t)i * g.mwa * mza + cb + kb - 1];
  column_sync<NW>();
  // phase 2: explicit W momentum and the tridiagonal coefficients (faces kb..mza-2)
  const int n = mza - 1 - kb;
  double ra = 0.0, rb = 1.0, rc = 0.0, rd = 0.0;
  if (i < n) {
    const float wnx = A.wn[iw * 3], wny = A.wn[iw * 3 + 1], wnz = A.wn[iw * 3 + 2];
    const float a = (float)(PEX[kd] - PEX[kd + 1]) * pwf;
    const float b = (float)(A.gdz_wgtm8[kd] * REX[kd] + A.gdz_wgtp8[kd] * REX[kd + 1]);
    const float c = (wnx * (vx + RKX[kd + 1]) + wny * (vy + RKY[kd + 1]) + wnz * (vz + RKZ[kd + 1])) * vwi;
    rd = (double)(wm0 + A.dts * (a - b + c));
    const float b7 = A.dts * vwi;
    const float b8 = A.c8 * pwf;
    const float b21 = b7 * wcm;
    const float b22 = b7 * wcp;
    const float b23 = b8 * B15[kd];
    const float b24 = b8 * B15[kd + 1];
    const float b25 = A.c9 * vti * A.gdz_wgtm[kd];
    const float b26 = A.c9 * vtp * A.gdz_wgtp[kd];
    if (i > 0) ra = (double)(-arwm * (b21 + b25 + b23 * U[kd - 1]));
    rb = (double)(A.b20[kd] + arw0 * (b25 - b26 + (b23 + b24) * u[0]));
    if (i < n - 1) rc = (double)(arwp * (b22 + b26 - b24 * U[kd + 1]));
  } else if (i == 0) {
    A.wc[x - 1] = wcp;   // a column of one level, whose wcp is its own
  }
  column_sync<NW>();
  // phase 3: tridiffo's system across the column's lanes
  column_solve<NW>(base, n, i, ra, rb, rc, rd, WMF + kb);
  const float wf = i < n ? WMF[kd] : 0.f;
  // phase 4: implicit fluxes and the updates of rho, press, thil and vm*et_rk
  if (in) {
    const float wma = i < n ? wf * arw0 : 0.f;
    const float wmam = i > 0 ? WMF[kd - 1] * arwm : 0.f;
    const double vft = i < n ? (double)(wma * u[0]) : 0.0;
    const double vftm = i > 0 ? (double)(wmam * U[kd - 1]) : 0.0;
    const float vfx = i < n ? wma * u[1] : 0.f;
    const float vfxm = i > 0 ? wmam * U[mza + kd - 1] : 0.f;
    const float vfy = i < n ? wma * u[2] : 0.f;
    const float vfym = i > 0 ? wmam * U[2 * mza + kd - 1] : 0.f;
    const float vfz = i < n ? wma * u[3] : 0.f;
    const float vfzm = i > 0 ? wmam * U[3 * mza + kd - 1] : 0.f;
    if (A.istage == A.nrk && i < n) A.wmasc[x] = A.wmasc[x] + wma;
    const double rhon = rho0 + b10 * (hf + (double)wmam - (double)wma);
    A.rho[x] = rhon;
    RHON[kd] = rhon;
    drt = drt + b10 * (vftm - vft);
    A.press[x] = b5 * (rt + A.pc3 * drt);
    const float thn = (float)((rt + drt) * recip(rhon));
    A.thil[x] = thn;
    if (i == 0)
      for (int k = 0; k < kb; ++k) A.thil[cb + k] = thn;   // bottom values
    A.rk_vx[x] = vx + vfxm - vfx;
    A.rk_vy[x] = vy + vfym - vfy;
    A.rk_vz[x] = vz + vfzm - vfz;
  }
  column_sync<NW>();
  // phase 5: W momentum and velocity
  if (i < n) {
    A.wmc[x] = wf;
    const float w = wf / (float)(A.zwgt_bot8[kd] * RHON[kd] + A.zwgt_top8[kd] * RHON[kd + 1]);
    A.wc[x] = w;
    if (i == 0) A.wc[x - 1] = w;
  }
}

// prog_v_begs (prog_wrtv_rk.f90:888-946)
__global__ void k_prog_v(DynK g, const int* __restrict__ vprog, int nv, float dts, const float* vmc0,
                         const float* vmt_short, const double* press,
                         const float* __restrict__ pvfac, const float* __restrict__ vn,
                         const float* rkx, const float* rky,
                         const float* rkz, const float* __restrict__ volvi,
                         const double* rho, float* vmc, float* vc) {
  grid_wait();
  PK(j, kd, nv);
  const int iv = VPTAB(j);
  if (kd < LPV(iv)) return;
  const int mza = g.mza;
  const int iw1 = g.v_iw[iv * 2], iw2 = g.v_iw[iv * 2 + 1];
  const size_t x = (size_t)iv * mza + kd, x1 = (size_t)iw1 * mza + kd, x2 = (size_t)iw2 * mza + kd;
  // every load before the first store (the arrays may alias for the compiler)
  const double rs = rho[x1] + rho[x2];
  const float pgf = (float)(press[x1] - press[x2]) * pvfac[x];
  const float v = vmc0[x] + dts * (vmt_short[x] + pgf +
                                   (vn[iv * 3] * (rkx[x1] + rkx[x2]) + vn[iv * 3 + 1] * (rky[x1] + rky[x2]) +
                                    vn[iv * 3 + 2] * (rkz[x1] + rkz[x2])) * volvi[x]);
  vmc[x] = v;
  vc[x] = 2.0f * v / (float)rs;
}

// Prognostic shaved-cell method (prog_wrtv_rk.f90:202-211): the momentum of
// the lve2 lowest levels of a column with closed V faces at the step's start.
// A thread per (column, shaved level).
__global__ void k_shaved_save(DynK g, const int* __restrict__ prog, int nprog, const int* __restrict__ lve2,
                              int nve2, const float* __restrict__ vxe, const float* __restrict__ vye,
                              const float* __restrict__ vze, const double* __restrict__ rho, float* __restrict__ vm0) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nprog * nve2) return;
  const int j = (int)(i / nve2), ks = (int)(i % nve2);
  const int iw = prog[j];
  if (ks >= lve2[iw]) return;
  const size_t x = (size_t)iw * g.mza + LPW(iw) + ks;
  const float rs = (float)rho[x];
  float* o = vm0 + ((size_t)iw * nve2 + ks) * 3;
  o[0] = vxe[x] * rs; o[1] = vye[x] * rs; o[2] = vze[x] * rs;
}

// the shaved-cell inputs of k_vel_t3d: lve2 == nullptr on grids without
// closed faces; prog != 0 in a stage of prog_wrtv_rk (the velocities of the
// shaved levels are prognosed first, update_vxe_undrgnd), 0 in diagvel_t3d
// (the cell's current velocities)
struct Shaved {
  const int* lve2;
  const float* vm0;
  const float *rkx, *rky, *rkz;
  const double* rho;
  const float* vn;
  int nve2, prog;
  float dts;
};

static Shaved shaved_args(const Dyn& y, const Transport& tp, int prog, float dts) {
  Shaved a{};
  if (y.nve2_max > 0) { a.lve2 = y.lve2.p; a.vm0 = y.vm0.p; a.nve2 = y.nve2_max; }
  a.rkx = y.rk_vx.p; a.rky = y.rk_vy.p; a.rkz = y.rk_vz.p;
  a.rho = tp.rho.p; a.vn = y.vn.p; a.prog = prog; a.dts = dts;
  return a;
}

// update_vxe_undrgnd (prog_wrtv_rk.f90:1558-1595) and vel_t3d_hex
// (vel_t3d.f90:39-108): a closed face (below its lpv) contributes the normal
// component of the cell's prognosed velocity at that level
// ecv: four floats per edge (x, y, z, 0), 7 edges per column
template <int R>
__global__ void __launch_bounds__(256) k_vel_t3d(DynK g, const int* __restrict__ prog, int nprog, const float* wc,
                          const float* vc, const float* __restrict__ wno2,
                          const float4* __restrict__ ecv, float* vxe, float* vye,
                          float* vze, Shaved sh) {
  grid_wait();
  WARP_POINT(nprog, 0u);
  const int mza = g.mza;
  const int iw = WTAB((int)w_), kb = LPW(iw), np = g.npoly[iw];
  const size_t cb = (size_t)iw * mza;
  const int4* E = g.edge + (size_t)iw * (7 * EDGE_W / 4);
  edges_ahead(g, E, iw);
  const float wx = wno2[iw * 3], wy = wno2[iw * 3 + 1], wz = wno2[iw * 3 + 2];
  const int lve = sh.lve2 ? sh.lve2[iw] : 0;
  int4 e[6];
  float4 ec[6];
#pragma unroll
  for (int n = 0; n < 6; ++n) { e[n] = __ldg(E + 2 * n); ec[n] = __ldg(ecv + iw * 7 + n); }
  float wl[R], wu[R], v[R][6];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int kd = lane + 32 * r;
    wl[r] = wu[r] = 0.f;
    if (kd >= kb && kd < mza) { wl[r] = wc[cb + kd - 1]; wu[r] = wc[cb + kd]; }
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      v[r][n] = 0.f;
      if (kd >= e[n].z && kd < mza) v[r][n] = vc[(size_t)(e[n].y & 0x7fffffff) * mza + kd];
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int kd = lane + 32 * r;
    if (kd < kb || kd >= mza) continue;
    const int ks = kd - kb;
    const bool shaved = ks < lve;
    float p1x = 0.f, p1y = 0.f, p1z = 0.f;
    if (shaved) {
      if (sh.prog) {
        const float rsi = 1.0f / (float)sh.rho[cb + kd];
        const float vt = g.volti[cb + kd];
        const float* m = sh.vm0 + ((size_t)iw * sh.nve2 + ks) * 3;
        p1x = (m[0] + sh.dts * (sh.rkx[cb + kd] * vt)) * rsi;
        p1y = (m[1] + sh.dts * (sh.rky[cb + kd] * vt)) * rsi;
        p1z = (m[2] + sh.dts * (sh.rkz[cb + kd] * vt)) * rsi;
      } else {
        p1x = vxe[cb + kd]; p1y = vye[cb + kd]; p1z = vze[cb + kd];
      }
    }
    const float wst = wl[r] + wu[r];
    float x = wst * wx, y = wst * wy, z = wst * wz;
    auto add = [&](const int4& q, const float4& c, float u) {
      if (kd < q.z) {   // a face under ground
        if (!shaved) return;
        const int iv = q.y & 0x7fffffff;
        u = sh.vn[iv * 3] * p1x + sh.vn[iv * 3 + 1] * p1y + sh.vn[iv * 3 + 2] * p1z;
      }
      x = x + c.x * u;
      y = y + c.y * u;
      z = z + c.z * u;
    };
#pragma unroll
    for (int n = 0; n < 6; ++n) if (n < np) add(e[n], ec[n], v[r][n]);
    if (np > 6) {
      const int4 q = __ldg(E + 12);
      add(q, __ldg(ecv + iw * 7 + 6), kd >= q.z ? vc[(size_t)(q.y & 0x7fffffff) * mza + kd] : 0.f);
    }
    vxe[cb + kd] = x; vye[cb + kd] = y; vze[cb + kd] = z;
    if (kd == kb)
      for (int k2 = 0; k2 < kb; ++k2) { vxe[cb + k2] = x; vye[cb + k2] = y; vze[cb + k2] = z; }
  }
}

// tend0 (timestep.f90:430-496) for the hot-path arrays
__global__ void k_tend0_w(DynK g, float* thilt, float* vmxet, float* vmyet, float* vmzet,
                          const double* rho, float* rho_old, float* wmasc) {
  grid_wait();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)(g.mwa - 1) * g.mza) return;
  const int iw = 1 + (int)(i / g.mza), kd = (int)(i % g.mza);
  if (kd < LPW(iw)) return;
  const size_t x = (size_t)iw * g.mza + kd;
  thilt[x] = 0.f; vmxet[x] = 0.f; vmyet[x] = 0.f; vmzet[x] = 0.f;
  rho_old[x] = (float)rho[x];
  wmasc[x] = 0.f;
}

__global__ void k_tend0_v(DynK g, float* vmt, float* vmasc) {
  grid_wait();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)(g.mva - 1) * g.mza) return;
  const int iv = 1 + (int)(i / g.mza), kd = (int)(i % g.mza);
  if (kd < LPV(iv)) return;
  const size_t x = (size_t)iv * g.mza + kd;
  vmt[x] = 0.f;
  vmasc[x] = 0.f;
}

// timeavg_momsc (timestep.f90:563-612)
__global__ void k_timeavg_v(DynK g, const int* __restrict__ vadj, int nv, float a, float* vmasc) {
  grid_wait();
  PK(j, kd, nv);
  const int iv = VATAB(j);
  if (kd < LPV(iv)) return;
  vmasc[(size_t)iv * g.mza + kd] = vmasc[(size_t)iv * g.mza + kd] / a;
}

__global__ void k_timeavg_w(DynK g, const int* __restrict__ prog, int nprog, float a, float* wmasc) {
  grid_wait();
  PK(j, kd, nprog);
  const int iw = WTAB(j);
  if (kd < LPW(iw) || kd > g.mza - 2) return;
  wmasc[(size_t)iw * g.mza + kd] = wmasc[(size_t)iw * g.mza + kd] / a;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <class T>
static int up(DevBuf<T>& b, const T* h, size_t n, cudaStream_t s, const char* name) {
  if (!h) {
    set_error(std::string("olamgpu_grid/opts: ") + name + " is NULL (needed by prog_wrtv_rk)");
    return OLAMGPU_E_ARG;
  }
  return upload(b, h, n, s);
}

int dyn_setup(const olamgpu_grid* g, const olamgpu_opts* o, cudaStream_t s) {
  Context& C = ctx();
  Dyn& y = C.dy;
  const int mza = g->mza, mwa = g->mwa, mva = g->mva, mma = g->mma;
  if (!g->itab_m_iv || !g->jtm_prog || g->nm_prog <= 0 || !g->lpm) {
    set_error("prog_wrtv_rk needs the M-point tables (itab_m, jtm_prog, lpm)");
    return OLAMGPU_E_ARG;
  }
  for (int i = 1; i < mma; ++i)
    if (g->lpm[i] < 2 || g->lpm[i] > mza) { set_error("lpm out of range [2,mza] at M point " + std::to_string(i + 1)); return OLAMGPU_E_ARG; }
  y.lpm_flat = true;
  for (int i = 1; i < mma; ++i) if (g->lpm[i] != 2) y.lpm_flat = false;
  // shaved cells: lve2(iw) levels from lpw up have closed V faces; every
  // closed face must lie within them (hex_grid.f90 sets lve2 to the largest
  // lpv - lpw of the column's faces)
  int nve2 = 0;
  std::vector<int> lve2(mwa, 0);
  for (int i = 1; i < mwa; ++i) {
    const int l = g->lve2 ? g->lve2[i] : 0;
    if (l < 0 || l > mza) { set_error("lve2 out of range [0,mza] at W point " + std::to_string(i + 1)); return OLAMGPU_E_ARG; }
    for (int n = 0; n < g->npoly[i]; ++n) {
      const int iv = g->itab_w_iv[(size_t)i * 7 + n] - 1;
      if (iv >= 1 && iv < mva && g->lpv[iv] - g->lpw[i] > l) {
        set_error("lve2 at W point " + std::to_string(i + 1) + " does not cover its closed V faces (lpv - lpw)");
        return OLAMGPU_E_ARG;
      }
    }
    lve2[i] = l;
    nve2 = std::max(nve2, l);
  }
  y.nve2_max = nve2;
  if (nve2 > 0) {
    OG_CHECK(upload(y.lve2, lve2.data(), lve2.size(), s));
    OG_CHECK(y.vm0.alloc((size_t)mwa * nve2 * 3));
    OG_CUDA(cudaMemsetAsync(y.vm0.p, 0, y.vm0.bytes(), s));
  }
  if (mza > 128) { set_error("prog_wrtv_rk supports mza <= 128"); return OLAMGPU_E_UNSUPPORTED; }
  if ((size_t)std::max(std::max(mwa, mva), mma) * mza >= (1ull << 31)) {
    set_error("prog_wrtv_rk supports grids with max(mwa, mva, mma) * mza < 2^31");
    return OLAMGPU_E_UNSUPPORTED;
  }
  OG_CHECK(up(y.arv, g->arv, (size_t)mza * mva, s, "arv"));
  OG_CHECK(up(y.arw, g->arw, (size_t)mza * mwa, s, "arw"));
  OG_CHECK(up(y.volwi, g->volwi, (size_t)mza * mwa, s, "volwi"));
  OG_CHECK(up(y.volvi, g->volvi, (size_t)mza * mva, s, "volvi"));
  OG_CHECK(up(y.volt, g->volt, (size_t)mza * mwa, s, "volt"));
  {
    if (!g->wnx || !g->wnxo2 || !g->vnx || !g->ecvec_vx) { set_error("normals/ecvec missing"); return OLAMGPU_E_ARG; }
    std::vector<float> wn((size_t)mwa * 3), wno2((size_t)mwa * 3), vn((size_t)mva * 3), ec((size_t)mwa * 28, 0.f);
    for (int i = 0; i < mwa; ++i) {
      wn[i * 3] = g->wnx[i]; wn[i * 3 + 1] = g->wny[i]; wn[i * 3 + 2] = g->wnz[i];
      wno2[i * 3] = g->wnxo2[i]; wno2[i * 3 + 1] = g->wnyo2[i]; wno2[i * 3 + 2] = g->wnzo2[i];
      for (int n = 0; n < 7; ++n) {
        ec[(i * 7 + n) * 4] = g->ecvec_vx[i * 7 + n];
        ec[(i * 7 + n) * 4 + 1] = g->ecvec_vy[i * 7 + n];
        ec[(i * 7 + n) * 4 + 2] = g->ecvec_vz[i * 7 + n];
      }
    }
    for (int i = 0; i < mva; ++i) { vn[i * 3] = g->vnx[i]; vn[i * 3 + 1] = g->vny[i]; vn[i * 3 + 2] = g->vnz[i]; }
    OG_CHECK(upload(y.wn, wn.data(), wn.size(), s));
    OG_CHECK(upload(y.wno2, wno2.data(), wno2.size(), s));
    OG_CHECK(upload(y.vn, vn.data(), vn.size(), s));
    OG_CHECK(upload(y.ecv, ec.data(), ec.size(), s));
    OG_CUDA(cudaStreamSynchronize(s));
  }
  OG_CHECK(up(y.gdz_wgtm, g->gdz_wgtm, mza, s, "gdz_wgtm"));
  OG_CHECK(up(y.gdz_wgtp, g->gdz_wgtp, mza, s, "gdz_wgtp"));
  OG_CHECK(up(y.gdz_wgtm8, g->gdz_wgtm8, mza, s, "gdz_wgtm8"));
  OG_CHECK(up(y.gdz_wgtp8, g->gdz_wgtp8, mza, s, "gdz_wgtp8"));
  OG_CHECK(up(y.zwgt_top8, g->zwgt_top8, mza, s, "zwgt_top8"));
  OG_CHECK(up(y.zwgt_bot8, g->zwgt_bot8, mza, s, "zwgt_bot8"));
  OG_CHECK(up(y.dniv, g->dniv, mva, s, "dniv"));
  OG_CHECK(up(y.dniu, g->dniu, mva, s, "dniu"));
  OG_CHECK(up(y.dnv, g->dnv, mva, s, "dnv"));
  OG_CHECK(up(y.arw0, g->arw0, mwa, s, "arw0"));
  OG_CHECK(up(y.arm0, g->arm0, mma, s, "arm0"));
  OG_CHECK(up(y.zfacit, g->zfacit, mza, s, "zfacit"));
  OG_CHECK(up(y.dzit, g->dzit, mza, s, "dzit"));
  OG_CHECK(up(y.xx_yy, g->xx_yy, (size_t)mwa * 7, s, "xx_yy"));
  OG_CHECK(up(y.xx_yy_m, g->xx_yy_m, (size_t)mma * 3, s, "xx_yy_m"));
  // init_wrtv_rk (prog_wrtv_rk.f90:36-54): b20 = 1 + dtsm * rayf_cofw
  std::vector<float> b20(mza, 1.0f);
  if (o->rayf_cofw)
    for (int k = o->krayfw_bot; k <= mza - 1; ++k) b20[k - 1] = 1.0f + (float)o->dtsm * o->rayf_cofw[k - 1];
  OG_CHECK(upload(y.b20, b20.data(), b20.size(), s));
  if (o->rayf_cof) {
    OG_CHECK(up(y.rayf_cof, o->rayf_cof, mza, s, "rayf_cof"));
    if (o->initial == 1) {
      OG_CHECK(up(y.dn01d, o->dn01d, mza, s, "dn01d"));
      OG_CHECK(up(y.th01d, o->th01d, mza, s, "th01d"));
    }
    OG_CHECK(up(y.vc03d, o->vc03d, (size_t)mza * mva, s, "vc03d"));
  }
  OG_CUDA(cudaStreamSynchronize(s));
  y.div_first = y.vort_first = true;
  y.uploaded = false;
  y.ready = true;
  return OLAMGPU_OK;
}

static int ensure_dyn_buffers(Context& C) {
  Dyn& y = C.dy;
  Transport& tp = C.tp;
  const size_t wz = (size_t)C.g.mza * C.g.mwa, vz = (size_t)C.g.mza * C.g.mva, mz = (size_t)C.g.mza * C.g.mma;
  auto A = [](auto& b, size_t n) { return b.p ? OLAMGPU_OK : b.alloc(n); };
  OG_CHECK(A(tp.rho, wz)); OG_CHECK(A(tp.vmasc, vz)); OG_CHECK(A(tp.wmasc, wz)); OG_CHECK(A(tp.wc, wz));
  OG_CHECK(A(tp.rho_old, wz));
  OG_CHECK(A(y.press, wz)); OG_CHECK(A(y.rho0, wz)); OG_CHECK(A(y.rth0, wz));
  DevBuf<float>* w[] = {&y.thil, &y.wmc, &y.vxe, &y.vye, &y.vze, &y.alpha_press, &y.pwfac, &y.thilt,
                        &y.vmxet, &y.vmyet, &y.vmzet, &y.wmc0, &y.sh_th, &y.sh_vx, &y.sh_vy, &y.sh_vz,
                        &y.rk_vx, &y.rk_vy, &y.rk_vz};
  for (auto* b : w) OG_CHECK(A(*b, wz));
  DevBuf<float>* v[] = {&y.vmc, &y.vc, &y.pvfac, &y.vmt, &y.vmc0, &y.vmca, &y.sh_vmt, &y.fdivh};
  for (auto* b : v) OG_CHECK(A(*b, vz));
  OG_CHECK(A(y.upw, 4 * wz));
  OG_CHECK(A(y.upv, 4 * vz));
  OG_CHECK(A(y.div2d, 2 * wz));
  OG_CHECK(A(y.vort2d, 2 * mz));
  OG_CHECK(A(y.fvorth, C.g.mva)); OG_CHECK(A(y.fvortl, C.g.mva));
  OG_CHECK(A(y.vfact, 3 * (size_t)C.g.mma));
  return OLAMGPU_OK;
}

// host <-> device copies of the registered mem_basic / mem_tend arrays
int dyn_state_to_device(unsigned mask, cudaStream_t s) {
  Context& C = ctx();
  if (!C.have_state) return OLAMGPU_OK;
  OG_CHECK(ensure_dyn_buffers(C));
  const olamgpu_state& h = C.hstate;
  Dyn& y = C.dy;
  Transport& tp = C.tp;
  const size_t wz = (size_t)C.g.mza * C.g.mwa, vz = (size_t)C.g.mza * C.g.mva;
  auto cp = [&](void* d, const void* hp, size_t bytes) -> int {
    if (!hp) return OLAMGPU_OK;
    OG_CUDA(cudaMemcpyAsync(d, hp, bytes, cudaMemcpyHostToDevice, s));
    return OLAMGPU_OK;
  };
  if (mask & OLAMGPU_F_RHO) OG_CHECK(cp(tp.rho.p, h.rho, wz * 8));
  if (mask & OLAMGPU_F_PRESS) OG_CHECK(cp(y.press.p, h.press, wz * 8));
  if (mask & OLAMGPU_F_THIL) OG_CHECK(cp(y.thil.p, h.thil, wz * 4));
  if (mask & OLAMGPU_F_WC) OG_CHECK(cp(tp.wc.p, h.wc, wz * 4));
  if (mask & OLAMGPU_F_WMC) OG_CHECK(cp(y.wmc.p, h.wmc, wz * 4));
  if (mask & OLAMGPU_F_VXE) {
    OG_CHECK(cp(y.vxe.p, h.vxe, wz * 4)); OG_CHECK(cp(y.vye.p, h.vye, wz * 4)); OG_CHECK(cp(y.vze.p, h.vze, wz * 4));
  }
  if (mask & OLAMGPU_F_VMC) OG_CHECK(cp(y.vmc.p, h.vmc, vz * 4));
  if (mask & OLAMGPU_F_VC) OG_CHECK(cp(y.vc.p, h.vc, vz * 4));
  if (mask & OLAMGPU_F_VMASC) OG_CHECK(cp(tp.vmasc.p, h.vmasc, vz * 4));
  if (mask & OLAMGPU_F_WMASC) OG_CHECK(cp(tp.wmasc.p, h.wmasc, wz * 4));
  if (mask & OLAMGPU_F_FACS) {
    OG_CHECK(cp(y.alpha_press.p, h.alpha_press, wz * 4)); OG_CHECK(cp(y.pwfac.p, h.pwfac, wz * 4));
    OG_CHECK(cp(y.pvfac.p, h.pvfac, vz * 4));
  }
  if (mask & OLAMGPU_F_TEND) {
    OG_CHECK(cp(y.thilt.p, h.thilt, wz * 4)); OG_CHECK(cp(y.vmxet.p, h.vmxet, wz * 4));
    OG_CHECK(cp(y.vmyet.p, h.vmyet, wz * 4)); OG_CHECK(cp(y.vmzet.p, h.vmzet, wz * 4));
    OG_CHECK(cp(y.vmt.p, h.vmt, vz * 4));
  }
  // the registered arrays are page-locked: the copies read them when they
  // run, so they must end before the caller may write them again
  OG_CUDA(cudaStreamSynchronize(s));
  return OLAMGPU_OK;
}

int dyn_state_to_host(unsigned mask, cudaStream_t s) {
  Context& C = ctx();
  if (!C.have_state || !C.dy.thil.p) return OLAMGPU_OK;
  const olamgpu_state& h = C.hstate;
  Dyn& y = C.dy;
  Transport& tp = C.tp;
  const size_t wz = (size_t)C.g.mza * C.g.mwa, vz = (size_t)C.g.mza * C.g.mva;
  auto cp = [&](void* hp, const void* d, size_t bytes) -> int {
    if (!hp || !d) return OLAMGPU_OK;
    OG_CUDA(cudaMemcpyAsync(hp, d, bytes, cudaMemcpyDeviceToHost, s));
    return OLAMGPU_OK;
  };
  if (mask & OLAMGPU_F_RHO) OG_CHECK(cp(h.rho, tp.rho.p, wz * 8));
  if (mask & OLAMGPU_F_PRESS) OG_CHECK(cp(h.press, y.press.p, wz * 8));
  if (mask & OLAMGPU_F_THIL) OG_CHECK(cp(h.thil, y.thil.p, wz * 4));
  if (mask & OLAMGPU_F_WC) OG_CHECK(cp(h.wc, tp.wc.p, wz * 4));
  if (mask & OLAMGPU_F_WMC) OG_CHECK(cp(h.wmc, y.wmc.p, wz * 4));
  if (mask & OLAMGPU_F_VXE) {
    OG_CHECK(cp(h.vxe, y.vxe.p, wz * 4)); OG_CHECK(cp(h.vye, y.vye.p, wz * 4)); OG_CHECK(cp(h.vze, y.vze.p, wz * 4));
  }
  if (mask & OLAMGPU_F_VMC) OG_CHECK(cp(h.vmc, y.vmc.p, vz * 4));
  if (mask & OLAMGPU_F_VC) OG_CHECK(cp(h.vc, y.vc.p, vz * 4));
  if (mask & OLAMGPU_F_VMASC) OG_CHECK(cp(h.vmasc, tp.vmasc.p, vz * 4));
  if (mask & OLAMGPU_F_WMASC) OG_CHECK(cp(h.wmasc, tp.wmasc.p, wz * 4));
  if (mask & OLAMGPU_F_TEND) {
    OG_CHECK(cp(h.thilt, y.thilt.p, wz * 4)); OG_CHECK(cp(h.vmxet, y.vmxet.p, wz * 4));
    OG_CHECK(cp(h.vmyet, y.vmyet.p, wz * 4)); OG_CHECK(cp(h.vmzet, y.vmzet.p, wz * 4));
    OG_CHECK(cp(h.vmt, y.vmt.p, vz * 4));
  }
  return OLAMGPU_OK;
}

#define DYN_IN_MASK (OLAMGPU_F_RHO | OLAMGPU_F_PRESS | OLAMGPU_F_THIL | OLAMGPU_F_WC | OLAMGPU_F_WMC | \
                     OLAMGPU_F_VXE | OLAMGPU_F_VMC | OLAMGPU_F_VC | OLAMGPU_F_VMASC | OLAMGPU_F_WMASC | \
                     OLAMGPU_F_FACS | OLAMGPU_F_TEND)
#define DYN_OUT_MASK (OLAMGPU_F_RHO | OLAMGPU_F_PRESS | OLAMGPU_F_THIL | OLAMGPU_F_WC | OLAMGPU_F_WMC | \
                      OLAMGPU_F_VXE | OLAMGPU_F_VMC | OLAMGPU_F_VC | OLAMGPU_F_VMASC | OLAMGPU_F_WMASC | \
                      OLAMGPU_F_TEND)

// a kernel template's instance for the levels of the grid
#define BY_ROWS(mza, ...)               \
  do {                                  \
    if ((mza) <= 32) { constexpr int R = 1; __VA_ARGS__; }      \
    else if ((mza) <= 64) { constexpr int R = 2; __VA_ARGS__; } \
    else { constexpr int R = 4; __VA_ARGS__; }                  \
    OG_LAUNCHED();                      \
  } while (0)

static bool divh_on(const olamgpu_opts& o) { return o.divh_damp_fact > 1.e-7f && o.divh_damp_level > 0; }
static bool vort_on(const olamgpu_opts& o) { return !(o.vort_damp_fact < 1.e-7f) && o.vort_damp_level > 0; }

// divh_damp and / or vort_damp of a step dtm, added to the V tendency src ->
// dst.  With setup also prog_wrtv_rk's V set-up: the Rayleigh term on the
// tendency and the start momentum vmc0.
static int v_tendency(Context& C, bool div, bool vor, bool setup, const float* src, float* dst, double dtm,
                      cudaStream_t s) {
  const olamgpu_opts& o = C.opts;
  const DevGrid& d = C.g;
  Dyn& y = C.dy;
  const DynK g = dynk(d);
  const int mza = d.mza;
  const size_t wz = (size_t)mza * d.mwa, mz = (size_t)mza * d.mma;
  div = div && divh_on(o);
  vor = vor && vort_on(o);
  if (div && y.div_first) {
    y.div_first = false;
    cudaMemsetAsync(y.div2d.p, 0, 2 * wz * sizeof(float), s);
    float p = 1.f;
    for (int i = 0; i < o.divh_damp_level; ++i) p = p * (-o.divh_damp_fact);
    const double facth = -((double)p / dtm);
    const float fact2 = o.divh_damp_fact / (float)dtm;
    k_div_fdivh<<<cdiv((size_t)d.nv_prog * mza, 256), 256, 0, s>>>(g, d.jtv_prog.p, d.nv_prog, y.arw0.p, y.dniv.p,
                                                                   y.zfacit.p, y.dzit.p, y.volt.p, facth,
                                                                   o.divh_damp_level, fact2, y.fdivh.p);
    OG_LAUNCHED();
  }
  if (vor && y.vort_first) {
    y.vort_first = false;
    k_vort_first_m<<<cdiv(d.nm_prog, 128), 128, 0, s>>>(g, d.jtm_prog.p, d.nm_prog, y.dnv.p, y.arm0.p, y.vfact.p);
    k_vort_first_v<<<cdiv(d.nv_prog, 128), 128, 0, s>>>(g, d.jtv_prog.p, d.nv_prog, y.dniu.p, y.arm0.p, (float)dtm,
                                                        o.vort_damp_fact, o.vort_damp_level, y.fvorth.p, y.fvortl.p);
    OG_LAUNCHED(); OG_LAUNCHED();
  }
  // the planes each Laplacian step reads and writes: 1 -> 2 -> 1 ...
  auto plane = [](float* p, size_t n, int i) { return p + (size_t)(i - 1) * n; };
  DampArgs A;
  A.wprog = d.jtw_prog.p; A.mprog = d.jtm_prog.p; A.off_m = d.off_mprog;
  A.arv = y.arv.p; A.vmc = y.vmc.p; A.vc = y.vc.p;
  A.xx_yy = y.xx_yy.p; A.xx_yy_m = y.xx_yy_m.p; A.vfact = y.vfact.p;
  auto run = [&](int step, bool dw, bool dm) -> int {   // step 0: the first planes
    A.nw = dw ? d.nw_prog : 0;
    A.nm = dm ? d.nm_prog : 0;
    A.mblock = cdiv(A.nw, 8);
    const unsigned nb = A.mblock + cdiv(A.nm, 8);
    const int il = step == 0 ? 1 : (step - 1) % 2 + 1, ih = step == 0 ? 1 : step % 2 + 1;
    A.wsrc = plane(y.div2d.p, wz, il); A.wdst = plane(y.div2d.p, wz, ih);
    A.msrc = plane(y.vort2d.p, mz, il); A.mdst = plane(y.vort2d.p, mz, ih);
    if (nb == 0) return OLAMGPU_OK;
    if (step == 0) BY_ROWS(mza, launch_next(k_damp_first<R>, nb, 256, 0, s, g, A));
    else BY_ROWS(mza, launch_next(k_damp_lap<R>, nb, 256, 0, s, g, A));
    // border planes for the Laplacian and the apply (vort_div_damp.f90:150, 208)
    if (dw) { HField f[1] = {{A.wdst, 4}}; OG_CHECK(halo_exchange_fields(C, HALO_W, f, 1, s)); }
    if (dm) { HField f[1] = {{A.mdst, 4}}; OG_CHECK(halo_exchange_fields(C, HALO_M, f, 1, s)); }
    return OLAMGPU_OK;
  };
  const int ld = div ? o.divh_damp_level : 0, lv = vor ? o.vort_damp_level : 0;
  for (int step = 0; step < std::max(ld, lv); ++step) OG_CHECK(run(step, step < ld, step < lv));
  if (!div && !vor && !setup) return OLAMGPU_OK;
  VtendArgs V{};
  V.vprog = d.jtv_prog.p; V.nv = d.nv_prog; V.src = src; V.dst = dst;
  V.vmc = y.vmc.p; V.rho = C.tp.rho.p; V.vc = y.vc.p;
  if (setup) {
    V.vmc0 = y.vmc0.p;
    V.rayf_cof = (o.rayf_cof && o.vc03d) ? y.rayf_cof.p : nullptr;
    V.vc03d = y.vc03d.p;
    V.krayf_bot = o.krayf_bot;
  }
  if (div) { V.fdivh = y.fdivh.p; V.dh = plane(y.div2d.p, wz, ld == 1 ? 1 : (ld - 1) % 2 + 1); }
  if (vor) {
    V.fvorth = y.fvorth.p; V.fvortl = y.fvortl.p;
    V.lpm = lv == 3 && !(g.flat && y.lpm_flat);
    V.vl = plane(y.vort2d.p, mz, lv == 1 ? 1 : (lv - 2) % 2 + 1);
    V.vh = plane(y.vort2d.p, mz, lv == 1 ? 1 : (lv - 1) % 2 + 1);
  }
  if (d.nv_prog > 0) { launch_next(k_vtend, cdiv((size_t)d.nv_prog * ((mza + 31) / 32), 8), 256, 0, s, g, V); OG_LAUNCHED(); }
  return OLAMGPU_OK;
}

static void launch_vel_t3d(Context& C, const Shaved& sh, cudaStream_t s) {
  const DevGrid& d = C.g;
  Dyn& y = C.dy;
  BY_ROWS(d.mza, launch_next(k_vel_t3d<R>, cdiv(d.nw_prog, 8), 256, 0, s, dynk(d), d.jtw_prog.p, d.nw_prog, C.tp.wc.p, y.vc.p, y.wno2.p,
                                                                 reinterpret_cast<const float4*>(y.ecv.p), y.vxe.p,
                                                                 y.vye.p, y.vze.p, sh));
}

int dyn_prog_wrtv_rk(int istp) {
  Context& C = ctx();
  if (!C.initialised) { set_error("olamgpu_init has not been called"); return OLAMGPU_E_STATE; }
  if (!C.dy.ready) { set_error("prog_wrtv_rk was not set up (see olamgpu_init's status)"); return OLAMGPU_E_STATE; }
  if (!C.have_state) { set_error("prog_wrtv_rk needs the state arrays registered at init"); return OLAMGPU_E_STATE; }
  const olamgpu_opts& o = C.opts;
  if (o.nrk_wrtv != 2 && o.nrk_wrtv != 3) { set_error("acoust_timestep_level must be 2 or 3"); return OLAMGPU_E_UNSUPPORTED; }
  if (C.halo.on && (!C.halo.dyn || o.ithil_monot > 0 || o.iwind_monot > 0)) {
    set_error("prog_wrtv_rk on a rank with a halo needs the V and M plans and no flux-corrected faces");
    return OLAMGPU_E_UNSUPPORTED;
  }
  cudaStream_t s = C.stream;
  OG_CHECK(ensure_dyn_buffers(C));
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL || !C.dy.uploaded) {
    OG_CHECK(dyn_state_to_device(DYN_IN_MASK, s));
    OG_CHECK(dyn_eddy_to_device(s));
  }
  C.dy.uploaded = true;
  const DevGrid& d = C.g;
  Dyn& y = C.dy;
  Transport& tp = C.tp;
  const DynK g = dynk(d);
  const int mza = d.mza;
  const unsigned nbw = cdiv((size_t)d.nw_prog * mza, 256), nbv = cdiv((size_t)d.nv_prog * mza, 256),
                 nbva = cdiv((size_t)d.nv_wadj * mza, 256);
  OG_PROF("prog_wrtv_rk", s);
  if (istp == 1 && (!o.divh_damp_short || !o.vort_damp_short)) {
    OG_PROF("v_tendency", s);
    OG_CHECK(v_tendency(C, !o.divh_damp_short, !o.vort_damp_short, false, y.vmt.p, y.vmt.p, o.dtlm, s));
  }
  SetupW sw{tp.rho.p, y.thil.p, y.wmc.p, y.thilt.p, y.vmxet.p, y.vmyet.p, y.vmzet.p, y.volt.p, y.rho0.p,
            y.rth0.p, y.wmc0.p, y.sh_th.p, y.sh_vx.p, y.sh_vy.p, y.sh_vz.p, y.rayf_cof.p, y.dn01d.p, y.th01d.p,
            o.krayf_bot};
  const bool rayleigh_th = o.rayf_cof && o.initial == 1;
  // with eddy diffusion the Rayleigh term on thil follows the eddy terms
  if (!rayleigh_th || y.eddy_on) sw.rayf_cof = nullptr;
  if (y.nve2_max > 0 && d.nw_prog > 0) {
    k_shaved_save<<<cdiv((size_t)d.nw_prog * y.nve2_max, 256), 256, 0, s>>>(g, d.jtw_prog.p, d.nw_prog, y.lve2.p,
                                                                             y.nve2_max, y.vxe.p, y.vye.p, y.vze.p,
                                                                             tp.rho.p, y.vm0.p);
    OG_LAUNCHED();
  }
  // Without eddy, Rayleigh or flux-corrected terms the column kernel forms
  // the start values, the tendencies and the W-face values itself.
  const bool lean = !y.eddy_on && !rayleigh_th && o.ithil_monot <= 0 && o.iwind_monot <= 0;
  if (!lean) { OG_PROF("setup_w", s); k_setup_w<<<nbw, 256, 0, s>>>(g, d.jtw_prog.p, d.nw_prog, sw); OG_LAUNCHED(); }
  if (y.eddy_on) {
    OG_PROF("eddy_columns", s);
    OG_CHECK(dyn_eddy_columns(C, rayleigh_th, s));
  }
  {
    OG_PROF("v_tendency", s);
    OG_CHECK(v_tendency(C, o.divh_damp_short != 0, o.vort_damp_short != 0, true, y.vmt.p, y.sh_vmt.p, o.dtsm, s));
  }
  // start values of the fields fluxes_wrtv_monot limits (prog_wrtv_rk.f90:186-198)
  const bool thil_monot = o.ithil_monot > 0, wind_monot = o.iwind_monot > 0;
  const size_t wzb = (size_t)mza * d.mwa * sizeof(float);
  if (thil_monot) {
    OG_CHECK(y.th0.alloc((size_t)mza * d.mwa));
    OG_CUDA(cudaMemcpyAsync(y.th0.p, y.thil.p, wzb, cudaMemcpyDeviceToDevice, s));
  }
  if (wind_monot) {
    DevBuf<float>* b0[3] = {&y.vx0, &y.vy0, &y.vz0};
    const float* src[3] = {y.vxe.p, y.vye.p, y.vze.p};
    for (int i = 0; i < 3; ++i) {
      OG_CHECK(b0[i]->alloc((size_t)mza * d.mwa));
      OG_CUDA(cudaMemcpyAsync(b0[i]->p, src[i], wzb, cudaMemcpyDeviceToDevice, s));
    }
  }

  const int nrk = o.nrk_wrtv;
  const double third = 1.0 / 3.0;
  const double xstg3[3] = {third, 0.5, 1.0}, xstg2[2] = {0.5, 1.0};
  for (int istage = 1; istage <= nrk; ++istage) {
    const double dt8 = (nrk <= 2 ? xstg2[istage - 1] : xstg3[istage - 1]) * o.dtsm;
    const float dts = (float)dt8;
    const int last = istage == nrk;
    // vmca = vmc arv, added to vmasc on the last stage: formed with the face
    // values by the face's upwind column, or over jtv_wadj where that may be
    // a column k_grad_upv4 does not run (a border column) and on a rank with
    // a halo, whose ring-1 columns have faces outside the table
    FaceFlux ffx{y.arv.p, y.vmca.p, last ? tp.vmasc.p : nullptr};
    if (C.halo.on || !d.v_closed) {
      ffx = FaceFlux{};
      OG_PROF("vmca", s);
      k_vmca<<<nbva, 256, 0, s>>>(g, d.jtv_wadj.p, d.nv_wadj, y.vmc.p, y.arv.p, y.vmca.p, tp.vmasc.p, last);
      OG_LAUNCHED();
    }
    Four f{{y.thil.p, y.vxe.p, y.vye.p, y.vze.p}};
    // fields by reconstruction order: thil has thil_horiz_adv_order, the
    // winds wind_horiz_adv_order (order 1: no gradient)
    const int ordf[4] = {o.thil_horiz_adv_order, o.wind_horiz_adv_order, o.wind_horiz_adv_order,
                         o.wind_horiz_adv_order};
    unsigned m2 = 0, m3 = 0;
    for (int q = 0; q < 4; ++q) { if (ordf[q] == 2) m2 |= 1u << q; if (ordf[q] >= 3) m3 |= 1u << q; }
    if (!lean) {
      OG_PROF("upw4", s);
      k_upw4<<<nbw, 256, 0, s>>>(g, d.jtw_prog.p, d.nw_prog, f, y.wmc.p, y.upw.p);
      OG_LAUNCHED();
    }
    {
      OG_PROF("grad_upv4", s);
      // every face of jtv_wadj is written by its upwind cell: the columns
      // (and on a rank with a halo, ring 1, whose gradients the reference
      // exchanges) hold the gradients of their own faces' upwind sides
      DynK gg = g;
      const int* gt = d.jtw_prog.p;
      int gn = d.nw_prog;
      if (C.halo.on) {
        gg.off_w = d.off_wwadj;
        gt = d.jtw_wadj.p;
        gn = d.nw_wadj;
      }
      const int nch = (mza + 31) / 32;
      const unsigned nbg = cdiv((size_t)gn * nch, 8);
      VSide vs{d.dxps.p, d.dyps.p, d.xx0_v.p, d.xy0_v.p, d.yy0_v.p};
      float4* upv = reinterpret_cast<float4*>(y.upv.p);
      const unsigned plain = 0xFu & ~(m2 | m3);
      if (m2 || plain) {
        if (m2 == 0xFu) launch_next(k_grad_upv4<2, true>, nbg, 256, 0, s, gg, gt, gn, nch, f, m2, plain, d.xy_hu.p, vs, y.vmc.p, upv, ffx);
        else launch_next(k_grad_upv4<2, false>, nbg, 256, 0, s, gg, gt, gn, nch, f, m2, plain, d.xy_hu.p, vs, y.vmc.p, upv, ffx);
        OG_LAUNCHED();
        ffx = FaceFlux{};   // once a stage
      }
      if (m3) {
        launch_next(k_grad_upv4<3, false>, nbg, 256, 0, s, gg, gt, gn, nch, f, m3, 0u, d.xy_hu.p, vs, y.vmc.p, upv, ffx);
        OG_LAUNCHED();
      }
    }
    // last stage: flux-corrected face values replace those of the limited fields (370-399)
    if (last && thil_monot) {
      OG_PROF("monot_faces", s);
      OG_CHECK(dyn_monot_faces(C, 0, y.thil.p, y.th0.p, y.sh_th.p, dts, o.thil_horiz_adv_order, s));
    }
    if (last && wind_monot) {
      OG_PROF("monot_faces", s);
      OG_CHECK(dyn_monot_faces(C, 1, y.vxe.p, y.vx0.p, y.sh_vx.p, dts, o.wind_horiz_adv_order, s));
      OG_CHECK(dyn_monot_faces(C, 2, y.vye.p, y.vy0.p, y.sh_vy.p, dts, o.wind_horiz_adv_order, s));
      OG_CHECK(dyn_monot_faces(C, 3, y.vze.p, y.vz0.p, y.sh_vz.p, dts, o.wind_horiz_adv_order, s));
    }
    WrtArgs A;
    A.istage = istage; A.nrk = nrk; A.dt8 = dt8; A.dts = dts; A.fcoriol = o.fcoriol;
    A.fr = (double)0.70f;
    const float cpocv = 1004.f / 717.f;
    A.pc2 = A.fr * (double)cpocv;
    A.pc3 = A.fr * (double)cpocv;
    A.rocv = (1004.f - 717.f) / 717.f;
    A.c8 = dts * (float)A.pc2;
    A.c9 = -dts * dts * (float)A.fr;
    A.prog = d.jtw_prog.p; A.nprog = d.nw_prog;
    A.vmca = y.vmca.p; A.upv = reinterpret_cast<const float4*>(y.upv.p); A.upw = y.upw.p;
    A.sh_th = lean ? y.thilt.p : y.sh_th.p; A.sh_vx = lean ? y.vmxet.p : y.sh_vx.p;
    A.sh_vy = lean ? y.vmyet.p : y.sh_vy.p; A.sh_vz = lean ? y.vmzet.p : y.sh_vz.p;
    A.rk_vx = y.rk_vx.p; A.rk_vy = y.rk_vy.p; A.rk_vz = y.rk_vz.p;
    A.rho = tp.rho.p; A.press = y.press.p; A.rho0 = y.rho0.p; A.rth0 = y.rth0.p;
    A.thil = y.thil.p; A.wc = tp.wc.p; A.wmc = y.wmc.p; A.wmc0 = y.wmc0.p; A.vxe = y.vxe.p; A.vye = y.vye.p;
    A.vze = y.vze.p;
    A.wmasc = tp.wmasc.p; A.alpha_press = y.alpha_press.p; A.pwfac = y.pwfac.p;
    A.volt = y.volt.p; A.volwi = y.volwi.p; A.arw = y.arw.p; A.wn = y.wn.p;
    A.gdz_wgtm8 = y.gdz_wgtm8.p; A.gdz_wgtp8 = y.gdz_wgtp8.p; A.gdz_wgtm = y.gdz_wgtm.p; A.gdz_wgtp = y.gdz_wgtp.p;
    A.zwgt_bot8 = y.zwgt_bot8.p; A.zwgt_top8 = y.zwgt_top8.p; A.b20 = y.b20.p;
    {
      OG_PROF("wrt_begs", s);
      BY_ROWS(mza, {
        constexpr int cols = WRT_COLS(R);
        const size_t smem = (size_t)cols * ((R == 1 ? 224 : 128 * R) + 4 * mza) * sizeof(double);   // 11.2 KB or less
        const unsigned nb = cdiv(d.nw_prog, cols);
        if (lean) launch_next(k_wrt_begs<R, true>, nb, 32 * R * cols, smem, s, g, A);
        else launch_next(k_wrt_begs<R, false>, nb, 32 * R * cols, smem, s, g, A);
      });
    }
    if (C.halo.on) {
      // prog_wrtv_rk.f90:418-429: what prog_v_begs reads at border V points
      OG_PROF("halo_exchange", s);
      HField f5[5] = {{y.press.p, 8}, {tp.rho.p, 8}, {y.rk_vx.p, 4}, {y.rk_vy.p, 4}, {y.rk_vz.p, 4}};
      OG_CHECK(halo_exchange_fields(C, HALO_W, f5, 5, s));
    }
    {
      OG_PROF("prog_v", s);
      launch_next(k_prog_v, nbv, 256, 0, s, g, d.jtv_prog.p, d.nv_prog, dts, y.vmc0.p, y.sh_vmt.p, y.press.p, y.pvfac.p,
                                   y.vn.p, y.rk_vx.p, y.rk_vy.p, y.rk_vz.p, y.volvi.p, tp.rho.p, y.vmc.p, y.vc.p);
      OG_LAUNCHED();
    }
    if (C.halo.on) {   // prog_wrtv_rk.f90:442-447
      OG_PROF("halo_exchange", s);
      HField f2[2] = {{y.vmc.p, 4}, {y.vc.p, 4}};
      OG_CHECK(halo_exchange_fields(C, HALO_V, f2, 2, s));
    }
    {
      OG_PROF("vel_t3d", s);
      launch_vel_t3d(C, shaved_args(y, tp, 1, dts), s);
    }
    if (C.halo.on) {   // prog_wrtv_rk.f90:464-472
      OG_PROF("halo_exchange", s);
      HField f6[6] = {{y.vxe.p, 4}, {y.vye.p, 4}, {y.vze.p, 4}, {y.wmc.p, 4}, {tp.wc.p, 4}, {y.thil.p, 4}};
      OG_CHECK(halo_exchange_fields(C, HALO_W, f6, 6, s));
    }
  }
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) {
    OG_CHECK(dyn_state_to_host(DYN_OUT_MASK, s));
    OG_CUDA(cudaStreamSynchronize(s));
  }
  OG_CUDA(cudaGetLastError());
  return OLAMGPU_OK;
}

int dyn_tend0(float* rho_old_host) {
  Context& C = ctx();
  if (!C.initialised || !C.dy.ready || !C.have_state) { set_error("tend0 before init"); return OLAMGPU_E_STATE; }
  cudaStream_t s = C.stream;
  OG_CHECK(ensure_dyn_buffers(C));
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) {
    // the kernels write levels k >= lpw only: the rest of each array it
    // returns keeps the caller's values
    OG_CHECK(dyn_state_to_device(OLAMGPU_F_RHO | OLAMGPU_F_TEND | OLAMGPU_F_VMASC | OLAMGPU_F_WMASC, s));
    if (rho_old_host)
      OG_CUDA(cudaMemcpyAsync(C.tp.rho_old.p, rho_old_host, (size_t)C.g.mza * C.g.mwa * 4, cudaMemcpyHostToDevice, s));
  } else if (!C.dy.uploaded) { OG_CHECK(dyn_state_to_device(DYN_IN_MASK, s)); C.dy.uploaded = true; }
  const DynK g = dynk(C.g);
  Dyn& y = C.dy;
  Transport& tp = C.tp;
  launch_next(k_tend0_w, cdiv((size_t)(C.g.mwa - 1) * C.g.mza, 256), 256, 0, s, g, y.thilt.p, y.vmxet.p, y.vmyet.p,
                                                                      y.vmzet.p, tp.rho.p, tp.rho_old.p,
                                                                      tp.wmasc.p);
  launch_next(k_tend0_v, cdiv((size_t)(C.g.mva - 1) * C.g.mza, 256), 256, 0, s, g, y.vmt.p, tp.vmasc.p);
  OG_LAUNCHED(); OG_LAUNCHED();
  // scalar tendencies var_t = 0 for k >= lpw (the device copies)
  // (a window's adjoint lends the per-tracer arrays' memory out while it
  // runs the dynamics again: there are none to clear then)
  for (int n = 0; n < C.tr.n; ++n)
    if (C.tr.t[n].p) OG_CUDA(cudaMemsetAsync(C.tr.t[n].p, 0, (size_t)C.g.mza * C.g.mwa * 4, s));
  if (C.tr.q_valid && C.tr.qt.p) OG_CUDA(cudaMemsetAsync(C.tr.qt.p, 0, C.tr.qt.bytes(), s));
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) {
    OG_CHECK(dyn_state_to_host(OLAMGPU_F_TEND | OLAMGPU_F_VMASC | OLAMGPU_F_WMASC, s));
    if (rho_old_host)
      OG_CUDA(cudaMemcpyAsync(rho_old_host, tp.rho_old.p, (size_t)C.g.mza * C.g.mwa * 4, cudaMemcpyDeviceToHost, s));
    for (int n = 0; n < C.tr.n; ++n)
      OG_CUDA(cudaMemcpyAsync(C.tr.h_t[n], C.tr.t[n].p, (size_t)C.g.mza * C.g.mwa * 4, cudaMemcpyDeviceToHost, s));
    OG_CUDA(cudaStreamSynchronize(s));
  }
  return OLAMGPU_OK;
}

int dyn_timeavg_momsc() {
  Context& C = ctx();
  if (!C.initialised || !C.dy.ready) { set_error("timeavg_momsc before init"); return OLAMGPU_E_STATE; }
  if (C.opts.nacoust <= 1) return OLAMGPU_OK;
  cudaStream_t s = C.stream;
  OG_CHECK(ensure_dyn_buffers(C));
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) OG_CHECK(dyn_state_to_device(OLAMGPU_F_VMASC | OLAMGPU_F_WMASC, s));
  else if (!C.dy.uploaded) { OG_CHECK(dyn_state_to_device(DYN_IN_MASK, s)); C.dy.uploaded = true; }
  const DynK g = dynk(C.g);
  const float a = (float)C.opts.nacoust;
  launch_next(k_timeavg_v, cdiv((size_t)C.g.nv_wadj * C.g.mza, 256), 256, 0, s, g, C.g.jtv_wadj.p, C.g.nv_wadj, a, C.tp.vmasc.p);
  launch_next(k_timeavg_w, cdiv((size_t)C.g.nw_prog * C.g.mza, 256), 256, 0, s, g, C.g.jtw_prog.p, C.g.nw_prog, a, C.tp.wmasc.p);
  OG_LAUNCHED(); OG_LAUNCHED();
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) {
    OG_CHECK(dyn_state_to_host(OLAMGPU_F_VMASC | OLAMGPU_F_WMASC, s));
    OG_CUDA(cudaStreamSynchronize(s));
  }
  return OLAMGPU_OK;
}

// diagvel_t3d (vel_t3d.f90:7-35): vel_t3d_hex over jtw_prog
int dyn_diagvel_t3d() {
  Context& C = ctx();
  if (!C.initialised || !C.dy.ready || !C.have_state) { set_error("diagvel_t3d before init"); return OLAMGPU_E_STATE; }
  cudaStream_t s = C.stream;
  OG_CHECK(ensure_dyn_buffers(C));
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) OG_CHECK(dyn_state_to_device(OLAMGPU_F_WC | OLAMGPU_F_VC | OLAMGPU_F_VXE, s));
  else if (!C.dy.uploaded) { OG_CHECK(dyn_state_to_device(DYN_IN_MASK, s)); C.dy.uploaded = true; }
  const DevGrid& d = C.g;
  Dyn& y = C.dy;
  if (d.nw_prog > 0) launch_vel_t3d(C, shaved_args(y, C.tp, 0, 0.f), s);
  if (C.coherence == OLAMGPU_SYNC_EACH_CALL) {
    OG_CHECK(dyn_state_to_host(OLAMGPU_F_VXE, s));
    OG_CUDA(cudaStreamSynchronize(s));
  }
  OG_CUDA(cudaGetLastError());
  return OLAMGPU_OK;
}

void dyn_release() {
  Dyn& y = ctx().dy;
  DevBuf<double>* d8[] = {&y.press, &y.rho0, &y.rth0, &y.volt, &y.zwgt_top8, &y.zwgt_bot8, &y.gdz_wgtm8, &y.gdz_wgtp8};
  for (auto* b : d8) b->release();
  DevBuf<float>* f[] = {&y.thil, &y.wmc, &y.vxe, &y.vye, &y.vze, &y.vmc, &y.vc, &y.alpha_press, &y.pwfac,
                        &y.pvfac, &y.thilt, &y.vmxet, &y.vmyet, &y.vmzet, &y.vmt, &y.wmc0, &y.vmc0, &y.vmca,
                        &y.sh_th, &y.sh_vx, &y.sh_vy, &y.sh_vz, &y.sh_vmt, &y.rk_vx, &y.rk_vy,
                        &y.rk_vz, &y.upw, &y.upv, &y.div2d, &y.fdivh, &y.vort2d, &y.fvorth, &y.fvortl,
                        &y.vfact, &y.arv, &y.arw, &y.volwi, &y.volvi, &y.wn, &y.wno2, &y.vn, &y.ecv,
                        &y.gdz_wgtm, &y.gdz_wgtp, &y.dniv, &y.dniu, &y.dnv, &y.arw0, &y.arm0, &y.zfacit,
                        &y.dzit, &y.xx_yy, &y.xx_yy_m, &y.b20, &y.rayf_cof, &y.dn01d, &y.th01d, &y.vc03d,
                        &y.th0, &y.vx0, &y.vy0, &y.vz0, &y.m_scpt, &y.m_gx, &y.m_hiw, &y.m_sfw, &y.m_hiv,
                        &y.m_sfv, &y.m_sin, &y.m_sout};
  for (auto* b : f) b->release();
  y.lve2.release();
  y.vm0.release();
  dyn_eddy_release();
  y = Dyn();
}

}  // namespace olamgpu
