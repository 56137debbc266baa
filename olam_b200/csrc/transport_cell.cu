// transport_cell.cu -- update_scalar as passes over cells, a thread per
// (column, level, tracer quad).
//
// Restates omodel/scalar_transport_rk.F90 in two passes for an unlimited
// stage and three for a limited one:
//   k_face    grad_t2d / grad_t2d_quadratic (grad_lib.f90:236-341) and the
//             upwind V-face values (scalar_v_column 474-534,
//             scalar_vflux_monot 749-832, scalar_vflux_pd 1215-1285): a cell
//             forms its gradients in registers and writes the values of the
//             faces it is upwind of, so no gradient plane goes through memory
//             and each face is written once
//   k_scale   the limiters' scale factors (scalar_wflux_and_scales_monot
//             835-1022, scalar_wflux_and_scale_pd 1288-1414)
//   k_update  grad_z_quadratic (grad_lib.f90:166-229), scalar_w_column
//             (537-612) or the renormalised faces and the tendency of the
//             limited stage (711-724, 1025-1078, 1177-1190, 1417-1469)
// None of them has a recurrence in k, so the levels of a column run in
// parallel, and a limited face's low-order value (scp0 of the upwind cell) is
// read again instead of being stored.
//
// They run one tracer in OLAM's (mza, n) layout (V = 1), the batched layout
// with few tracers, where the tiled kernel leaves lanes idle (V = 4 tracers
// per thread), and the limited last stage of the batched layout.
//
// Bound: the neighbour gathers through L1 and L2, then HBM (a face value is
// written once and read by two cells: 44 B per tracer cell unlimited).
//
// Device level index kd = Fortran k - 1.
#include <algorithm>
#include <type_traits>

#include "transport_kernels.cuh"

namespace olamgpu {

struct CellArgs {
  int mza, mwa;
  int ncol, nq, nch;                // columns, tracer quads (V = 1: 1), item chunks per column
  int off, flat;                    // cols is off, off + 1, ... (-1: not); every floor is level 1
  const int* __restrict__ cols;
  const int* __restrict__ npoly;
  const int* __restrict__ lpw;
  const int4* __restrict__ edge;    // EDGE_W words per edge
  const float4* __restrict__ edge3; // order 3: EDGE3_W words per edge
  const float* vmasc;
  const float* wmasc;
  const float* __restrict__ volti;
  const float* __restrict__ a_w;    // bounded or unbounded, as the pass needs
  const float* rhos;
  const float* ff;     // (mwa, nrk), NULL: every column explicit
  const int* __restrict__ mode;     // limited stage: mode of each tracer
  const float* S;
  const float* S0;
  const float* SCT;
  float* out;
  float* face;         // (mva, mza, nq V)
  float* scale;        // (mwa, mza, nq V), two planes with the monotonic limiter
  int ld, nt;                       // row length of S, S0, SCT, out; tracers
  int istage, nrk;
  float dtr;
};

template <int V>
struct Vec { float v[V]; };

template <int V>
__device__ __forceinline__ Vec<V> ldv(const float* p) {
  Vec<V> r;
  if constexpr (V == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int V>
__device__ __forceinline__ void stv(float* p, const Vec<V>& r) {
  if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else *p = r.v[0];
}
template <int V>
__device__ __forceinline__ Vec<V> zerov() {
  Vec<V> r;
#pragma unroll
  for (int c = 0; c < V; ++c) r.v[c] = 0.f;
  return r;
}
// acc + w x, two tracers per instruction
template <int V>
__device__ __forceinline__ Vec<V> fmav(float w, const Vec<V>& x, const Vec<V>& acc) {
  Vec<V> r;
  if constexpr (V == 4) {
    const float2 w2 = make_float2(w, w);
    const float2 a = __ffma2_rn(w2, make_float2(x.v[0], x.v[1]), make_float2(acc.v[0], acc.v[1]));
    const float2 b = __ffma2_rn(w2, make_float2(x.v[2], x.v[3]), make_float2(acc.v[2], acc.v[3]));
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = b.x; r.v[3] = b.y;
  } else {
    r.v[0] = fmaf(w, x.v[0], acc.v[0]);
  }
  return r;
}
template <int V>
__device__ __forceinline__ Vec<V> subv(const Vec<V>& x, const Vec<V>& y) { return fmav<V>(-1.f, y, x); }

// a warp's chunk of 32 items of one column: item -> (level, quad).  OFF: the
// type of element offsets, unsigned where every array has fewer than 2^32
// elements (half the address instructions of size_t).
#define CELL_ITEM(A)                                                                      \
  const unsigned warp_ = blockIdx.x * 8u + (threadIdx.x >> 5);                            \
  const unsigned j_ = warp_ / (unsigned)A.nch;                                            \
  if (j_ >= (unsigned)A.ncol) return;                                                     \
  const unsigned i_ = (warp_ - j_ * (unsigned)A.nch) * 32u + (threadIdx.x & 31u);         \
  const int kd = (int)(i_ / (unsigned)A.nq), q = (int)(i_ - (unsigned)kd * (unsigned)A.nq); \
  const int iw = A.off >= 0 ? A.off + (int)j_ : __ldg(A.cols + j_);                       \
  const int mza = A.mza;                                                                  \
  grid_wait();                                                                            \
  if (kd >= mza) return;
#define CELL_FLOOR(A) (A.flat ? 1 : __ldg(A.lpw + iw))

// per-tracer modes of a quad; tracers past the count are PLAIN
template <int V>
__device__ __forceinline__ void quad_modes(const CellArgs& A, int q, int (&m)[V]) {
#pragma unroll
  for (int c = 0; c < V; ++c) m[c] = V * q + c < A.nt ? __ldg(A.mode + V * q + c) : MODE_PLAIN;
}

// The edges of a column go in batches of N: every load of a batch is issued
// before any of its values is used, and a closed edge (a face under ground, a
// pentagon's sixth edge) is a predicated load, not a branch -- a warp waits
// once per batch instead of once per edge.  A column has six edges (OLAM
// allows seven).
#define CELL_EDGES(np, body)                 \
  body(std::integral_constant<int, 6>(), 0); \
  if (np > 6) body(std::integral_constant<int, 1>(), 6);
#define CELL_EDGES2(np, body)                \
  body(std::integral_constant<int, 2>(), 0); \
  body(std::integral_constant<int, 2>(), 2); \
  body(std::integral_constant<int, 2>(), 4); \
  if (np > 6) body(std::integral_constant<int, 1>(), 6);
#define CELL_EDGES3(np, body)                \
  body(std::integral_constant<int, 3>(), 0); \
  body(std::integral_constant<int, 3>(), 3); \
  if (np > 6) body(std::integral_constant<int, 1>(), 6);

// LIM: the limited last stage -- the face array holds, for a limited tracer,
// the high-order correction (value minus scp0 of the upwind cell)
template <int V, int ORDER, bool LIM, typename OFF>
__global__ void __launch_bounds__(256, ORDER == 2 ? 4 : 3) k_face(CellArgs A) {
  CELL_ITEM(A);
  constexpr int M = ORDER == 2 ? 2 : 5;
  const int np = __ldg(A.npoly + iw);
  const OFF row = (OFF)A.ld;
  const float* S = A.S + V * q;
  const OFF x0 = ((OFF)iw * mza + kd) * row;
  const Vec<V> s0 = ldv<V>(S + x0);
  Vec<V> lo = zerov<V>();
  if (LIM) {
    int md[V];
    quad_modes<V>(A, q, md);
    lo = ldv<V>(A.S0 + x0 + V * q);
#pragma unroll
    for (int c = 0; c < V; ++c) if (md[c] == MODE_PLAIN) lo.v[c] = 0.f;
  }
  Vec<V> g[M];
#pragma unroll
  for (int m = 0; m < M; ++m) g[m] = zerov<V>();
  const int4* E = A.edge + (size_t)iw * (7 * EDGE_W / 4);
  const float4* E3 = A.edge3 + (size_t)iw * (7 * EDGE3_W / 4);
  auto gradient = [&](auto cnt, int n0) {
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    Vec<V> x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));   // neighbour, face | side << 31, floor, dirv
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = s0;                                                  // a closed edge adds nothing
      if (kd >= e[i].z) x[i] = ldv<V>(S + ((OFF)e[i].x * mza + kd) * row);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float w[M];
      if (ORDER == 2) {
        const int4 b = __ldg(E + 2 * (n0 + i) + 1);               // gradient weights, face offsets
        w[0] = __int_as_float(b.x);
        w[1] = __int_as_float(b.y);
      } else {
        const float4 a = __ldg(E3 + 3 * (n0 + i)), b = __ldg(E3 + 3 * (n0 + i) + 1);
        w[0] = a.x; w[1] = a.y; w[M - 3] = a.z; w[M - 2] = a.w; w[M - 1] = b.x;
      }
      const Vec<V> d = subv<V>(x[i], s0);
#pragma unroll
      for (int m = 0; m < M; ++m) g[m] = fmav<V>(w[m], d, g[m]);
    }
  };
  if constexpr (ORDER == 2) { CELL_EDGES(np, gradient); }
  else { CELL_EDGES3(np, gradient); }
  auto faces = [&](auto cnt, int n0) {
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    float vm[N];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));
#pragma unroll
    for (int i = 0; i < N; ++i)
      vm[i] = kd >= e[i].z ? A.vmasc[(OFF)(e[i].y & 0x7fffffff) * mza + kd] : 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (kd < e[i].z || (vm[i] < 0.f) != (e[i].y < 0)) continue;  // closed, or the other cell is upwind
      float o[M];
      if (ORDER == 2) {
        const int4 b = __ldg(E + 2 * (n0 + i) + 1);
        o[0] = __int_as_float(b.z);
        o[1] = __int_as_float(b.w);
      } else {
        const float4 b = __ldg(E3 + 3 * (n0 + i) + 1), d = __ldg(E3 + 3 * (n0 + i) + 2);
        o[0] = b.y; o[1] = b.z; o[M - 3] = b.w; o[M - 2] = d.x; o[M - 1] = d.y;
      }
      Vec<V> v = s0;
#pragma unroll
      for (int m = 0; m < M; ++m) v = fmav<V>(o[m], g[m], v);
      if (LIM) v = subv<V>(v, lo);
      stv<V>(A.face + (((OFF)(e[i].y & 0x7fffffff) * mza + kd) * A.nq + q) * V, v);
    }
  };
  CELL_EDGES(np, faces);
}

// grad_z_quadratic's value at the face above level f from the upwind level
// lev (f + 1 where the air sinks, else f): its coefficients, and which of the
// level's two differences exist.  UNB: the unbounded coefficients with
// constant-gradient ends (monotonic limiter).
struct ZFace {
  bool down, has_up, has_dn;
  float c1, c2;
};
__device__ __forceinline__ ZFace zface(const float* a, int mza, int f, int kb, float w) {
  ZFace z;
  z.down = w < 0.f;
  const int lev = min(max(z.down ? f + 1 : f, 0), mza - 1);
  z.c1 = __ldg(a + lev + (z.down ? 0 : 2 * mza));
  z.c2 = __ldg(a + lev + (z.down ? mza : 3 * mza));
  z.has_up = lev <= mza - 2;
  z.has_dn = lev >= kb + 1;
  return z;
}
// sm1 .. s2: S(f-1) .. S(f+2)
template <bool UNB>
__device__ __forceinline__ float zvalue(const ZFace& z, float sm1, float s0, float s1, float s2) {
  const float c = z.down ? s1 : s0, lo = z.down ? s0 : sm1, hi = z.down ? s2 : s1;
  const float up = hi - c, dn = c - lo;
  const float dk = z.has_up ? up : (UNB ? dn : 0.f);
  const float dkm1 = z.has_dn ? dn : (UNB ? up : 0.f);
  return c + dk * z.c1 + dkm1 * z.c2;
}

// a field's rows kd-M .. kd+M of the column, the end levels repeating; base:
// the column's first element
template <int V, int M, typename OFF>
__device__ __forceinline__ void window(const float* p, OFF base, OFF row, int kd, int kb, int mza, Vec<V> (&w)[2 * M + 1]) {
#pragma unroll
  for (int m = 0; m < 2 * M + 1; ++m) w[m] = ldv<V>(p + (base + (OFF)min(max(kd - M + m, kb), mza - 1) * row));
}

// the vertical flux wm (lower face) - wp (upper face) of grad_z_quadratic's
// values as coefficients on S(kd-2 .. kd+2); they add up to wm - wp
__device__ __forceinline__ void zbeta(const float* a, int mza, int kd, int kb, float wm, float wp, float (&b)[5]) {
  const ZFace l = zface(a, mza, kd - 1, kb, wm), u = zface(a, mza, kd, kb, wp);
  // face value c + c1 (S(lev+1) - c) + c2 (c - S(lev-1)), c = S(lev)
  const float l1 = l.has_up ? l.c1 : 0.f, l2 = l.has_dn ? l.c2 : 0.f, u1 = u.has_up ? u.c1 : 0.f, u2 = u.has_dn ? u.c2 : 0.f;
  const float lm = -wm * l2, lc = wm * (1.f - l1 + l2), lp = wm * l1;
  const float um = wp * u2, uc = -wp * (1.f - u1 + u2), up = -wp * u1;
  const bool bot = kd == kb, top = kd == mza - 1;   // scp_upw(kb-1) = scp(kb), scp_upw(mza) = scp(mza)
  b[0] = bot || l.down ? 0.f : lm;
  b[1] = bot ? 0.f : (l.down ? lm : lc);
  b[2] = bot ? wm : (l.down ? lc : lp);
  b[3] = bot || !l.down ? 0.f : lp;
  b[4] = 0.f;
  b[1] += top || u.down ? 0.f : um;
  b[2] += top ? -wp : (u.down ? um : uc);
  b[3] += top ? 0.f : (u.down ? uc : up);
  b[4] += top || !u.down ? 0.f : up;
}

// an unlimited stage (scalar_w_column)
template <int V, typename OFF>
__global__ void __launch_bounds__(256) k_update(CellArgs A) {
  CELL_ITEM(A);
  const int kb = CELL_FLOOR(A);
  if (kd < kb) return;                                // written by the thread of level kb
  const int np = __ldg(A.npoly + iw);
  const float fexpl = A.ff ? 1.0f - A.ff[(size_t)iw * A.nrk + A.istage - 1] : 1.0f;
  const OFF row = (OFF)A.ld, cb = (OFF)iw * mza, x = cb + kd;
  const Vec<V> s00 = ldv<V>(A.S0 + V * q + x * row), tend = ldv<V>(A.SCT + V * q + x * row);
  Vec<V> w[5];
  window<V, 2, OFF>(A.S + V * q, cb * row, row, kd, kb, mza, w);
  const float wm = A.wmasc[x - 1], wp = A.wmasc[x];
  const float vt = __ldg(A.volti + x), rh = A.rhos[x];
  Vec<V> fd = zerov<V>();
  const int4* E = A.edge + (size_t)iw * (7 * EDGE_W / 4);
  auto edges = [&](auto cnt, int n0) {
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    float vm[N];
    Vec<V> up[N];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const OFF xv = (OFF)(e[i].y & 0x7fffffff) * mza + kd;
      vm[i] = 0.f;
      up[i] = s00;
      if (kd >= e[i].z) { vm[i] = A.vmasc[xv]; up[i] = ldv<V>(A.face + (xv * A.nq + q) * V); }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) fd = fmav<V>(__int_as_float(e[i].w) * vm[i], subv<V>(up[i], s00), fd);
  };
  CELL_EDGES(np, edges);
  // differences from scp0: the coefficients add up to the S0 term's
  float b[5];
  zbeta(A.a_w, mza, kd, kb, wm, wp, b);
  // The level two away on the downwind side of a face is not in the stencil:
  // its coefficient is zero, but a NaN there times zero would reach this cell.
  if (wm < 0.f || kd == kb) w[0] = s00;
  if (!(wp < 0.f) || kd == mza - 1) w[4] = s00;
#pragma unroll
  for (int m = 0; m < 5; ++m) fd = fmav<V>(fexpl * b[m], subv<V>(w[m], s00), fd);
  const Vec<V> o = fmav<V>(A.dtr / rh, fmav<V>(vt, fd, tend), s00);
  float* out = A.out + V * q;
  stv<V>(out + x * row, o);
  if (kd == kb)
    for (int k = 0; k < kb; ++k) stv<V>(out + (cb + k) * row, o);
}

// the vertical faces of a limited cell: low-order values and high-order
// corrections of the faces below (0) and above (1) level kd; s: S(kd-2 ..
// kd+2), z: scp0(kd-1 .. kd+1)
template <bool MONOT>
__device__ __forceinline__ void lim_faces(int mza, int kd, int kb, const ZFace& zl, const ZFace& zu,
                                          const float (&s)[5], const float (&z)[3], float (&lo)[2], float (&hi)[2]) {
  const float vl = zvalue<MONOT>(zl, s[0], s[1], s[2], s[3]), vu = zvalue<MONOT>(zu, s[1], s[2], s[3], s[4]);
  const float end = MONOT ? z[1] : s[2];
  lo[0] = kd == kb ? end : (zl.down ? z[1] : z[0]);
  hi[0] = kd == kb ? 0.f : vl - lo[0];
  lo[1] = kd == mza - 1 ? end : (zu.down ? z[2] : z[1]);
  hi[1] = kd == mza - 1 ? 0.f : vu - lo[1];
}

// scale factors of the limited stage: plane 0 the inflow (monotonic) or
// outflow (positive-definite) factor, plane 1 the monotonic outflow factor.
// The vertical faces come first, so that their nine rows are spent before the
// edges' values are loaded (80 registers, 24 warps an SM, against 128-163).
template <int V, bool MONOT, typename OFF>
__global__ void __launch_bounds__(256, 3) k_scale(CellArgs A) {
  CELL_ITEM(A);
  const int kb = CELL_FLOOR(A);
  if (kd < kb) return;
  const int np = __ldg(A.npoly + iw);
  const float fimpl = A.ff[(size_t)iw * A.nrk + A.istage - 1], fexpl = 1.0f - fimpl;
  const bool impl = fimpl > .001f;
  const OFF row = (OFF)A.ld, cb = (OFF)iw * mza, x = cb + kd;
  const float* S0 = A.S0 + V * q;
  const float wm = A.wmasc[x - 1], wp = A.wmasc[x];
  const float rh = A.rhos[x], vt = __ldg(A.volti + x);
  float fl[V], fin[V], fout[V], smax[V], smin[V];
  Vec<V> s00;
  {
    Vec<V> w[5], z[3];
    window<V, 2, OFF>(A.S + V * q, cb * row, row, kd, kb, mza, w);
    window<V, 1, OFF>(S0, cb * row, row, kd, kb, mza, z);
    const ZFace zl = zface(A.a_w, mza, kd - 1, kb, wm), zu = zface(A.a_w, mza, kd, kb, wp);
    s00 = z[1];
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const float s[5] = {w[0].v[c], w[1].v[c], w[2].v[c], w[3].v[c], w[4].v[c]};
      const float z3[3] = {z[0].v[c], z[1].v[c], z[2].v[c]};
      smax[c] = smin[c] = z3[1];
      if (MONOT) {
        if (kd >= kb + 1 && wm > 0.f) { smax[c] = fmaxf(smax[c], z3[0]); smin[c] = fminf(smin[c], z3[0]); }
        if (kd <= mza - 2 && wp < 0.f) { smax[c] = fmaxf(smax[c], z3[2]); smin[c] = fminf(smin[c], z3[2]); }
      }
      float lo[2], hi[2];
      lim_faces<MONOT>(mza, kd, kb, zl, zu, s, z3, lo, hi);
      // 0 at the column's ends
      const float sfm = kd == kb ? 0.f : fexpl * wm * hi[0], sfp = kd == mza - 1 ? 0.f : fexpl * wp * hi[1];
      fin[c] = fmaxf(sfm, 0.f) - fminf(sfp, 0.f);
      fout[c] = fminf(sfm, 0.f) - fmaxf(sfp, 0.f);
      const float lv = wm * (lo[0] - z3[1]) - wp * (lo[1] - z3[1]);
      fl[c] = impl ? fexpl * lv + fimpl * z3[1] * (wp - wm) : lv;
    }
  }
  const int4* E = A.edge + (size_t)iw * (7 * EDGE_W / 4);
  auto edges = [&](auto cnt, int n0) {
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    float vm[N];
    Vec<V> hv[N], sn[N];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const OFF xv = (OFF)(e[i].y & 0x7fffffff) * mza + kd;
      vm[i] = 0.f;
      hv[i] = zerov<V>();
      sn[i] = s00;
      if (kd >= e[i].z) {
        vm[i] = A.vmasc[xv];
        hv[i] = ldv<V>(A.face + (xv * A.nq + q) * V);
        sn[i] = ldv<V>(S0 + ((OFF)e[i].x * mza + kd) * row);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float dv = __int_as_float(e[i].w);
      // the neighbour is upwind: its scp0 is the face's low-order value
      const bool far = kd >= e[i].z && (vm[i] < 0.f) != (e[i].y < 0);
      const bool inflow = MONOT && dv * vm[i] > 0.f;
#pragma unroll
      for (int c = 0; c < V; ++c) {
        if (far) fl[c] = fl[c] + dv * vm[i] * (sn[i].v[c] - s00.v[c]);
        const float sf = dv * (vm[i] * hv[i].v[c]);
        if (MONOT) fin[c] = fin[c] + fmaxf(sf, 0.f);
        fout[c] = fout[c] + fminf(sf, 0.f);
        if (inflow) { smax[c] = fmaxf(smax[c], sn[i].v[c]); smin[c] = fminf(smin[c], sn[i].v[c]); }
      }
    }
  };
  CELL_EDGES3(np, edges);
  const float dtrp = (1.0f + kEps1) * A.dtr;
  // the monotonic bounds of an implicit column count its mass change
  const float rhb = MONOT && impl ? rh + A.dtr * vt * (fimpl * (wp - wm)) : rh;
  Vec<V> r0, r1;
#pragma unroll
  for (int c = 0; c < V; ++c) {
    const float low = s00.v[c] * rh + A.dtr * vt * fl[c];
    if (MONOT) {
      const float flux_in = fmaxf(dtrp * vt * fin[c], kEps0);
      const float flux_out = fminf(dtrp * vt * fout[c], -kEps0);
      const float epsr = kEps1 * fabsf(low);
      const float sc_in = fmaxf(rhb * smax[c] - (low + epsr) - kEps0, 0.f);
      const float sc_out = fminf(rhb * smin[c] - (low - epsr) + kEps0, 0.f);
      r0.v[c] = fminf(1.f, sc_in / fmaxf(flux_in, 0.01f * sc_in));
      r1.v[c] = fminf(1.f, sc_out / fminf(flux_out, 0.01f * sc_out));
    } else {
      const float flux_out = fmaxf(-dtrp * vt * fout[c], kEps0);
      const float sc_out = fmaxf((1.0f - kEps1) * low - kEps0, 0.f);
      r0.v[c] = fminf(1.f, sc_out / fmaxf(flux_out, 0.01f * sc_out));
    }
  }
  float* o = A.scale + (x * A.nq + q) * V;
  stv<V>(o, r0);
  if (MONOT) stv<V>(o + (size_t)A.mwa * mza * A.nq * V, r1);
}

// the update of the limited stage: the scaled faces and the tendency.  PLAIN
// tracers of the group (without pdef under the positive-definite option)
// take the unlimited update.
template <int V, bool MONOT, typename OFF>
__global__ void __launch_bounds__(256, 3) k_update_lim(CellArgs A) {
  CELL_ITEM(A);
  const int kb = CELL_FLOOR(A);
  if (kd < kb) return;
  const int np = __ldg(A.npoly + iw);
  const float fimpl = A.ff[(size_t)iw * A.nrk + A.istage - 1], fexpl = 1.0f - fimpl;
  const bool impl = fimpl > .001f;
  const OFF row = (OFF)A.ld, cb = (OFF)iw * mza, x = cb + kd;
  const size_t plane = (size_t)A.mwa * mza * A.nq * V;
  const float* S0 = A.S0 + V * q;
  const float* sc = A.scale + (size_t)V * q;
  const OFF srow = (OFF)A.nq * V;
  unsigned pl = 0;                                     // the quad's PLAIN tracers
  if (!MONOT) {
    int md[V];
    quad_modes<V>(A, q, md);
#pragma unroll
    for (int c = 0; c < V; ++c) if (md[c] == MODE_PLAIN) pl |= 1u << c;
  }
  const float wm = A.wmasc[x - 1], wp = A.wmasc[x];
  const float vt = __ldg(A.volti + x), rh = A.rhos[x];
  Vec<V> s00, a0, b0;                                  // scp0 and the factors of this cell
  float fd[V];
  {
    Vec<V> w[5], z[3], a[3], b[3];
    window<V, 2, OFF>(A.S + V * q, cb * row, row, kd, kb, mza, w);
    window<V, 1, OFF>(S0, cb * row, row, kd, kb, mza, z);
    window<V, 1, OFF>(sc, cb * srow, srow, kd, kb, mza, a);
    if (MONOT) window<V, 1, OFF>(sc + plane, cb * srow, srow, kd, kb, mza, b);
    const ZFace zl = zface(A.a_w, mza, kd - 1, kb, wm), zu = zface(A.a_w, mza, kd, kb, wp);
    s00 = z[1];
    a0 = a[1];
    b0 = MONOT ? b[1] : a[1];
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const float s[5] = {w[0].v[c], w[1].v[c], w[2].v[c], w[3].v[c], w[4].v[c]};
      const float z3[3] = {z[0].v[c], z[1].v[c], z[2].v[c]};
      float lo[2], hi[2];
      lim_faces<MONOT>(mza, kd, kb, zl, zu, s, z3, lo, hi);
      const bool bm = fexpl * wm * hi[0] < 0.f, bp = fexpl * wp * hi[1] < 0.f;
      float cm, cp;
      if (MONOT) {
        cm = bm ? fminf(a[0].v[c], b[1].v[c]) : fminf(a[1].v[c], b[0].v[c]);
        cp = bp ? fminf(a[1].v[c], b[2].v[c]) : fminf(a[2].v[c], b[1].v[c]);
      } else {
        cm = bm ? a[1].v[c] : a[0].v[c];
        cp = bp ? a[2].v[c] : a[1].v[c];
      }
      float ul = kd == kb ? lo[0] : lo[0] + hi[0] * cm;
      float uu = kd == mza - 1 ? lo[1] : lo[1] + hi[1] * cp;
      if (!MONOT && ((pl >> c) & 1u)) {
        ul = kd == kb ? s[2] : zvalue<false>(zl, s[0], s[1], s[2], s[3]);
        uu = kd == mza - 1 ? s[2] : zvalue<false>(zu, s[1], s[2], s[3], s[4]);
      }
      const float f = wm * (ul - z3[1]) - wp * (uu - z3[1]);
      fd[c] = impl || ((pl >> c) & 1u) ? fexpl * f : f;
    }
  }
  const int4* E = A.edge + (size_t)iw * (7 * EDGE_W / 4);
  auto edges = [&](auto cnt, int n0) {   // two or three at a time: five or four quads each
    constexpr int N = decltype(cnt)::value;
    int4 e[N];
    float vm[N];
    Vec<V> hv[N], sn[N], an[N], bn[N];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = __ldg(E + 2 * (n0 + i));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const OFF xv = (OFF)(e[i].y & 0x7fffffff) * mza + kd, xn = (OFF)e[i].x * mza + kd;
      vm[i] = 0.f;
      hv[i] = an[i] = bn[i] = zerov<V>();
      sn[i] = s00;
      if (kd >= e[i].z) {
        vm[i] = A.vmasc[xv];
        hv[i] = ldv<V>(A.face + (xv * A.nq + q) * V);
        an[i] = ldv<V>(sc + xn * srow);
        if (MONOT) bn[i] = ldv<V>(sc + plane + xn * srow);
        // scp0 of the neighbour where it is upwind
        if ((vm[i] < 0.f) != (e[i].y < 0)) sn[i] = ldv<V>(S0 + xn * row);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const bool open = kd >= e[i].z;
      const float f = __int_as_float(e[i].w) * vm[i];
      const bool second = e[i].y < 0;                  // this cell is side 2 of the face
#pragma unroll
      for (int c = 0; c < V; ++c) {
        // the correction runs from side 1 to side 2, or back where it is negative
        const bool back = vm[i] * hv[i].v[c] < 0.f;
        const bool from_here = back == second;         // this cell gives the corrected flux
        const float s = MONOT ? (from_here ? fminf(an[i].v[c], b0.v[c]) : fminf(a0.v[c], bn[i].v[c]))
                              : (from_here ? a0.v[c] : an[i].v[c]);
        const float up = (pl >> c) & 1u ? hv[i].v[c] : sn[i].v[c] + hv[i].v[c] * s;
        if (open) fd[c] = fd[c] + f * (up - s00.v[c]);
      }
    }
  };
  if constexpr (MONOT) { CELL_EDGES2(np, edges); }
  else { CELL_EDGES3(np, edges); }
  Vec<V> o, tend = zerov<V>();
  if (pl) tend = ldv<V>(A.SCT + V * q + x * row);
  const float dr = A.dtr / rh;
#pragma unroll
  for (int c = 0; c < V; ++c)
    o.v[c] = (pl >> c) & 1u ? s00.v[c] + dr * (tend.v[c] + vt * fd[c]) : s00.v[c] + dr * vt * fd[c];
  float* out = A.out + V * q;
  stv<V>(out + x * row, o);
  // Below the floor the reference updates in place: scp(2:kb-1) = scp(kb) in
  // the explicit branch only (an unlimited tracer: scp(1:kb-1)), and levels
  // it does not write keep the stage input.
  if (kd == kb)
    for (int k = 0; k < kb; ++k) {
      Vec<V> y = ldv<V>(A.S + V * q + (cb + k) * row);
#pragma unroll
      for (int c = 0; c < V; ++c)
        if (((pl >> c) & 1u) || (!impl && k >= 1)) y.v[c] = o.v[c];
      stv<V>(out + (cb + k) * row, y);
    }
}

// last-stage low-order pre-update of scp0 for the tracers flagged in mode
// (scalar_transport_rk.F90:297-314), in place
__global__ void __launch_bounds__(256) k_preupdate(CellArgs A, float* S0, const float* rho_old) {
  CELL_ITEM(A);
  const int kb = CELL_FLOOR(A);
  if (kd < kb) return;
  constexpr int V = 4;
  const size_t row = (size_t)A.ld;
  float* p = S0 + (size_t)iw * mza * row + V * q;
  Vec<V> s = ldv<V>(p + (size_t)kd * row);
  const Vec<V> t = ldv<V>(A.SCT + ((size_t)iw * mza + kd) * row + V * q);
  const float ro = rho_old[(size_t)iw * mza + kd];
  int md[V];
  quad_modes<V>(A, q, md);
#pragma unroll
  for (int c = 0; c < V; ++c) if (md[c]) s.v[c] = s.v[c] + A.dtr * t.v[c] / ro;
  stv<V>(p + (size_t)kd * row, s);
  if (kd == kb)
    for (int k = 1; k < kb; ++k) {
      Vec<V> y = ldv<V>(p + (size_t)k * row);
#pragma unroll
      for (int c = 0; c < V; ++c) if (md[c]) y.v[c] = s.v[c];
      stv<V>(p + (size_t)k * row, y);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static CellArgs cell_args(const DevGrid& d, int nq, int V) {
  CellArgs A{};
  A.mza = d.mza; A.mwa = d.mwa;
  A.nq = nq;
  A.nch = (int)cdiv((size_t)d.mza * nq, 32);
  A.npoly = d.npoly.p; A.lpw = d.lpw.p;
  A.edge = reinterpret_cast<const int4*>(d.edge.p);
  A.volti = d.volti.p;
  A.ld = nq * V;
  A.flat = ctx().tp.flat ? 1 : 0;
  return A;
}

static void over(CellArgs& A, const DevBuf<int>& cols, int n, int off) { A.cols = cols.p; A.ncol = n; A.off = off; }
static unsigned cell_blocks(const CellArgs& A) { return cdiv((size_t)A.ncol * A.nch, 8); }

bool cell_stage_available(const DevGrid& d, int order) {
  return d.w_covered && (order == 2 || order == 3);
}

template <int V, typename OFF>
static int run_stage(const DevGrid& d, int order, const CellStage& c, cudaStream_t s) {
  const int nq = V == 1 ? 1 : (c.nt + 3) / 4;
  CellArgs A = cell_args(d, nq, V);
  A.ld = c.ld; A.nt = c.nt;
  A.vmasc = c.vmasc; A.wmasc = c.wmasc; A.rhos = c.rhos; A.ff = c.ff; A.mode = c.mode;
  A.S = c.S; A.S0 = c.S0; A.SCT = c.SCT; A.out = c.out; A.face = c.face; A.scale = c.scale;
  A.istage = c.istage; A.nrk = c.nrk; A.dtr = c.dtr;
  const bool lim = c.limited != 0, monot = c.limited == 1;
  A.a_w = monot ? d.a_wu.p : d.a_w.p;
  A.edge3 = reinterpret_cast<const float4*>(monot ? d.edge3_u.p : d.edge3_b.p);
  // Every face's upwind cell is in jtw_wadj.  A caller of the no-allocation
  // stage may leave the table out: on a domain without borders jtw_prog holds
  // them too.
  if (d.w_covered || lim) over(A, d.jtw_wadj, d.nw_wadj, d.off_wwadj);
  else over(A, d.jtw_prog, d.nw_prog, d.off_wprog);
  {
    OG_PROF(lim ? "lim_face" : "cell_face", s);
    const unsigned nb = cell_blocks(A);
    if (!lim) {
      if (order == 2) launch_next(k_face<V, 2, false, OFF>, nb, 256, 0, s, A);
      else launch_next(k_face<V, 3, false, OFF>, nb, 256, 0, s, A);
    } else if constexpr (V == 4) {
      if (order == 2) launch_next(k_face<V, 2, true, OFF>, nb, 256, 0, s, A);
      else launch_next(k_face<V, 3, true, OFF>, nb, 256, 0, s, A);
    }
    OG_LAUNCHED();
  }
  if constexpr (V == 4) {
    if (lim) {
      // the factors of both cells of every face of a prognosed column
      OG_PROF("lim_scale", s);
      const unsigned nb = cell_blocks(A);
      if (monot) launch_next(k_scale<V, true, OFF>, nb, 256, 0, s, A);
      else launch_next(k_scale<V, false, OFF>, nb, 256, 0, s, A);
      OG_LAUNCHED();
    }
  }
  over(A, d.jtw_prog, d.nw_prog, d.off_wprog);
  {
    OG_PROF(lim ? "lim_update" : "cell_update", s);
    const unsigned nb = cell_blocks(A);
    if (!lim) launch_next(k_update<V, OFF>, nb, 256, 0, s, A);
    else if constexpr (V == 4) {
      if (monot) launch_next(k_update_lim<V, true, OFF>, nb, 256, 0, s, A);
      else launch_next(k_update_lim<V, false, OFF>, nb, 256, 0, s, A);
    }
    OG_LAUNCHED();
  }
  OG_CUDA(cudaGetLastError());
  return OLAMGPU_OK;
}

int launch_cell_stage(const DevGrid& d, int order, const CellStage& c, cudaStream_t s) {
  if (d.nw_prog <= 0 || c.nt <= 0) return OLAMGPU_OK;
  if (c.ld == 1 && c.limited) { set_error("cell stage: limited stages run the batched layout"); return OLAMGPU_E_UNSUPPORTED; }
  if (c.ld == 1) return run_stage<1, unsigned>(d, order, c, s);   // one plane: under 2^32 elements
  const double most = (double)d.mza * std::max((double)d.mwa * std::max(c.ld, 2 * cell_width(c.nt)), (double)d.mva * cell_width(c.nt));
  return most < 4294967296.0 ? run_stage<4, unsigned>(d, order, c, s) : run_stage<4, size_t>(d, order, c, s);
}

void launch_cell_preupdate(const DevGrid& d, const Transport& tp, float* S0, const float* SCT, int ld, int nt,
                           const int* mode, float dtr, cudaStream_t s) {
  if (d.nw_wadj <= 0 || nt <= 0) return;
  CellArgs A = cell_args(d, (nt + 3) / 4, 4);
  A.ld = ld; A.nt = nt; A.mode = mode; A.SCT = SCT; A.dtr = dtr;
  over(A, d.jtw_wadj, d.nw_wadj, d.off_wwadj);
  OG_PROF("lim_preupdate", s);
  launch_next(k_preupdate, cell_blocks(A), 256, 0, s, A, S0, tp.rho_old.p);
  OG_LAUNCHED();
}

}  // namespace olamgpu
