// Batched horizontal 2-D real FFT passes with fused prologues/epilogues.
//
// A 2-D r2c/c2r of the reference (decomp_2d_fft_2d.f90:498-577: x r2c,
// transpose X->Y, y c2c) becomes three kernel families that work on every
// level of a field in one launch:
//
//   xfwd  : physical rows (length NX) -> half-spectrum rows, first nk modes.
//           The load step computes the transformed quantity on the fly
//           (scaling, vorticity, fine-grid products, SGS test-filter inputs).
//   ypass : columns of a spectral buffer -> y FFT (length NY) -> spectral op
//           (i*k multiply, Nyquist kill, filter, 3/2 pad or truncate) ->
//           inverse y FFT (length NYO) -> spectral buffer.  This is where the
//           2DECOMP X<->Y pencil transpose happens: columns are staged through
//           shared memory, no global transpose is ever written.
//   xinv  : half-spectrum rows -> c2r (length NX) -> fused store op
//           (plain store, rhs accumulation, stress divergence with its dz
//           term and pressure-BC layers, SGS dynamic-procedure contraction).
//
// Spectral buffers are [level][ky row][kx] with kx fastest, so the x passes
// read and write whole contiguous rows and the y pass reads C consecutive kx
// columns per row (128-byte segments).
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fft2.cuh"
#include "tc05.cuh"

namespace les {

constexpr int MAXIN = 24;
constexpr int MAXOUT = 48;

// ---- asynchronous global -> shared copies (cp.async) ----
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int n = valid ? BYTES : 0;  // 0: zero fill, nothing read
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gmem), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(gmem), "n"(BYTES), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- bulk global -> shared copies (cp.async.bulk, completion on an mbarrier) ----
// One instruction moves a whole contiguous row: both addresses 16-byte
// aligned, the size a multiple of 16.  No multicast: the destination is this
// CTA's shared memory only.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(mbar))
               : "memory");
}
// the one arrival of a stage's mbarrier, announcing the bytes its copies bring
__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(mbar)), "r"(bytes)
               : "memory");
}

// r2c split of a length-2M real row transformed as M complex values Z:
// X_k = (Z_k + conj Z_{M-k}) / 2 + W^k (Z_k - conj Z_{M-k}) / (2i), with
// wh = W^k / 2 (W = exp(-2 pi i / 2M)).  The sums with the sign pairs are
// packed FP32x2 instructions in single precision.
template <typename T>
__device__ __forceinline__ cplx<T> r2c_split(cplx<T> zk, cplx<T> zm, cplx<T> wh) {
  const cplx<T> sp = c_fma(zm, cplx<T>{T(1), T(-1)}, zk);  // Z_k + conj Z_{M-k}
  const cplx<T> dp = c_fma(zm, cplx<T>{T(-1), T(1)}, zk);  // Z_k - conj Z_{M-k}
  const cplx<T> q = {dp.y * wh.x + dp.x * wh.y, dp.y * wh.y - dp.x * wh.x};  // dp wh / i
  return c_fma(sp, cplx<T>{T(0.5), T(0.5)}, q);
}
// c2r split, the inverse of the above without the halving:
// Z_m = (X_m + conj X_{M-m}) + i W^{-m} (X_m - conj X_{M-m}).
template <typename T>
__device__ __forceinline__ cplx<T> c2r_split(cplx<T> xk, cplx<T> xm, cplx<T> w) {
  const cplx<T> s1 = c_fma(xm, cplx<T>{T(1), T(-1)}, xk);
  const cplx<T> d1 = c_fma(xm, cplx<T>{T(-1), T(1)}, xk);
  // t = d1 conj(w), held swapped as (t.y, t.x); Z = s1 + i t
  const cplx<T> ts = {d1.y * w.x - d1.x * w.y, d1.x * w.x + d1.y * w.y};
  return c_fma(ts, cplx<T>{T(-1), T(1)}, s1);
}

// r2c split and store of the first nk modes of a sequence whose FFT output
// Z sits in natural order in its slot: lane t writes modes k = t + TL i
// (i <= E: mode M, the Nyquist bin, falls on lane 0 at i = E), an unrolled
// loop with compile-time offsets; Z_M is Z_0 and the partner of mode 0 is
// Z_0 itself
template <typename T, int M, int TL, int E>
__device__ __forceinline__ void xf_split_store(const cplx<T>* seq, const cplx<T>* tw, cplx<T>* orow, int t, int nk) {
#pragma unroll
  for (int i = 0; i <= E; ++i) {
    const int k = t + TL * i;
    if (k < nk) {
      if (i == 0) orow[k] = r2c_split(seq[k], seq[k == 0 ? 0 : M - k], tw[k]);
      else if (i < E) orow[k] = r2c_split(seq[k], seq[M - k], tw[k]);
      else orow[k] = r2c_split(seq[0], seq[0], tw[M]);  // k = M (t = 0)
    }
  }
}

// ---------------------------------------------------------------- xfwd ----
enum XFOp : int {
  XF_SCALE = 0,   // field f = c0 * in[f]
  XF_CONV_IN = 1, // u,v,w scaled by -c0 and the three vorticity components (c0 scaled)
  XF_PROD = 2,    // fine-grid u x omega products (inputs on the padded grid)
  XF_LASD = 3,    // the 21 test-filter inputs of the dynamic procedure
  XF_PRESS = 4,   // pressure right-hand side: u*, v*, dw*/dz -> i kx u^ + (dw*/dz)^ and v^
  XF_PROD_SC = 5, // fine-grid scalar advection -(u . grad theta) (inputs on the padded grid)
  XF_SCDYN = 6,   // the 19 test-filter inputs of the dynamic Prandtl model
  XF_PRESS_INC = 7,  // pressure right-hand side from the AB2 increment and div u^n
};

template <typename T>
struct XFArgs {
  FastDiv d_rows, d_nf, d_ns;  // division by rows_pp, nf, nsrc (set by the launcher)
  int dep;         // launched by launch_dep: the tables are constant
  int op, nf, R;
  int lfast;       // k_xfwd: a CTA's rows are one row of R consecutive levels
  long nrows;      // rows to process = nplanes * rows_pp
  int rows_pp;     // rows per plane of the input grid
  int plane0;      // first level
  int nk;          // modes stored per output row
  int opitch;      // complex values between output rows (>= nk; 0: nk)
  int nz;
  int wall;        // wall-law special rows at k=1
  int use_ref;     // subtract each field's value at (i,j)=(0,0) of the level
  int fluct;       // XF_LASD: form products of u, v, w minus their (0,0) values
  double ref_mul;  // refout = ref * ref_mul (the value the inverse adds back)
  T* refout[MAXIN];
  long in_pstride; // elements per plane of the input grid
  long in_rstride; // elements per row of the input grid (== NX)
  double c0, c1, c2, c3;
  double rc1;      // XF_PRESS: 1 / c1
  const T* in[16];
  const float* inf[16];  // FP32 inputs of an FP64 transform (in_f32 = 1; whole rows only)
  int in_f32;
  cplx<T>* out[MAXIN];
  long out_pstride;  // rows_pp * nk
  const T* kxr;      // x wavenumbers (XF_PRESS), Nyquist zero
  int nsrc, nbuf, stage_rows;  // k_xfwd_row: staged rows per grid row, stages, slots per stage (set by the launcher)
  unsigned* status;  // device status word (ST_COPY_WAIT), may be null
  const cplx<T>* tw; // exp(-2 pi i m / NX), m < NX
};

// Four consecutive x points of one row, moved with 16-byte loads and stores.
template <typename T>
struct V4 {
  T e[4];
};
template <typename T>
__device__ __forceinline__ V4<T> operator+(const V4<T>& a, const V4<T>& b) {
  return {{a.e[0] + b.e[0], a.e[1] + b.e[1], a.e[2] + b.e[2], a.e[3] + b.e[3]}};
}
template <typename T>
__device__ __forceinline__ V4<T> operator-(const V4<T>& a, const V4<T>& b) {
  return {{a.e[0] - b.e[0], a.e[1] - b.e[1], a.e[2] - b.e[2], a.e[3] - b.e[3]}};
}
template <typename T>
__device__ __forceinline__ V4<T> operator*(const V4<T>& a, const V4<T>& b) {
  return {{a.e[0] * b.e[0], a.e[1] * b.e[1], a.e[2] * b.e[2], a.e[3] * b.e[3]}};
}
template <typename T>
__device__ __forceinline__ V4<T> operator*(T c, const V4<T>& b) {
  return {{c * b.e[0], c * b.e[1], c * b.e[2], c * b.e[3]}};
}
template <typename T>
__device__ __forceinline__ V4<T> operator/(const V4<T>& a, T c) {
  return {{a.e[0] / c, a.e[1] / c, a.e[2] / c, a.e[3] / c}};
}
template <typename T>
__device__ __forceinline__ V4<T> operator-(const V4<T>& a) {
  return {{-a.e[0], -a.e[1], -a.e[2], -a.e[3]}};
}

// value type V (T: one point, V4<T>: four points) loaded from S* at off
template <typename V, typename S>
struct VLd;
template <typename S>
struct VLd<float, S> {
  static __device__ __forceinline__ float ld(const S* p, long o) { return float(p[o]); }
};
template <typename S>
struct VLd<double, S> {
  static __device__ __forceinline__ double ld(const S* p, long o) { return double(p[o]); }
};
template <>
struct VLd<V4<float>, float> {
  static __device__ __forceinline__ V4<float> ld(const float* p, long o) {
    const float4 q = *reinterpret_cast<const float4*>(p + o);
    return {{q.x, q.y, q.z, q.w}};
  }
};
template <>
struct VLd<V4<double>, double> {
  static __device__ __forceinline__ V4<double> ld(const double* p, long o) {
    const double2 q0 = *reinterpret_cast<const double2*>(p + o);
    const double2 q1 = *reinterpret_cast<const double2*>(p + o + 2);
    return {{q0.x, q0.y, q1.x, q1.y}};
  }
};
template <>
struct VLd<V4<double>, float> {
  static __device__ __forceinline__ V4<double> ld(const float* p, long o) {
    const float4 q = *reinterpret_cast<const float4*>(p + o);
    return {{double(q.x), double(q.y), double(q.z), double(q.w)}};
  }
};
template <typename V, typename S>
__device__ __forceinline__ V vld(const S* p, long o) {
  return VLd<V, S>::ld(p, o);
}
// the same through the read-only data path (ld.global.nc): for inputs that
// no thread of the kernel writes; the compiler may then schedule these
// loads across shared-memory stores
template <typename V, typename S>
__device__ __forceinline__ V vldg(const S* p, long o) {
  if constexpr (std::is_same<V, V4<float>>::value && std::is_same<S, float>::value) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p + o));
    return {{q.x, q.y, q.z, q.w}};
  } else if constexpr (std::is_same<V, V4<double>>::value && std::is_same<S, double>::value) {
    const double2 q0 = __ldg(reinterpret_cast<const double2*>(p + o));
    const double2 q1 = __ldg(reinterpret_cast<const double2*>(p + o + 2));
    return {{q0.x, q0.y, q1.x, q1.y}};
  } else if constexpr (std::is_same<V, V4<double>>::value && std::is_same<S, float>::value) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p + o));
    return {{double(q.x), double(q.y), double(q.z), double(q.w)}};
  } else {
    return V(__ldg(p + o));
  }
}
template <typename T>
__device__ __forceinline__ void vst(T* p, T x) {
  *p = x;
}
__device__ __forceinline__ void vst(float* p, const V4<float>& x) {
  *reinterpret_cast<float4*>(p) = make_float4(x.e[0], x.e[1], x.e[2], x.e[3]);
}
__device__ __forceinline__ void vst(double* p, const V4<double>& x) {
  reinterpret_cast<double2*>(p)[0] = make_double2(x.e[0], x.e[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(x.e[2], x.e[3]);
}
template <typename V, typename T>
__device__ __forceinline__ V vsplat(T x) {
  if constexpr (std::is_same<V, T>::value) return x;
  else return V{{x, x, x, x}};
}

// Values of every field of op OP at level l, row j, columns i (one point for
// V = T, four for V = V4<T>; i a multiple of 4 then), stored at v + f * vs,
// minus sub[f] when SUB (the per-level references of the mixed-precision
// transforms).  The op is a template parameter so that a pass's load loop
// is compiled per op, with no dispatch per point.
template <typename T, typename V, int OP, bool SUB>
__device__ __forceinline__ void xf_load_op(const XFArgs<T>& a, int l, int j, int i, T* v, int vs, const T* sub) {
  const long off = (long)l * a.in_pstride + (long)j * a.in_rstride + i;
  auto put = [&](int f, const V& x) {
    if constexpr (SUB) vst(v + f * vs, x - vsplat<V>(sub[f]));
    else vst(v + f * vs, x);
  };
  {
    if constexpr (OP == XF_CONV_IN) {
      // compute_convective_padd.f90:133-165
      const T c = T(a.c0);
      put(0, -c * vldg<V>(a.in[0], off));
      put(1, -c * vldg<V>(a.in[1], off));
      put(2, -c * vldg<V>(a.in[2], off));
      const T* dwdy = a.in[3];
      const T* dvdz = a.in[4];
      const T* dudz = a.in[5];
      const T* dwdx = a.in[6];
      const T* dvdx = a.in[7];
      const T* dudy = a.in[8];
      if (a.wall && l == 0) {
        put(3, vsplat<V>(T(0)));
        put(4, vsplat<V>(T(0)));
      } else if (a.wall && l == 1) {
        const long up = off + a.in_pstride;
        put(3, c * (T(0.5) * (vldg<V>(dwdy, off) + vldg<V>(dwdy, up)) - vldg<V>(dvdz, off)));
        put(4, c * (vldg<V>(dudz, off) - T(0.5) * (vldg<V>(dwdx, off) + vldg<V>(dwdx, up))));
      } else {
        put(3, c * (vldg<V>(dwdy, off) - vldg<V>(dvdz, off)));
        put(4, c * (vldg<V>(dudz, off) - vldg<V>(dwdx, off)));
      }
      put(5, c * (vldg<V>(dvdx, off) - vldg<V>(dudy, off)));
    } else if constexpr (OP == XF_PROD) {
      // compute_convective_padd.f90:180-249 on the fine grid; inputs are
      // ub, vb, wb, o1, o2, o3 (padded -c*u, -c*v, -c*w and vorticity).
      const T c = T(a.c0);
      const T* ub = a.in[0];
      const T* vb = a.in[1];
      const T* wb = a.in[2];
      const T* o1 = a.in[3];
      const T* o2 = a.in[4];
      const T* o3 = a.in[5];
      const long up = off + a.in_pstride;
      const long dn = off - a.in_pstride;
      const V vb0 = vldg<V>(vb, off), o30 = vldg<V>(o3, off), ub0 = vldg<V>(ub, off);
      const V wbu = vldg<V>(wb, up), o2u = vldg<V>(o2, up), o1u = vldg<V>(o1, up);
      if (l == 1) {
        put(0, c * (-vb0 * o30 + T(0.5) * wbu * o2u));
        put(1, c * (ub0 * o30 + T(0.5) * wbu * (-o1u)));
        put(2, vsplat<V>(T(0)));
      } else {
        const V wb0 = vldg<V>(wb, off), o20 = vldg<V>(o2, off), o10 = vldg<V>(o1, off);
        put(0, c * (-vb0 * o30 + T(0.5) * (wbu * o2u + wb0 * o20)));
        put(1, c * (ub0 * o30 + T(0.5) * (wb0 * (-o10) + wbu * (-o1u))));
        put(2, c * T(0.5) * ((ub0 + vldg<V>(ub, dn)) * (-o20) + (vb0 + vldg<V>(vb, dn)) * o10));
      }
    } else if constexpr (OP == XF_PROD_SC) {
      // scalar advection on the fine grid, uvp level l: inputs ub, vb, wb
      // (padded -u, -v, -w), tx, ty (padded d theta/dx, dy, uvp nodes) and
      // tz (padded d theta/dz, w nodes): ub tx + vb ty + (wb tz at l, l+1)/2
      const T c = T(a.c0);
      const long up = off + a.in_pstride;
      const V r = vldg<V>(a.in[0], off) * vldg<V>(a.in[3], off) + vldg<V>(a.in[1], off) * vldg<V>(a.in[4], off) +
                  T(0.5) * (vldg<V>(a.in[2], off) * vldg<V>(a.in[5], off) + vldg<V>(a.in[2], up) * vldg<V>(a.in[5], up));
      put(0, c * r);
    } else if constexpr (OP == XF_PRESS_INC) {
      // u* = u^n + dt (t1 r + t2 r_f), so u* / (dt t1) = u^n / (dt t1) + r +
      // (t2/t1) r_f: the increment parts (inputs 0..5: rx ry rz rfx rfy rfz)
      // and the divergence of u^n (inputs 6..8: dudx dvdy dwdz, uvp nodes)
      // over dt t1 as a fourth field; c0 = 1/(nx ny), c1 = t2/t1,
      // c2 = 1/(dt t1).  Nothing large cancels in any of the four.
      const T c = T(a.c0), r21 = T(a.c1), idt = T(a.c2);
      put(0, c * (vldg<V>(a.in[0], off) + r21 * vldg<V>(a.in[3], off)));
      put(1, c * (vldg<V>(a.in[1], off) + r21 * vldg<V>(a.in[4], off)));
      put(2, c * (vldg<V>(a.in[2], off) + r21 * vldg<V>(a.in[5], off)));
      put(3, (c * idt) * ((vldg<V>(a.in[6], off) + vldg<V>(a.in[7], off)) + vldg<V>(a.in[8], off)));
    } else if constexpr (OP == XF_SCDYN) {
      // dynamic Prandtl model on the nodes of compute_dynamic_mum
      // (compute_LagScaleDep.f90:501-520: level 1 on uvp nodes with w(2)/4,
      // levels >= 2 on w nodes).  Inputs: 0 u, 1 v, 2 w, 3 theta, 4..9 S_ij,
      // 10 |S|, 11 d theta/dx, 12 d theta/dy, 13 d theta/dz (w nodes).
      // Outputs: u, v, w, theta, u theta, v theta, w theta, S_ij (6),
      // d_j theta (3), |S| d_j theta (3).
      const long pl = a.in_pstride;
      auto at_w = [&](const T* f, long o) -> V {
        return l == 1 ? vldg<V>(f, o) : T(0.5) * (vldg<V>(f, o) + vldg<V>(f, o - pl));
      };
      V uf = at_w(a.in[0], off), vf = at_w(a.in[1], off), tf = at_w(a.in[3], off);
      V wf = l == 1 ? T(0.25) * vldg<V>(a.in[2], off + pl) : vldg<V>(a.in[2], off);
      if (a.fluct) {
        // K_j = filt(u_j theta) - filt(u_j) filt(theta) does not change when
        // per-level constants are removed from u_j and theta (the filter
        // keeps the mean); FP32 keeps the fluctuations
        const long o0 = (long)l * pl;
        auto at_w0 = [&](const T* f) -> T { return l == 1 ? f[o0] : T(0.5) * (f[o0] + f[o0 - pl]); };
        const T w0 = l == 1 ? T(0.25) * a.in[2][o0 + pl] : a.in[2][o0];
        uf = uf - vsplat<V>(at_w0(a.in[0]));
        vf = vf - vsplat<V>(at_w0(a.in[1]));
        tf = tf - vsplat<V>(at_w0(a.in[3]));
        wf = wf - vsplat<V>(w0);
      }
      put(0, uf);
      put(1, vf);
      put(2, wf);
      put(3, tf);
      put(4, uf * tf);
      put(5, vf * tf);
      put(6, wf * tf);
#pragma unroll
      for (int q = 0; q < 6; ++q) put(7 + q, vldg<V>(a.in[4 + q], off));
      const V S = vldg<V>(a.in[10], off);
      const V tx = at_w(a.in[11], off), ty = at_w(a.in[12], off), tz = vldg<V>(a.in[13], off);
      put(13, tx);
      put(14, ty);
      put(15, tz);
      put(16, S * tx);
      put(17, S * ty);
      put(18, S * tz);
    } else if constexpr (OP == XF_LASD) {
      // compute_LagScaleDep.f90:501-584: u_ft, A_ij, S_ij, |S| S_ij
      const T* u = a.in[0];
      const T* vv = a.in[1];
      const T* w = a.in[2];
      V uf, vf, wf;
      if (l == 1) {
        uf = vldg<V>(u, off);
        vf = vldg<V>(vv, off);
        wf = T(0.25) * vldg<V>(w, off + a.in_pstride);
      } else {
        const long dn = off - a.in_pstride;
        uf = T(0.5) * (vldg<V>(u, off) + vldg<V>(u, dn));
        vf = T(0.5) * (vldg<V>(vv, off) + vldg<V>(vv, dn));
        wf = vldg<V>(w, off);
      }
      if (a.fluct) {
        // L_ij = filt(u_i u_j) - filt(u_i) filt(u_j) is unchanged when a
        // per-level constant is removed from u_i; FP32 keeps the fluctuation.
        const long o0 = (long)l * a.in_pstride;
        T u0, v0, w0;
        if (l == 1) {
          u0 = u[o0];
          v0 = vv[o0];
          w0 = T(0.25) * w[o0 + a.in_pstride];
        } else {
          u0 = T(0.5) * (u[o0] + u[o0 - a.in_pstride]);
          v0 = T(0.5) * (vv[o0] + vv[o0 - a.in_pstride]);
          w0 = w[o0];
        }
        uf = uf - vsplat<V>(u0);
        vf = vf - vsplat<V>(v0);
        wf = wf - vsplat<V>(w0);
      }
      put(0, uf);
      put(1, vf);
      put(2, wf);
      put(3, uf * uf);  // A11
      put(4, uf * vf);  // A12
      put(5, uf * wf);  // A13
      put(6, vf * vf);  // A22
      put(7, vf * wf);  // A23
      put(8, wf * wf);  // A33
      const V S = vldg<V>(a.in[9], off);
#pragma unroll
      for (int q = 0; q < 6; ++q) {  // s11 s12 s13 s22 s23 s33
        const V sq = vldg<V>(a.in[3 + q], off);
        put(9 + q, sq);
        put(15 + q, S * sq);
      }
    }
  }
}

// the same with the op chosen at run time (the per-row references)
template <typename T, typename V>
__device__ __forceinline__ void xf_load(const XFArgs<T>& a, int l, int j, int i, T* v, int vs) {
  switch (a.op) {
    case XF_CONV_IN: xf_load_op<T, V, XF_CONV_IN, false>(a, l, j, i, v, vs, nullptr); break;
    case XF_PROD: xf_load_op<T, V, XF_PROD, false>(a, l, j, i, v, vs, nullptr); break;
    case XF_LASD: xf_load_op<T, V, XF_LASD, false>(a, l, j, i, v, vs, nullptr); break;
    case XF_PROD_SC: xf_load_op<T, V, XF_PROD_SC, false>(a, l, j, i, v, vs, nullptr); break;
    case XF_SCDYN: xf_load_op<T, V, XF_SCDYN, false>(a, l, j, i, v, vs, nullptr); break;
    case XF_PRESS_INC: xf_load_op<T, V, XF_PRESS_INC, false>(a, l, j, i, v, vs, nullptr); break;
    default: break;
  }
}

// number of sequence slots in an x pass: rounded up to whole warps
template <int M>
__host__ __device__ constexpr int seq_pad(int nseq) {
  constexpr int spw = 32 / Geo<M>::T;  // sequences per warp
  return ((nseq + spw - 1) / spw) * spw;
}

template <typename T, int NX>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? (NX <= 256 ? 4 : 3) : 2) k_xfwd(const XFArgs<T> a) {
  constexpr int M = NX / 2;
  constexpr int TL = Geo<M>::T;
  constexpr int E = Geo<M>::E;
  constexpr int RI = Layout<M, false>::in;
  constexpr int RO = Layout<M, false>::out;
  constexpr int SL = slot_stride(M, int(sizeof(cplx<T>)));  // complex values per sequence slot
  constexpr int XS = 2 * SL;         // the same slot viewed as reals
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* twm = tw + NX;  // twiddle matrices of the M-point transform
  cplx<T>* buf = twm + Twm<M, false>::len;
  const int nseq = a.R * a.nf;
  const int npad = seq_pad<M>(nseq);
  T* refs = reinterpret_cast<T*>(buf + (long)npad * SL);  // R * nf per-row references
  int* rowl = reinterpret_cast<int*>(refs + a.R * a.nf);  // level of row r (-1: beyond the grid)
  int* rowj = rowl + a.R;
  for (int i = threadIdx.x; i < NX; i += blockDim.x) tw[i] = c_scl(a.tw[i], T(0.5));  // W^k / 2 for the split
  twm_build<T, M, false, 2>(a.tw, twm, threadIdx.x, blockDim.x);
  // rows of this CTA: consecutive rows of the grid, or (lfast) one row of R
  // consecutive levels
  const int nlev = a.d_rows(a.nrows);
  for (int r = threadIdx.x; r < a.R; r += blockDim.x) {
    int q, j;  // level index and row
    if (a.lfast) {
      q = a.d_rows(blockIdx.x);
      j = blockIdx.x - q * a.rows_pp;
      q = q * a.R + r;
    } else {
      const long g = (long)blockIdx.x * a.R + r;
      q = a.d_rows(g);
      j = int(g) - q * a.rows_pp;
    }
    rowl[r] = q < nlev ? a.plane0 + q : -1;
    rowj[r] = q < nlev ? j : 0;
  }
  dep_wait();
  __syncthreads();
  if (a.use_ref) {
    for (int r = threadIdx.x; r < a.R; r += blockDim.x) {
      const int l = rowl[r];
      if (l < 0) continue;
      xf_load<T, T>(a, l, 0, 0, refs + r * a.nf, 1);
      for (int f = 0; f < a.nf; ++f) {
        if (!a.refout[f]) refs[r * a.nf + f] = T(0);
        else if (rowj[r] == 0) a.refout[f][l] = T(double(refs[r * a.nf + f]) * a.ref_mul);
      }
    }
    __syncthreads();
  }
  // load: four consecutive points per thread (16-byte accesses); sequence
  // s = r*nf + f holds the packed row z_m = x_{2m} + i x_{2m+1}, i.e. the
  // real row itself viewed as complex.
  T* xr = reinterpret_cast<T*>(buf);
  // the load loop is compiled per op and per reference mode (no dispatch
  // per point); references are subtracted in registers before the store
  auto load_rows = [&](auto op_c, auto ref_c) {
    constexpr int OP = decltype(op_c)::value;
    constexpr bool REF = decltype(ref_c)::value;
    for (int idx = threadIdx.x; idx < a.R * (NX / 4); idx += blockDim.x) {
      const int r = idx / (NX / 4);
      const int i = 4 * (idx - r * (NX / 4));
      T* dst = xr + (long)(r * a.nf) * XS + i;
      const int l = rowl[r];
      if (l >= 0) xf_load_op<T, V4<T>, OP, REF>(a, l, rowj[r], i, dst, XS, refs + r * a.nf);
      else
        for (int f = 0; f < a.nf; ++f) vst(dst + f * XS, vsplat<V4<T>>(T(0)));
    }
  };
  auto load_op = [&](auto op_c) {
    if (a.use_ref) load_rows(op_c, std::true_type{});
    else load_rows(op_c, std::false_type{});
  };
  switch (a.op) {
    case XF_CONV_IN: load_op(std::integral_constant<int, XF_CONV_IN>{}); break;
    case XF_PROD: load_op(std::integral_constant<int, XF_PROD>{}); break;
    case XF_LASD: load_op(std::integral_constant<int, XF_LASD>{}); break;
    case XF_PROD_SC: load_op(std::integral_constant<int, XF_PROD_SC>{}); break;
    case XF_SCDYN: load_op(std::integral_constant<int, XF_SCDYN>{}); break;
    case XF_PRESS_INC: load_op(std::integral_constant<int, XF_PRESS_INC>{}); break;
    default: break;
  }
  for (int idx = nseq * SL + threadIdx.x; idx < npad * SL; idx += blockDim.x) buf[idx] = cplx<T>{T(0), T(0)};
  __syncthreads();
  // complex FFT of length M per sequence in registers, then the r2c split
  const int lane_t = threadIdx.x % TL;
  for (int base = 0; base < npad; base += blockDim.x / TL) {
    const int s = base + threadIdx.x / TL;
    if (base + (threadIdx.x / 32) * (32 / TL) >= npad) break;  // whole warp beyond the slots
    cplx<T>* seq = buf + (long)s * SL;
    cplx<T> v[E];
#pragma unroll
    for (int g = 0; g < E / RI; ++g)
#pragma unroll
      for (int r = 0; r < RI; ++r) v[g * RI + r] = seq[lane_t + TL * g + r * (M / RI)];
    reg_fft<T, M, false>(v, seq, lane_t, twm);
    __syncwarp();
#pragma unroll
    for (int g = 0; g < E / RO; ++g)
#pragma unroll
      for (int r = 0; r < RO; ++r) seq[lane_t + TL * g + r * (M / RO)] = v[g * RO + r];
    __syncwarp();
    if (s < nseq) {
      const int r = a.d_nf(s);
      const int f = s - r * a.nf;
      const int l = rowl[r];
      if (l >= 0) {
        const int j = rowj[r];
        cplx<T>* orow = a.out[f] + (long)l * a.out_pstride + (long)j * a.opitch;
        xf_split_store<T, M, TL, E>(seq, tw, orow, lane_t, a.nk);
      }
    }
  }
}

// ---- x forward pass of whole rows (k_xfwd_row) ----
// For ops whose inputs are rows as they stand: scalings (XF_SCALE) and the
// pressure right-hand side (XF_PRESS).  A bulk copy brings each input row
// straight into the shared slot its transform works in; the scale, the
// reference and the conversion of FP32 rows are applied as the registers are
// loaded.  Source row f of level l, row j (nullptr: none).
template <typename T, typename S>
__device__ __forceinline__ const S* xr_source(const XFArgs<T>& a, int f, int l, int j) {
  const S* const* in;
  if constexpr (std::is_same<S, T>::value) in = a.in;
  else in = a.inf;
  const long row = (long)l * a.in_pstride + (long)j * a.in_rstride;
  if (a.op != XF_PRESS) return in[f] + row;
  // XF_PRESS: sources u, v, w at l, w at l + 1 (none above level nz: w(nz+1)
  // counts as zero); the plane past level nz holds the two boundary layers,
  // the top one in place of v, the bottom one in place of w
  if (l > a.nz) return f == 1 ? in[4] + (long)j * a.in_rstride : (f == 2 ? in[3] + (long)j * a.in_rstride : nullptr);
  if (f < 3) return in[f] + row;
  return l < a.nz ? in[2] + row + a.in_pstride : nullptr;
}

// warp 0: announce the bytes of batch `item` and start one bulk copy per row
template <typename T, typename S, int NX, int SL>
__device__ __forceinline__ void xr_issue(const XFArgs<T>& a, long item, cplx<T>* stage, uint64_t* mbar) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const int ns = a.nsrc;
  const long left = a.nrows - item * a.R;
  const int nrow = int(left < a.R ? left : a.R) * ns;
  constexpr unsigned RB = NX * sizeof(S);
  auto source = [&](int s) {
    const int r = a.d_ns(s), f = s - r * ns;
    const int g = int(item) * a.R + r, q = a.d_rows(g);
    return xr_source<T, S>(a, f, a.plane0 + q, g - q * a.rows_pp);
  };
  unsigned bytes = nrow * RB;
  if (a.op == XF_PRESS) {  // some have no source
    bytes = 0;
    for (int s = lane; s < nrow; s += 32)
      if (source(s)) bytes += RB;
    for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
  }
  if (lane == 0) mbar_expect_tx(mbar, bytes);
  __syncwarp();
  tc::fence_async_smem();  // earlier generic accesses of this stage come first
  for (int s = lane; s < nrow; s += 32) {
    const S* src = source(s);
    if (src) bulk_g2s(stage + (long)s * SL, src, RB, mbar);
  }
}

// x / c for a fixed c with rc = 1/c: Markstein's correction of the product
// (P. Markstein, IBM J. Res. Dev. 34, 1990), the correctly rounded quotient
// for a correctly rounded rc.  The pressure inputs are velocities over dt
// whose divergence cancels; rounded as the reference's division rounds them
// they cancel as its do (a plain product moved p's gradients by 2e-12).
__device__ __forceinline__ double quot(double x, double c, double rc) {
  const double q = x * rc;
  return fma(fma(-q, c, x), rc, q);
}

// Persistent CTAs over batches of R rows with one or two stages of slots (two:
// the next batch is copied while this one is transformed).  Against loading
// through registers into the slots (k_xfwd) the pass has no load phase: at
// 256^3 the gradients' pass went from 0.166 to 0.111, the stresses' from 0.213
// to 0.203, the pressure's from 0.311 to 0.222 ms per step (mixed; FP64 0.298
// to 0.203, 0.438 to 0.323, 0.326 to 0.228).  The smallest launches pay for
// the barrier set-up (32^3: 8.9 -> 10.7 us).
template <typename T, int NX, typename S>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_xfwd_row(const XFArgs<T> a) {
  constexpr int M = NX / 2;
  constexpr int TL = Geo<M>::T;
  constexpr int E = Geo<M>::E;
  constexpr int RI = Layout<M, false>::in;
  constexpr int RO = Layout<M, false>::out;
  constexpr int SL = slot_stride(M, int(sizeof(cplx<T>)));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* twm = tw + NX;  // twiddle matrices of the M-point transform
  const int ns = a.nsrc;   // staged rows per grid row
  const int nseq = a.R * a.nf;
  const int npad = seq_pad<M>(nseq);
  const long stage_len = (long)a.stage_rows * SL;
  cplx<T>* stage0 = twm + Twm<M, false>::len;
  cplx<T>* stage1 = stage0 + (a.nbuf > 1 ? stage_len : 0L);  // stage 0 again when single
  uint64_t* bars = reinterpret_cast<uint64_t*>(stage0 + a.nbuf * stage_len);
  T* refs = reinterpret_cast<T*>(bars + 2);  // R * nf per-level references
  int* rowl = reinterpret_cast<int*>(refs + ((nseq + 1) & ~1));
  int* rowj = rowl + a.R;
  const long nitems = (a.nrows + a.R - 1) / a.R;
  for (int i = threadIdx.x; i < NX; i += blockDim.x) tw[i] = c_scl(a.tw[i], T(0.5));  // W^k / 2 for the split
  twm_build<T, M, false, 2>(a.tw, twm, threadIdx.x, blockDim.x);
  dep_wait();
  // warp 0 sets up the barriers and issues the first copies
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      tc::mbar_init(&bars[0], 1);
      tc::mbar_init(&bars[1], 1);
      tc::fence_mbar_init();
    }
    __syncwarp();
    if ((long)blockIdx.x < nitems) xr_issue<T, S, NX, SL>(a, blockIdx.x, stage0, &bars[0]);
  }
  // the reference of row r, field f of a batch (one per thread; R nf <= 256)
  auto ref_of = [&](long item) -> T {
    if (!a.use_ref || item >= nitems || threadIdx.x >= nseq) return T(0);
    const int r = a.d_nf(threadIdx.x), f = threadIdx.x - r * a.nf;
    const long g = item * a.R + r;
    if (g >= a.nrows || !a.refout[f]) return T(0);
    return T(a.c0) * a.in[f][(long)(a.plane0 + a.d_rows(g)) * a.in_pstride];
  };
  T ref_next = ref_of(blockIdx.x);
  __syncthreads();
  unsigned phase = 0;  // bit b: parity of the next completion of bars[b]
  int stg = 0;
  for (long item = blockIdx.x; item < nitems; item += gridDim.x) {
    const long next = item + gridDim.x;
    cplx<T>* stage = stg ? stage1 : stage0;
    if (a.nbuf > 1 && next < nitems) xr_issue<T, S, NX, SL>(a, next, stg ? stage0 : stage1, &bars[stg ^ 1]);
    const long g0 = item * a.R;
    for (int r = blockDim.x - 1 - threadIdx.x; r < a.R; r += blockDim.x) {  // (not warp 0, which issues)
      const long g = g0 + r;
      const int q = a.d_rows(g);
      rowl[r] = (g < a.nrows) ? a.plane0 + q : -1;
      rowj[r] = (g < a.nrows) ? int(g) - q * a.rows_pp : 0;
    }
    if (a.use_ref && threadIdx.x < nseq) {
      const int r = a.d_nf(threadIdx.x), f = threadIdx.x - r * a.nf;
      const long g = g0 + r;
      const int q = a.d_rows(g);
      refs[threadIdx.x] = ref_next;
      if (g < a.nrows && a.refout[f] && int(g) == q * a.rows_pp)
        a.refout[f][a.plane0 + q] = T(double(ref_next) * a.ref_mul);
    }
    ref_next = ref_of(next);
    const bool late = !tc::mbar_wait(&bars[stg], (phase >> stg) & 1u);
    phase ^= 1u << stg;
    if (__syncthreads_or(late)) {
      // as in k_xinv: record it, a last bounded wait for the copies in
      // flight, and every thread of the CTA leaves
      if (threadIdx.x == 0 && a.status) atomicOr(a.status, unsigned(ST_COPY_WAIT));
      tc::mbar_wait(&bars[stg], (phase >> stg) & 1u ^ 1u);
      if (a.nbuf > 1 && next < nitems) tc::mbar_wait(&bars[stg ^ 1], (phase >> (stg ^ 1)) & 1u);
      return;
    }
    const int lane_t = threadIdx.x % TL;
    for (int base = 0; base < npad; base += blockDim.x / TL) {
      const int s = base + threadIdx.x / TL;
      if (base + (threadIdx.x / 32) * (32 / TL) >= npad) break;  // whole warp beyond the slots
      const bool valid = s < nseq;
      const int r = valid ? a.d_nf(s) : 0;
      const int f = valid ? s - r * a.nf : 0;
      const int l = valid ? rowl[r] : -1;
      // slots past the last sequence follow the staged rows
      cplx<T>* seq = stage + (long)(valid ? r * ns + f : a.R * ns + (s - nseq)) * SL;
      cplx<T> v[E];
      if (l < 0) {
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = cplx<T>{T(0), T(0)};
      } else {
        // the row as pairs: z_m = x_2m + i x_2m+1
        const cplx<S>* row = reinterpret_cast<const cplx<S>*>(seq);
        auto at = [&](const cplx<S>* p, int m) { return cplx<T>{T(p[m].x), T(p[m].y)}; };
        auto load = [&](auto get) {
#pragma unroll
          for (int g = 0; g < E / RI; ++g)
#pragma unroll
            for (int q = 0; q < RI; ++q) v[g * RI + q] = get(lane_t + TL * g + q * (M / RI));
        };
        const T c0 = T(a.c0);
        if (a.op == XF_SCALE) {
          const T rf = a.use_ref ? -refs[s] : T(0);
          const cplx<T> cc = {c0, c0}, rr = {rf, rf};
          load([&](int m) { return c_fma(at(row, m), cc, rr); });
        } else if constexpr (sizeof(T) == 8) {  // XF_PRESS
          if (l > a.nz) {
            // boundary layers: nothing, the top one over nx ny, the bottom
            // one scaled in place (compute_pressure.f90:151-165)
            if (f == 0) {
              load([&](int) { return cplx<T>{T(0), T(0)}; });
            } else if (f == 1) {
              load([&](int m) { return c_scl(at(row, m), T(a.c2)); });
            } else {
              cplx<S>* plane = reinterpret_cast<cplx<S>*>(const_cast<S*>(xr_source<T, S>(a, 2, l, rowj[r])));
              const S sc = S(a.c2);
              load([&](int m) {
                const cplx<S> b = {sc * row[m].x, sc * row[m].y};
                plane[m] = b;
                return cplx<T>{T(b.x), T(b.y)};
              });
            }
          } else {
            // compute_pressure.f90:138-140: c0 (x / dt)
            const double dt = a.c1, rdt = a.rc1;
            auto h = [&](cplx<T> x) { return cplx<T>{c0 * quot(x.x, dt, rdt), c0 * quot(x.y, dt, rdt)}; };
            if (f < 2) {
              load([&](int m) { return h(at(row, m)); });
            } else {
              // (w(l+1) - w(l)) / dz, w(nz+1) = 0
              const cplx<S>* up = reinterpret_cast<const cplx<S>*>(seq + SL);
              const T cz = T(a.c3);
              if (l < a.nz) load([&](int m) { return h(c_scl(c_sub(at(up, m), at(row, m)), cz)); });
              else load([&](int m) { return h(c_scl(at(row, m), -cz)); });
            }
          }
        }
      }
      reg_fft<T, M, false>(v, seq, lane_t, twm);
      __syncwarp();
#pragma unroll
      for (int g = 0; g < E / RO; ++g)
#pragma unroll
        for (int q = 0; q < RO; ++q) seq[lane_t + TL * g + q * (M / RO)] = v[g * RO + q];
      __syncwarp();
      if (l >= 0 && a.op == XF_SCALE) {
        cplx<T>* orow = a.out[f] + (long)l * a.out_pstride + (long)rowj[r] * a.opitch;
        xf_split_store<T, M, TL, E>(seq, tw, orow, lane_t, a.nk);
      }
    }
    __syncthreads();
    if constexpr (sizeof(T) == 8) {
      if (a.op == XF_PRESS) {
        // two spectra leave for the three transforms of a row: i kx u^ + w'^
        // and v^ (one warp per row, consecutive modes on consecutive lanes)
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
        for (int r = warp; r < a.R; r += nwarps) {
          const int l = rowl[r];
          if (l < 0) continue;
          const cplx<T>* zu = stage + (long)(r * ns) * SL;
          const cplx<T>* zv = zu + SL;
          const cplx<T>* zw = zv + SL;
          const long o = (long)l * a.out_pstride + (long)rowj[r] * a.opitch;
          for (int k = lane; k <= M; k += 32) {
            const int k0 = k == M ? 0 : k, k1 = k == 0 ? 0 : M - k;  // Z_M is Z_0
            const cplx<T> h = tw[k];
            a.out[0][o + k] = c_add(ik_mul(a.kxr[k], r2c_split(zu[k0], zu[k1], h)), r2c_split(zw[k0], zw[k1], h));
            a.out[1][o + k] = r2c_split(zv[k0], zv[k1], h);
          }
        }
        __syncthreads();
      }
    }
    if (a.nbuf > 1) stg ^= 1;
    else if (next < nitems) xr_issue<T, S, NX, SL>(a, next, stage0, &bars[0]);
  }
}

// --------------------------------------------------------------- ypass ----
enum YPOp : int {
  YP_DIV2 = 1,     // (fx, fy) -> i kx fx + i ky fy     (Nyquist killed)
  YP_FWDKILL = 2,  // f -> f, no inverse y transform    (Nyquist killed)
  YP_PGRAD = 3,    // p^ (already y-spectral) -> p, i ky p   (i kx p in the x inverse)
  YP_FILTER2 = 4,  // f -> G0 f, G1 f
  YP_PAD = 5,      // ny -> 3ny/2 zero padding (ky Nyquist dropped)
  YP_TRUNC = 6,    // 3ny/2 -> ny truncation (ky Nyquist zeroed)
  YP_MASK = 7,     // keep |ky| <= tt (2/3-rule truncation)
  YP_FILTER1 = 8,  // f -> G0 f
  YP_GRADY = 9,    // f -> f, i ky f                    (Nyquist killed; i kx f in the x inverse)
  YP_PADY = 11,    // YP_PAD of f and of i ky f (second output optional)
  YP_MASKY = 12,   // YP_MASK of f and of i ky f (second output optional)
  YP_PRESS = 10,   // (f, v) -> f + i ky v, no inverse y transform (Nyquist killed); the last plane's two
                   // inputs are the pressure-BC layers: f -> plane 0, v -> its own plane
};

template <typename T>
struct YPArgs {
  FastDiv d_ncb, d_np;  // division by the column blocks, nplanes (set by the launcher)
  int dep;         // launched by launch_dep: the tables are constant
  int op, nin, nout, C, lc;  // C = 1 << lc columns per CTA
  int SI;                    // column stride of the shared stages (>= both lengths' slots)
  int ncols;           // columns processed
  int ncols1;          // columns stored for the second FILTER2 output
  int nk_in, nk_out, nk_out1;
  int ipitch, opitch, opitch1;  // complex values between rows of in / out / second out (0: the nk)
  int nplanes, ngroups;         // work items: column blocks x planes x groups
  int plane0;
  int nstage;  // input stages (set by the launcher): 2 = the next item's columns load during this one
  long in_pstride, out_pstride, out_pstride1;
  int nxh, lhx;        // base-grid Nyquist column and row length of kkx/kky/G
  int tt;              // YP_MASK: largest |ky| kept
  const cplx<T>* in[MAXIN];
  cplx<T>* out[MAXOUT];
  const T* kkx;        // [ny][lhx]
  const T* kky;
  // YP_GRADY, group < 2: a third output on level 1, the column times G0 gs
  // (nullptr: none), one plane of rows opitch1 apart, columns below ncols1
  cplx<T>* wall[2];
  T gs;
  const T* G0;         // [ny][lhx] filter kernels (include 1/(nx ny))
  const T* G1;
  const cplx<T>* tw_in;   // length NY table
  const cplx<T>* tw_out;  // length NYO table
};

// The ops of the y passes in classes, each compiled on its own (FP64: with every
// op in one kernel 200-350 bytes per thread spilled at the register limit that
// three blocks per SM need; the test-filtered fields at 128^3 took 312 us so,
// 183 apart, at 256^3 1978 and 1850, FP32 at 512 x 512 x 96 1835 and 1490).
// Length-changing passes are YC_OTHER.
enum YPClass : int { YC_FWD = 0, YC_GRADY = 1, YC_PGRAD = 2, YC_FILTER = 3, YC_DIV2 = 4, YC_OTHER = 5 };
inline int yp_class(int op) {
  switch (op) {
    case YP_FWDKILL: case YP_PRESS: return YC_FWD;
    case YP_GRADY: return YC_GRADY;
    case YP_PGRAD: return YC_PGRAD;
    case YP_FILTER1: case YP_FILTER2: return YC_FILTER;
    case YP_DIV2: return YC_DIV2;
    default: return YC_OTHER;
  }
}

// Output q at (kx, ky) of a column's forward transform F0, kyv = kky(ky) of the
// row (column 0 of the table).  The tables hold 2 pi / l times the wrapped
// index, zeroed on the Nyquist row / column only, so away from those the
// values are the table's; the kills below reproduce the zeros.
template <typename T, int NY, int CLS>
__device__ __forceinline__ cplx<T> yp_op(const YPArgs<T>& a, int q, int kx, int ky, cplx<T> F0, T kyv) {
  const cplx<T> zero = {T(0), T(0)};
  if constexpr (CLS == YC_GRADY) {
    if (ky == NY / 2 || kx == a.nxh) return zero;
    if (q == 0) return F0;
    return ik_mul(kyv, F0);
  } else if constexpr (CLS == YC_PGRAD) {  // no kill, the Nyquist row / column of the tables are zero
    if (q == 0) return F0;
    return ik_mul(kx == a.nxh ? T(0) : kyv, F0);
  } else if constexpr (CLS == YC_FILTER) {
    const T g = (q == 0 ? a.G0 : a.G1)[ky * a.lhx + kx];
    return cplx<T>{F0.x * g, F0.y * g};
  } else {  // YP_MASK, YP_MASKY: columns and kept rows below the Nyquist ones
    if (!(ky <= a.tt || ky >= NY - a.tt)) return zero;
    return q == 0 ? F0 : ik_mul(kyv, F0);
  }
}

// y pass: start the copies of work item `item` (C columns x NY rows of every
// input field) into the shared stage `bin` ([nin][C][SI])
template <typename T, int NY>
__device__ __forceinline__ void yp_issue(const YPArgs<T>& a, long item, int ncb, cplx<T>* bin) {
  const int C = a.C, SI = a.SI;
  const int pq = a.d_ncb(item), grp = a.d_np(pq);
  const int col0 = (int(item) - pq * ncb) * C;
  const int l = a.plane0 + pq - grp * a.nplanes;
  // thread -> fixed column c, rows ky0 + TL i: the CTA has C x TL threads,
  // so every thread copies NY / TL rows at a compile-time count and the
  // addresses advance by constant strides (an unrolled loop)
  constexpr int TL = Geo<NY>::T;
  const int c = threadIdx.x & (C - 1);
  const int ky0 = threadIdx.x >> a.lc;
  const int kx = col0 + c;
  const bool valid = kx < a.ncols;
  const long step = (long)TL * a.ipitch;
  for (int q = 0; q < a.nin; ++q) {
    const cplx<T>* base = a.in[grp * a.nin + q];
    const cplx<T>* src = valid ? base + (long)l * a.in_pstride + kx + (long)ky0 * a.ipitch : base;
    cplx<T>* dst = bin + (q * C + c) * SI + ky0;
#pragma unroll
    for (int i = 0; i < NY / TL; ++i)
      cp_async<int(sizeof(cplx<T>))>(dst + TL * i, valid ? src + i * step : base, valid);
  }
}

// YC_FWD: forward transforms only, compiled without the inverse so that it
// keeps fewer registers.  FP64: 168 registers (three CTAs of 128 threads) where
// the compiler would take 255 (two); the 21 test-filtered fields at 256^3: 2965
// -> 2286 us, 1993 without the columns past the narrower filter, 1850 in a
// class of their own.
template <typename T, int NY, int NYO, int CLS>
__global__ void __launch_bounds__(sizeof(T) == 8 ? 128 : 256, sizeof(T) == 8 ? 3 : 2)
    k_ypass(const YPArgs<T> a) {
  constexpr int TL = Geo<NY>::T;
  static_assert(Geo<NYO>::T == TL, "pad/truncate pairs must share the lanes per sequence");
  constexpr int EI = Geo<NY>::E;
  constexpr int EO = Geo<NYO>::E;
  constexpr int FI = Layout<NY, false>::in;    // forward input groups
  constexpr int FO = Layout<NY, false>::out;   // forward output groups
  constexpr int II = Layout<NYO, true>::in;    // inverse input groups
  constexpr int IO = Layout<NYO, true>::out;   // inverse output groups
  constexpr bool SAME = (NY == NYO), FWD = CLS == YC_FWD;
  static_assert(SAME || CLS == YC_OTHER, "a class keeps the length");
  static_assert(!SAME || FO == II, "forward output layout must feed the inverse");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* twi = reinterpret_cast<cplx<T>*>(smem_raw);  // twiddle matrices, forward NY
  cplx<T>* two = twi + Twm<NY, false>::len;                 // and inverse NYO
  const int SI = a.SI;  // >= the slots of NY and NYO
  const int C = a.C;
  T* kyrow = reinterpret_cast<T*>(two + Twm<NYO, true>::len);  // kky(ky), column 0 of the table
  cplx<T>* bin0 = reinterpret_cast<cplx<T>*>(kyrow + ((NY + 3) & ~3));  // input stage 0: [nin][C][SI]
  cplx<T>* bin1 = bin0 + (a.nstage > 1 ? a.nin * C * SI : 0);  // input stage 1 (stage 0 again when single)
  // the inverse transform, its output layout and the coalesced copy-out use
  // the first input row of each column of the current stage, free once the
  // forward transforms hold their values in registers
  twm_build<T, NY, false>(a.tw_in, twi, threadIdx.x, blockDim.x);
  if constexpr (!FWD) twm_build<T, NYO, true>(a.tw_out, two, threadIdx.x, blockDim.x);
  if (a.kky)
    for (int i = threadIdx.x; i < NY; i += blockDim.x) kyrow[i] = a.kky[(long)i * a.lhx];
  dep_wait();
  // persistent CTAs: work item = (column block, plane, group); with two
  // stages the columns of the next item are copied into the other input
  // stage asynchronously while this one is transformed, with one stage they
  // are copied after this item's last read of it (more resident CTAs where
  // shared memory limits them)
  const int ncb = (a.ncols + C - 1) / C;
  const long nitems = (long)ncb * a.nplanes * a.ngroups;
  if ((long)blockIdx.x < nitems) {
    yp_issue<T, NY>(a, blockIdx.x, ncb, bin0);
    cp_async_commit();
  }
  int stage = 0;
  for (long item = blockIdx.x; item < nitems; item += gridDim.x) {
  const long next = item + gridDim.x;
  cplx<T>* bin = stage ? bin1 : bin0;
  if (a.nstage > 1 && next < nitems) {
    yp_issue<T, NY>(a, next, ncb, stage ? bin0 : bin1);
    cp_async_commit();
    cp_async_wait<1>();
  } else {
    cp_async_wait<0>();
  }
  __syncthreads();
  const int pq = a.d_ncb(item), grp = a.d_np(pq);
  const int col0 = (int(item) - pq * ncb) * C;
  const int l = a.plane0 + pq - grp * a.nplanes;
  const int c = threadIdx.x / TL;
  const int lt = threadIdx.x % TL;
  const int kx = col0 + c;
  // forward transform in registers; the stress divergence folds its second
  // input into w = i kx F0 + i ky F1 before the output loop
  cplx<T> f0[EI];
  cplx<T> w[EO];
  {
    cplx<T>* seq = bin + c * SI;
    if constexpr (CLS == YC_PGRAD) {
      // input is already y-spectral: load it in the inverse input layout
#pragma unroll
      for (int g = 0; g < EI / II; ++g)
#pragma unroll
        for (int r = 0; r < II; ++r) f0[g * II + r] = seq[lt + TL * g + r * (NY / II)];
    } else {
#pragma unroll
      for (int g = 0; g < EI / FI; ++g)
#pragma unroll
        for (int r = 0; r < FI; ++r) f0[g * FI + r] = seq[lt + TL * g + r * (NY / FI)];
      reg_fft<T, NY, false>(f0, seq, lt, twi);
      if constexpr (FWD) {
        if (a.op == YP_PRESS) {
          // the first transform rests in its slot (natural order, as the
          // copy-out wants it) while the registers take the second
          __syncwarp();
#pragma unroll
          for (int g = 0; g < EI / FO; ++g)
#pragma unroll
            for (int r = 0; r < FO; ++r) seq[lt + TL * g + r * (NY / FO)] = f0[g * FO + r];
          cplx<T>* seq1 = bin + (C + c) * SI;
#pragma unroll
          for (int g = 0; g < EI / FI; ++g)
#pragma unroll
            for (int r = 0; r < FI; ++r) f0[g * FI + r] = seq1[lt + TL * g + r * (NY / FI)];
          reg_fft<T, NY, false>(f0, seq1, lt, twi);
        }
      } else if constexpr (CLS == YC_DIV2) {
        const cplx<T> zero = {T(0), T(0)};
#pragma unroll
        for (int g = 0; g < EI / FO; ++g)
#pragma unroll
          for (int r = 0; r < FO; ++r) {
            const int ky = lt + TL * g + r * (NY / FO);
            const bool kill = (ky == NY / 2) || (kx == a.nxh) || (kx >= a.ncols);
            w[g * FO + r] = kill ? zero : ik_mul(a.kkx[kx], f0[g * FO + r]);
          }
        cplx<T>* seq1 = bin + (C + c) * SI;
#pragma unroll
        for (int g = 0; g < EI / FI; ++g)
#pragma unroll
          for (int r = 0; r < FI; ++r) f0[g * FI + r] = seq1[lt + TL * g + r * (NY / FI)];
        reg_fft<T, NY, false>(f0, seq1, lt, twi);
#pragma unroll
        for (int g = 0; g < EI / FO; ++g)
#pragma unroll
          for (int r = 0; r < FO; ++r) {
            const int ky = lt + TL * g + r * (NY / FO);
            const bool kill = (ky == NY / 2) || (kx == a.nxh) || (kx >= a.ncols);
            if (!kill) w[g * FO + r] = c_add(w[g * FO + r], ik_mul(kyrow[ky], f0[g * FO + r]));
          }
      }
    }
  }
  __syncwarp();  // the column's forward reads are done before its slot is rewritten
  cplx<T>* sout = bin + c * SI;
  const bool layers = FWD && a.op == YP_PRESS && l == a.plane0 + a.nplanes - 1;
  const bool wall = CLS == YC_GRADY && l == 1 && grp < 2 && a.wall[grp] && col0 < a.ncols1;
  const int nout = layers ? 2 : a.nout + (wall ? 1 : 0);
  for (int q = 0; q < nout; ++q) {
    const bool third = wall && q == a.nout;
    if (!layers && !third && !a.out[grp * a.nout + q]) continue;  // an optional output left out (the whole CTA)
    if (CLS == YC_FILTER && a.op == YP_FILTER2 && q == 1 && col0 >= a.ncols1) continue;  // all columns beyond the narrower filter
    if constexpr (SAME) {
      // forward output layout (groups FO) == inverse input layout; the
      // stress divergence already holds its result in w
      if constexpr (FWD) {
        // YP_FWDKILL: the killed forward output goes straight to the slot in
        // the forward output layout (groups FO).  YP_PRESS: the slot holds
        // the first transform; i ky times the second is added, or, on the
        // plane of the boundary layers, both leave one after the other.
        const bool press = a.op == YP_PRESS;
#pragma unroll
        for (int g = 0; g < EI / FO; ++g)
#pragma unroll
          for (int r = 0; r < FO; ++r) {
            const int ky = lt + TL * g + r * (NY / FO);
            const bool kill = (ky == NY / 2) || (kx == a.nxh) || (kx >= a.ncols);
            cplx<T>& slot = sout[lt + TL * g + r * (NYO / FO)];
            cplx<T> x = f0[g * FO + r];
            if (press && !(layers && q == 1)) {
              x = slot;
              if (!layers) x = c_add(x, ik_mul(kyrow[ky], f0[g * FO + r]));
            }
            slot = kill ? cplx<T>{T(0), T(0)} : x;
          }
      } else if constexpr (CLS != YC_DIV2) {
        if (third) {
#pragma unroll
          for (int g = 0; g < EI / FO; ++g)
#pragma unroll
            for (int r = 0; r < FO; ++r) {
              const int ky = lt + TL * g + r * (NY / FO);
              const T gv = (kx < a.ncols1) ? a.G0[ky * a.lhx + kx] * a.gs : T(0);
              w[g * FO + r] = c_scl(f0[g * FO + r], gv);
            }
        } else {
#pragma unroll
          for (int g = 0; g < EI / FO; ++g)
#pragma unroll
            for (int r = 0; r < FO; ++r) {
              const int ky = lt + TL * g + r * (NY / FO);
              const T kyv = CLS == YC_FILTER ? T(0) : kyrow[ky];
              w[g * FO + r] = (kx < a.ncols) ? yp_op<T, NY, CLS>(a, q, kx, ky, f0[g * FO + r], kyv)
                                             : cplx<T>{T(0), T(0)};
            }
        }
      }
    } else {
      // 3/2 pad or truncate.  Lane lt holds the forward output at ky = lt +
      // TL m (m < EI) and the inverse wants ko = lt + TL m' (m' < EO); pad
      // and truncation map ky to ko by a shift of whole multiples of TL, so
      // the remap stays in the lane: a permutation of registers with zeros.
      // PAD: ko = ky (ky < NY/2), ky + NY/2 (ky > NY/2), ky = NY/2 dropped;
      // TRUNC: ko = ky (ky < NYO/2), ky - NYO/2 (ky > NYO), ky = NYO dropped.
      constexpr int GI = EI / FO;  // forward output: f0[g FO + r] holds m = g + r GI
      constexpr int GO = EO / II;  // inverse input: w[g II + r] wants m' = g + r GO
      const bool live = kx < a.ncols;
      auto remap = [&](auto ddy) {  // ddy: the output is i ky f
      static_for<EO>([&](auto mc) {
        constexpr int mo = decltype(mc)::value;
        constexpr int wi = (mo % GO) * II + mo / GO;
        constexpr bool PAD = NYO > NY;
        // source m of output m' (-1: zero), and whether lane 0 drops it
        constexpr int ms = PAD ? (mo < EI / 2 ? mo : (mo < EI ? -1 : mo - EI / 2))
                               : (mo < EO / 2 ? mo : mo + EO / 2);
        constexpr bool drop0 = PAD ? (mo == EI) : (mo == EO / 2);
        if constexpr (ms < 0) {
          w[wi] = cplx<T>{T(0), T(0)};
        } else {
          constexpr int fi = (ms % GI) * FO + ms / GI;
          const bool keep = live && !(drop0 && lt == 0);
          cplx<T> x = f0[fi];
          if constexpr (decltype(ddy)::value) x = ik_mul(kyrow[lt + TL * ms], x);
          w[wi] = keep ? x : cplx<T>{T(0), T(0)};
        }
      });
      };
      if constexpr (NYO > NY) {
        if (a.op == YP_PADY && q == 1) remap(std::true_type{});
        else remap(std::false_type{});
      } else {
        remap(std::false_type{});
      }
    }
    if constexpr (FWD) {
      // no inverse: stored above
    } else {
      reg_fft<T, NYO, true>(w, sout, lt, two);
      __syncwarp();
#pragma unroll
      for (int g = 0; g < EO / IO; ++g)
#pragma unroll
        for (int r = 0; r < IO; ++r) sout[lt + TL * g + r * (NYO / IO)] = w[g * IO + r];
    }
    __syncthreads();
    // coalesced store of output q
    const bool second = (CLS == YC_FILTER && a.op == YP_FILTER2 && q == 1) || third;
    const int lim = second ? a.ncols1 : a.ncols;
    {
      // thread -> fixed column cc, rows ky0 + TL i (as in yp_issue)
      const int cc = threadIdx.x & (C - 1);
      const int kxx = col0 + cc;
      if (kxx < lim) {
        const int ky0 = threadIdx.x >> a.lc;
        const long opitch = second ? a.opitch1 : a.opitch;
        const int lo = (layers && q == 0) ? 0 : l;
        cplx<T>* plane = third ? a.wall[grp]
                               : a.out[layers ? 0 : grp * a.nout + q] +
                                     (long)lo * (second ? a.out_pstride1 : a.out_pstride);
        cplx<T>* dst = plane + kxx + (long)ky0 * opitch;
        const cplx<T>* srow = bin + cc * SI + ky0;
        const long step = (long)TL * opitch;
#pragma unroll
        for (int i = 0; i < NYO / TL; ++i) dst[i * step] = srow[TL * i];
      }
    }
    __syncthreads();
  }
  if (a.nstage > 1) {
    stage ^= 1;
  } else if (next < nitems) {
    // single stage: every thread is past the last read of it (barrier above)
    yp_issue<T, NY>(a, next, ncb, bin0);
    cp_async_commit();
  }
  }
}

// ------------------------------------------------ right-hand side in y ----
// One y pass for a whole right-hand side: per column the forward transform of
// the convective products (NF rows, truncated or masked to N), of the two
// stresses (i kx t_x + i ky t_y), their sum, and one inverse transform.
template <typename T>
struct YRArgs {
  FastDiv d_ncb, d_np;  // division by the column blocks, nplanes (set by the launcher)
  int dep;         // launched by launch_dep: the tables are constant
  int C, lc, SI;       // C = 1 << lc columns per CTA, column stride of a shared slot
  int nslot;           // shared slots (set by the launcher): 2 = a copy runs under every transform
  int ncols;           // output columns
  int nkp;             // columns of the products (the rest are zero)
  int ppitch, spitch, opitch;  // complex values between rows of products / stresses / output
  long pstride, sstride, ostride;  // complex values between planes
  int plane0, nplanes, ngroups, lp;  // products exist on levels up to lp
  int tt;              // 2/3 rule (NF == N): largest |ky| of the products kept
  int nxh, lhx;
  const cplx<T>* p[4];
  const cplx<T>* sx[4];
  const cplx<T>* sy[4];
  cplx<T>* out[4];
  const T* kkx;
  const T* kky;
  const cplx<T>* tw_p;  // length NF table
  const cplx<T>* tw_s;  // length N table
};

// start the copy of one input's columns (C columns x NR rows) into a slot
template <typename T, int NR, int TL>
__device__ __forceinline__ void yr_copy(const YRArgs<T>& a, const cplx<T>* base, long plane, int pitch, int col0,
                                        int lim, cplx<T>* slot) {
  const int c = threadIdx.x & (a.C - 1);
  const int ky0 = threadIdx.x >> a.lc;
  const int kx = col0 + c;
  const bool valid = kx < lim;
  const cplx<T>* src = valid ? base + plane + kx + (long)ky0 * pitch : base;
  cplx<T>* dst = slot + c * a.SI + ky0;
  const long step = (long)TL * pitch;
#pragma unroll
  for (int i = 0; i < NR / TL; ++i) cp_async<int(sizeof(cplx<T>))>(dst + TL * i, valid ? src + i * step : base, valid);
}

// Persistent CTAs over (column block, level, equation).  The three inputs of
// an item and of the next ones pass through a ring of two shared slots, each
// refilled with the input after next as soon as its transform has left it, so
// that a copy runs under every transform; the inverse transform and the
// copy-out use the slot of the item's last input.  Two slots of the longer
// length per column keep 16 warps per SM in FP32 (three inputs side by side:
// 12), the register limit.  Where two slots leave room for fewer warps, one
// slot refilled between transforms takes their place: FP32 at 512 points 12
// -> 16 warps (814 -> 651 us, 512 x 512 x 96), FP64 at 512 points 4 -> 8 (400
// -> 335 us, 512 x 512 x 24), at 256 points 6 -> 12 (198 -> 181 us at 64
// levels, 741 -> 763 us at 256), at 64 points 22.9 -> 25.1 us.
template <typename T, int NF, int N>
__global__ void __launch_bounds__(sizeof(T) == 8 ? 128 : 256, sizeof(T) == 8 ? 3 : 2) k_yrhs(const YRArgs<T> a) {
  constexpr int TL = Geo<N>::T;
  static_assert(Geo<NF>::T == TL, "both lengths must share the lanes per sequence");
  constexpr int EF = Geo<NF>::E, E = Geo<N>::E;
  constexpr int PI_ = Layout<NF, false>::in, PO = Layout<NF, false>::out;
  constexpr int FI = Layout<N, false>::in, FO = Layout<N, false>::out;
  constexpr int II = Layout<N, true>::in, IO = Layout<N, true>::out;
  static_assert(FO == II, "forward output layout must feed the inverse");
  constexpr bool SAME = NF == N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* twp = reinterpret_cast<cplx<T>*>(smem_raw);  // forward NF (shared with forward N where equal)
  cplx<T>* tws = twp + (SAME ? 0 : Twm<NF, false>::len);
  cplx<T>* twi = tws + Twm<N, false>::len;
  T* kyrow = reinterpret_cast<T*>(twi + Twm<N, true>::len);
  cplx<T>* ring = reinterpret_cast<cplx<T>*>(kyrow + ((N + 3) & ~3));
  const int C = a.C, SI = a.SI;
  if constexpr (!SAME) twm_build<T, NF, false>(a.tw_p, twp, threadIdx.x, blockDim.x);
  twm_build<T, N, false>(a.tw_s, tws, threadIdx.x, blockDim.x);
  twm_build<T, N, true>(a.tw_s, twi, threadIdx.x, blockDim.x);
  for (int i = threadIdx.x; i < N; i += blockDim.x) kyrow[i] = a.kky[(long)i * a.lhx];
  dep_wait();
  const int ncb = (a.ncols + C - 1) / C;
  const long nitems = (long)ncb * a.nplanes * a.ngroups;
  // input `in` (0 products, 1 t_x, 2 t_y) of item `item` into ring slot `sl`
  auto issue = [&](long item, int in, int sl) {
    if (item < nitems) {
      const int pq = a.d_ncb(item), grp = a.d_np(pq);
      const int col0 = (int(item) - pq * ncb) * C;
      const int l = a.plane0 + pq - grp * a.nplanes;
      cplx<T>* slot = ring + sl * C * SI;
      if (in == 0)
        yr_copy<T, NF, TL>(a, a.p[grp], (long)l * a.pstride, a.ppitch, col0, l <= a.lp ? a.nkp : 0, slot);
      else
        yr_copy<T, N, TL>(a, in == 1 ? a.sx[grp] : a.sy[grp], (long)l * a.sstride, a.spitch, col0, a.ncols, slot);
    }
    cp_async_commit();
  };
  // the next input to copy; a slot is free again when its input is transformed
  const int flip = a.nslot - 1;
  long aitem = blockIdx.x;
  int ain = 0, asl = 0;
  auto issue_next = [&]() {
    issue(aitem, ain, asl);
    asl ^= flip;
    if (++ain == 3) {
      ain = 0;
      aitem += gridDim.x;
    }
  };
  auto arrived = [&]() {
    if (flip) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
  };
  issue_next();
  if (flip) issue_next();
  const int c = threadIdx.x / TL;
  const int lt = threadIdx.x % TL;
  int sl = 0;  // slot of the current input
  for (long item = blockIdx.x; item < nitems; item += gridDim.x, sl ^= flip) {
    const int pq = a.d_ncb(item), grp = a.d_np(pq);
    const int col0 = (int(item) - pq * ncb) * C;
    const int kx = col0 + c;
    const bool live = kx < a.ncols && kx != a.nxh;
    cplx<T> w[E];  // the sum, forward output layout of N (groups FO)
    {
      arrived();
      cplx<T>* seq = ring + (sl * C + c) * SI;
      cplx<T> f[EF];
#pragma unroll
      for (int g = 0; g < EF / PI_; ++g)
#pragma unroll
        for (int r = 0; r < PI_; ++r) f[g * PI_ + r] = seq[lt + TL * g + r * (NF / PI_)];
      reg_fft<T, NF, false>(f, seq, lt, SAME ? tws : twp);
      if constexpr (SAME) {
#pragma unroll
        for (int g = 0; g < E / FO; ++g)
#pragma unroll
          for (int r = 0; r < FO; ++r) {
            const int ky = lt + TL * g + r * (N / FO);
            const bool keep = ky <= a.tt || ky >= N - a.tt;
            w[g * FO + r] = keep ? f[g * FO + r] : cplx<T>{T(0), T(0)};
          }
      } else {
        // truncation NF -> N in the lane (as in k_ypass): m' < E/2 from m',
        // the rest from m' + E/2; lane 0 drops ky = N/2
        constexpr int GP = EF / PO, GO = E / II;
        static_for<E>([&](auto mc) {
          constexpr int mo = decltype(mc)::value;
          constexpr int ms = mo < E / 2 ? mo : mo + E / 2;
          constexpr int wi = (mo % GO) * II + mo / GO, fi = (ms % GP) * PO + ms / GP;
          w[wi] = (mo == E / 2 && lt == 0) ? cplx<T>{T(0), T(0)} : f[fi];
        });
      }
      __syncthreads();
      issue_next();
    }
#pragma unroll 1
    for (int in = 1; in <= 2; ++in) {
      sl ^= flip;
      arrived();
      cplx<T>* seq = ring + (sl * C + c) * SI;
      cplx<T> f[E];
#pragma unroll
      for (int g = 0; g < E / FI; ++g)
#pragma unroll
        for (int r = 0; r < FI; ++r) f[g * FI + r] = seq[lt + TL * g + r * (N / FI)];
      reg_fft<T, N, false>(f, seq, lt, tws);
      const T kxv = live ? a.kkx[kx] : T(0);
#pragma unroll
      for (int g = 0; g < E / FO; ++g)
#pragma unroll
        for (int r = 0; r < FO; ++r) {
          const int ky = lt + TL * g + r * (N / FO);
          if (live && ky != N / 2)
            w[g * FO + r] = c_add(w[g * FO + r], ik_mul(in == 1 ? kxv : kyrow[ky], f[g * FO + r]));
        }
      if (in == 1) {
        __syncthreads();
        issue_next();
      }
    }
    {
      cplx<T>* seq = ring + (sl * C + c) * SI;
      __syncwarp();
      reg_fft<T, N, true>(w, seq, lt, twi);
      __syncwarp();
#pragma unroll
      for (int g = 0; g < E / IO; ++g)
#pragma unroll
        for (int r = 0; r < IO; ++r) seq[lt + TL * g + r * (N / IO)] = w[g * IO + r];
      __syncthreads();
      const int l = a.plane0 + pq - grp * a.nplanes;
      const int cc = threadIdx.x & (C - 1);
      const int kxx = col0 + cc;
      if (kxx < a.ncols) {
        const int ky0 = threadIdx.x >> a.lc;
        cplx<T>* dst = a.out[grp] + (long)l * a.ostride + kxx + (long)ky0 * a.opitch;
        const cplx<T>* srow = ring + (sl * C + cc) * SI + ky0;
        const long step = (long)TL * a.opitch;
#pragma unroll
        for (int i = 0; i < N / TL; ++i) dst[i * step] = srow[TL * i];
      }
      __syncthreads();
      issue_next();
    }
  }
}

// ---------------------------------------------------------------- xinv ----
enum XIOp : int {
  XI_STORE = 0,  // out[f](l) = x_f for lo[f] <= l <= hi[f]
  XI_CONV = 1,   // -u, -v, -w and the vorticity from the spectra of u, v, w and their y derivatives
  XI_CONVS = 6,  // the gradient of theta from the spectra of theta and i ky theta
  XI_DIV = 2,    // rhs += x + dz(tz) + pf ; pressure-BC layers of the w equation
  XI_LASD = 3,   // 21 filtered fields -> L:M and M:M
  XI_WALL = 4,   // filtered u1, v1 -> u*, Neumann ghost value, wall stress
  XI_SCDYN = 5,  // 19 filtered fields of the dynamic Prandtl model -> K.X and X.X
};

enum : int { ADV_KEEP = 0, ADV_ZERO = 1, ADV_LID = 2 };
template <typename T>
struct XIArgs {
  FastDiv d_rows, d_ns, d_nin, d_nk;  // division by rows_pp, the staged rows per grid row, nin, nk (set by the launcher)
  int dep;         // launched by launch_dep: the tables are constant
  int op, nin, R;
  long nrows;
  int rows_pp;
  int plane0;
  int nk;          // modes present in the input rows (rest zero)
  int ipitch;      // complex values between input rows (>= nk; 0: nk)
  int nkc;         // values of a row that are copied: nk, in FP32 rounded up to whole 16 bytes where the pitch allows (set by the launcher)
  int nks;         // complex values between staged rows in shared memory (set by the launcher)
  int stage_rows;  // staged rows per stage (set by the launcher)
  int nbuf;        // input stages (set by the launcher): 2 = the next item's rows load during this one
  int merged;      // 1: each sequence is transformed in its own staged row (plain store, nstage 0)
  int nz;
  long in_pstride;
  long out_pstride;  // elements per plane of the output grid
  double c0, c1, c2, c3;
  double pf[4];
  int lo[MAXIN], hi[MAXIN];
  const cplx<T>* in[MAXIN];
  const T* refin[MAXIN];  // per-level values added back to input field f
  int lo_ref, hi_ref;     // combining ops: on these levels
  int fresh;              // XI_DIV: the input is the whole horizontal part, out is not read
  // XI_DIV inside a time step: equation q's variable adv_v[q] (nullptr: not
  // here) advances by dt (t1 rhs + t2 adv_f[q]); its levels 0 and nz + 1 stay
  // (ADV_KEEP), become zero (ADV_ZERO) or zero and level nz plus adv_top
  // (ADV_LID).  adv_ghosts: the ghost levels of the right-hand sides as their
  // buffers change roles: adv_f takes out's, and out takes BOGUS (2) or keeps
  // its own (1).
  T* adv_v[3];
  T* adv_f[3];
  int adv_lid[3];
  int adv_ghosts;
  double adv_dt, adv_t1, adv_t2, adv_top;
  T* out[16];
  const T* aux[8];
  const cplx<T>* tw;  // exp(-2 pi i m / NX), m < NX
  // several transforms of one staged row: nstage rows per grid row are
  // staged (0: nin); transform f reads staged row src[f] and, with dx[f],
  // multiplies it by i kx (kxr[m], the x wavenumbers, Nyquist zero) first
  int nstage;
  int src[MAXIN];
  int dx[MAXIN];
  const T* kxr;
  // XI_CONVS: staged rows theta, i ky theta at level l, theta at l - 1;
  // XI_CONV: staged rows u, v, w, i ky u, i ky w at level l, then u, v at
  // l - 1; refin[0..2] the per-plane references of u, v, w; c0 = 1/dz,
  // c1 the scale of the spectra
  int wall;
  // set by the launcher: every output (and the plane stride) admits stores of
  // whole (x_2m, x_2m+1) pairs
  int pair_store;
  // set by the launcher: stage the spectral rows with bulk copies (every
  // input and stage row 16-byte aligned); else per-thread cp.async copies
  int bulk;
  unsigned* status;  // device status word (ST_COPY_WAIT), may be null
};

// Plane of the spectrum that staged row f of level l comes from.  XI_CONV:
// the values of w on its two boundary levels lie apart (plane 0: level 1,
// plane nz + 2: level nz + 1), since the planes of those levels keep the w
// whose derivatives the gradients hold.
template <typename T>
__device__ __forceinline__ int xi_plane(const XIArgs<T>& a, int f, int l) {
  if (a.op == XI_CONVS) return f == 2 ? l - 1 : l;
  if (a.op != XI_CONV) return l;
  if (f >= 5) return l - 1;
  if (f == 2) return l == 1 ? 0 : (l == a.nz + 1 ? l + 1 : l);
  return l;
}
template <typename T>
__device__ __forceinline__ const cplx<T>* xi_row(const XIArgs<T>& a, int f, long g) {
  const int q = a.d_rows(g), j = int(g) - q * a.rows_pp;
  return a.in[f] + (long)xi_plane(a, f, a.plane0 + q) * a.in_pstride + (long)j * a.ipitch;
}

// x inverse pass: start the copies of the spectral rows of batch `item`
// (R rows x nin fields, nk values each) into the shared stage
template <typename T>
__device__ __forceinline__ void xi_issue(const XIArgs<T>& a, long item, cplx<T>* stage) {
  // one warp per row: the row address is formed once, the lanes copy its
  // nk values
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int ns = a.nstage ? a.nstage : a.nin;
  const int nrow = a.R * ns;
  for (int s = warp; s < nrow; s += nwarps) {
    const int r = a.d_ns(s);
    const int f = s - r * ns;
    const long g = item * a.R + r;
    const bool valid = g < a.nrows;
    const cplx<T>* base = a.in[f];
    const cplx<T>* row = valid ? xi_row(a, f, g) : base;
    cplx<T>* dst = stage + (long)s * a.nks;
    for (int m = lane; m < a.nk; m += 32) cp_async<int(sizeof(cplx<T>))>(dst + m, valid ? row + m : base, valid);
  }
}

// the same with bulk copies, issued by warp 0 (the other warps wait for what it
// issues, so nothing is looked at twice): lane 0 announces the bytes of every
// valid row's whole 16-byte parts, then each lane copies whole rows (their
// addresses are 16-byte aligned: a.bulk); the last value of an odd FP32 row
// without one to spare goes by a plain load and store (visible after the
// barrier that follows the wait)
template <typename T>
__device__ __forceinline__ void xi_issue_bulk(const XIArgs<T>& a, long item, cplx<T>* stage, uint64_t* mbar) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const int ns = a.nstage ? a.nstage : a.nin;
  const long rows_left = a.nrows - item * a.R;
  const int nrow = int(rows_left < a.R ? rows_left : a.R) * ns;
  const unsigned rb = unsigned(a.nkc * sizeof(cplx<T>));
  const unsigned rbulk = rb & ~15u;
  // the barrier's one arrival carries every byte the copies below bring (an
  // item always has a valid row, so the phase completes)
  if (lane == 0) mbar_expect_tx(mbar, nrow * rbulk);
  __syncwarp();
  tc::fence_async_smem();  // earlier generic reads of this stage come first
  for (int s = lane; s < nrow; s += 32) {
    const int r = a.d_ns(s), f = s - r * ns;
    const cplx<T>* row = xi_row(a, f, item * a.R + r);
    cplx<T>* dst = stage + (long)s * a.nks;
    bulk_g2s(dst, row, rbulk, mbar);
    if (rb != rbulk) dst[a.nkc - 1] = row[a.nkc - 1];
  }
}

// The ops of the x inverse in classes, each compiled on its own.  With every op
// in one kernel the register limit that its occupancy needs (64 in FP32, 128
// in FP64, at 256 threads) spilled 30-190 bytes per thread into each of them;
// apart, at 256^3 FP64: convective inputs 954 -> 870 us, the
// contractions of the LASD model 1485 -> 1273, stress divergence 346 -> 324; at 512 x 512
// x 96 FP32 convective inputs 807 -> 763, gradients 487 -> 457, scalar 268 ->
// 245, stress divergence 299 -> 270.
enum XIClass : int { XC_STORE = 0, XC_CONV = 1, XC_DIV = 2, XC_DYN = 3, XC_WALL = 4 };
inline int xi_class(int op) {
  switch (op) {
    case XI_CONV: case XI_CONVS: return XC_CONV;
    case XI_DIV: return XC_DIV;
    case XI_LASD: case XI_SCDYN: return XC_DYN;
    case XI_WALL: return XC_WALL;
    default: return XC_STORE;
  }
}

template <typename T, int NX, int CLS>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? (NX <= 256 ? 4 : 3) : 2) k_xinv(const XIArgs<T> a) {
  constexpr int M = NX / 2;
  constexpr int TL = Geo<M>::T;
  constexpr int E = Geo<M>::E;
  constexpr int RI = Layout<M, true>::in;
  constexpr int RO = Layout<M, true>::out;
  constexpr int SL = slot_stride(M, int(sizeof(cplx<T>)));  // complex values per sequence slot
  constexpr int XS = 2 * SL;         // the same slot viewed as reals
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* twm = tw + NX;  // twiddle matrices of the M-point inverse transform
  const int nseq = a.R * a.nin;
  const int npad = seq_pad<M>(nseq);
  const int ns = a.nstage ? a.nstage : a.nin;        // staged rows per grid row
  // a stage holds an even number of complex values, so the sequence slots
  // after the stages keep the 16-byte alignment of their four-point accesses
  // whatever the stage count (FP32 rows of an odd nks)
  const long stage_len = ((long)a.stage_rows * a.nks + 1) & ~1L;
  cplx<T>* stage0 = twm + Twm<M, true>::len;         // input rows of a work item: [R][ns][nk]
  cplx<T>* stage1 = stage0 + (a.nbuf > 1 ? stage_len : 0L);  // stage 0 again when single
  cplx<T>* buf = stage0 + a.nbuf * stage_len;        // sequence slots (none when merged)
  int* rowl = reinterpret_cast<int*>(buf + (a.merged ? 0L : (long)npad * SL));  // level of row r (-1: beyond the grid)
  int* rowj = rowl + a.R;
  T* kxs = reinterpret_cast<T*>(rowj + a.R);          // x wavenumbers (nstage > 0)
  // one mbarrier per input stage (bulk staging)
  uint64_t* bars = reinterpret_cast<uint64_t*>(
      (reinterpret_cast<uintptr_t>(kxs + (a.nstage ? a.nk + 2 : 0)) + 7) & ~uintptr_t(7));
  // persistent CTAs over batches of R rows; with two stages the spectral
  // rows of the next batch are copied into the other stage while this one
  // is transformed, with one stage after this batch's last read of it (warp 0
  // sets up the barriers and issues the bulk copies).
  const long nitems = (a.nrows + a.R - 1) / a.R;
  for (int i = threadIdx.x; i < NX; i += blockDim.x) tw[i] = a.tw[i];
  twm_build<T, M, true, 2>(a.tw, twm, threadIdx.x, blockDim.x);
  if (a.nstage)
    for (int i = threadIdx.x; i < a.nk; i += blockDim.x) kxs[i] = a.kxr[i];
  dep_wait();
  if (a.bulk) {
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0) {
        tc::mbar_init(&bars[0], 1);
        tc::mbar_init(&bars[1], 1);
        tc::fence_mbar_init();
      }
      __syncwarp();
      if ((long)blockIdx.x < nitems) xi_issue_bulk<T>(a, blockIdx.x, stage0, &bars[0]);
    }
  } else if ((long)blockIdx.x < nitems) {
    xi_issue<T>(a, blockIdx.x, stage0);
    cp_async_commit();
  }
  __syncthreads();
  unsigned phase = 0;  // bit b: parity of the next completion of bars[b]
  int stg = 0;
  for (long item = blockIdx.x; item < nitems; item += gridDim.x) {
  const long next = item + gridDim.x;
  const cplx<T>* stage = stg ? stage1 : stage0;
  bool late = false;  // this thread's wait for the item's rows ran out
  if (a.bulk) {
    if (a.nbuf > 1 && next < nitems) xi_issue_bulk<T>(a, next, stg ? stage0 : stage1, &bars[stg ^ 1]);
    late = !tc::mbar_wait(&bars[stg], (phase >> stg) & 1u);
    phase ^= 1u << stg;
  } else if (a.nbuf > 1 && next < nitems) {
    xi_issue<T>(a, next, stg ? stage0 : stage1);
    cp_async_commit();
    cp_async_wait<1>();
  } else {
    cp_async_wait<0>();
  }
  const long g0 = item * a.R;
  for (int r = blockDim.x - 1 - threadIdx.x; r < a.R; r += blockDim.x) {  // (not warp 0, which issues)
    const long g = g0 + r;
    const int q = a.d_rows(g);
    rowl[r] = (g < a.nrows) ? a.plane0 + q : -1;
    rowj[r] = (g < a.nrows) ? int(g) - q * a.rows_pp : 0;
  }
  if (__syncthreads_or(late)) {
    // the copies did not complete within the limit: record it, give the
    // copies in flight a last bounded wait (they write this CTA's shared
    // memory) and leave, every thread of the CTA together
    if (threadIdx.x == 0 && a.status) atomicOr(a.status, unsigned(ST_COPY_WAIT));
    tc::mbar_wait(&bars[stg], (phase >> stg) & 1u ^ 1u);
    if (a.nbuf > 1 && next < nitems) tc::mbar_wait(&bars[stg ^ 1], (phase >> (stg ^ 1)) & 1u);
    return;
  }
  // a plain store writes straight from registers; the other ops combine
  // fields per point through shared memory
  constexpr bool conv = CLS == XC_CONV;
  constexpr bool direct = CLS == XC_STORE || conv;
  if (conv && a.op == XI_CONVS) {
    // i kx theta over theta, d theta / dz over theta(l - 1); plane 0 holds the
    // wall's d theta / dz(1) itself
    cplx<T>* rows = const_cast<cplx<T>*>(stage);
    const T rdz = T(a.c0);
    for (int idx = threadIdx.x; idx < a.R * a.nk; idx += blockDim.x) {
      const int r = a.d_nk(idx);
      const int m = idx - r * a.nk;
      const int l = rowl[r];
      if (l < 0) continue;
      cplx<T>* q = rows + (long)r * 3 * a.nks + m;
      const cplx<T> t = q[0];
      if (l > 1) q[2 * a.nks] = c_scl(c_sub(t, q[2 * a.nks]), rdz);
      q[0] = ik_mul(kxs[m], t);
    }
    __syncthreads();
  }
  if (conv && a.op == XI_CONV) {
    // the vorticity in the staged rows: o1 over i ky w, o2 over u(l - 1), o3
    // over i ky u (compute_convective_padd.f90:145-165; the wall rows' means
    // of w derivatives over levels 1 and 2).  Boundary levels take the w of
    // the gradients from global memory.
    cplx<T>* rows = const_cast<cplx<T>*>(stage);
    const T rdz = T(a.c0);
    for (int idx = threadIdx.x; idx < a.R * a.nk; idx += blockDim.x) {
      const int r = a.d_nk(idx);
      const int m = idx - r * a.nk;
      const int l = rowl[r];
      if (l < 0) continue;
      cplx<T>* q = rows + (long)r * 7 * a.nks + m;
      const int n = a.nks;
      cplx<T> wp = q[2 * n], yw = q[4 * n];
      if (l == 1 || l == a.nz + 1) {
        const long o = (long)l * a.in_pstride + (long)rowj[r] * a.ipitch + m;
        wp = a.in[2][o];
        if (a.wall && l == 1) {
          wp = c_scl(c_add(wp, a.in[2][o + a.in_pstride]), T(0.5));
          yw = c_scl(c_add(yw, a.in[4][o + a.in_pstride]), T(0.5));
        }
      }
      const cplx<T> uz = c_scl(c_sub(q[0], q[5 * n]), rdz), vz = c_scl(c_sub(q[n], q[6 * n]), rdz);
      const T kx = kxs[m];
      q[3 * n] = c_sub(ik_mul(kx, q[n]), q[3 * n]);
      q[4 * n] = c_sub(yw, vz);
      q[5 * n] = c_sub(uz, ik_mul(kx, wp));
    }
    __syncthreads();
  }
  const int lane_t = threadIdx.x % TL;
  for (int base = 0; base < npad; base += blockDim.x / TL) {
    const int s = base + threadIdx.x / TL;
    if (base + (threadIdx.x / 32) * (32 / TL) >= npad) break;  // whole warp beyond the slots
    const int r = a.d_nin(s);
    const int f = s - r * a.nin;
    const bool valid = (s < nseq) && (rowl[r < a.R ? r : 0] >= 0);
    int l = 0, j = 0;
    if (valid) {
      l = rowl[r];
      j = rowj[r];
    }
    // merged: the staged row of sequence s is its slot (slots past the last
    // sequence follow the staged rows)
    const int srow = conv ? (s < nseq ? r * ns + a.src[f] : a.R * ns + (s - nseq)) : s;
    cplx<T>* seq = a.merged ? const_cast<cplx<T>*>(stage) + (long)srow * a.nks : buf + (long)s * SL;
    // c2r split: Z_m = (X_m + conj X_{M-m}) + i W^{-m} (X_m - conj X_{M-m}),
    // imaginary parts of the DC and Nyquist bins ignored
    cplx<T> v[E];
    const int fs = a.nstage ? a.src[f] : f;
    const bool dxf = CLS == XC_STORE && a.nstage && a.dx[f];
    const cplx<T>* row = valid ? stage + (long)(r * ns + fs) * a.nks : nullptr;  // the staged spectral row
    // The per-sequence choices (d/dx, whether every mode below M is present)
    // are made once here, not inside the unrolled element loop: with nk >= M
    // the partner X_{M-m} exists for every element but m = 0, which only the
    // first element of lane 0 can hold.
    auto split = [&](auto dx_c, auto full_c) {
      constexpr bool DX = decltype(dx_c)::value;
      constexpr bool FULL = decltype(full_c)::value;
#pragma unroll
      for (int gg = 0; gg < E / RI; ++gg)
#pragma unroll
        for (int rr = 0; rr < RI; ++rr) {
          const int m = lane_t + TL * gg + rr * (M / RI);
          const bool first = (gg == 0 && rr == 0);  // the only element that can hold m = 0
          cplx<T> xk, xm;
          if constexpr (FULL) {
            xk = row[m];
            xm = (first && m == 0 && a.nk == M) ? cplx<T>{T(0), T(0)} : row[M - m];
          } else {
            xk = (m < a.nk) ? row[m] : cplx<T>{T(0), T(0)};
            xm = (M - m < a.nk) ? row[M - m] : cplx<T>{T(0), T(0)};
          }
          if constexpr (DX) {  // d/dx: i kx X (compute_derivatives.f90:94-137)
            if constexpr (FULL) {
              xk = ik_mul(kxs[m], xk);
              if (!(first && m == 0 && a.nk == M)) xm = ik_mul(kxs[M - m], xm);
            } else {
              xk = (m < a.nk) ? ik_mul(kxs[m], xk) : xk;
              xm = (M - m < a.nk) ? ik_mul(kxs[M - m], xm) : xm;
            }
          }
          if (first && m == 0) {
            xk.y = T(0);
            xm.y = T(0);
          }
          v[gg * RI + rr] = c2r_split(xk, xm, tw[m]);
        }
    };
    if constexpr (sizeof(T) == 8) {
      // FP64: one generic loop (the specialised copies spill at the
      // 128-register budget: 256^3 gradients 511 -> 603 us)
#pragma unroll
      for (int gg = 0; gg < E / RI; ++gg)
#pragma unroll
        for (int rr = 0; rr < RI; ++rr) {
          const int m = lane_t + TL * gg + rr * (M / RI);
          cplx<T> z = {T(0), T(0)};
          if (valid) {
            cplx<T> xk = (m < a.nk) ? row[m] : cplx<T>{T(0), T(0)};
            cplx<T> xm = (M - m < a.nk) ? row[M - m] : cplx<T>{T(0), T(0)};
            if (dxf) {  // d/dx: i kx X (compute_derivatives.f90:94-137)
              xk = (m < a.nk) ? ik_mul(kxs[m], xk) : xk;
              xm = (M - m < a.nk) ? ik_mul(kxs[M - m], xm) : xm;
            }
            if (m == 0) {
              xk.y = T(0);
              xm.y = T(0);
            }
            z = c2r_split(xk, xm, tw[m]);
          }
          v[gg * RI + rr] = z;
        }
    } else if (!valid) {
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = cplx<T>{T(0), T(0)};
    } else if (a.nk >= M) {
      if (dxf) split(std::true_type{}, std::true_type{});
      else split(std::false_type{}, std::true_type{});
    } else {
      if (dxf) split(std::true_type{}, std::false_type{});
      else split(std::false_type{}, std::false_type{});
    }
    reg_fft<T, M, true>(v, seq, lane_t, twm);
    if constexpr (direct) {
      if (valid && l >= a.lo[f] && l <= a.hi[f]) {
        T ref = T(0);
        if (conv && a.op == XI_CONVS) {
          if (f == 2 && l > 1 && a.refin[0]) ref = T((double(a.refin[0][l]) - double(a.refin[0][l - 1])) * a.c0);
        } else if (conv) {
          // -u, -v, -w and their levels' references; the vertical differences'
          if (f < 3) ref = a.refin[f] ? -a.refin[f][xi_plane(a, f, l)] : T(0);
          else if (f < 5 && a.refin[0]) {
            const T* rf = a.refin[f == 3 ? 1 : 0];
            const double d = (double(rf[l]) - double(rf[l - 1])) * a.c0;
            ref = T(f == 3 ? -d : d);
          }
        } else if (a.refin[f]) {
          ref = a.refin[f][l];
        }
        const cplx<T> ref2 = {ref, ref};
        const T sg = conv ? T(a.op == XI_CONV && f < 3 ? -a.c1 : a.c1) : T(1);
        const cplx<T> sg2 = {sg, sg};
        const long off = (long)l * a.out_pstride + (long)j * NX;
        // the store form is chosen once per sequence (outside the unrolled loop)
        auto store = [&](auto pair_c) {
#pragma unroll
          for (int gg = 0; gg < E / RO; ++gg)
#pragma unroll
            for (int rr = 0; rr < RO; ++rr) {
              const int m = lane_t + TL * gg + rr * (M / RO);
              const cplx<T> z = c_fma(v[gg * RO + rr], sg2, ref2);
              if constexpr (decltype(pair_c)::value) {
                // one 8-byte (FP32) / 16-byte (FP64) store per output pair
                *reinterpret_cast<cplx<T>*>(a.out[f] + off + 2 * m) = z;
              } else {
                a.out[f][off + 2 * m] = z.x;
                a.out[f][off + 2 * m + 1] = z.y;
              }
            }
        };
        if (a.pair_store) store(std::true_type{});
        else store(std::false_type{});
      }
    } else {
      __syncwarp();
#pragma unroll
      for (int gg = 0; gg < E / RO; ++gg)
#pragma unroll
        for (int rr = 0; rr < RO; ++rr) seq[lane_t + TL * gg + rr * (M / RO)] = v[gg * RO + rr];
    }
  }
  if constexpr (!direct) {
  __syncthreads();
  const T* xs = reinterpret_cast<const T*>(buf);  // x_i of sequence s at xs[s*XS + i]
  if constexpr (CLS == XC_DIV) {
    // compute_derivatives.f90:544-574 + LES_engine.f90:546-551, one equation
    // per input (up to three): out[q] = rhs, aux[q] = tz, lo[q] = stag, pf[q]
    // = forcing; out[8]/out[9] = bottom/top pressure-BC layers of the
    // non-staggered (w) equation.  c0 = 1/dz.  Four consecutive points of one
    // equation per thread, everything it reads requested before its first
    // store (all equations of a point per thread spilled 70-240 bytes).
    using V = V4<T>;
    const T rdz = T(a.c0);
    const long pl = a.out_pstride;
    for (int idx = threadIdx.x; idx < nseq * (NX / 4); idx += blockDim.x) {
      const int s = idx / (NX / 4);
      const int i0 = 4 * (idx - s * (NX / 4));
      const int r = a.d_nin(s), q = s - r * a.nin;
      const int l = rowl[r];
      if (l < 0) continue;
      const long p2 = (long)rowj[r] * NX + i0;
      const long off = (long)l * pl + p2;
      T* out = a.out[q];
      T* u = a.adv_v[q];
      V xq = vld<V>(xs, (long)s * XS + i0);
      if (l >= 1 && l <= a.nz) {
        const T* tz = a.aux[q];
        const V t0 = vldg<V>(tz, off), t1 = vldg<V>(tz, a.lo[q] ? off + pl : off - pl);
        V uo = vsplat<V>(T(0)), fo = uo;
        if (u) {
          uo = vld<V>(u, off);
          fo = vld<V>(a.adv_f[q], off);
        }
        if (a.refin[q] && l >= a.lo_ref && l <= a.hi_ref) xq = xq + vsplat<V>(a.refin[q][l]);
        const V dzq = rdz * (a.lo[q] ? t1 - t0 : t0 - t1);  // ddz_w, ddz_uv
        const V base = a.fresh ? xq : vld<V>(out, off) + xq;
        const V rhs = (base + dzq) + vsplat<V>(T(a.pf[q]));
        vst(out + off, rhs);
        if (u) {
          const V un = uo + T(a.adv_dt) * (T(a.adv_t1) * rhs + T(a.adv_t2) * fo);
          vst(u + off, un);
          if (a.adv_lid[q] == ADV_LID && l == a.nz) vst(u + off + pl, un + vsplat<V>(T(a.adv_top)));
          if (a.adv_lid[q] != ADV_KEEP && l == 1) vst(u + p2, vsplat<V>(T(0)));
        }
        if (!a.lo[q] && l == 1 && a.out[8]) vst(a.out[8] + p2, xq + dzq);
      } else {
        if (a.refin[q] && l >= a.lo_ref && l <= a.hi_ref) xq = xq + vsplat<V>(a.refin[q][l]);
        if (!a.lo[q] && l == a.nz + 1 && a.out[9]) vst(a.out[9] + p2, xq);
        if (u && a.adv_lid[q] == ADV_ZERO && l == a.nz + 1) vst(u + off, vsplat<V>(T(0)));
      }
      if (a.adv_ghosts && (l == 1 || l == a.nz + 1)) {
        const long gh = l == 1 ? p2 : off;
        vst(a.adv_f[q] + gh, vld<V>(out, gh));
        if (a.adv_ghosts == 2) vst(out + gh, vsplat<V>(T(BOGUS)));
      }
    }
  }
  if constexpr (CLS == XC_DYN) {
    // one point per thread: consecutive lanes read consecutive values of
    // every field's slot (four points per thread read them at a stride of
    // four, four lanes to a bank, and left most threads of a one-row item
    // idle: the 21-field contraction at 256^3 FP64 went from 1836 to 1485 us)
    for (int idx = threadIdx.x; idx < a.R * NX; idx += blockDim.x) {
      const int r = idx / NX;
      const int i = idx - r * NX;
      const int l = rowl[r];
      if (l < 0) continue;
      const long off = (long)l * a.out_pstride + (long)rowj[r] * NX + i;
      const T* x = xs + (long)(r * a.nin) * XS + i;  // field f at x[f*XS]
      if (a.op == XI_LASD) {
        // compute_LagScaleDep.f90:541-594; c0 = 2 delta^2, c1 = alpha^2
        const T uf = x[0], vf = x[XS], wf = x[2 * XS];
        const T a11 = x[3 * XS] - uf * uf;
        const T a12 = x[4 * XS] - uf * vf;
        const T a13 = x[5 * XS] - uf * wf;
        const T a22 = x[6 * XS] - vf * vf;
        const T a23 = x[7 * XS] - vf * wf;
        const T a33 = x[8 * XS] - wf * wf;
        const T s11 = x[9 * XS], s12 = x[10 * XS], s13 = x[11 * XS];
        const T s22 = x[12 * XS], s23 = x[13 * XS], s33 = x[14 * XS];
        const T sft = sqrt(T(2) * (s11 * s11 + s22 * s22 + s33 * s33 +
                                   T(2) * (s12 * s12 + s13 * s13 + s23 * s23)));
        const T cst = T(a.c0), tf2 = T(a.c1);
        const T b11 = cst * (x[15 * XS] - tf2 * sft * s11);
        const T b12 = cst * (x[16 * XS] - tf2 * sft * s12);
        const T b13 = cst * (x[17 * XS] - tf2 * sft * s13);
        const T b22 = cst * (x[18 * XS] - tf2 * sft * s22);
        const T b23 = cst * (x[19 * XS] - tf2 * sft * s23);
        const T b33 = cst * (x[20 * XS] - tf2 * sft * s33);
        a.out[0][off] = a11 * b11 + a22 * b22 + a33 * b33 + T(2) * (a12 * b12 + a13 * b13 + a23 * b23);
        a.out[1][off] = b11 * b11 + b22 * b22 + b33 * b33 + T(2) * (b12 * b12 + b13 * b13 + b23 * b23);
      } else {
        // K_j = filt(u_j theta) - filt(u_j) filt(theta),
        // X_j = Delta^2 (filt(|S| d_j theta) - alpha^2 |S~| filt(d_j theta));
        // c0 = Delta^2, c1 = alpha^2
        const T uf = x[0], vf = x[XS], wf = x[2 * XS], tf = x[3 * XS];
        const T k1 = x[4 * XS] - uf * tf;
        const T k2 = x[5 * XS] - vf * tf;
        const T k3 = x[6 * XS] - wf * tf;
        const T s11 = x[7 * XS], s12 = x[8 * XS], s13 = x[9 * XS];
        const T s22 = x[10 * XS], s23 = x[11 * XS], s33 = x[12 * XS];
        const T sft = sqrt(T(2) * (s11 * s11 + s22 * s22 + s33 * s33 +
                                   T(2) * (s12 * s12 + s13 * s13 + s23 * s23)));
        const T d2 = T(a.c0), tf2 = T(a.c1);
        const T x1 = d2 * (x[16 * XS] - tf2 * sft * x[13 * XS]);
        const T x2 = d2 * (x[17 * XS] - tf2 * sft * x[14 * XS]);
        const T x3 = d2 * (x[18 * XS] - tf2 * sft * x[15 * XS]);
        a.out[0][off] = k1 * x1 + k2 * x2 + k3 * x3;
        a.out[1][off] = x1 * x1 + x2 * x2 + x3 * x3;
      }
    }
  }
  if constexpr (CLS == XC_WALL) {
    // compute_wall_law.f90:143-183, 247-251 on the filtered first level, one
    // point per thread (a plane is few rows, and the FP64 logarithm and
    // divisions of a point are a long dependent chain): c0 = dz, aux[0] = z0
    // plane; out: u_star_avg, lbc_u, lbc_v, txz(1), tyz(1), dudz(1), dvdz(1)
    for (int idx = threadIdx.x; idx < a.R * NX; idx += blockDim.x) {
      const int r = idx / NX;
      const int i = idx - r * NX;
      if (rowl[r] < 0) continue;
      const long p2 = (long)rowj[r] * NX + i;
      const T* x = xs + (long)(r * a.nin) * XS + i;
      const T ru = a.refin[0] ? a.refin[0][rowl[r]] : T(0), rv = a.refin[1] ? a.refin[1][rowl[r]] : T(0);
      const double u1 = double(x[0] + ru), v1 = double(x[XS] + rv);
      const double uavg = sqrt(u1 * u1 + v1 * v1);
      const double dz = a.c0;
      const double ustar = KVONK * uavg / log((0.5 * dz) / double(a.aux[0][p2]));
      double bu = 0.0, bv = 0.0, tx = 0.0, ty = 0.0;
      if (uavg != 0.0) {
        bu = ustar / (0.5 * dz * KVONK) * u1 / uavg;
        bv = ustar / (0.5 * dz * KVONK) * v1 / uavg;
        tx = (ustar * ustar) * u1 / uavg;
        ty = (ustar * ustar) * v1 / uavg;
      }
      a.out[0][p2] = T(ustar);
      a.out[1][p2] = T(bu);
      a.out[2][p2] = T(bv);
      const long o1 = a.out_pstride + p2;  // level 1 of a field
      a.out[3][o1] = T(tx);
      a.out[4][o1] = T(ty);
      a.out[5][o1] = T(bu);
      a.out[6][o1] = T(bv);
    }
  }
  }  // the combining ops
  __syncthreads();
  if (a.nbuf > 1) {
    stg ^= 1;
  } else if (next < nitems) {
    // single stage: every thread is past the last read of it (barrier above)
    if (a.bulk) {
      xi_issue_bulk<T>(a, next, stage0, &bars[0]);
    } else {
      xi_issue<T>(a, next, stage0);
      cp_async_commit();
    }
  }
  }
}

}  // namespace les
