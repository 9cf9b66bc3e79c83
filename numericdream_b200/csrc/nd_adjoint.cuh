// Adjoint of the Lambert image with respect to formula @params and an orbit camera
// pose, by implicit differentiation at the hit point.
//
// For every hit ray, with t the forward's hit distance, p = o + d t, g = grad DE(p):
//   the march stops where DE(p(t); theta) = eps(t) = coef t + floor, so
//     dt/dtheta = -(dDE/dtheta|_t fixed) / (g . d - coef)
//   dp/dtheta = do/dtheta + t dd/dtheta + d dt/dtheta
//   the normal is n = D / |D| with D_i = DE(p + h e_i) - DE(p - h e_i), h = hc t
//   (central differences), so dD_i/dtheta is the difference of the DE's total
//   derivatives at the two taps, the taps moving with dp/dtheta +- e_i dh/dtheta
//   dn = (dD - n (n . dD)) / |D|
//   I = a + (1 - a) max(n . L, 0)  =>  dI = (1 - a) [n . L > 0] (L . dn)
// and dLoss/dtheta = sum over rays of dLoss/dI * dI/dtheta.  Every DE total
// derivative is ONE evaluation of the formula code with T = Dual<S>, the position
// seeded with its tangent and the parameters with theirs.  Silhouette (visibility)
// changes are not differentiated: the gradient is that of the image's interior.
// Neither are hits where DE - eps(t) changes sign by a jump rather than through
// zero: a DE can be discontinuous (a Mandelbulb of non-integer power jumps where an
// iterate crosses atan2's branch cut, the half-plane y = 0, x < 0), and a hit on such
// a sheet moves with the sheet, not with the level set.  Such hits are recognised by
// their residual |DE(p) - eps(t)|, which a root reached by bisection does not have.
#pragma once

#include "nd_dual.h"
#include "nd_rayprog.h"

namespace nd {

constexpr int kMaxAdjParams = 4;  // formula @params per backward call
constexpr int kPoseParams = 3;    // yaw, pitch, distance of the orbit camera

// Derivatives of a view's camera with respect to yaw, pitch and distance.
struct PoseTangents {
  double dorg[kPoseParams][3];
  double dfwd[kPoseParams][3];
  double dright[kPoseParams][3];
  double dup[kPoseParams][3];
};

struct AdjointArgs {
  const DevView* views;
  int32_t nviews;
  int64_t total_rays;
  const PoseTangents* tangents;  // per view (launch order)
  const double* depth64;         // forward G-buffer (by G-buffer index)
  const float* normal4;
  const float* dL_dshade;        // nullable when grad is null
  double* grad;                  // nullable: [user view][nparam + 3], added to
  double* dshade;                // nullable: dI/dtheta per G-buffer slot [slot][nparam + 3]
  int32_t param_idx[kMaxAdjParams];
  int32_t nparam;
  int32_t num_sms;
  int32_t inline_thetas;  // 0: adjoint_surface leaves the thetas to the second kernel
  int64_t first;  // the rays [first, last) of the launch are worked on at a time
  int64_t last;
  unsigned* counts;     // entries in hits and in lit
  int32_t* hits;        // contributing rays, as indices from first
  struct LitRay* lit;   // those whose derivatives are not zero
};

// A listed ray that reached its derivatives: what the first adjoint kernel found.
struct LitRay {
  int32_t ray, view;
  double denom, D[3];
};
// Rays worked on at a time: it bounds the scratch (44 bytes a ray).
constexpr int64_t kAdjointRays = int64_t(1) << 22;
// Blocks of 128 threads per SM the adjoint kernels are compiled for: surface FP32 and
// FP64, thetas FP32 and FP64.  Measured for the thetas: FP32 5 / 6 / 8 blocks 978 / 1024 /
// 1003 us a backward of 4 views of 512 x 512; FP64 3 / 4 blocks (146 registers; 128 with 12
// bytes spilled) 1717 / 1530 us a backward of 2 views of 256 x 256.
constexpr int kSurfaceBlocks32 = 6, kSurfaceBlocks64 = 4, kThetaBlocks32 = 5, kThetaBlocks64 = 4;

// Parameter accessor with one dual tangent: parameter `seed` gets tangent 1.
template <class S> struct DualParams {
  const float* v;
  int seed;
  ND_DEV_INLINE ndw::Dual<S> operator[](int i) const { return ndw::mkd(S(v[i]), i == seed ? S(1) : S(0)); }
};

// The DE of view v at p and its derivative along (position tangent tan, parameter seed).
template <class Set, class S>
ND_DEV_INLINE ndw::Dual<S> de_dir_full(const DevView& v, D3 p, D3 tan, int seed) {
  typedef ndw::Dual<S> DS;
  const ndw::v3<DS> q = ndw::v3<DS>(ndw::mkd(S(p.x), S(tan.x)), ndw::mkd(S(p.y), S(tan.y)), ndw::mkd(S(p.z), S(tan.z)));
  return Set::template de_with<DS, DualParams<S>>(v.code, q, DualParams<S>{v.params, seed}, v).d;
}
template <class Set, class S>
ND_DEV_INLINE S de_dir(const DevView& v, D3 p, D3 tan, int seed) {
  return de_dir_full<Set, S>(v, p, tan, seed).d;
}

// Largest |DE(p) - eps(t)| / eps(t) at a hit that is a root of the level set.  FP64
// bisection leaves ~1e-13.  An FP32 DE near the surface carries rounding of ~1e-3 of
// eps (12 iterations amplify each ulp by about dr), so FP32 tells only jumps above
// 1e-2 of eps from roots; the smaller jumps it misses are the FP32 adjoint's limit.
template <class S> struct RootTol;
template <> struct RootTol<double> { static constexpr double value = 1e-6; };
template <> struct RootTol<float> { static constexpr double value = 1e-2; };

ND_DEV_INLINE D3 axpy(D3 a, double s, D3 b) { return D3{a.x + s * b.x, a.y + s * b.y, a.z + s * b.z}; }
ND_DEV_INLINE double dot3(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
ND_DEV_INLINE D3 axis(int i, double s) { return D3{i == 0 ? s : 0.0, i == 1 ? s : 0.0, i == 2 ? s : 0.0}; }

// The ray of a listed hit: what both adjoint kernels start from.
struct AdjointRay {
  double ux, uy, wn, t, hc, h;
  D3 d, p;
};
ND_DEV_INLINE AdjointRay adjoint_ray(const DevView& v, int64_t local, double t) {
  AdjointRay r;
  ray_uv(v, local, &r.ux, &r.uy);
  const D3 w = D3{v.fwd[0] + v.right[0] * r.ux + v.up[0] * r.uy, v.fwd[1] + v.right[1] * r.ux + v.up[1] * r.uy,
                  v.fwd[2] + v.right[2] * r.ux + v.up[2] * r.uy};
  r.wn = sqrt(dot3(w, w));
  r.d = ray_dir(v, local);  // w / |w| exactly as the forward computed it
  r.p = fmadd(D3{v.org[0], v.org[1], v.org[2]}, r.d, t);
  r.t = t;
  const bool central = v.normal_h_coef > 0.0f;
  r.hc = central ? double(v.normal_h_coef) : double(v.eps_coef);
  r.h = central ? r.hc * t : double(v.eps_coef) * t + double(v.eps_floor);
  return r;
}

// dp/dtheta_k with t held fixed (k < nparam: params[param_idx[k]]; then yaw, pitch, dist).
ND_DEV_INLINE D3 adjoint_tangent(const PoseTangents& T, const AdjointRay& r, int k, int nparam) {
  D3 dorg = D3{0, 0, 0}, dd = D3{0, 0, 0};
  if (k >= nparam && k < nparam + kPoseParams) {
    const int j = k - nparam;
    dorg = D3{T.dorg[j][0], T.dorg[j][1], T.dorg[j][2]};
    const D3 dw = D3{T.dfwd[j][0] + r.ux * T.dright[j][0] + r.uy * T.dup[j][0],
                     T.dfwd[j][1] + r.ux * T.dright[j][1] + r.uy * T.dup[j][1],
                     T.dfwd[j][2] + r.ux * T.dright[j][2] + r.uy * T.dup[j][2]};
    const double dd_par = dot3(r.d, dw);
    dd = D3{(dw.x - r.d.x * dd_par) / r.wn, (dw.y - r.d.y * dd_par) / r.wn, (dw.z - r.d.z * dd_par) / r.wn};
  }
  return axpy(dorg, r.t, dd);
}

// dI/dtheta_k of one ray, one tangent to an evaluation.  Three FP64 tangents to an evaluation
// would share its arccosine, powers and sines (0.83 ms where one takes 1.53), but the compiler
// then fuses other products, in the values too, and a grazing ray turns an ulp of those into
// 1e-9 to 1e-7 of its derivatives.
template <class Set, class S>
ND_DEV_INLINE double adjoint_theta(const DevView& v, const PoseTangents& T, const int32_t* param_idx, int nparam,
                                   const AdjointRay& r, double denom, const D3& D, int k) {
  // |D| as adjoint_surface has it: its sum is fused in this order there, left to the compiler
  // in another one here
  const double Dn = sqrt(fma_d(D.z, D.z, fma_d(D.x, D.x, rn_mul(D.y, D.y))));
  const D3 n = D3{D.x / Dn, D.y / Dn, D.z / Dn};
  const D3 L = D3{v.light[0], v.light[1], v.light[2]};
  const int seed = k < nparam ? param_idx[k] : -1;
  const D3 ptan0 = adjoint_tangent(T, r, k, nparam);
  const double a_k = double(de_dir<Set, S>(v, r.p, ptan0, seed));
  const double dt = -a_k / denom;
  const D3 dp = axpy(ptan0, dt, r.d);
  const double dh = r.hc * dt;
  double dD[3];
  for (int i = 0; i < 3; ++i) {
    const D3 tp = axpy(dp, dh, axis(i, 1.0));
    const D3 tm = axpy(dp, -dh, axis(i, 1.0));
    dD[i] = double(de_dir<Set, S>(v, axpy(r.p, r.h, axis(i, 1.0)), tp, seed)) -
            double(de_dir<Set, S>(v, axpy(r.p, -r.h, axis(i, 1.0)), tm, seed));
  }
  const double nd = n.x * dD[0] + n.y * dD[1] + n.z * dD[2];
  const D3 dn = D3{(dD[0] - n.x * nd) / Dn, (dD[1] - n.y * nd) / Dn, (dD[2] - n.z * nd) / Dn};
  return (1.0 - kSimpleAmbient) * dot3(L, dn);
}

// What the derivatives along every theta share: g . d - coef and the normal's
// central-difference vector D.  False when the pixel contributes nothing (a back-lit
// normal, a degenerate gradient, a hit on a jump of the DE).
//
// The FP32 form ends in the loop over the first `thetas` derivatives, which the kernels
// run zero times (adjoint_theta computes them for the lit rays): the compiler contracts the
// gradient's products into FMAs by what surrounds them, and with the loop there the
// derivatives keep the rounding they had when one lane computed all of them.  Without it
// the gradient's x component is up to 16 ulps off and the rows 1e-6 in norm (an opaque
// seed or axis, a function of its own, another order of the axes and fused operators of the
// duals move them as much or more); it costs 15 us of 884.  FP64 rows keep their bits
// without it.
template <class Set, class S>
ND_DEV_INLINE bool adjoint_surface(const DevView& v, const PoseTangents& T, const int32_t* param_idx, int nparam,
                                   int thetas, const AdjointRay& r, double* denom, double* Dv, double* dI) {
  // value and gradient of the DE at the hit
  const ndw::Dual<S> gx = de_dir_full<Set, S>(v, r.p, axis(0, 1.0), -1);
  const D3 g = D3{double(gx.d), double(de_dir<Set, S>(v, r.p, axis(1, 1.0), -1)),
                  double(de_dir<Set, S>(v, r.p, axis(2, 1.0), -1))};
  const double eps_t = double(v.eps_coef) * r.t + double(v.eps_floor);
  if (eps_t > 0.0 && !(fabs(double(gx.v) - eps_t) <= RootTol<S>::value * eps_t)) return false;
  *denom = dot3(g, r.d) - double(v.eps_coef);
  // the normal's central-difference vector D
  for (int i = 0; i < 3; ++i)
    Dv[i] = double(de_dir_full<Set, S>(v, axpy(r.p, r.h, axis(i, 1.0)), D3{0, 0, 0}, -1).v) -
            double(de_dir_full<Set, S>(v, axpy(r.p, -r.h, axis(i, 1.0)), D3{0, 0, 0}, -1).v);
  const D3 D = D3{Dv[0], Dv[1], Dv[2]};
  const double Dn = sqrt(dot3(D, D));
  if (!(Dn > 0.0) || *denom == 0.0) return false;
  const D3 n = D3{D.x / Dn, D.y / Dn, D.z / Dn};
  if (!(dot3(n, D3{v.light[0], v.light[1], v.light[2]}) > 0.0)) return false;
  if constexpr (sizeof(S) == 4 || Set::kCount > 1)
    for (int k = 0; k < thetas; ++k) dI[k] = adjoint_theta<Set, S>(v, T, param_idx, nparam, r, *denom, D, k);
  return true;
}

#if defined(__CUDACC__)
// Appends a block's wanted rays to a list: one atomic per block, so that the list keeps
// runs of neighbouring rays together.  Returns this thread's slot (when it wants one).
__device__ __forceinline__ unsigned block_append(bool want, unsigned* count) {
  __shared__ unsigned warp_want[32], base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, want);
  __syncthreads();  // the last call's slots have been read
  if (lane == 0) warp_want[warp] = unsigned(__popc(m));
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned n = 0;
    for (int w = 0; w < warps; ++w) n += warp_want[w];
    base = n ? atomicAdd(count, n) : 0u;
  }
  __syncthreads();
  unsigned at = base + __popc(m & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) at += warp_want[w];
  return at;
}

// The rays of [first, last) that may contribute (hits with a loss weight, or every hit
// when the Jacobian is asked for), as indices from first, in hits[0 .. *count).  The
// Jacobian rows of every ray are zeroed here.
__global__ static void __launch_bounds__(256) adjoint_list_kernel(const __grid_constant__ AdjointArgs a) {
  const int64_t it = a.first + int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int K = a.nparam + kPoseParams;
  bool want = false;
  if (it < a.last) {
    const DevView& v = a.views[find_view(a.views, a.nviews, it)];
    const int64_t r = v.out_offset + it - v.ray_offset;
    want = a.normal4[4 * r + 3] > 0.5f && (a.dshade || a.dL_dshade[r] != 0.0f);
    if (a.dshade)
      for (int k = 0; k < K; ++k) a.dshade[r * K + k] = 0.0;
  }
  const unsigned at = block_append(want, a.counts);
  if (want) a.hits[at] = int(it - a.first);
}

// The adjoint of a listed hit is two kernels.  The first, one lane per hit, does what all
// thetas share: the DE's value and gradient at the hit and its values at the six normal
// taps.  About half of the hits end there (back-lit normals).  The second does a lit ray's
// K = nparam + 3 derivatives, 7 dual evaluations each.  Both lists are dense, so that no
// lane waits for a neighbour that missed, was back-lit or had no weight: one kernel with one
// lane per ray of the image ran with 15 (FP32) and 13 (FP64) of 32 lanes active.  The
// kernels are bound by instruction issue (FP32) and by the FP64 pipe's latency (FP64).  A
// backward call with two parameters: 4 views of 512 x 512, FP32, 2.19 -> 0.89 ms; 2 views of
// 256 x 256, FP64, 4.12 -> 1.53 ms.
template <class Set, class S>
__global__ void __launch_bounds__(128, sizeof(S) == 4 ? kSurfaceBlocks32 : kSurfaceBlocks64)
    adjoint_surface_kernel(const __grid_constant__ AdjointArgs a) {
  const int n = int(a.counts[0]);
  const int stride = int(gridDim.x) * int(blockDim.x);
  for (int first = int(blockIdx.x) * int(blockDim.x); first < n; first += stride) {  // block-uniform
    const int entry = first + int(threadIdx.x);
    bool lit = false;
    LitRay o;
    if (entry < n) {
      const int64_t it = a.first + a.hits[entry];
      o.ray = int(it - a.first);
      o.view = find_view(a.views, a.nviews, it);
      const DevView& v = a.views[o.view];
      const int64_t local = it - v.ray_offset;
      double none[kMaxAdjParams + kPoseParams];
      lit = adjoint_surface<Set, S>(v, a.tangents[o.view], a.param_idx, a.nparam, a.inline_thetas,
                                    adjoint_ray(v, local, a.depth64[v.out_offset + local]), &o.denom, o.D, none);
      if (a.inline_thetas > 0) o.denom = none[0];  // never taken: it keeps the loop's results in use
    }
    const unsigned at = block_append(lit, a.counts + 1);
    if (lit) a.lit[at] = o;
  }
}

// One lane per lit ray and theta; the thetas of a ray are neighbours.  A lane keeps its
// theta from one ray to the next (the stride is a multiple of the thetas), so it sums its
// view's gradient in a register.
template <class Set, class S>
__global__ void __launch_bounds__(128, sizeof(S) == 4 ? kThetaBlocks32 : kThetaBlocks64)
    adjoint_theta_kernel(const __grid_constant__ AdjointArgs a) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int K = a.nparam + kPoseParams;
  const int64_t items = int64_t(a.counts[1]) * K;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x / K * K;
  const int64_t me = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int mine = int(me % K);
  double acc = 0.0;
  int cur = -1;
  // adds the sums of the lanes whose view is not `keep`: one atomic per view and theta
  auto flush = [&](int keep) {
    unsigned left = __ballot_sync(full, cur >= 0 && cur != keep);
    while (left) {
      const int src = __ffs(left) - 1;
      const int view = __shfl_sync(full, cur, src), k = __shfl_sync(full, mine, src);
      const bool in = cur == view && mine == k && cur != keep;
      left &= ~__ballot_sync(full, in);
      double x = in ? acc : 0.0;
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(full, x, o);
      if (lane == 0 && x != 0.0) atomicAdd(&a.grad[int64_t(a.views[view].user_index) * K + k], x);
      if (in) cur = -1;
    }
  };
  for (int64_t base = me - lane; base < items; base += stride) {  // warp-uniform
    const int64_t item = base + lane;
    const bool live = item < items && me < stride;
    LitRay o;
    if (live) o = a.lit[item / K];
    if (a.grad) {
      const int view = live ? o.view : cur;
      if (__any_sync(full, cur >= 0 && view != cur)) flush(view);
      if (live && cur < 0) {
        cur = view;
        acc = 0.0;
      }
    }
    if (live) {
      const DevView& v = a.views[o.view];
      const int64_t local = a.first + o.ray - v.ray_offset;
      const int64_t r = v.out_offset + local;
      const double dI = adjoint_theta<Set, S>(v, a.tangents[o.view], a.param_idx, a.nparam,
                                              adjoint_ray(v, local, a.depth64[r]), o.denom,
                                              D3{o.D[0], o.D[1], o.D[2]}, mine);
      if (a.dshade) a.dshade[r * K + mine] = dI;
      acc += (a.grad ? double(a.dL_dshade[r]) : 0.0) * dI;
    }
  }
  if (a.grad) flush(-2);
}

// A formula group's adjoint: one lane per listed ray does all of it.  Split in two like a
// single formula's, the group's kernels are compiled with other fused products: the rows of
// its Mandelbulbs moved by 2e-4 (FP32, 2-norm) and 1e-12 (FP64).  Four small views of the
// four-formula group: one lane per image ray 0.45 (FP32) and 1.72 ms (FP64), this 0.25 and
// 1.57, split 0.18 and 0.85.
template <class Set, class S>
__global__ void __launch_bounds__(128) adjoint_ray_kernel(const __grid_constant__ AdjointArgs a) {
  const unsigned full = 0xffffffffu;
  const int K = a.nparam + kPoseParams;
  const int n = int(a.counts[0]);
  const int stride = int(gridDim.x) * int(blockDim.x);
  for (int first = int(blockIdx.x) * int(blockDim.x); first < n; first += stride) {  // block-uniform
    const int entry = first + int(threadIdx.x);
    double dI[kMaxAdjParams + kPoseParams];
    for (int k = 0; k < kMaxAdjParams + kPoseParams; ++k) dI[k] = 0.0;
    int vi = -1;
    if (entry < n) {
      const int64_t it = a.first + a.hits[entry];
      const int at = find_view(a.views, a.nviews, it);
      const DevView& v = a.views[at];
      const int64_t local = it - v.ray_offset;
      const int64_t r = v.out_offset + local;
      double denom, D[3];
      if (adjoint_surface<Set, S>(v, a.tangents[at], a.param_idx, a.nparam, K, adjoint_ray(v, local, a.depth64[r]), &denom,
                                  D, dI)) {
        vi = at;
        if (a.dshade)
          for (int k = 0; k < K; ++k) a.dshade[r * K + k] = dI[k];
        if (a.grad)
          for (int k = 0; k < K; ++k) dI[k] *= double(a.dL_dshade[r]);
      }
    }
    if (!a.grad) continue;
    // one atomic per theta where the warp's lit rays are of one view, else one per ray
    const int view = __reduce_max_sync(full, vi);
    const bool one = __all_sync(full, vi < 0 || vi == view);
    if (view < 0) continue;
    for (int k = 0; k < K; ++k) {
      double x = vi >= 0 ? dI[k] : 0.0;
      if (one) {
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(full, x, o);
        if ((threadIdx.x & 31) == 0 && x != 0.0) atomicAdd(&a.grad[int64_t(a.views[view].user_index) * K + k], x);
      } else if (x != 0.0) {
        atomicAdd(&a.grad[int64_t(a.views[vi].user_index) * K + k], x);
      }
    }
  }
}

// A resident grid of a kernel that strides over at most `most` lanes of work.
template <class Kernel> cudaError_t launch_listed(Kernel kernel, const AdjointArgs& a, int64_t most, cudaStream_t s) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, 0);
  if (e != cudaSuccess) return e;
  const int64_t needed = (most + 127) / 128, resident = int64_t(a.num_sms) * (per_sm < 1 ? 1 : per_sm);
  kernel<<<unsigned(needed < resident ? needed : resident), 128, 0, s>>>(a);
  return cudaGetLastError();
}

template <class Set, class S> cudaError_t launch_adjoint(AdjointArgs a, cudaStream_t s) {
  for (a.first = 0; a.first < a.total_rays; a.first = a.last) {
    a.last = a.total_rays - a.first > kAdjointRays ? a.first + kAdjointRays : a.total_rays;
    const int64_t n = a.last - a.first;
    cudaError_t e = cudaMemsetAsync(a.counts, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    adjoint_list_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(a);
    e = cudaGetLastError();
    if constexpr (Set::kCount > 1) {
      if (e == cudaSuccess) e = launch_listed(adjoint_ray_kernel<Set, S>, a, n, s);
    } else {
      if (e == cudaSuccess) e = launch_listed(adjoint_surface_kernel<Set, S>, a, n, s);
      if (e == cudaSuccess) e = launch_listed(adjoint_theta_kernel<Set, S>, a, n * (a.nparam + kPoseParams), s);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

typedef cudaError_t (*AdjointFn)(AdjointArgs, cudaStream_t);
#endif

}  // namespace nd
