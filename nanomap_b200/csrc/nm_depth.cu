// nm_depth.cu -- soft expected-depth renderer over the device map, its adjoint, and the
// per-step kernel of scan-to-map pose refinement (sm_100a).  No reference counterpart.
//
// Per pixel ray (sensor pixel model, double): voxel DDA from the voxel holding the eye.  Every
// voxel after it, entered at t_in < t_max and left at t_out (clamped to t_max), carries the
// density sigma = softplus(scale L + bias) (L the map's log-odds, 0 for voxels of absent
// leaves), so that sigmoid(scale L + bias) is the probability of the ray ending within one
// voxel length of it; the start voxel holds the sensor and is empty.  The expected depth
// (remaining probability placed at t_max) is the integral of the transmittance:
//   D = res (t_1 + sum_k T_k (1 - exp(-sigma_k D_k)) / sigma_k),  T_{k+1} = T_k exp(-sigma_k D_k)
// with D_k = t_out - t_in, accumulated in FP32.  D is continuous in the pose.
// The adjoint replays the traversal twice instead of storing it: the first replay rebuilds D;
// the second walks front to back with the running prefix P of the transmittance integral, so
// the tail S = D/res - t_1 - P needs no per-ray storage:
//   dD/dsigma_k = res (T_k D_k^2 g(sigma_k D_k) - D_k S_k),  g(u) = (u e^-u - 1 + e^-u) / u^2
//   crossing c from voxel A into B: dD/dc = res (sigma_B - sigma_A) * (tail after c),
//     c = (b - e_a) / d_a  ->  dc/de_a = -1/d_a,  dc/dd_a = -c/d_a
// and for a left world-frame pose perturbation (rho, phi): dD/drho = dD_idx/de,
// dD/dphi = res (d x dD_idx/dd).  The DDA runs in double with explicit round-to-nearest
// operations (no contraction), so its voxel sequence equals the FP64 CPU definition's.
#include <math_constants.h>

#include <cstdint>

#include "nm_device.cuh"
#include "nm_internal.h"

namespace nm {

namespace {

// 8 x 8 pixels per CTA: many small CTAs balance the uneven ray lengths (forward 11 % faster
// than 16 x 16 on the headline frame)
constexpr int kDepthTile = 8;

__device__ __forceinline__ void pixel_dir(const DepthParams& p, int w, int h, double d[3]) {
  double x, y, z;
  if (p.type == NM_SENSOR_FRUSTUM) {
    const double u = __dmul_rn((double)w, (double)p.su);
    const double v = __dmul_rn((double)h, (double)p.sv);
    x = __dadd_rn(__dmul_rn(u, (double)p.c0), -(double)p.hw);
    y = __dadd_rn(__dmul_rn(v, (double)p.c1), -(double)p.hh);
    z = 1.0;
  } else {
    x = __dmul_rn((double)__ldg(&p.sinu[w]), (double)__ldg(&p.cosv[h]));
    y = (double)__ldg(&p.sinv[h]);
    z = __dmul_rn((double)__ldg(&p.cosu[w]), (double)__ldg(&p.cosv[h]));
  }
  const double n = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z)));
  x = __ddiv_rn(x, n);
  y = __ddiv_rn(y, n);
  z = __ddiv_rn(z, n);
#pragma unroll
  for (int i = 0; i < 3; ++i)
    d[i] = __dadd_rn(__dadd_rn(__dmul_rn(p.R[3 * i], x), __dmul_rn(p.R[3 * i + 1], y)),
                     __dmul_rn(p.R[3 * i + 2], z));
}

__device__ __forceinline__ float softplus(float x) {
  return x > 0.0f ? x + log1pf(expf(-x)) : log1pf(expf(x));
}

// g(u) = (u e^-u - 1 + e^-u) / u^2 given em1 = e^-u - 1; -1/2 at u = 0.
__device__ __forceinline__ float seg_g(float u, float em1) {
  if (u < 1e-2f) return -0.5f + u * (1.0f / 3.0f) - u * u * 0.125f;
  return (u * (1.0f + em1) + em1) / (u * u);
}

// A segment of length D >= 0 in a medium of density sg >= 0, u = sg D: returns em1 = expm1(-u) and
// sets *len to the integral of the transmittance over it, -em1 / sg (D at sg = 0).  A long ray runs
// through observed free space, where u is far below 2^-10 on every lane of the warp, and the series
// (next terms below 1e-10 of em1 and of len) replace the function and the division, the longest parts
// of a step's chain.  Each value is its leading term and a correction below 2^-11 of it, added by
// one fma, and no quotient is formed: sg may be as thin as a denormal, whose reciprocal is out of range.
// Error against 64 bits over u from 1e-9 to 2^-10 (mean / worst, 2^-24 relative): len 0.30 / 1.0, by
// division 0.48 / 2.9; em1 0.46 / 2.0, as expm1f's.  (Denser voxels divide: a reciprocal kept with the
// density took 94 us against 99.5 for the depths of one 640x480 frame, but rounds twice.)
__device__ __forceinline__ float segment(float sg, float D, float u, float* len) {
  if (u < 0x1p-10f) {
    const float h = fmaf(u, 1.0f / 6.0f, -0.5f);
    *len = fmaf(D * u, h, D);
    return -fmaf(u * u, h, u);
  }
  const float em1 = expm1f(-u);
  *len = sg > 0.0f ? -em1 / sg : D;
  return em1;
}

// Every walk of a ray (forward, adjoint replays, refinement) ends where its transmittance
// falls below this: what the rest of the ray could add to the expected depth is at most
// kStopTransmittance x its remaining length (< 1e-6 voxel lengths for rays up to 1000
// voxels), each such FP32 term being below half an ulp of the running integral once that
// exceeds 0.01 voxels, and the rest's gradients carry the factor T too (there, the FP32 tail
// A - P is rounding noise).  The forward and the adjoint compute T with the same operations, so
// they stop at the same voxel.
constexpr float kStopTransmittance = 1e-9f;

// Density of a log-odds value, memoised on the last value seen: along a ray most voxels share
// a few values (the clamp of observed free space, 0 for unknown space), so the softplus and
// sigmoid are mostly reused and each visit costs one expm1.
struct DensityCache {
  bool has = false;
  float L = 0.0f;
  float sg = 0.0f, sig = 0.5f;
  __device__ __forceinline__ void at(const DepthParams& p, float l) {
    if (!has || l != L) {
      has = true;
      L = l;
      const float x = p.scale * l + p.bias;
      sg = softplus(x);
      sig = 1.0f / (1.0f + expf(-x));
    }
  }
};

// Slot of a leaf in the map's table, or -1.  No depth kernel writes the table, so the keys may come
// from L1 (neighbouring rays look the same leaves up).
__device__ __forceinline__ int depth_find(const MapView& m, unsigned long long key) {
  uint32_t h = hash_key(key) & m.mask;
  const uint32_t limit = m.capacity < kMaxProbe ? m.capacity : kMaxProbe;
  for (uint32_t probe = 0; probe < limit; ++probe) {
    const unsigned long long k = __ldg(&m.keys[h]);
    if (k == key) return (int)h;
    if (k == kEmptyKey) return -1;
    h = (h + 1) & m.mask;
  }
  return -1;
}

// Visits the voxels of the ray after the start voxel: f(slot, l, L, t_in, a_in, t_out), the voxel
// (leaf slot or -1, index inside the leaf, log-odds) entered at t_in < t_max across axis a_in and
// left at t_out = min(next crossing, t_max); f returns false to end the walk.  Crossings are
// (boundary - e) * (1 / d), the reciprocal taken once per ray.
//
// A ray is a chain of steps, and a frame waits for its longest one (600 steps through observed free
// space).  Ahead: the voxel after the current one is found, and its log-odds loaded, before the
// current one is handed to f, so the load and the leaf look-up stay out of the chain (not for the
// adjoint, whose gradient atomics bound it and whose registers are the tighter for it: 190 against
// 185 us).  Times of one launch on the B200, before -> now: refinement step, 640x480 at 10 m and
// 0.05 m, 140.7 -> 92 us (84.6 with kRefineBlocks), expected depth of
// 1280x720 at 15 m and 0.02 m 868 -> 665 us, of 640x480 64.1 -> 60.1 us, its adjoint 185.4 -> 187.1.
template <bool Ahead, class F>
__device__ __forceinline__ void walk(const MapView& m, const float* __restrict__ vals,
                                     const double e[3], const double d[3], double t_max, F&& f) {
  const int vx = (int)floor(e[0]), vy = (int)floor(e[1]), vz = (int)floor(e[2]);
  const int sx = d[0] > 0.0 ? 1 : (d[0] < 0.0 ? -1 : 0);
  const int sy = d[1] > 0.0 ? 1 : (d[1] < 0.0 ? -1 : 0);
  const int sz = d[2] > 0.0 ? 1 : (d[2] < 0.0 ? -1 : 0);
  const double rx = sx ? __drcp_rn(d[0]) : 0.0;
  const double ry = sy ? __drcp_rn(d[1]) : 0.0;
  const double rz = sz ? __drcp_rn(d[2]) : 0.0;
  // next plane per axis, and the time of its crossing
  int qx = vx + (sx > 0 ? 1 : 0), qy = vy + (sy > 0 ? 1 : 0), qz = vz + (sz > 0 ? 1 : 0);
  double tx = sx ? __dmul_rn(__dadd_rn((double)qx, -e[0]), rx) : CUDART_INF;
  double ty = sy ? __dmul_rn(__dadd_rn((double)qy, -e[1]), ry) : CUDART_INF;
  double tz = sz ? __dmul_rn(__dadd_rn((double)qz, -e[2]), rz) : CUDART_INF;
  int lx = vx >> 3, ly = vy >> 3, lz = vz >> 3;  // leaf of the voxel entered last
  int l = local_index(vx, vy, vz);
  int slot = depth_find(m, leaf_key(lx, ly, lz));
  int a;  // axis crossed next
  double t;
  auto next = [&]() {
    a = 2;
    t = tz;
    if (ty < t) {
      a = 1;
      t = ty;
    }
    if (tx < t) {
      a = 0;
      t = tx;
    }
  };
  // enters the voxel across axis a: its leaf, index and log-odds
  auto enter = [&]() -> float {
    int msk, ds;
    if (a == 0) {
      qx += sx;
      tx = __dmul_rn(__dadd_rn((double)qx, -e[0]), rx);
      msk = 0x1C0;
      ds = sx * 64;
    } else if (a == 1) {
      qy += sy;
      ty = __dmul_rn(__dadd_rn((double)qy, -e[1]), ry);
      msk = 0x38;
      ds = sy * 8;
    } else {
      qz += sz;
      tz = __dmul_rn(__dadd_rn((double)qz, -e[2]), rz);
      msk = 0x7;
      ds = sz;
    }
    const int vv = (l & msk) + ds;
    l = (l & ~msk) | (vv & msk);
    if ((unsigned)vv > (unsigned)msk) {
      lx += a == 0 ? sx : 0;
      ly += a == 1 ? sy : 0;
      lz += a == 2 ? sz : 0;
      slot = depth_find(m, leaf_key(lx, ly, lz));
    }
    return slot >= 0 ? __ldg(&vals[(size_t)slot * kLeafVoxels + l]) : 0.0f;
  };
  next();
  if (!(t < t_max)) return;
  const long long cap = 3ll * (long long)t_max + 16;
  if (Ahead) {
    float L = enter();
    for (long long it = 0; it < cap; ++it) {
      const int slot0 = slot, l0 = l, a_in = a;
      const double t_in = t;
      const float L0 = L;
      next();
      const bool more = t < t_max;
      if (more) L = enter();
      if (!f(slot0, l0, L0, t_in, a_in, more ? t : t_max) || !more) break;
    }
  } else {
    for (long long it = 0; it < cap && t < t_max; ++it) {
      const float L = enter();
      const int a_in = a;
      const double t_in = t;
      next();
      if (!f(slot, l, L, t_in, a_in, t < t_max ? t : t_max)) break;
    }
  }
}

// Expected depth in index units (integral of the transmittance over [0, t_max]), FP32.
__device__ __forceinline__ float expected_index_depth(const DepthParams& p, const MapView& m,
                                                      const float* vals, const double d[3],
                                                      float* t1_out, uint32_t* visits) {
  DensityCache dc;
  float T = 1.0f, acc = 0.0f;
  double t1 = p.t_max;
  bool first = true;
  uint32_t n = 0;
  walk<true>(m, vals, p.eye, d, p.t_max, [&](int, int, float L, double t_in, int, double t_out) {
    ++n;
    dc.at(p, L);
    const float sg = dc.sg;
    const float Dk = (float)(t_out - t_in);
    if (first) {
      t1 = t_in;
      first = false;
    }
    float len;
    const float em1 = segment(sg, Dk, sg * Dk, &len);
    acc += T * len;
    T *= 1.0f + em1;
    return T >= kStopTransmittance;
  });
  *t1_out = (float)t1;
  *visits += n;
  return (float)t1 + acc;
}

// The time of the ray's first voxel crossing (the t_in of walk()'s first visit, the same
// operations), or t_max when the ray stays in its start voxel.
__device__ __forceinline__ double first_crossing(const double e[3], const double d[3],
                                                 double t_max) {
  double t = CUDART_INF;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int s = d[a] > 0.0 ? 1 : (d[a] < 0.0 ? -1 : 0);
    if (!s) continue;
    const int v = (int)floor(e[a]);
    const double c = __dmul_rn(__dadd_rn((double)(v + (s > 0 ? 1 : 0)), -e[a]), __drcp_rn(d[a]));
    t = c < t ? c : t;
  }
  return t < t_max ? t : t_max;
}

// Voxels nearer the eye than this (index units) take their log-odds gradient through
// scatter_gradient: there the rays of a warp share voxels and thousands of rays add into the
// same voxel.  Farther out lanes rarely share a voxel at the same step and a plain atomic is
// cheaper (headline frame, given depths: 1.59 ms plain, 1.44 ms aggregated everywhere,
// 1.09 ms aggregated within this span).
constexpr double kGatherSpan = 48.0;

// Adds x into grad_vals[slot * 512 + l] (nothing for slot < 0) with one atomic per voxel
// among the warp's lanes at this call: lanes holding the same voxel (rays near the eye and
// neighbouring rays walk the same voxels at the same step) are summed by a shuffle tree first,
// in rounds that each fold every second remaining lane of a group into the one before it.
__device__ __forceinline__ void scatter_gradient(float* grad_vals, int slot, int l, float x) {
  const unsigned act = __activemask();
  const int lane = (int)((threadIdx.y * blockDim.x + threadIdx.x) & 31u);
  const unsigned long long key =
      slot >= 0 ? (unsigned long long)slot * kLeafVoxels + (unsigned)l : ~0ull;
  const unsigned peers = __match_any_sync(act, key);
  int rank = __popc(peers & ((1u << lane) - 1u));  // position among the voxel's lanes
  unsigned above = lane == 31 ? 0u : peers & (~0u << (lane + 1));
  while (__any_sync(act, above != 0u)) {
    const int nxt = __ffs(above);
    const float y = __shfl_sync(act, x, nxt ? nxt - 1 : lane);
    if (nxt) x += y;
    above &= ~__ballot_sync(act, rank & 1);  // odd ranks have been folded into their left
    rank >>= 1;
  }
  if (slot >= 0 && lane == __ffs(peers) - 1) atomicAdd(&grad_vals[key], x);
}

// Gradient replay of one ray: adds gd-weighted log-odds gradients into grad_vals (when given)
// and returns the ray's pose gradient (6: rho, phi) times gd.
__device__ __forceinline__ void replay_gradients(const DepthParams& p, const MapView& m,
                                                 const float* vals, const double d[3], float D,
                                                 float t1, float gd, float* grad_vals,
                                                 float g6[6], uint32_t* visits) {
  DensityCache dc;
  uint32_t n = 0;
  float T = 1.0f, P = 0.0f, sg_prev = 0.0f;
  float ge[3] = {0.f, 0.f, 0.f}, gdir[3] = {0.f, 0.f, 0.f};
  const float inv_d[3] = {(float)(1.0 / d[0]), (float)(1.0 / d[1]), (float)(1.0 / d[2])};
  const float gv = gd * (float)p.res * p.scale;
  const float tail0 = D - t1;
  walk<false>(m, vals, p.eye, d, p.t_max, [&](int slot, int l, float L, double t_in, int a_in, double t_out) {
    dc.at(p, L);
    ++n;
    const float sg = dc.sg;
    const float Dk = (float)(t_out - t_in);
    // entry crossing: the density steps from sg_prev to sg
    const float gc = (sg - sg_prev) * (tail0 - P) * (a_in == 0 ? inv_d[0] : (a_in == 1 ? inv_d[1] : inv_d[2]));
    const float ti = (float)t_in;
    if (a_in == 0) {
      ge[0] -= gc;
      gdir[0] -= gc * ti;
    } else if (a_in == 1) {
      ge[1] -= gc;
      gdir[1] -= gc * ti;
    } else {
      ge[2] -= gc;
      gdir[2] -= gc * ti;
    }
    const float u = sg * Dk;
    float len;
    const float em1 = segment(sg, Dk, u, &len);
    const float Pn = P + T * len;
    if (grad_vals) {
      const float dsig = T * Dk * Dk * seg_g(u, em1) - Dk * (tail0 - Pn);
      if (t_in < kGatherSpan)
        scatter_gradient(grad_vals, slot, l, gv * dc.sig * dsig);
      else if (slot >= 0)
        atomicAdd(&grad_vals[(size_t)slot * kLeafVoxels + l], gv * dc.sig * dsig);
    }
    P = Pn;
    T *= 1.0f + em1;
    sg_prev = sg;
    return T >= kStopTransmittance;
  });
  *visits += n;
  const float r = gd * (float)p.res;
  const float dx = (float)d[0], dy = (float)d[1], dz = (float)d[2];
  g6[0] = gd * ge[0];
  g6[1] = gd * ge[1];
  g6[2] = gd * ge[2];
  g6[3] = r * (dy * gdir[2] - dz * gdir[1]);
  g6[4] = r * (dz * gdir[0] - dx * gdir[2]);
  g6[5] = r * (dx * gdir[1] - dy * gdir[0]);
}

// Adds the active lanes' visit counts to the map's counter (one atomic per warp).
__device__ __forceinline__ void add_depth_visits(const MapView& m, uint32_t n) {
  const unsigned act = __activemask();
  const uint32_t sum = __reduce_add_sync(act, n);
  if (((threadIdx.y * blockDim.x + threadIdx.x) & 31) == (unsigned)(__ffs(act) - 1))
    atomicAdd(&m.ctr->depth_visits, (unsigned long long)sum);
}

// Sum of N doubles over the CTA (blockDim.x * blockDim.y threads, a multiple of 32); thread 0
// writes the CTA's partials to out[blockIdx * N ...].
template <int N>
__device__ __forceinline__ void block_partials(double (&x)[N], double* out) {
  __shared__ double s[32][N];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int nw = (blockDim.x * blockDim.y) >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i)
    for (int o = 16; o > 0; o >>= 1) x[i] += __shfl_down_sync(0xffffffffu, x[i], o);
  if ((tid & 31) == 0)
#pragma unroll
    for (int i = 0; i < N; ++i) s[tid >> 5][i] = x[i];
  __syncthreads();
  if (tid == 0) {
    const size_t b = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    for (int i = 0; i < N; ++i) {
      double acc = 0.0;
      for (int w = 0; w < nw; ++w) acc += s[w][i];
      out[b * N + i] = acc;
    }
  }
}

__global__ void __launch_bounds__(kDepthTile * kDepthTile) k_depth_forward(DepthParams p, MapView m,
                                                                           const float* vals,
                                                                           float* depth) {
  const int w = blockIdx.x * kDepthTile + threadIdx.x;
  const int h = blockIdx.y * kDepthTile + threadIdx.y;
  if (w >= p.width || h >= p.height) return;
  double d[3];
  pixel_dir(p, w, h, d);
  float t1;
  uint32_t n = 0;
  depth[(size_t)h * p.width + w] = expected_index_depth(p, m, vals, d, &t1, &n) * (float)p.res;
  add_depth_visits(m, n);
}

// `depth` (may be null): the forward's output at this pose and these values; the ray's
// expected depth is then taken from it instead of a first replay.  16 CTAs per SM (64 registers): 187
// us for a 640x480 adjoint given depths; about 10 us more at 79 registers.
__global__ void __launch_bounds__(kDepthTile * kDepthTile, 16) k_depth_backward(
    DepthParams p, MapView m, const float* vals, const float* grad_depth, const float* depth,
    float* grad_vals, double* partials) {
  const int w = blockIdx.x * kDepthTile + threadIdx.x;
  const int h = blockIdx.y * kDepthTile + threadIdx.y;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  uint32_t n = 0;
  if (w < p.width && h < p.height) {
    const float gd = grad_depth[(size_t)h * p.width + w];
    if (gd != 0.0f) {
      double d[3];
      pixel_dir(p, w, h, d);
      float t1, D;
      if (depth) {
        D = depth[(size_t)h * p.width + w] / (float)p.res;
        t1 = (float)first_crossing(p.eye, d, p.t_max);
      } else {
        D = expected_index_depth(p, m, vals, d, &t1, &n);
      }
      float g6[6];
      replay_gradients(p, m, vals, d, D, t1, gd, grad_vals, g6, &n);
#pragma unroll
      for (int i = 0; i < 6; ++i) acc[i] = (double)g6[i];
    }
  }
  add_depth_visits(m, n);
  block_partials<6>(acc, partials);
}

// One walk giving the expected depth (as expected_index_depth, with the entry step) and the
// ray's pose gradient for a unit depth gradient, for the refinement step.  replay_gradients'
// crossing term is c (A - P) with c = (sigma_B - sigma_A) / d_a, P the transmittance integral
// before the crossing and A the whole integral (D / res - t_1), so per axis the sums of c,
// c P, c t and c t P (in double: A and P are close where c is large) give the gradient once
// A is known at the end of the walk.  Returns D (index units); g6 as replay_gradients' for
// gd = 1.
__device__ __forceinline__ float depth_and_pose_gradient(const DepthParams& p, const MapView& m,
                                                         const float* vals, const double d[3],
                                                         uint32_t* visits, float* entry_step,
                                                         float g6[6]) {
  DensityCache dc;
  float T = 1.0f, acc = 0.0f, W = 0.0f, sg_prev = 0.0f;
  double t1 = p.t_max;
  bool first = true;
  uint32_t n = 0;
  const float step[3] = {(float)(1.0 / fabs(d[0])), (float)(1.0 / fabs(d[1])),
                         (float)(1.0 / fabs(d[2]))};
  const float inv_d[3] = {(float)(1.0 / d[0]), (float)(1.0 / d[1]), (float)(1.0 / d[2])};
  double sc[3] = {0.0, 0.0, 0.0}, scp[3] = {0.0, 0.0, 0.0};
  double sct[3] = {0.0, 0.0, 0.0}, sctp[3] = {0.0, 0.0, 0.0};
  walk<true>(m, vals, p.eye, d, p.t_max, [&](int, int, float L, double t_in, int a_in, double t_out) {
    ++n;
    dc.at(p, L);
    const float sg = dc.sg;
    const float Dk = (float)(t_out - t_in);
    if (first) {
      t1 = t_in;
      first = false;
    }
    if (sg != sg_prev) {
      const double cd = (double)((sg - sg_prev) * (a_in == 0 ? inv_d[0] : (a_in == 1 ? inv_d[1] : inv_d[2])));
      const double P = (double)acc, ti = (double)(float)t_in;
      if (a_in == 0) {
        sc[0] += cd;
        scp[0] += cd * P;
        sct[0] += cd * ti;
        sctp[0] += cd * ti * P;
      } else if (a_in == 1) {
        sc[1] += cd;
        scp[1] += cd * P;
        sct[1] += cd * ti;
        sctp[1] += cd * ti * P;
      } else {
        sc[2] += cd;
        scp[2] += cd * P;
        sct[2] += cd * ti;
        sctp[2] += cd * ti * P;
      }
    }
    // The refinement's path doubles differences of rounding from step to step, so the segment's
    // integral keeps the division and the function; -u is expm1f(-u)'s own value for u this small.
    const float u = sg * Dk;
    const float em1 = u < 0x1p-26f ? -u : expm1f(-u);
    acc += T * (sg > 0.0f ? -em1 / sg : Dk);
    W -= T * em1 * step[a_in];
    T *= 1.0f + em1;
    sg_prev = sg;
    return T >= kStopTransmittance;
  });
  *visits += n;
  *entry_step = T < 1.0f ? W / (1.0f - T) : 0.0f;
  const double A = (double)acc;
  float ge[3], gdir[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    ge[a] = (float)(scp[a] - A * sc[a]);
    gdir[a] = (float)(sctp[a] - A * sct[a]);
  }
  const float r = (float)p.res;
  const float dx = (float)d[0], dy = (float)d[1], dz = (float)d[2];
  g6[0] = ge[0];
  g6[1] = ge[1];
  g6[2] = ge[2];
  g6[3] = r * (dy * gdir[2] - dz * gdir[1]);
  g6[4] = r * (dz * gdir[0] - dx * gdir[2]);
  g6[5] = r * (dx * gdir[1] - dy * gdir[0]);
  return (float)t1 + acc;
}

// Whether pixel (w, h) of the target lies on a silhouette: a 4-neighbour inside the image
// without a return, or with a range more than `edge` metres away.
__device__ __forceinline__ bool target_edge(const float* target, int W, int H, int w, int h,
                                            float r, float edge) {
  const int nx[4] = {w - 1, w + 1, w, w};
  const int ny[4] = {h, h, h - 1, h + 1};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (nx[k] < 0 || nx[k] >= W || ny[k] < 0 || ny[k] >= H) continue;
    const float q = target[(size_t)ny[k] * W + nx[k]];
    if (!(q > 0.0f && q < CUDART_INF_F) || fabsf(q - r) > edge) return true;
  }
  return false;
}

// One refinement step: L1 loss against `target` (metres; <= 0 or NaN = no return), truncated
// at max_residual when it is positive (residuals beyond it add max_residual and no gradient),
// its pose gradient, and the number of pixels that took part.  The prediction is the expected
// depth plus `surface_offset` times the entry step of the voxel where the ray ends (0: the
// surface at the face the ray enters; 0.5: at the middle of the voxel), the offset held fixed
// for the gradient.  Silhouette pixels of the target are left out when edge > 0.  Partials:
// loss, count, 6 gradients.
//
// A chain of steps per ray, so the blocks resident set the rate: 8 per SM (115 registers) 92 us for 640x480
// at 10 m and 0.05 m, 10 (96) 88, 12 (80, with spills) 85, 14 84, 16 (64) 85.
// (The forward kernel has 18 without a limit and the adjoint 16: more of them only spilled.)
constexpr int kRefineBlocks = 12;
__global__ void __launch_bounds__(kDepthTile * kDepthTile, kRefineBlocks) k_depth_refine(
    DepthParams p0, MapView m, const float* vals, const float* target, float max_residual,
    float surface_offset, float edge, const RefineState* st, double* partials) {
  // the pose of this step, from the device state (the eye as the host computes it)
  DepthParams p = p0;
#pragma unroll
  for (int a = 0; a < 3; ++a) p.eye[a] = __ddiv_rn(st->position[a], p.res);
#pragma unroll
  for (int i = 0; i < 9; ++i) p.R[i] = st->R[i];
  const int w = blockIdx.x * kDepthTile + threadIdx.x;
  const int h = blockIdx.y * kDepthTile + threadIdx.y;
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  uint32_t n = 0;
  if (w < p.width && h < p.height) {
    const float r = target[(size_t)h * p.width + w];
    if (r > 0.0f && r < CUDART_INF_F &&
        !(edge > 0.0f && target_edge(target, p.width, p.height, w, h, r, edge))) {
      double d[3];
      pixel_dir(p, w, h, d);
      float step, g6[6];
      const float D = depth_and_pose_gradient(p, m, vals, d, &n, &step, g6);
      const float res = (D + surface_offset * step) * (float)p.res - r;
      const bool clipped = max_residual > 0.0f && fabsf(res) > max_residual;
      acc[0] = clipped ? (double)max_residual : fabs((double)res);
      acc[1] = 1.0;
      const float gd = clipped ? 0.0f : (res > 0.0f ? 1.0f : (res < 0.0f ? -1.0f : 0.0f));
      if (gd != 0.0f) {
#pragma unroll
        for (int i = 0; i < 6; ++i) acc[2 + i] = (double)(gd * g6[i]);
      }
    }
  }
  add_depth_visits(m, n);
  block_partials<8>(acc, partials);
}

// exp([phi]x) R (Rodrigues), row-major, in place.
__device__ void rotate_left(const double phi[3], double R[9]) {
  const double th = sqrt(phi[0] * phi[0] + phi[1] * phi[1] + phi[2] * phi[2]);
  const double K[9] = {0, -phi[2], phi[1], phi[2], 0, -phi[0], -phi[1], phi[0], 0};
  double E[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  if (th > 0.0) {
    const double a = sin(th) / th, b = (1.0 - cos(th)) / (th * th);
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c)
        E[3 * r + c] += a * K[3 * r + c] +
                        b * (K[3 * r] * K[c] + K[3 * r + 1] * K[3 + c] + K[3 * r + 2] * K[6 + c]);
  }
  double out[9];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c)
      out[3 * r + c] = E[3 * r] * R[c] + E[3 * r + 1] * R[3 + c] + E[3 * r + 2] * R[6 + c];
  for (int i = 0; i < 9; ++i) R[i] = out[i];
}

// Column sums of an (n, N) array of partials, N <= 8, by one block of kSumThreads threads in a
// fixed order (deterministic); h[c] = sum of column c, on every thread.  Thread t adds rows t / 8,
// t / 8 + 128, ... of column t % 8 (neighbouring threads read neighbouring words, four rows in
// flight), then a shuffle tree and one over the warps.  Bound by the latency of its 10 dependent
// loads: 43.5 -> 10 us in the refinement step's update and 28 -> 12 us after an adjoint, both for
// the 4800 rows of a 640x480 image (one column at a time over 256 threads before).
constexpr int kSumThreads = 1024;
template <int N>
__device__ __forceinline__ void column_sums(const double* __restrict__ partials, int n, double h[N]) {
  __shared__ double s[kSumThreads / 32][8];
  const int c = threadIdx.x & 7, r0 = threadIdx.x >> 3;
  constexpr int kRows = kSumThreads / 8;
  double x[4] = {0.0, 0.0, 0.0, 0.0};
  if (c < N) {
    int i = r0;
    for (; i + 3 * kRows < n; i += 4 * kRows)
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] += partials[(size_t)(i + k * kRows) * N + c];
    for (int k = 0; i < n; i += kRows, ++k) x[k] += partials[(size_t)i * N + c];
  }
  double sum = (x[0] + x[1]) + (x[2] + x[3]);
  sum += __shfl_xor_sync(0xffffffffu, sum, 8);
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
  if ((threadIdx.x & 31) < 8) s[threadIdx.x >> 5][c] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {  // 4 warps' sums a lane, then the four lanes of a column
    double y = 0.0;
#pragma unroll
    for (int k = 0; k < kSumThreads / 128; ++k) y += s[(threadIdx.x >> 3) + 4 * k][c];
    y += __shfl_xor_sync(0xffffffffu, y, 8);
    y += __shfl_xor_sync(0xffffffffu, y, 16);
    if (threadIdx.x < 8) s[0][c] = y;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) h[k] = s[0][k];
}

// One block: the step's partials summed in a fixed order (loss, count, 6 gradients), then
// the mean loss is recorded and, before the last step, Adam is applied on the left world-frame
// increment (rho, phi), a component per lane, with the learning rates cosine-decayed to zero.
__global__ void __launch_bounds__(kSumThreads) k_refine_update(const double* partials, int n,
                                                               RefineState* st, float* losses,
                                                               int it) {
  double h[8];
  column_sums<8>(partials, n, h);
  if (threadIdx.x >= 32 || st->error) return;
  if (h[1] < 1.0) {
    if (threadIdx.x == 0) st->error |= kRefineNoPixels;
    return;
  }
  if (threadIdx.x == 0) losses[it] = (float)(h[0] / h[1]);
  if (it >= st->steps) return;
  const double b1 = 0.9, b2 = 0.999, eps = 1e-8;
  const double t = (double)(it + 1);
  double step = 0.0;
  const int i = threadIdx.x;
  if (i < 6) {
    const double decay = 0.5 * (1.0 + cos(CUDART_PI * it / st->steps));
    double gi = h[2];
#pragma unroll
    for (int k = 1; k < 6; ++k) gi = i == k ? h[2 + k] : gi;
    const double g = gi / h[1];
    const double mom = b1 * st->mom[i] + (1.0 - b1) * g;
    const double var = b2 * st->var[i] + (1.0 - b2) * g * g;
    st->mom[i] = mom;
    st->var[i] = var;
    const double mh = mom / (1.0 - pow(b1, t));
    const double vh = var / (1.0 - pow(b2, t));
    step = -decay * (i < 3 ? st->lr_position : st->lr_rotation) * mh / (sqrt(vh) + eps);
  }
  const bool out = i < 3 && fabs((st->position[i < 3 ? i : 0] + step) / st->res) + st->t_max + 2.0 >
                                (double)(1 << 23) - 16.0;
  if (__any_sync(0xffffffffu, out)) {
    if (i == 0) st->error |= kRefineOutOfRange;
    return;
  }
  if (i < 3) st->position[i] += step;
  double phi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) phi[k] = __shfl_sync(0xffffffffu, step, 3 + k);
  if (i == 0) rotate_left(phi, st->R);
}

__global__ void __launch_bounds__(kSumThreads) k_sum_partials(const double* partials, int n,
                                                              double* out) {
  double h[6];
  column_sums<6>(partials, n, h);
  if (threadIdx.x == 0)
#pragma unroll
    for (int c = 0; c < 6; ++c) out[c] = h[c];
}

dim3 depth_grid(const DepthParams& p) {
  return dim3((p.width + kDepthTile - 1) / kDepthTile, (p.height + kDepthTile - 1) / kDepthTile);
}

}  // namespace

int depth_partial_blocks(const DepthParams& p) {
  const dim3 g = depth_grid(p);
  return (int)(g.x * g.y);
}

cudaError_t launch_depth_forward(const DepthParams& p, const MapView& m, const float* vals,
                                 float* depth, cudaStream_t s) {
  k_depth_forward<<<depth_grid(p), dim3(kDepthTile, kDepthTile), 0, s>>>(p, m, vals, depth);
  return cudaGetLastError();
}

cudaError_t launch_depth_backward(const DepthParams& p, const MapView& m, const float* vals,
                                  const float* grad_depth, const float* depth, float* grad_vals,
                                  double* partials, double* out6, cudaStream_t s) {
  const dim3 g = depth_grid(p);
  k_depth_backward<<<g, dim3(kDepthTile, kDepthTile), 0, s>>>(p, m, vals, grad_depth, depth,
                                                              grad_vals, partials);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_sum_partials<<<1, kSumThreads, 0, s>>>(partials, (int)(g.x * g.y), out6);
  return cudaGetLastError();
}

cudaError_t launch_depth_refine(const DepthParams& p, const MapView& m, const float* vals,
                                const float* target, float max_residual, float surface_offset,
                                float edge, double* partials, RefineState* st, float* losses,
                                int it, cudaStream_t s) {
  const dim3 g = depth_grid(p);
  k_depth_refine<<<g, dim3(kDepthTile, kDepthTile), 0, s>>>(p, m, vals, target, max_residual,
                                                            surface_offset, edge, st, partials);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_refine_update<<<1, kSumThreads, 0, s>>>(partials, (int)(g.x * g.y), st, losses, it);
  return cudaGetLastError();
}

}  // namespace nm
