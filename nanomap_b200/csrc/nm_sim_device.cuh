// nm_sim_device.cuh -- simulated-depth ray casting and range noise (device functions),
// shared by the render kernels (nm_sim.cu) and the traversal's fused render (nm_traverse.cu).
//
// Replaces getActiveCrossing / viewSimKernel (generateCloud.cu:20-82).  The ray cast is an
// exact hierarchical form of the closed-form voxel DDA the oracle runs: crossing times are
// always recomputed from the plane index, t(p) = (p - eye) / dir, so the walk has no
// accumulated state, and a skip over an empty leaf or brick lands on the same voxel the
// voxel-by-voxel walk reaches when it leaves that cube.  The landing voxel is found by
// ordering crossing events by (time, higher axis first): on each other axis the walk has
// crossed every plane whose time is below the exit time, or equal to it on a higher axis
// than the exit axis.
#pragma once

#include <cfloat>
#include <cstdint>

#include "nm_sim.h"

namespace nm {
namespace {

// ---- ray casting -----------------------------------------------------------------------------

__device__ __forceinline__ float plane_time(int p, float e, float inv) {
  return __fmul_rn(__fadd_rn((float)p, -e), inv);
}

__device__ __forceinline__ float plane_time_f(float p, float e, float inv) {
  return __fmul_rn(__fadd_rn(p, -e), inv);
}

// Crossed-before-exit predicate for a plane on axis j (see the header comment).
__device__ __forceinline__ bool crossed(int p, float e, float inv, float T, bool higher) {
  const float t = plane_time(p, e, inv);
  return t < T || (t == T && higher);
}

// Voxel index on axis j after the walk has processed every event before the exit event
// (T, exit axis a), starting from voxel k inside [k .. far] (s = +1) or [far .. k] (s = -1).
__device__ __forceinline__ int advance_axis(int k, int far, int s, float e, float dir, float inv,
                                            float T, bool higher) {
  int est = (int)floorf(__fadd_rn(e, __fmul_rn(dir, T)));
  if (s > 0) {
    est = max(k, min(far, est));
    while (est < far && crossed(est + 1, e, inv, T, higher)) ++est;
    while (est > k && !crossed(est, e, inv, T, higher)) --est;
  } else {
    est = min(k, max(far, est));
    while (est > far && crossed(est, e, inv, T, higher)) --est;
    while (est < k && !crossed(est + 1, e, inv, T, higher)) ++est;
  }
  return est;
}

// Block of leaves of the brick that holds a voxel, -1 for an empty brick or outside the map.
__device__ __forceinline__ int32_t sim_brick(const SimMapView& v, int x, int y, int z) {
  const int bx = (x >> 6) - v.blo[0], by = (y >> 6) - v.blo[1], bz = (z >> 6) - v.blo[2];
  if ((unsigned)bx >= (unsigned)v.bdim[0] || (unsigned)by >= (unsigned)v.bdim[1] ||
      (unsigned)bz >= (unsigned)v.bdim[2])
    return -1;
  return __ldg(&v.brick_index[((long long)bx * v.bdim[1] + by) * v.bdim[2] + bz]);
}

// Distance (metres) to the first active voxel entered along the ray from `eye` (index space)
// in the unit direction `dir`, at a ray time within [tmin, tmax] (voxel units), or 0.  The
// voxel holding the eye is not tested.  With nseg > 1 the walk covers only the seg-th of nseg parts of
// the ray: the voxels entered in (start, end] of the part.  Crossing times have no accumulated state,
// so the voxel that the whole walk is in at the part's start is found directly: on each axis it
// has crossed every plane whose time is not above the start.  *found: an active voxel ended the walk
// (also one whose distance is 0).
__device__ __forceinline__ float sim_cast(const SimMapView& v, const float eye[3], float dir[3],
                                          float tmin, float tmax, int seg = 0, int nseg = 1,
                                          bool* found = nullptr) {
  float result = 0.0f;
  float inv[3];
  int st[3];
  // Nothing past tmax can be a result, so the walk ends there and not only where the ray leaves the
  // map (a NaN tmax leaves it the map's end): 512 rays of 5 m in a 20 m world 94 -> 62 us, a frame
  // whose rays mostly end on something 64.2 -> 63.2 us (before the figures below).
  float t_in = 0.0f, t_out = fminf(INFINITY, tmax);
  bool miss = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (fabsf(dir[a]) < 1e-30f) dir[a] = 0.0f;
    if (dir[a] == 0.0f) {
      st[a] = 0;
      inv[a] = 0.0f;
      if (eye[a] < v.box_lo[a] || eye[a] > v.box_hi[a]) miss = true;
    } else {
      inv[a] = __frcp_rn(dir[a]);
      st[a] = dir[a] > 0.0f ? 1 : -1;
      float ta = plane_time_f(v.box_lo[a], eye[a], inv[a]);
      float tb = plane_time_f(v.box_hi[a], eye[a], inv[a]);
      if (ta > tb) {
        const float x = ta;
        ta = tb;
        tb = x;
      }
      if (ta > t_in) t_in = ta;
      if (tb < t_out) t_out = tb;
    }
  }
  if (!miss && !(t_in > t_out)) {
    t_out = fminf(t_out, FLT_MAX);  // an axis that is never crossed has the time infinity
    int k[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) k[a] = (int)floorf(__fadd_rn(eye[a], __fmul_rn(dir[a], t_in)));
    float t = t_in;
    if (nseg > 1 && !(t_out < 1e6f)) {  // no end to divide: the first lane takes the whole ray
      if (seg > 0) return 0.0f;
    } else if (nseg > 1) {
      const float part = __fdiv_rn(__fadd_rn(t_out, -t_in), (float)nseg);
      const float t0 = __fadd_rn(t_in, __fmul_rn(part, (float)seg));
      // (the parts' ends do not fall with seg, and neighbours compute the same value)
      if (seg + 1 < nseg) t_out = fminf(t_out, __fadd_rn(t_in, __fmul_rn(part, (float)(seg + 1))));
      if (seg > 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if (st[a] != 0)
            k[a] = advance_axis(k[a], k[a] + st[a] * (1 << 22), st[a], eye[a], dir[a], inv[a], t0, true);
        t = t0;
      }
    }
    // A position e + dir * T this near the middle of a voxel lies in that voxel for the planes' times
    // too: those and T carry at most 5 roundings of dir * T, the position one of itself.  (Below zero
    // for coordinates past 5e5, where kFloor would not do either.)
    constexpr float kFloor = 12582912.0f;  // 1.5 * 2^23: x + this, rounded down, has floor(x) in its bits
    float sure[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
      sure[a] = st[a] == 0 ? (fabsf(eye[a]) < 1e6f ? 1.0f : -1.0f)
                           : 0.5f - 1e-6f * (t_out + fabsf(eye[a]) + 1.0f);
    bool first = true;
    int32_t blk = -1;
    int last[3] = {k[0] ^ 64, k[1], k[2]};  // a voxel of blk's brick (at first of another one)
    for (int iter = 0; iter < (1 << 22); ++iter) {
      if ((unsigned)((k[0] ^ last[0]) | (k[1] ^ last[1]) | (k[2] ^ last[2])) > 63u) {
        blk = sim_brick(v, k[0], k[1], k[2]);
#pragma unroll
        for (int a = 0; a < 3; ++a) last[a] = k[a];
      }
      // leaf index, or -d (d >= 1): every leaf within Chebyshev distance d - 1 of this one is empty
      int leaf = -8;
      if (blk >= 0) {
        const int e = (((k[0] >> 3) & 7) << 6) | (((k[1] >> 3) & 7) << 3) | ((k[2] >> 3) & 7);
        leaf = __ldg(&v.brick_leaves[(size_t)blk * 512 + e]);
      }
      if (leaf >= 0) {
        // Voxel steps inside a leaf with active voxels: the leaf's words come from L1, and
        // only the stepped axis's next crossing changes (each crossing is the closed form of
        // its own plane, so the event sequence is the one the generic step takes).  l holds the voxel in
        // three fields of 4 bits: the high bit of one is set once the step on its axis left the leaf.
        // Everything under predicates: as three branches each of them was taken by some lane.  Bound by
        // issue: 640x480 rays of at most 10 m at 0.05 m 63.2 -> 51.5 us with this and the brick kept
        // between lookups.
        const uint32_t* lw = v.leaf_words + (size_t)leaf * 16;
        int p0 = k[0] + (st[0] > 0), p1 = k[1] + (st[1] > 0), p2 = k[2] + (st[2] > 0);
        float T0 = st[0] == 0 ? INFINITY : plane_time(p0, eye[0], inv[0]);
        float T1 = st[1] == 0 ? INFINITY : plane_time(p1, eye[1], inv[1]);
        float T2 = st[2] == 0 ? INFINITY : plane_time(p2, eye[2], inv[2]);
        const int d0 = st[0] * 256, d1 = st[1] * 16, d2 = st[2];
        int l = ((k[0] & 7) << 8) | ((k[1] & 7) << 4) | (k[2] & 7);
        bool hit = false, done = false;
        do {
          const uint32_t word = __ldg(&lw[(l >> 7) + ((l >> 6) & 1)]);
          if (!first && ((word >> (((l >> 1) & 0x18) | (l & 7))) & 1u)) {
            hit = true;
            break;
          }
          first = false;
          const bool c01 = T0 < T1;
          const bool is0 = c01 && T0 < T2, is1 = !c01 && T1 < T2;
          const float Tx = is0 ? T0 : (is1 ? T1 : T2);
          if (!(Tx <= t_out)) {
            done = true;
            break;
          }
          t = Tx;
          l += is0 ? d0 : (is1 ? d1 : d2);
          if (is0) {
            p0 += st[0];
            T0 = plane_time(p0, eye[0], inv[0]);
          }
          if (is1) {
            p1 += st[1];
            T1 = plane_time(p1, eye[1], inv[1]);
          }
          if (!is0 && !is1) {
            p2 += st[2];
            T2 = plane_time(p2, eye[2], inv[2]);
          }
        } while (!(l & 0x888));
        k[0] = p0 - (st[0] > 0);
        k[1] = p1 - (st[1] > 0);
        k[2] = p2 - (st[2] > 0);
        if (hit) {
          if (found) *found = true;
          if (t >= tmin && t <= tmax) result = __fmul_rn(t, v.res);
          break;
        }
        if (done) break;
        continue;  // left the leaf: the outer walk takes the next level
      }
      first = false;
      // (About half of the walk's instructions: 51.5 -> 45.3 us, 16 sensors' 5.1 M rays 527 -> 461 us with
      // the three axes done alike and the planes' own times left for the places where they decide.)
      // the empty cube to leave: the brick (64^3 voxels), or the leaves within Chebyshev
      // distance d - 1 of this empty leaf (all empty; d = 1: the leaf itself)
      const int cell = blk < 0 ? 64 : 8, ahead = blk < 0 ? 64 : -8 * leaf, back = cell - ahead;
      int pl[3];  // plane of the cube that the ray can leave it through, per axis
      float T[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        pl[a] = (k[a] & -cell) + (st[a] < 0 ? back : ahead);
        T[a] = st[a] == 0 ? INFINITY : plane_time(pl[a], eye[a], inv[a]);
      }
      const bool c01 = T[0] < T[1];
      const bool is0 = c01 && T[0] < T[2], is1 = !c01 && T[1] < T[2];
      const float Tx = is0 ? T[0] : (is1 ? T[1] : T[2]);
      if (!(Tx <= t_out)) break;
      int to[3];
      bool easy = true;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const bool exit = a == 0 ? is0 : (a == 1 ? is1 : !is0 && !is1);
        const float at = __fmaf_rn(dir[a], Tx, eye[a]);
        const float fl = __fadd_rd(at, kFloor);
        easy &= exit || fabsf(at - (fl - kFloor) - 0.5f) < sure[a];
        to[a] = exit ? pl[a] - (st[a] < 0) : __float_as_int(fl) - __float_as_int(kFloor);
      }
      if (!easy) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const bool exit = a == 0 ? is0 : (a == 1 ? is1 : !is0 && !is1);
          if (exit) continue;
          to[a] = k[a];
          if (st[a] != 0)
            to[a] = advance_axis(k[a], st[a] > 0 ? pl[a] - 1 : pl[a], st[a], eye[a], dir[a], inv[a], Tx,
                                 a > (is0 ? 0 : (is1 ? 1 : 2)));
        }
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) k[a] = to[a];
      t = Tx;
    }
  }
  return result;
}

// Range of pixel (w, h): the first active voxel entered along the pixel ray, or 0.
__device__ __forceinline__ float sim_ray(const SimMapView& v, const SimRayParams& rp, int w, int h) {
  if (!v.any) return 0.0f;
  float d0, d1, d2;
  if (rp.type == NM_SENSOR_FRUSTUM) {
    const float u = __fmul_rn((float)w, rp.su);
    const float vv = __fmul_rn((float)h, rp.sv);
    d0 = __fadd_rn(__fmul_rn(u, rp.c0), -rp.hw);
    d1 = __fadd_rn(__fmul_rn(vv, rp.c1), -rp.hh);
    d2 = 1.0f;
  } else {
    const float cv = __ldg(&rp.cosv[h]);
    d0 = __fmul_rn(__ldg(&rp.sinu[w]), cv);
    d1 = __ldg(&rp.sinv[h]);
    d2 = __fmul_rn(__ldg(&rp.cosu[w]), cv);
  }
  const float* R = rp.R;
  const float m0 = __fadd_rn(__fadd_rn(__fmul_rn(R[0], d0), __fmul_rn(R[1], d1)), __fmul_rn(R[2], d2));
  const float m1 = __fadd_rn(__fadd_rn(__fmul_rn(R[3], d0), __fmul_rn(R[4], d1)), __fmul_rn(R[5], d2));
  const float m2 = __fadd_rn(__fadd_rn(__fmul_rn(R[6], d0), __fmul_rn(R[7], d1)), __fmul_rn(R[8], d2));
  const float norm = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(m0, m0), __fmul_rn(m1, m1)), __fmul_rn(m2, m2)));
  float dir[3] = {__fdiv_rn(m0, norm), __fdiv_rn(m1, norm), __fdiv_rn(m2, norm)};
  const float eye[3] = {rp.eye[0], rp.eye[1], rp.eye[2]};  // pos / res
  float tmin = rp.tmin, tmax = rp.tmax;                     // range limits / res
  if (rp.type == NM_SENSOR_FRUSTUM) {
    tmin = __fmul_rn(tmin, norm);
    tmax = __fmul_rn(tmax, norm);
  }
  return sim_cast(v, eye, dir, tmin, tmax);
}

// splitmix64 (Steele, Lea, Flood 2014) as a counter-based generator.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

__device__ __forceinline__ float noisy(float x, uint64_t seed, long long i, float sigma_coef,
                                       float drop) {
  const uint64_t a = mix64(seed ^ mix64((uint64_t)i));
  const uint64_t b = mix64(a);
  const float u1 = ((float)(a >> 40) + 0.5f) * (1.0f / 16777216.0f);
  const float u2 = (float)((a >> 16) & 0xFFFFFFu) * (1.0f / 16777216.0f);
  const float u3 = (float)(b >> 40) * (1.0f / 16777216.0f);
  if (x > 0.0f) {
    const float g = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
    x = x + g * sigma_coef * x * x;
    if (u3 < drop || !(x > 0.0f)) x = 0.0f;
  }
  return x;
}

}  // namespace
}  // namespace nm
