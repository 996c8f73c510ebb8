// nm_traverse.cu -- persistent traversal + per-frame labelling kernel (sm_100a).
//
// Replaces nodePassHDDA / voxelPassHDDA and the CUB compaction between them
// (frustumCastCloud.cu:44-246): one pass walks every ray voxel by voxel with the insertion
// DDA of Handler.cpp:58-85 and records one label per voxel (hit overrides miss), allocating
// map leaves on the fly.
//
// Work distribution: CTAs stay resident and take tiles of neighbouring pixels from a device
// counter, longest rays first.  A tile of short rays is walked: one thread per ray, the DDA step by
// step (walk_counted), the rays ordered by range (a counting sort on 32 range buckets) so the 32
// lanes of a warp walk rays of about the same length.  A step compares the three crossing times
// (non-negative doubles, ties to the higher axis), advances the chosen axis with one rounded double
// add, and keeps the voxel as (leaf code, index inside the leaf); labels collect per 32-voxel word
// in a register and go to shared memory with one shared atomic when the walk leaves the word.
//
// A tile with long rays (tile_split_bucket) is taken apart in quarters and marched (march_*): every
// voxel a ray enters is entered through a lattice plane, and on plane j of axis a the ray's other
// two coordinates are linear in j, so the planes of a ray are independent and are spread over
// all warps of the CTA; the walk's chain of dependent steps, which made a frame of few tiles wait
// for its longest rays, is gone.  Neighbouring rays also pass the same voxels many times over
// (24.2 M voxel visits label 181 K voxels of a 640x480 frame at 0.05 m): planes lie on lanes, and a
// lane ORs the cells of its plane over the tile's rays in a register, 14 instructions a ray, before
// it writes them to the leaf table once.
//
// The march's labels are those of the double-precision DDA under the map's rounding mode bit for
// bit.  The DDA's crossing times carry an absolute error below 2e-9 voxels over the longest ray (4000
// rounded adds of at most 2^-41 each), so wherever the exact line stays further from the deciding
// lattice plane than that and than the march's own arithmetic can be off, both choose the same
// voxel.  A ray with any coordinate closer than 1e-8 voxels, or whose last crossing is as close to a
// tie, or whose length or last time is as close to the maximum range, is walked by the DDA itself
// (setup_ray, walk_ray).  walk_counted takes its number of steps from the same test.
//
// Leaves are named by a leaf code lx*2^20 + ly*2^10 + lz (mod 2^32) relative to the eye's leaf,
// one-to-one over every leaf a frame can reach while max_range / res stays below kNarrowMaxTime
// voxels; it is both the tag and the hash source of a per-CTA shared-memory leaf table (32 label
// words per leaf).  A leaf that finds no room in the table goes straight to the device table.
// After a tile, one lane per cached leaf looks its slot up and puts it on the touched list (the
// lookups overlap), then one warp per leaf ORs its 32 words into the device label buffer.
//
// Frames whose reach exceeds the code's range (max_range / res >= kNarrowMaxTime) take
// k_traverse_wide: one thread per ray with device-table lookups and label atomics.
//
// k_traverse_render renders each tile's ranges from the sim map into shared memory first
// (nm_sim_insert), so one launch does the simulated frame and its insertion.
#include <cfloat>
#include <climits>
#include <algorithm>
#include <cstdint>
#include <mutex>

#include "nm_device.cuh"
#include "nm_internal.h"
#include "nm_sim_device.cuh"

namespace nm {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kSortBuckets = 32;
// Word index of a leaf whose labels were lost (device table full): flushes skip it.
constexpr int kLostWord = INT_MIN;
// Word indices at or above kGlobFloor and below 0 name a device-table leaf g as
// -(g + 1) * 16 + w (w = miss word 0..15); capacities are at most 2^26 slots.
constexpr int kGlobFloor = -(1 << 30);

__device__ __forceinline__ uint32_t leaf_code(int lx, int ly, int lz) {
  return ((uint32_t)lx << 20) + ((uint32_t)ly << 10) + (uint32_t)lz;
}

// Table position of a leaf code: Fibonacci hashing, top bits (`sh` = 32 - log2 entries).
__device__ __forceinline__ uint32_t code_slot(uint32_t code, int sh) {
  return (code * 0x9E3779B1u) >> sh;
}

__device__ __forceinline__ int sext(uint32_t v, int bits) {
  return (int)(v << (32 - bits)) >> (32 - bits);
}

// Tag of an empty table entry: the code of no leaf within reach.
constexpr uint32_t kNoLeaf = 1536u << 20;

// Shared leaf table of a CTA.  Leaf codes are relative to the eye's leaf, so the table's state
// between tiles (every tag kNoLeaf, every word 0) does not depend on the frame.
struct TileTable {
  uint32_t* tags;    // leaf code per entry, kNoLeaf = empty
  uint32_t* words;   // 32 label words per entry: 0..15 hit, 16..31 miss
  uint32_t* used;    // entries in use, in order of first use
  uint32_t* n_used;
  uint32_t smask;
  int sh;
  int elx, ely, elz;  // the eye's leaf

  __device__ __forceinline__ uint32_t code(int lx, int ly, int lz) const {
    return leaf_code(lx - elx, ly - ely, lz - elz);
  }
  // Absolute leaf key of a code (every reachable leaf lies within 511 leaves of the eye's on each
  // axis, where the code is one-to-one).
  __device__ __forceinline__ unsigned long long key(uint32_t c) const {
    const int dz = sext(c & 0x3FFu, 10);
    const uint32_t c1 = (c - (uint32_t)dz) >> 10;
    const int dy = sext(c1 & 0x3FFu, 10);
    const int dx = sext(((c1 - (uint32_t)dy) >> 10) & 0xFFFu, 12);
    return leaf_key(elx + dx, ely + dy, elz + dz);
  }
};

// Probe / insert of a code the inline probe missed.  Returns the miss-word base of the leaf:
// e * 32 + 16 for table entry e, -(g + 1) * 16 for device-table slot g, kLostWord when the
// device table is full.
__device__ __noinline__ int leaf_base_slow(const TileTable& tt, const MapView& m, uint32_t code,
                                           uint32_t epoch, int plane) {
  uint32_t h = code_slot(code, tt.sh);
  const uint32_t limit = (tt.smask + 1) < 16u ? (tt.smask + 1) : 16u;
  for (uint32_t i = 0; i < limit; ++i) {
    const uint32_t k = ((volatile uint32_t*)tt.tags)[h];
    if (k == code) return (int)(h * kLabelWords + 16);
    if (k == kNoLeaf) {
      const uint32_t old = atomicCAS(&tt.tags[h], kNoLeaf, code);
      if (old == kNoLeaf) {
        tt.used[atomicAdd(tt.n_used, 1u)] = h;
        return (int)(h * kLabelWords + 16);
      }
      if (old == code) return (int)(h * kLabelWords + 16);
    }
    h = (h + 1) & tt.smask;
  }
  const int g = map_find_or_insert(m, tt.key(code));
  if (g < 0) return kLostWord;
  mark_touched(m, g, epoch, plane);
  return -(g + 1) * 16;
}

// (Two probes inline: a leaf whose home entry another one holds is mostly found next to it, and
// the call costs the whole warp.)
__device__ __forceinline__ int leaf_base(const TileTable& tt, const MapView& m, uint32_t code,
                                         uint32_t epoch, int plane) {
  uint32_t e = code_slot(code, tt.sh);
  if (((volatile uint32_t*)tt.tags)[e] == code) return (int)(e * kLabelWords + 16);
  e = (e + 1) & tt.smask;
  if (((volatile uint32_t*)tt.tags)[e] == code) return (int)(e * kLabelWords + 16);
  return leaf_base_slow(tt, m, code, epoch, plane);
}

// OR `bits` into label word `cw` (a table word, a device-table miss word, or lost).
__device__ __noinline__ void flush_device_word(const MapView& m, int cw, uint32_t bits, int plane) {
  if (cw < kGlobFloor) return;
  const uint32_t x = (uint32_t)(-cw - 1);
  const uint32_t g = x >> 4, w = 15u - (x & 15u);
  atomicOr(&m.labels[((size_t)plane * m.capacity + g) * kLabelWords + 16 + w], bits);
}

__device__ __forceinline__ void flush_word(uint32_t* s_words, const MapView& m, int cw,
                                           uint32_t bits, int plane) {
  if (cw >= 0)
    atomicOr(&s_words[cw], bits);
  else
    flush_device_word(m, cw, bits, plane);
}

// Hit label of voxel `l` of the leaf whose miss-word base is `wbase`.
__device__ __noinline__ void hit_device(const MapView& m, int wbase, int l, int plane) {
  if (wbase < kGlobFloor) return;
  const uint32_t g = (uint32_t)(-wbase / 16 - 1);
  atomicOr(&m.labels[((size_t)plane * m.capacity + g) * kLabelWords + (l >> 5)], 1u << (l & 31));
}

struct Ray {
  double t0, t1, t2;  // next crossing time per axis (never negative)
  double d0, d1, d2;  // crossing spacing per axis
  double len;         // ray length in voxels
  int ds0, ds1, ds2;  // step of the voxel index inside the leaf per axis: +-64, +-8, +-1 or 0
  int l;              // voxel index inside the leaf, x*64 + y*8 + z
  uint32_t hs0, hs1, hs2;  // leaf-code step per axis: +-2^20, +-2^10, +-1 or 0
  uint32_t code;           // leaf code of the current voxel, relative to the eye's leaf
};

// Ray set-up of the insertion DDA (Handler.cpp:64-76 restated; see trace_point in
// nm_device.cuh for the same arithmetic in one piece).  Returns false when the point is
// dropped (beyond range, NaN/Inf, shorter than 1e-7).
template <int RM>
__device__ __forceinline__ bool setup_ray(const FrameParams& f, const float p[3], Ray& r) {
  using A = Ar<RM>;
  const float* R = f.R;
  const float dxf = A::fadd(A::fadd(A::fmul(R[0], p[0]), A::fmul(R[1], p[1])), A::fmul(R[2], p[2]));
  const float dyf = A::fadd(A::fadd(A::fmul(R[3], p[0]), A::fmul(R[4], p[1])), A::fmul(R[5], p[2]));
  const float dzf = A::fadd(A::fadd(A::fmul(R[6], p[0]), A::fmul(R[7], p[1])), A::fmul(R[8], p[2]));
  const double dx = dxf, dy = dyf, dz = dzf;
  const double len = A::dsqrt(A::dadd(A::dadd(A::dmul(dx, dx), A::dmul(dy, dy)), A::dmul(dz, dz)));
  const double ray_len = A::ddiv(len, f.res_d);
  if (!(ray_len < (double)f.max_time)) return false;
  if (!(len > 1.0e-7)) return false;
  r.len = ray_len;
  const double inv_len = A::drcp(len);
  const double nd[3] = {A::dmul(dx, inv_len), A::dmul(dy, inv_len), A::dmul(dz, inv_len)};
  double tn[3], dl[3];
  int st[3], v[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    v[a] = (int)floor(f.eye[a]);
    if (nd[a] == 0.0) {
      st[a] = 0;
      tn[a] = DBL_MAX;
      dl[a] = DBL_MAX;
    } else {
      const double inv = A::drcp(nd[a]);
      if (inv > 0.0) {
        st[a] = 1;
        tn[a] = A::dmul(A::dadd((double)(v[a] + 1), -f.eye[a]), inv);
        dl[a] = inv;
      } else {
        st[a] = -1;
        tn[a] = A::dmul(A::dadd((double)v[a], -f.eye[a]), inv);
        dl[a] = -inv;
      }
      if (tn[a] == 0.0) tn[a] = 0.0;  // canonical +0
    }
  }
  r.t0 = tn[0];
  r.t1 = tn[1];
  r.t2 = tn[2];
  r.d0 = dl[0];
  r.d1 = dl[1];
  r.d2 = dl[2];
  r.ds0 = st[0] * 64;
  r.ds1 = st[1] * 8;
  r.ds2 = st[2];
  r.hs0 = (uint32_t)st[0] << 20;
  r.hs1 = (uint32_t)st[1] << 10;
  r.hs2 = (uint32_t)st[2];
  r.l = ((v[0] & 7) << 6) | ((v[1] & 7) << 3) | (v[2] & 7);
  r.code = 0u;  // the eye's leaf
  return true;
}

__device__ __forceinline__ bool pixel_point(const FrameParams& f, int w, int h, float p[3]) {
  if (f.input_kind == 1) return range_point(f, w, h, p);
  if (f.input_kind == 2 && (uint32_t)(h * f.width + w) >= __ldg(f.n_valid)) return false;
  return xyz_point(f, w, h, p);
}

// Walk one ray from its set-up to its end, labelling every voxel it leaves as a miss and its
// end voxel as a hit (when the crossing that leaves it lies below max_time).  Returns the
// number of label events.
template <int RM>
__device__ __forceinline__ uint32_t walk_ray(const Ray& r, const TileTable& tt, const MapView& m,
                                             double max_time, uint32_t epoch, int plane) {
  using A = Ar<RM>;
  double t0 = r.t0, t1 = r.t1, t2 = r.t2;
  const double d0 = r.d0, d1 = r.d1, d2 = r.d2, len = r.len;
  int l = r.l;
  uint32_t code = r.code;
  int wbase = leaf_base(tt, m, code, epoch, plane);
  int cw = kLostWord;  // word the pending bits belong to
  uint32_t acc = 0u;   // pending miss bits of word cw
  uint32_t n = 0u;
  double t;
  for (;;) {
    const bool c01 = t0 < t1, c02 = t0 < t2, c12 = t1 < t2;
    const bool is0 = c01 && c02;
    const bool is1 = !c01 && c12;
    t = is0 ? t0 : (is1 ? t1 : t2);
    if (!(t <= len)) break;
    // miss label of the voxel being left
    const int wi = wbase + (l >> 5);
    if (wi != cw) {
      // acc holds at least the bit of the step that set cw (none only for the initial
      // kLostWord, which flush_device_word drops)
      if (cw >= 0)
        atomicOr(&tt.words[cw], acc);
      else
        flush_device_word(m, cw, acc, plane);
      cw = wi;
      acc = 0u;
    }
    acc |= 1u << (l & 31);
    ++n;
    // advance along the chosen axis: crossing time, index inside the leaf, leaf on wrap
    const double dstep = is0 ? d0 : (is1 ? d1 : d2);
    const double tn = A::dadd(t, dstep);
    if (is0) t0 = tn;
    if (is1) t1 = tn;
    if (!is0 && !is1) t2 = tn;
    const int msk = is0 ? 0x1C0 : (is1 ? 0x38 : 0x7);
    const int ds = is0 ? r.ds0 : (is1 ? r.ds1 : r.ds2);
    const int vv = (l & msk) + ds;
    l = (l & ~msk) | (vv & msk);
    if ((unsigned)vv > (unsigned)msk) {
      code += is0 ? r.hs0 : (is1 ? r.hs1 : r.hs2);
      wbase = leaf_base(tt, m, code, epoch, plane);
    }
  }
  if (acc) flush_word(tt.words, m, cw, acc, plane);
  if (t < max_time) {
    if (wbase >= 0)
      atomicOr(&tt.words[wbase - 16 + (l >> 5)], 1u << (l & 31));
    else
      hit_device(m, wbase, l, plane);
    ++n;
  }
  return n;
}

// One step of the DDA: advances the crossing time of the axis crossed next (smallest time, ties to
// the higher axis) and gives that axis's mask and step of the voxel index inside the leaf.
template <int RM>
__device__ __forceinline__ void dda_step(double& t0, double& t1, double& t2, double d0, double d1,
                                         double d2, int ds0, int ds1, int ds2, int& msk, int& ds) {
#define NM_DDA_STEP(ADD)                                                        \
  asm("{\n\t.reg .pred c, p0, p1, p2;\n\t"                                       \
      "setp.lt.f64 c, %0, %1;\n\t"                                              \
      "setp.lt.and.f64 p0, %0, %2, c;\n\t"                                      \
      "setp.lt.and.f64 p1, %1, %2, !c;\n\t"                                     \
      "or.pred p2, p0, p1;\n\t"                                                 \
      "@p0 " ADD " %0, %0, %5;\n\t"                                             \
      "@p1 " ADD " %1, %1, %6;\n\t"                                             \
      "@!p2 " ADD " %2, %2, %7;\n\t"                                            \
      "selp.b32 %3, 56, 7, p1;\n\t"                                             \
      "selp.b32 %4, %9, %10, p1;\n\t"                                           \
      "selp.b32 %3, 448, %3, p0;\n\t"                                           \
      "selp.b32 %4, %8, %4, p0;\n\t}"                                           \
      : "+d"(t0), "+d"(t1), "+d"(t2), "=&r"(msk), "=&r"(ds)                     \
      : "d"(d0), "d"(d1), "d"(d2), "r"(ds0), "r"(ds1), "r"(ds2))
  if (RM == NM_ROUND_DOWN)
    NM_DDA_STEP("add.rm.f64");
  else
    NM_DDA_STEP("add.rn.f64");
#undef NM_DDA_STEP
}

// walk_ray for a ray whose number of crossings `n` is known: the loop counts down instead of comparing
// the next crossing's time with the ray's length, and needs that time only at its end, so each
// axis's time is advanced in place under a predicate.  Bound by issue; the 16-frame tick's
// traversal took 856 us with walk_ray alone and takes 783 us.
template <int RM>
__device__ __forceinline__ uint32_t walk_counted(const Ray& r, int n, const TileTable& tt,
                                                 const MapView& m, double max_time, uint32_t epoch,
                                                 int plane) {
  double t0 = r.t0, t1 = r.t1, t2 = r.t2;
  int l = r.l;
  uint32_t code = r.code;
  int wbase = leaf_base(tt, m, code, epoch, plane);
  int cw = wbase + (l >> 5);  // word the pending bits belong to
  uint32_t acc = 0u;          // pending miss bits of word cw
  for (int left = n; left > 0; --left) {
    const int wi = wbase + (l >> 5);
    if (wi != cw) {
      if (cw >= 0)
        atomicOr(&tt.words[cw], acc);
      else
        flush_device_word(m, cw, acc, plane);
      cw = wi;
      acc = 0u;
    }
    acc |= 1u << (l & 31);
    int msk, ds;
    dda_step<RM>(t0, t1, t2, r.d0, r.d1, r.d2, r.ds0, r.ds1, r.ds2, msk, ds);
    const int vv = (l & msk) + ds;
    l = (l & ~msk) | (vv & msk);
    if ((unsigned)vv > (unsigned)msk) {
      code += msk == 0x1C0 ? r.hs0 : (msk == 0x38 ? r.hs1 : r.hs2);
      wbase = leaf_base(tt, m, code, epoch, plane);
    }
  }
  if (acc) flush_word(tt.words, m, cw, acc, plane);
  if (!(fmin(fmin(t0, t1), t2) < max_time)) return (uint32_t)n;
  if (wbase >= 0)
    atomicOr(&tt.words[wbase - 16 + (l >> 5)], 1u << (l & 31));
  else
    hit_device(m, wbase, l, plane);
  return (uint32_t)n + 1u;
}

// ---- plane march -----------------------------------------------------------------------------

constexpr int kMarchThreads = 256;   // threads of a traversal CTA, whatever its tile
constexpr int kMarchRays = 256;      // rays of a tile handled at a time
constexpr int kMarchChunk = 16;      // planes per work item: half a warp, two rays at a time
constexpr int kMarchFew = 6;         // planes outside the window that one lane takes alone
constexpr int kMarchBins = 128;      // chunks of planes that the window takes, at most
constexpr float kMarchSpread = 1.98f;  // widest offset from the reference line (window of 5 x 5)
constexpr float kNearPlane = 1e-4f;  // first planes this close to the eye are ordered exactly
constexpr uint32_t kTie32 = 43u;     // 1e-8 voxels in units of 2^-32: closer to a lattice plane
                                     // counts as undecided (the DDA's crossings and the positions
                                     // here are each within 2e-9 of the exact line)
constexpr double kMagic = 1572864.0;  // 1.5 * 2^20: x + kMagic has floor(x) in the low 20 bits of
                                      // its high word and x's fraction (2^-32) in its low word

__device__ __forceinline__ int magic_floor(double q) {
  return (__double2hiint(q) & 0xFFFFF) - 0x80000;
}
__device__ __forceinline__ bool magic_tie(double q) {
  return (uint32_t)__double2loint(q) + kTie32 < 2u * kTie32;
}

// Eye constants of a frame.  Index [a][s]: axis a, rays of negative (0) or positive (1) direction.
struct MarchFrame {
  double fe[3];        // eye - floor(eye), plus kMagic
  double first[3][2];  // distance to the first plane crossed
  int v[3];            // the eye's voxel
  double inv_res;
  // squared lengths (m): below far2 a ray leaves its end voxel before the maximum range, below sure2
  // it ends before it, above drop2 the point is out of range
  float far2, sure2, drop2;
  bool near[3][2];     // the first plane is closer than kNearPlane: the set-up marks it, or sends the
                       // ray to the DDA, and the march leaves it out
};

// Rays of a round.  Per axis and ray: `d` = end minus eye (m), `n` = planes to mark (bit 15: positive
// direction).  `rel`, `take` = the rays of an axis that the tile's window takes, by falling
// number of chunks: slopes relative to the reference line; planes | ray << 16.  `rest` = planes
// outside the window: axis | ray << 2 | first plane << 16.
struct MarchRays {
  float2* rel;
  float* d;
  uint32_t* take;
  uint32_t* rest;
  uint16_t* n;
  int count;
};

__host__ __device__ constexpr size_t march_bytes(int rays) {
  return (size_t)rays * 3 * (8 + 4 + 4 + 4 + 2);
}

__device__ __forceinline__ MarchRays march_rays(void* mem, int rays) {
  MarchRays mr;
  mr.rel = reinterpret_cast<float2*>(mem);
  mr.d = reinterpret_cast<float*>(mr.rel + 3 * rays);
  mr.take = reinterpret_cast<uint32_t*>(mr.d + 3 * rays);
  mr.rest = mr.take + 3 * rays;
  mr.n = reinterpret_cast<uint16_t*>(mr.rest + 3 * rays);
  mr.count = rays;
  return mr;
}

struct MarchShared {
  int maxn[3][2];
  uint32_t ref[3][2];  // reference ray: the one with planes nearest the tile's middle
  uint32_t n_rest[2];                   // rays with many / with few planes outside the window
  uint32_t next;                        // next work item
  uint32_t dda;                         // some ray went to the DDA
  uint32_t bins[3][2][kMarchBins];      // rays by chunks taken, then: rays taking more than this
  uint32_t walk[kMarchRays / 32];       // rays left to the DDA by their set-up (not counted yet)
  uint32_t undecided[kMarchRays / 32];  // rays left to the DDA by one of their planes
};

// Clears what a round accumulates into.
__device__ __forceinline__ void march_reset(MarchShared& ms) {
  for (int i = threadIdx.x; i < 6 * kMarchBins; i += blockDim.x) (&ms.bins[0][0][0])[i] = 0u;
  if (threadIdx.x < kMarchRays / 32) ms.undecided[threadIdx.x] = ms.walk[threadIdx.x] = 0u;
  if (threadIdx.x < 6) {
    (&ms.maxn[0][0])[threadIdx.x] = 0;
    (&ms.ref[0][0])[threadIdx.x] = 0xFFFFFFFFu;
  }
  if (threadIdx.x == 6) ms.n_rest[0] = ms.n_rest[1] = ms.next = 0u;
}

// Fills `mf`: an axis per thread, the divisions and lengths on two more (of different warps, so
// they run side by side); every thread of the CTA calls it.
__device__ __forceinline__ void march_frame(const FrameParams& f, MarchFrame& mf) {
  const int a = threadIdx.x;
  if (a < 3) {
    const double v = floor(f.eye[a]);
    mf.v[a] = (int)v;
    mf.fe[a] = f.eye[a] - v + kMagic;
    mf.first[a][0] = f.eye[a] - v;
    mf.first[a][1] = (v + 1.0) - f.eye[a];
    mf.near[a][0] = f.eye[a] - v < (double)kNearPlane;
    mf.near[a][1] = (v + 1.0) - f.eye[a] < (double)kNearPlane;
  } else if (a == 32) {
    mf.inv_res = 1.0 / f.res_d;
  } else if (a == 33) {
    // a ray of this length leaves its end voxel (2 voxels across at most) before max_time
    const double reach = (double)f.max_time * f.res_d, far = reach - 2.0 * f.res_d;
    mf.far2 = far > 0.0 ? (float)(far * far * (1.0 - 1e-5)) : 0.0f;
    mf.sure2 = (float)(reach * reach * (1.0 - 1e-5));
    mf.drop2 = (float)(reach * reach * (1.0 + 1e-5));
  }
}

// Number of lattice planes that a ray which passes the DDA's length checks crosses (end minus eye `d`,
// m), or -1 where its end is too close to a plane, or it is too short, to tell without the DDA's own
// arithmetic.  (Rays that end near the maximum range have a count too, and walk_counted tells from its
// last time whether they hit.  Left to walk_ray they made each warp that held one go through both
// loops: one 320x240 frame of 50 voxels' reach, 0.8 % of its rays ending there, 38.4 -> 27.3 us.)
__device__ __forceinline__ int march_count(const MarchFrame& mf, const float d[3]) {
  const float len2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
  bool sure = len2 > 1e-13f;
  int n = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double q = fma((double)d[a], mf.inv_res, mf.fe[a]);
    sure &= d[a] == 0.0f || !magic_tie(q);
    n += d[a] == 0.0f ? 0 : abs(magic_floor(q));
  }
  return sure ? n : -1;
}

// OR `bits` into miss word `w` (0..15) of the leaf whose miss-word base is `base`.  Most bits are
// there already (the patches of a tile share voxels): a read costs less than an atomic.
__device__ __forceinline__ void or_word(const TileTable& tt, const MapView& m, int base, int w,
                                        uint32_t bits, int plane) {
  const int cw = base + w;
  if (cw >= 0) {
    if ((((volatile uint32_t*)tt.words)[cw] & bits) != bits) atomicOr(&tt.words[cw], bits);
  } else {
    flush_device_word(m, cw, bits, plane);
  }
}

// Miss label of one voxel.
__device__ __forceinline__ void mark_voxel(const TileTable& tt, const MapView& m, int x, int y,
                                           int z, uint32_t epoch, int plane) {
  const int base = leaf_base(tt, m, tt.code(x >> 3, y >> 3, z >> 3), epoch, plane);
  or_word(tt, m, base, (x & 7) * 2 + ((y >> 2) & 1), 1u << (((y & 3) << 3) | (z & 7)), plane);
}

// Bits 0..3 of n moved to bits 0, 8, 16, 24.
__device__ __forceinline__ uint32_t spread_bytes(uint32_t n) {
  return (n * 0x00204081u) & 0x01010101u;
}

// Sets up ray `r` of a round (`ok`: it has the sensor-frame point p; `off`: its distance from the
// tile's middle, to choose a reference): its end `d` and planes per axis `n` (also into `mr`),
// its hit label, and its share of `visits` and `rays`.
template <int RM>
__device__ __forceinline__ void march_setup(const FrameParams& f, const MarchFrame& mf,
                                            const TileTable& tt, const MapView& m,
                                            const MarchRays& mr, MarchShared& ms, bool ok,
                                            const float p[3], int r, int off, float d[3],
                                            int n[3], uint32_t& visits, uint32_t& rays) {
  using A = Ar<RM>;
  const int lane = threadIdx.x & 31;
  int end[3] = {0, 0, 0};
  d[0] = d[1] = d[2] = 0.0f;
  n[0] = n[1] = n[2] = 0;
  bool walk = false;  // the DDA decides this ray
  bool live = false, hit = true;
  int total = 0;
  if (ok) {
    const float* R = f.R;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      d[a] = A::fadd(A::fadd(A::fmul(R[3 * a], p[0]), A::fmul(R[3 * a + 1], p[1])),
                     A::fmul(R[3 * a + 2], p[2]));
    const float len2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    if (len2 <= mf.drop2) {  // (NaN and Inf fall out here)
      live = len2 < mf.sure2 && len2 > 1e-13f;
      walk = !live;
    }
    if (live) {
      // the last crossing is the one least far behind the end, (end - plane) / |d|
      int last = -1;
      float lg = 0.0f, ld = 0.0f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (d[a] == 0.0f) continue;
        const double q = fma((double)d[a], mf.inv_res, mf.fe[a]);  // end, from the eye's voxel
        walk |= magic_tie(q);
        end[a] = magic_floor(q);
        n[a] = abs(end[a]);
        if (n[a] == 0) continue;
        const uint32_t lo = (uint32_t)__double2loint(q);
        const float g = (float)(d[a] > 0.0f ? lo : 0u - lo), da = fabsf(d[a]);
        const float x = g * ld, y = lg * da;
        if (last >= 0)  // 1e-6 relative for the products, 1e-8 voxels for the positions
          walk |= !(fabsf(x - y) > 1e-6f * (x + y) + 43.0f * (da + ld));
        if (last < 0 || x < y) {
          last = a;
          lg = g;
          ld = da;
        }
      }
      total = n[0] + n[1] + n[2];
      // Near the range a ray's end voxel is a hit only if the crossing that leaves it comes before the
      // range.  (The DDA's times are within 2e-9 of the exact line's.  With all such rays left to the DDA
      // each made its unit wait for one walk of full length: 640x480 at 10 m with 0.1 % of the rays
      // ending there 124 -> 113.5 us, voxel-filtered 104 -> 84, a 64x1024 spinning sensor's at 20 m
      // 71.5 -> 62.3.)
      if (!(len2 < mf.far2)) {
        const double dx = d[0], dy = d[1], dz = d[2], len = sqrt(dx * dx + dy * dy + dz * dz);
        double t = DBL_MAX;
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if (d[a] != 0.0f)
            t = fmin(t, (mf.first[a][d[a] > 0.0f] + (double)n[a]) * (len / fabs((double)d[a])));
        hit = t < (double)f.max_time;
        walk |= fabs(t - (double)f.max_time) < 1e-8;
      }
      live = !walk;
      // the voxel entered by the last crossing is the end voxel: no miss
#pragma unroll
      for (int a = 0; a < 3; ++a) n[a] -= last == a ? 1 : 0;
    }
  }
  if (!live) n[0] = n[1] = n[2] = total = 0;
  const unsigned w0 = __ballot_sync(kFull, walk);
  if (lane == 0 && w0) {
    ms.walk[r >> 5] = w0;
    ms.dda = 1u;
  }

  // First planes close to the eye: an eye near a lattice edge or corner crosses several of them
  // almost at once, which only their order decides.  (b, 0) comes before (a, 0) when
  // first_b / |d_b| < first_a / |d_a|; both zero: the higher axis first, as in the DDA.  (The products
  // below decide only while they are far from the denormals, where a factor has lost its precision.)
  if (live && (mf.near[0][d[0] > 0.0f] | mf.near[1][d[1] > 0.0f] | mf.near[2][d[2] > 0.0f])) {
    bool tie = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (!mf.near[a][d[a] > 0.0f] || n[a] <= 0) continue;
      const float fa = (float)mf.first[a][d[a] > 0.0f];
      int v[3];
      v[a] = d[a] > 0.0f ? 1 : -1;
      bool sure = true;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (b == a) continue;
        v[b] = 0;
        if (d[b] == 0.0f) continue;
        const float fb = (float)mf.first[b][d[b] > 0.0f];
        const float x = fb * fabsf(d[a]), y = fa * fabsf(d[b]);
        bool before = y > x;
        if (mf.first[a][d[a] > 0.0f] == 0.0 && mf.first[b][d[b] > 0.0f] == 0.0)
          before = b > a;
        else if (!(x + y > 1e-30f) || !(fabsf(x - y) > 1e-5f * (x + y)) ||
                 !(y < 0.99f * (x + fabsf(d[a]))))  // not so far that (b, 1) comes in question
          sure = false;
        if (before) v[b] = d[b] > 0.0f ? 1 : -1;
      }
      if (sure)
        mark_voxel(tt, m, mf.v[0] + v[0], mf.v[1] + v[1], mf.v[2] + v[2], f.epoch, f.plane);
      else
        tie = true;
    }
    if (tie) {
      atomicOr(&ms.undecided[r >> 5], 1u << lane);
      ms.dda = 1u;
    }
  }

  if (live) {
    visits += (uint32_t)total + (hit ? 1u : 0u);
    rays += 1u;
  }
  if (live && hit) {  // hit label of the end voxel
    const int x = mf.v[0] + end[0], y = mf.v[1] + end[1], z = mf.v[2] + end[2];
    const int base = leaf_base(tt, m, tt.code(x >> 3, y >> 3, z >> 3), f.epoch, f.plane);
    const int l = local_index(x, y, z);
    if (base >= 0) {
      const uint32_t bit = 1u << (l & 31);
      uint32_t* w = &tt.words[base - 16 + (l >> 5)];
      if (!(*(volatile uint32_t*)w & bit)) atomicOr(w, bit);
    } else {
      hit_device(m, base, l, f.plane);
    }
  }
  __syncwarp();
  // miss label of the eye's voxel, left by every ray with a crossing
  const unsigned left = __ballot_sync(kFull, total > 0);
  if (left && lane == __ffs(left) - 1)
    mark_voxel(tt, m, mf.v[0], mf.v[1], mf.v[2], f.epoch, f.plane);
  __syncwarp();

#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool up = d[a] > 0.0f;
    mr.d[a * mr.count + r] = d[a];
    mr.n[a * mr.count + r] = (uint16_t)(n[a] | (up ? 0x8000 : 0));
    const unsigned have = __ballot_sync(kFull, n[a] > 0);
    if (!have) continue;
    const uint32_t key = ((uint32_t)off << 16) | (uint32_t)r;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const bool mine = n[a] > 0 && (int)up == s;
      const int most = __reduce_max_sync(kFull, mine ? n[a] : 0);
      if (most == 0) continue;
      const uint32_t ref = __reduce_min_sync(kFull, mine ? key : 0xFFFFFFFFu);
      if (lane == 0) {
        atomicMax(&ms.maxn[a][s], most);
        atomicMin(&ms.ref[a][s], ref);
      }
    }
  }
}

// Slopes of the reference line of (axis, sign): those of the reference ray, rounded to floats.
__device__ __forceinline__ float2 march_reference(const MarchRays& mr, const MarchShared& ms, int a,
                                                  int s) {
  const int r = (int)(ms.ref[a][s] & 0xFFFFu), b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
  const float inv = __frcp_rn(fabsf(mr.d[a * mr.count + r]));
  return make_float2(mr.d[b * mr.count + r] * inv, mr.d[c * mr.count + r] * inv);
}

// Lists the round's rays for march_planes.  On each axis a ray's first planes, while it stays
// within kMarchSpread voxels of its sign's reference line, go to the tile's window; the rays are
// ordered by the chunks they take there (a counting sort), so a chunk's rays are the first of the
// list and none is looked at for nothing.  The planes left are listed apart.
__device__ __forceinline__ void march_list(const MarchRays& mr, MarchShared& ms, const float d[3],
                                           const int n[3]) {
  const int tid = threadIdx.x, lane = tid & 31;
  float2 rel[3];
  int fit[3] = {0, 0, 0}, rank[3];
  if (tid < mr.count) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int s = d[a] > 0.0f;
      if (!__any_sync(kFull, n[a] > 0)) continue;
      int bin = 0;
      if (n[a] > 0) {
        const float2 w = march_reference(mr, ms, a, s);
        const float da = fabsf(d[a]), inv = __frcp_rn(da);
        const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
        // one rounding of the small difference, one of the product
        rel[a] = make_float2(fmaf(-w.x, da, d[b]) * inv, fmaf(-w.y, da, d[c]) * inv);
        const float spread = fmaxf(fabsf(rel[a].x), fabsf(rel[a].y));
        // planes j with spread * (first + j) < kMarchSpread, first <= 1
        const float k = fminf(__fdividef(kMarchSpread, spread), (float)((kMarchBins - 1) * kMarchChunk));
        fit[a] = k < (float)n[a] ? (int)k : n[a];
        bin = (fit[a] + kMarchChunk - 1) / kMarchChunk;
      }
      // few planes left: from the list's end; many: from its front (one counter update per warp)
      const int left = n[a] - fit[a];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const bool out = k == 0 ? left > kMarchFew : left > 0 && left <= kMarchFew;
        const unsigned outs = __ballot_sync(kFull, out);
        if (!outs) continue;
        uint32_t at = 0u;
        if (lane == 0) at = atomicAdd(&ms.n_rest[k], (uint32_t)__popc(outs));
        at = __shfl_sync(kFull, at, 0) + __popc(outs & ((1u << lane) - 1u));
        if (k == 1) at = (uint32_t)(3 * mr.count - 1) - at;
        if (out) mr.rest[at] = (uint32_t)a | ((uint32_t)tid << 2) | ((uint32_t)fit[a] << 16);
      }
      const unsigned peers = __match_any_sync(kFull, s * kMarchBins + bin);
      const int leader = __ffs(peers) - 1;
      uint32_t base = 0u;
      if (lane == leader && bin) base = atomicAdd(&ms.bins[a][s][bin], (uint32_t)__popc(peers));
      rank[a] = (int)__shfl_sync(kFull, base, leader) + __popc(peers & ((1u << lane) - 1u));
    }
  }
  __syncthreads();
  // per axis and sign, bins -> rays in the bins above
  for (int k = tid >> 5; k < 6; k += blockDim.x >> 5) {
    if ((&ms.maxn[0][0])[k] == 0) continue;
    uint32_t* bins = &ms.bins[0][0][0] + k * kMarchBins + lane * (kMarchBins / 32);
    uint32_t c[kMarchBins / 32], own = 0u;
#pragma unroll
    for (int i = 0; i < kMarchBins / 32; ++i) own += c[i] = bins[i];
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_down_sync(kFull, incl, o);
      if (lane + o < 32) incl += u;
    }
    uint32_t above = incl - own;
#pragma unroll
    for (int i = kMarchBins / 32 - 1; i >= 0; --i) {
      bins[i] = above;
      above += c[i];
    }
  }
  __syncthreads();
  if (tid < mr.count) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (fit[a] == 0) continue;
      const int s = d[a] > 0.0f;
      const int bin = (fit[a] + kMarchChunk - 1) / kMarchChunk;
      // positive rays follow the negative ones (bins[.][0][0]: all of those)
      const int at = a * mr.count + (int)ms.bins[a][s][bin] + rank[a] + (s ? (int)ms.bins[a][0][0] : 0);
      mr.rel[at] = rel[a];
      mr.take[at] = (uint32_t)fit[a] | ((uint32_t)tid << 16);
    }
  }
}

// One lane's plane of a window: the reference line's cell and the offset of its fraction.
struct MarchWindow {
  int b0, c0;     // cell of the window's first row and column, relative to the eye's voxel
  float cb, cc;   // 8 + the reference line's position in the window, plus 2 units of 2^-20
};

__device__ __forceinline__ MarchWindow march_window(float2 slope, double F, double feb, double fec) {
  const double qb = fma((double)slope.x, F, feb), qc = fma((double)slope.y, F, fec);
  MarchWindow w;
  w.b0 = magic_floor(qb) - 2;
  w.c0 = magic_floor(qc) - 2;
  // 0x41200000 is 10.0f, a unit of its mantissa 2^-20
  const uint32_t fb = (uint32_t)__double2loint(qb), fc = (uint32_t)__double2loint(qc);
  w.cb = __uint_as_float(0x41200002u + (fb >> 12) + ((fb >> 11) & 1u));
  w.cc = __uint_as_float(0x41200002u + (fc >> 12) + ((fc >> 11) & 1u));
  return w;
}

// Writes a window's cells as miss labels: lane l the plane (l & 15).  `va`: the plane's voxel coordinate on axis a; b0, c0: the
// window's first row and column (absolute voxels).
__device__ __forceinline__ void march_write(int a, const TileTable& tt, const MapView& m,
                                            uint32_t mask, int va, int b0, int c0, uint32_t epoch,
                                            int plane) {
  const int cs = c0 & 7;
  uint32_t code0 = 0u;
  int base0 = kLostWord;
  bool cached = false;
  // rows with cells (bit 6 * row); the lower half-warp takes the first, third, ..., the upper the
  // second, fourth
  uint32_t rows = (mask | (mask >> 1) | (mask >> 2) | (mask >> 3) | (mask >> 4)) & 0x01041041u;
  if (threadIdx.x & 16) rows &= rows - 1u;
#pragma unroll 1
  for (; rows; rows &= rows - 1u, rows &= rows - 1u) {
    const int row6 = __ffs(rows) - 1;
    const uint32_t bits = (mask >> row6) & 31u;
    const int row = (row6 * 11) >> 6;  // row6 / 6
    const int gb = b0 + row;
    uint32_t by = (bits << cs) & 0xFFu, rest = (bits << cs) >> 8;
    int lc = c0 >> 3;
    if (!by) {
      by = rest;
      rest = 0u;
      ++lc;
    }
#pragma unroll 1
    while (by) {
      const uint32_t code = a == 0   ? tt.code(va >> 3, gb >> 3, lc)
                            : a == 1 ? tt.code(gb >> 3, va >> 3, lc)
                                     : tt.code(gb >> 3, lc, va >> 3);
      if (!cached || code != code0) {
        base0 = leaf_base(tt, m, code, epoch, plane);
        code0 = code;
        cached = true;
      }
      if (a == 2) {  // x rows of y cells at one z
        const int w = (gb & 7) * 2, sh = va & 7;
        if (by & 15u) or_word(tt, m, base0, w, spread_bytes(by & 15u) << sh, plane);
        if (by >> 4) or_word(tt, m, base0, w + 1, spread_bytes(by >> 4) << sh, plane);
      } else {  // runs of z
        const int x = a == 0 ? va : gb, y = a == 0 ? gb : va;
        or_word(tt, m, base0, (x & 7) * 2 + ((y >> 2) & 1), by << ((y & 3) * 8), plane);
      }
      by = rest;
      rest = 0u;
      ++lc;
    }
  }
  __syncwarp();
}

// Marks planes j, j + step, ... below n of one ray, two at a time (their table reads overlap);
// returns whether one was undecided.
__device__ __forceinline__ bool march_outside(const TileTable& tt, const MapView& m, int a, int s,
                                              double mb, double mc, double f0, double feb,
                                              double fec, int va0, int vb0, int vc0, int j,
                                              int step, int n, uint32_t epoch, int plane) {
  bool tie = false;
#pragma unroll 1
  for (; j < n; j += 2 * step) {
    uint32_t code[2], bit[2], tag[2], e[2];
    int w[2];
    bool ok[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int jk = j + k * step;
      const double F = f0 + (double)jk;
      const double qb = fma(mb, F, feb), qc = fma(mc, F, fec);
      const bool t = magic_tie(qb) || magic_tie(qc);
      ok[k] = jk < n && !t;
      tie |= jk < n && t;
      const int gb = vb0 + magic_floor(qb), gc = vc0 + magic_floor(qc);
      const int va = s ? va0 + 1 + jk : va0 - 1 - jk;
      const int x = a == 0 ? va : gb, y = a == 0 ? gb : (a == 1 ? va : gc), z = a == 2 ? va : gc;
      code[k] = tt.code(x >> 3, y >> 3, z >> 3);
      w[k] = (x & 7) * 2 + ((y >> 2) & 1);
      bit[k] = 1u << (((y & 3) << 3) | (z & 7));
      e[k] = code_slot(code[k], tt.sh);
      tag[k] = ((volatile uint32_t*)tt.tags)[e[k]];
    }
    int base[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      base[k] = (int)(e[k] * kLabelWords + 16);
      if (ok[k] && tag[k] != code[k]) base[k] = leaf_base(tt, m, code[k], epoch, plane);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (ok[k]) or_word(tt, m, base[k], w[k], bit[k], plane);
  }
  return tie;
}

// Miss labels of the voxels that the round's rays enter through lattice planes.  A work item is
// an axis, a sign and a chunk of 16 planes of the tile's window, over all rays that have it; the
// CTA's warps take items in turn.  Lane l holds plane j0 + (l & 15) and loops over every second
// ray: the rays' cells in the 5 x 5 window round the reference line are ORed in a register, a bit
// each, and written out once per plane.  The offset from the reference line is a product of two
// floats below 2 in size, exact to 1.5 units of 2^-20 with the window at [8, 16); 2 units are
// added, so a fraction below 4 units is too close to a cell's edge (one ray in 500 has such a
// crossing): the chunk is taken again with those crossings in double precision, and what is
// within 1e-8 voxels of an edge there sends its ray to the DDA.
//
// Planes outside the window (rays far apart at long range) are marked one by one from a
// double-precision position, 8 planes of 4 rays at a time.
//
// What bounds it: latency, at a third of the issue rate (33.5 M warp instructions for 14.7 M voxel
// visits of one 640x480 frame against the walk's 42 M, but eight barriers a unit); so it pays where
// the walk leaves SMs idle.  Traversal of one frame, walk alone -> now (B200): 64x1024 spinning sensor
// at 20 m and 0.05 m 114 -> 47.3 us, 1280x720 at 15 m and 0.02 m 1179 -> 410 us, voxel-filtered
// 640x480 at 10 m and 0.05 m 83.6 -> 58.1 us, unfiltered 94.5 -> 82.3 us.
__device__ __forceinline__ void march_planes(const MarchFrame& mf, const TileTable& tt,
                                             const MapView& m, const MarchRays& mr,
                                             MarchShared& ms, uint32_t epoch, int plane) {
  const int lane = threadIdx.x & 31, half = lane >> 4;
  int ends[6], chunks = 0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    chunks += min(((&ms.maxn[0][0])[k] + kMarchChunk - 1) / kMarchChunk, kMarchBins - 1);
    ends[k] = chunks;
  }
  const int many = (int)ms.n_rest[0], few = (int)ms.n_rest[1];
  const int wide = (many + 3) / 4;
  const int items = chunks + wide + (few + 31) / 32;
#pragma unroll 1
  for (;;) {
    int it = 0;
    if (lane == 0) it = (int)atomicAdd(&ms.next, 1u);
    it = __shfl_sync(kFull, it, 0);
    if (it >= items) break;
    if (it < chunks) {
      int k = 0, begin = 0;
#pragma unroll
      for (int q = 0; q < 5; ++q)
        if (it >= ends[q]) {
          k = q + 1;
          begin = ends[q];
        }
      const int a = k >> 1, s = k & 1, chunk = it - begin;
      const uint32_t* bins = ms.bins[a][s];
      const int cnt = (int)bins[chunk], whole = (int)bins[chunk + 1];
      if (cnt == 0) continue;
      const int j = chunk * kMarchChunk + (lane & 15);
      const double f0 = mf.first[a][s];
      const double F = f0 + (double)j;
      const float Ff = (float)F;
      const bool b1 = a == 0, cy = a == 2;  // the other two axes: b = b1 ? y : x, c = cy ? y : z
      const double feb = b1 ? mf.fe[1] : mf.fe[0], fec = cy ? mf.fe[1] : mf.fe[2];
      const MarchWindow w = march_window(march_reference(mr, ms, a, s), F, feb, fec);
      const int first = a * mr.count + (s ? (int)ms.bins[a][0][0] : 0);
      const float2* rel = mr.rel + first;
      const uint32_t* take = mr.take + first;
      uint32_t mask = 0u, z = 4u;
      // `whole` rays have all 16 planes; both words' top 12 bits are 0x410 + cell, and
      // 6 * 0x410 + 0x410 = 16 (mod 32)
#pragma unroll 4
      for (int i = half; i < whole; i += 2) {
        const float2 e = rel[i];
        const uint32_t ub = __float_as_uint(fmaf(e.x, Ff, w.cb));
        const uint32_t uc = __float_as_uint(fmaf(e.y, Ff, w.cc));
        mask |= 1u << (((ub >> 20) * 6u + (uc >> 20)) & 31u);
        z = min(z, min(ub & 0xFFFFCu, uc & 0xFFFFCu));
      }
#pragma unroll 4
      for (int i = whole + half; i < cnt; i += 2) {
        const float2 e = rel[i];
        const uint32_t ub = __float_as_uint(fmaf(e.x, Ff, w.cb));
        const uint32_t uc = __float_as_uint(fmaf(e.y, Ff, w.cc));
        const bool act = j < (int)(take[i] & 0xFFFFu);
        const uint32_t bit = 1u << (((ub >> 20) * 6u + (uc >> 20)) & 31u);
        const uint32_t edge = min(ub & 0xFFFFCu, uc & 0xFFFFCu);
        mask |= act ? bit : 0u;
        z = min(z, act ? edge : 4u);
      }
      __syncwarp();
      if (min(z, __shfl_xor_sync(kFull, z, 16)) == 0u) {  // the plane again, by both halves
        mask = 0u;
        unsigned long long edges = 0ull;  // up to 8 rays (list positions) close to a cell's edge
        int n_edges = 0;
#pragma unroll 2
        for (int i = half; i < cnt; i += 2) {
          const float2 e = rel[i];
          const uint32_t ub = __float_as_uint(fmaf(e.x, Ff, w.cb));
          const uint32_t uc = __float_as_uint(fmaf(e.y, Ff, w.cc));
          const bool act = j < (int)(take[i] & 0xFFFFu);
          const bool edge = !(ub & 0xFFFFCu) || !(uc & 0xFFFFCu);
          const uint32_t bit = 1u << (((ub >> 20) * 6u + (uc >> 20)) & 31u);
          mask |= act && !edge ? bit : 0u;
          if (act && edge) {
            if (n_edges < 8) {
              edges = (edges << 8) | (unsigned)i;
              ++n_edges;
            } else {
              const int r = (int)(take[i] >> 16);
              atomicOr(&ms.undecided[r >> 5], 1u << (r & 31));
              ms.dda = 1u;
            }
          }
        }
#pragma unroll 1
        for (; n_edges > 0; --n_edges, edges >>= 8) {
          const int i = (int)((unsigned)edges & 255u), r = (int)(take[i] >> 16);
          const float2 e = rel[i];
          // the nearest row and column edge, and the side of it that the ray passes on: the sign
          // of d_b F - (edge - eye_b) |d_a|
          const float vb = fmaf(e.x, Ff, w.cb), vc = fmaf(e.y, Ff, w.cc);
          const int eb = __float2int_rn(vb) - 8 + w.b0, ec = __float2int_rn(vc) - 8 + w.c0;
          const double da = fabs((double)mr.d[a * mr.count + r]);
          const double db = (double)mr.d[(b1 ? 1 : 0) * mr.count + r];
          const double dc = (double)mr.d[(cy ? 1 : 2) * mr.count + r];
          const double xb = fma(db, F, ((feb - kMagic) - (double)eb) * da);
          const double xc = fma(dc, F, ((fec - kMagic) - (double)ec) * da);
          const double room = 1e-8 * da;
          if (fabs(xb) < room || fabs(xc) < room) {
            atomicOr(&ms.undecided[r >> 5], 1u << (r & 31));
            ms.dda = 1u;
          } else {
            // away from its nearest edge a coordinate's float position decides as before
            const int cb = (__float_as_uint(vb) & 0xFFFFCu) ? (int)(__float_as_uint(vb) >> 20) - 0x410
                                                            : eb - w.b0 - (xb < 0.0 ? 1 : 0);
            const int cc = (__float_as_uint(vc) & 0xFFFFCu) ? (int)(__float_as_uint(vc) >> 20) - 0x410
                                                            : ec - w.c0 - (xc < 0.0 ? 1 : 0);
            mask |= 1u << ((cb * 6 + cc + 16) & 31);
          }
        }
      }
      __syncwarp();
      // a first plane close to the eye was marked by the set-up
      if (j == 0 && mf.near[a][s]) mask = 0u;
      mask |= __shfl_xor_sync(kFull, mask, 16);
      mask = (mask << 16) | (mask >> 16);
      march_write(a, tt, m, mask, s ? mf.v[a] + 1 + j : mf.v[a] - 1 - j,
                  (b1 ? mf.v[1] : mf.v[0]) + w.b0, (cy ? mf.v[1] : mf.v[2]) + w.c0, epoch, plane);
    } else {
      // 8 lanes a ray, or one
      const bool by8 = it < chunks + wide;
      const int e = by8 ? (it - chunks) * 4 + (lane >> 3) : (it - chunks - wide) * 32 + lane;
      if (e < (by8 ? many : few)) {
        const uint32_t entry = mr.rest[by8 ? e : 3 * mr.count - 1 - e];
        const int a = (int)(entry & 3u), r = (int)((entry >> 2) & 0x3FFFu);
        const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
        const uint32_t nn = mr.n[a * mr.count + r];
        const int s = (int)(nn >> 15), n = (int)(nn & 0x7FFFu);
        const double inv = 1.0 / fabs((double)mr.d[a * mr.count + r]);
        const double mb = (double)mr.d[b * mr.count + r] * inv;
        const double mc = (double)mr.d[c * mr.count + r] * inv;
        const double f0 = mf.first[a][s];
        // a first plane close to the eye was marked by the set-up
        const int first = max((int)(entry >> 16), mf.near[a][s] ? 1 : 0);
        if (march_outside(tt, m, a, s, mb, mc, f0, mf.fe[b], mf.fe[c], mf.v[a], mf.v[b], mf.v[c],
                          by8 ? first + (lane & 7) : first, by8 ? 8 : 1, n, epoch, plane)) {
          atomicOr(&ms.undecided[r >> 5], 1u << (r & 31));
          ms.dda = 1u;
        }
      }
      __syncwarp();
    }
  }
}

// Adds a thread's counts to the map's counters (one update per warp).
__device__ __forceinline__ void add_ray_counts(const MapView& m, uint32_t visits, uint32_t rays) {
  unsigned long long vv = visits, rr = rays;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vv += __shfl_xor_sync(kFull, vv, o);
    rr += __shfl_xor_sync(kFull, rr, o);
  }
  if ((threadIdx.x & 31) == 0 && (vv | rr)) {
    atomicAdd(&m.ctr->visits, vv);
    atomicAdd(&m.ctr->rays, rr);
  }
}

// Range bucket of a pixel for the tile's ray order: 0 = longest rays, kSortBuckets - 1 =
// shortest and rays without a return.
// `qs` = kSortBuckets / max_range (metres): the bucket is the range's fraction of max range.
__device__ __forceinline__ int range_bucket(float r_m, float qs) {
  if (!(r_m > 0.0f)) return kSortBuckets - 1;
  const float q = r_m * qs;
  const int k = q < (float)kSortBuckets ? (int)q : kSortBuckets - 1;
  return kSortBuckets - 1 - k;
}

// Units that the tiles of an order bucket are handed out in: whole, or in quarters.
template <int MaxF>
__device__ __forceinline__ uint32_t unit_count(const TickWork<MaxF>& work, int bucket) {
  return bucket < work.split_bucket ? 4u : 1u;
}

template <int RM, int MaxF, bool Render = false>
__device__ __forceinline__ void traverse_body(const TickWork<MaxF>& work, const MapView& m,
                                              const SimRender* sr = nullptr) {
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t smask = work.smask;
  const int nent = (int)smask + 1;
  uint32_t* s_words = reinterpret_cast<uint32_t*>(smem);
  uint32_t* s_tags = s_words + nent * kLabelWords;
  uint32_t* s_used = s_tags + nent;
  // then the walk's ray order and points, or the march's rays
  const int nrays = work.tile_w * work.tile_h;
  uint16_t* s_order = reinterpret_cast<uint16_t*>(s_used + nent);
  uint8_t* s_bkt = reinterpret_cast<uint8_t*>(s_order + nrays);
  // the tile's sensor-frame points, computed once by the range sort; x = NaN for a pixel
  // without a point
  float* s_pts = reinterpret_cast<float*>(s_bkt + nrays);
  MarchRays mr = march_rays(s_used + nent, min(nrays / 4, kMarchRays));
  __shared__ MarchShared s_march;
  __shared__ MarchFrame s_mf;
  __shared__ uint32_t s_n_used;
  const MarchFrame& mf = s_mf;
  __shared__ FrameParams s_f;
  __shared__ uint32_t s_tile;
  __shared__ int s_frame;
  __shared__ int s_sub;
  __shared__ uint32_t s_hist[kSortBuckets];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int nthreads = blockDim.x;
  uint32_t visits = 0, rays = 0;
  for (int i = tid; i < nent; i += nthreads) s_tags[i] = kNoLeaf;
  for (int i = tid; i < nent * kLabelWords; i += nthreads) s_words[i] = 0u;
  if (tid == 0) s_n_used = 0u;
  if (!Render && work.split_bucket > 0) march_reset(s_march);
  wait_prior_grid();
  // claim order: the first tiles of the queue are those of bucket 0 (longest walks), ...
  __shared__ uint32_t s_pre[kOrderBuckets + 1];
  if (work.order_counts) {
    if (tid < 32) {
      const uint32_t c0 = __ldcg(&work.order_counts[2 * lane]) * unit_count(work, 2 * lane);
      const uint32_t c1 = __ldcg(&work.order_counts[2 * lane + 1]) * unit_count(work, 2 * lane + 1);
      uint32_t incl = c0 + c1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += u;
      }
      s_pre[2 * lane] = incl - c0 - c1;
      s_pre[2 * lane + 1] = incl - c1;
      if (lane == 31) s_pre[kOrderBuckets] = incl;
    }
    __syncthreads();
  }

  for (;;) {
    if (tid == 0) {
      unsigned int* queue = &m.ctr->tile_queue;
      const uint32_t t = atomicAdd(queue, 1u);
      const uint32_t units = work.order_counts ? s_pre[kOrderBuckets] : work.total_tiles;
      uint32_t tl = t < units ? t : work.total_tiles;
      s_sub = -1;
      if (work.order_counts && t < units) {
        int lo = 0, hi = kOrderBuckets - 1;  // the bucket b with s_pre[b] <= t < s_pre[b + 1]
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (s_pre[mid] <= t) lo = mid; else hi = mid - 1;
        }
        const uint32_t o = t - s_pre[lo], n = unit_count(work, lo);
        tl = __ldcg(&work.order_lists[(size_t)lo * work.order_cap + o / n]);
        if (n > 1) s_sub = (int)(o % n);
      }
      int fi = 0;
      while (fi + 1 < work.n_frames && work.tile_start[fi + 1] <= tl) ++fi;
      s_tile = tl;
      s_frame = fi;
      if (t == units + gridDim.x - 1) {  // last reader resets
        *queue = 0u;
        // every CTA read the counts before its first claim: clear them for the next pass
        if (work.order_counts)
          for (int b = 0; b < kOrderBuckets; ++b) work.order_counts[b] = 0u;
      }
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= work.total_tiles) {
      allow_dependent_launch();  // the integration may start its CTAs on freed SMs
      break;
    }
    const int fi = s_frame;
    {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&work.fr[fi]);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&s_f);
      for (int i = tid; i < (int)(sizeof(FrameParams) / 4); i += nthreads) dst[i] = src[i];
    }
    if (tid < kSortBuckets) s_hist[tid] = 0u;
    if (tid == 0) s_march.dda = s_sub < 0;  // the walk may leave leaves without a label
    __syncthreads();
    const FrameParams& f = s_f;
    const uint32_t lt = tile - work.tile_start[fi];
    const int tx = (int)(lt % (uint32_t)work.tiles_x[fi]);
    const int ty = (int)(lt / (uint32_t)work.tiles_x[fi]);
    // the unit: the tile, or a quarter of it
    const int sub = s_sub;
    const int tw = sub < 0 ? work.tile_w : work.tile_w >> 1, th = sub < 0 ? work.tile_h : work.tile_h >> 1;
    const int x0 = tx * work.tile_w + (sub > 0 ? (sub & 1) * tw : 0);
    const int y0 = ty * work.tile_h + (sub > 0 ? (sub >> 1) * th : 0);
    // packed records (input kind 2) fill the first tiles only: later tiles have no work
    if (f.input_kind == 2 && (uint32_t)(y0 * f.width + x0) >= __ldg(f.n_valid)) {
      __syncthreads();
      continue;
    }
    TileTable tt;
    tt.tags = s_tags;
    tt.words = s_words;
    tt.used = s_used;
    tt.n_used = &s_n_used;
    tt.smask = smask;
    tt.sh = __clz((int)smask);
    tt.elx = (int)floor(f.eye[0]) >> 3;
    tt.ely = (int)floor(f.eye[1]) >> 3;
    tt.elz = (int)floor(f.eye[2]) >> 3;
    if (Render || sub < 0) {
      // the tile's ranges (Render: from the sim map, with the range noise), bucketed by length;
      // every thread runs the same number of iterations (nrays is a multiple of the block)
      const float qs = (float)kSortBuckets / (f.max_time * (float)f.res_d);
      const bool spread = f.type == NM_SENSOR_LASER;
      for (int k = tid; k < nrays; k += nthreads) {
        const int px = x0 + k % work.tile_w, py = y0 + k / work.tile_w;
        float rm = 0.0f;  // range in metres, 0 = no point
        float p[3] = {__int_as_float(0x7fffffff), 0.0f, 0.0f};
        if (px < f.width && py < f.height) {
          bool ok;
          if constexpr (Render) {
            float rr = sim_ray(sr->v, sr->rp, px, py);
            const long long i = (long long)py * f.width + px;
            if (sr->noise) rr = noisy(rr, sr->seed, i, sr->sigma_coef, sr->drop);
            if (sr->out) sr->out[i] = rr;
            rm = rr;
            ok = range_point_r(f, px, py, rr, p);
          } else if (f.input_kind == 1) {
            rm = __ldg(&f.ranges[(size_t)py * f.width + px]);
            ok = range_point_r(f, px, py, rm, p);
          } else {
            ok = pixel_point(f, px, py, p);
            if (ok) rm = sqrtf(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
          }
          if (!ok) p[0] = __int_as_float(0x7fffffff);
        }
        s_pts[3 * k] = p[0];
        s_pts[3 * k + 1] = p[1];
        s_pts[3 * k + 2] = p[2];
        const int b = range_bucket(rm, qs);
        s_bkt[k] = (uint8_t)b;
        const unsigned peers = __match_any_sync(kFull, b);
        if (lane == __ffs(peers) - 1) atomicAdd(&s_hist[b], (uint32_t)__popc(peers));
      }
      march_frame(f, s_mf);
      __syncthreads();
      if (tid < 32) {  // exclusive prefix over the buckets
        const uint32_t v = s_hist[lane];
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t u = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += u;
        }
        s_hist[lane] = incl - v;
      }
      __syncthreads();
      for (int k = tid; k < nrays; k += nthreads) {
        const int b = s_bkt[k];
        const unsigned peers = __match_any_sync(kFull, b);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&s_hist[b], (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        const int q = base + __popc(peers & ((1u << lane) - 1u));  // rank, longest first
        // one ray per thread: thread t walks the ray at s_order[t], so warp w gets ranks
        // 32w..32w+31 (rays of about one length per warp: best for camera frames); for a laser
        // frame ranks w, w + W, w + 2W, ... (W warps: every warp gets rays of all lengths; a
        // spinning sensor's tile mixes ground hits with far walls and its few tiles leave SMs
        // idle, so spreading the long rays over the warps wins: 0.32 against 0.46 ms for a
        // 64x1024 frame at 20 m)
        const int nw = nthreads >> 5;
        s_order[(spread && nrays == nthreads) ? (q % nw) * 32 + q / nw : q] = (uint16_t)k;
      }
      __syncthreads();

      const int plane = f.plane;
      const uint32_t epoch = f.epoch;
      const double max_time = (double)f.max_time;
      for (int j = 0; j < nrays / nthreads; ++j) {
        // alternate directions so every warp gets long and short rays
        const int pos = (j & 1) ? (j + 1) * nthreads - 1 - tid : j * nthreads + tid;
        const int k = s_order[pos];
        const float p[3] = {s_pts[3 * k], s_pts[3 * k + 1], s_pts[3 * k + 2]};
        Ray r;
        if (!isnan(p[0]) && setup_ray<RM>(f, p, r)) {
          using A = Ar<RM>;
          const float* R = f.R;
          float d[3];
#pragma unroll
          for (int a = 0; a < 3; ++a)
            d[a] = A::fadd(A::fadd(A::fmul(R[3 * a], p[0]), A::fmul(R[3 * a + 1], p[1])),
                           A::fmul(R[3 * a + 2], p[2]));
          const int c = march_count(mf, d);
          rays += 1;
          visits += c >= 0 ? walk_counted<RM>(r, c, tt, m, max_time, epoch, plane)
                           : walk_ray<RM>(r, tt, m, max_time, epoch, plane);
        }
      }
      __syncthreads();
    } else if constexpr (!Render) {
      march_frame(f, s_mf);
      __syncthreads();
      const int nray = min(tw * th, kMarchRays);  // rays of one round
      const int rounds = tw * th / nray;
      mr.count = nray;

      // a warp's 32 rays are a patch of 8 x 4 pixels where the tile is made of such patches
      const bool patches = (tw & 7) == 0 && (th & 3) == 0;
      for (int j = 0; j < rounds; ++j) {
        auto pixel = [&](int r, int& kx, int& ky) {
          if (patches) {
            const int q = j * (nray >> 5) + (r >> 5), pw = tw >> 3;
            kx = (q % pw) * 8 + (r & 7);
            ky = (q / pw) * 4 + ((r >> 3) & 3);
          } else {
            const int k = j * nray + r;
            kx = k % tw;
            ky = k / tw;
          }
        };
        float d[3];
        int n[3];
        if (tid < nray) {
          int kx, ky;
          pixel(tid, kx, ky);
          float p[3];
          const int px = x0 + kx, py = y0 + ky;
          const bool ok = px < f.width && py < f.height && pixel_point(f, px, py, p);
          const int ex = 2 * kx - tw, ey = 2 * ky - th;
          march_setup<RM>(f, mf, tt, m, mr, s_march, ok, p, tid, ex * ex + ey * ey, d, n, visits,
                          rays);
        }
        __syncthreads();
        march_list(mr, s_march, d, n);
        __syncthreads();
        march_planes(mf, tt, m, mr, s_march, f.epoch, f.plane);
        __syncthreads();
        // rays too close to a tie somewhere: the DDA labels all of their voxels (those marked
        // already are among them)
        if (s_march.dda && tid < nray) {
          const bool fresh = (s_march.walk[tid >> 5] >> lane) & 1u;
          if (fresh || ((s_march.undecided[tid >> 5] >> lane) & 1u)) {
            int kx, ky;
            pixel(tid, kx, ky);
            float p[3];
            Ray r;
            if (pixel_point(f, x0 + kx, y0 + ky, p) && setup_ray<RM>(f, p, r)) {
              const uint32_t c = walk_ray<RM>(r, tt, m, (double)f.max_time, f.epoch, f.plane);
              if (fresh) {
                visits += c;
                rays += 1u;
              }
            }
          }
        }
        __syncthreads();
        march_reset(s_march);
        if (j + 1 < rounds) __syncthreads();
      }
    }

    // Flush the tile's leaf table.  First one lane per leaf, so the device-table lookups of many
    // leaves overlap; the slot takes the place of the leaf's tag.  (Only the DDA enters leaves
    // that it may leave without a label: those are not inserted.)
    const int n_used = (int)s_n_used;
    for (int u = tid; u < n_used; u += nthreads) {
      const uint32_t e = s_used[u];
      bool has = s_march.dda == 0u;
      if (!has) {
        const uint32_t* sw = s_words + e * kLabelWords;
#pragma unroll 4
        for (int w = 0; w < kLabelWords; ++w) has |= sw[(w + lane) & (kLabelWords - 1)] != 0u;
      }
      int g = -1;
      if (has) {
        g = map_find_or_insert(m, tt.key(s_tags[e]));
        if (g >= 0) mark_touched(m, g, f.epoch, f.plane);
      }
      s_tags[e] = (uint32_t)g;
    }
    __syncthreads();
    // Then one warp per leaf, a lane per label word: whole 128-byte lines of atomics.  The entry is
    // left empty for the next tile.
    for (int u = tid >> 5; u < n_used; u += nthreads >> 5) {
      const uint32_t e = s_used[u];
      const int g = (int)s_tags[e];
      const uint32_t word = s_words[e * kLabelWords + lane];
      if (word) {
        s_words[e * kLabelWords + lane] = 0u;
        if (g >= 0) atomicOr(&m.labels[((size_t)f.plane * m.capacity + (size_t)g) * kLabelWords + lane], word);
      }
      __syncwarp();
      if (lane == 0) s_tags[e] = kNoLeaf;
    }
    if (tid == 0) s_n_used = 0u;
    __syncthreads();
  }

  add_ray_counts(m, visits, rays);
}

// ---- tile order (longest walks first) --------------------------------------------------------
//
// A frame's walk is bounded by its longest rays: a step costs a warp ~70 instructions issued
// at one per ~11 cycles while the SM's other warps run, so a 350-step ray takes most of a
// frame's traversal.  Claiming the tiles in decreasing order of their longest ray starts those
// rays first.  One CTA per tile takes the largest |R p|_1 / res over the tile's rays (the
// DDA's step count up to rounding) plus kSetupSteps, scales it to one of kOrderBuckets
// buckets, and appends the tile to that bucket's list (order inside a bucket is arbitrary).
constexpr float kSetupSteps = 8.0f;

// Tiles whose longest ray takes more steps than this go to the plane march, in quarters: a fixed
// share, and a share for the tiles that each resident CTA handles (592 CTAs: 148 SMs x 4).  The
// walk is the cheaper way to label a tile of short rays while enough tiles keep the SMs busy;
// what the march removes is the wait for the last long rays, which a frame of few tiles feels
// sooner.  Traversal times (us) by this limit, one frame each: 64x1024 spinning sensor at 20 m
// (256 tiles) 47 / 48 / 60 / 113 at 96 / 128 / 192 / never; 640x480 camera at 10 m (1200 tiles)
// 86 / 82 / 86 / 95, the same voxel-filtered (about 100 tiles with points) 58 / 62 / 72 / 75; 1280x720 at
// 0.02 m and 15 m (3600 tiles) 523 / 493 / 427 / 1143 (at 256: 411); the 16-frame tick (20 K tiles)
// 983 / 920 / 811 / 784.
constexpr float kSplitSteps = 64.0f;
constexpr float kSplitStepsPerTile = 32.0f / 592.0f;
constexpr int kOrderThreads = 128;

template <int MaxF>
__device__ __forceinline__ void tile_order_body(const TickWork<MaxF>& work, TileOrderBuffers b) {
  allow_dependent_launch();  // the walk's CTAs launch now and wait for this pass to finish
  // one CTA per tile, one thread per ray: every record load of the tile is in flight at once
  const uint32_t tile = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31;
  const int nrays = work.tile_w * work.tile_h;
  // the tile's frame, every start read at once: one after the other they were most of a CTA's time
  // (16-frame tick, 20 K tiles: 38.7 -> 30 us)
  static_assert(MaxF <= 32, "a lane per frame");
  const int fi = MaxF == 1 ? 0
                           : __popc(__ballot_sync(kFull, lane > 0 && lane < work.n_frames &&
                                                             work.tile_start[lane < MaxF ? lane : 0] <= tile));
  const FrameParams& f = work.fr[fi];
  const uint32_t lt = tile - work.tile_start[fi];
  const int x0 = (int)(lt % (uint32_t)work.tiles_x[fi]) * work.tile_w;
  const int y0 = (int)(lt / (uint32_t)work.tiles_x[fi]) * work.tile_h;
  const float inv_res = (float)(1.0 / f.res_d);
  float longest = 0.0f;
  for (int k = tid; k < nrays; k += kOrderThreads) {
    const int px = x0 + k % work.tile_w, py = y0 + k / work.tile_w;
    float p[3];
    if (px < f.width && py < f.height && pixel_point(f, px, py, p)) {
      const float* R = f.R;
      const float x = R[0] * p[0] + R[1] * p[1] + R[2] * p[2];
      const float y = R[3] * p[0] + R[4] * p[1] + R[5] * p[2];
      const float z = R[6] * p[0] + R[7] * p[1] + R[8] * p[2];
      const float len = sqrtf(x * x + y * y + z * z) * inv_res;
      if (len < f.max_time)
        longest = fmaxf(longest, (fabsf(x) + fabsf(y) + fabsf(z)) * inv_res + kSetupSteps);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) longest = fmaxf(longest, __shfl_xor_sync(kFull, longest, o));
  __shared__ float s_max[kOrderThreads / 32];
  if (lane == 0) s_max[tid >> 5] = longest;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < kOrderThreads / 32; ++w) longest = fmaxf(longest, s_max[w]);
    const float q = longest * work.order_scale;
    const int bkt = kOrderBuckets - 1 - (q < (float)(kOrderBuckets - 1) ? (int)q : kOrderBuckets - 1);
    const uint32_t r = atomicAdd(&b.counts[bkt], 1u);
    if (r < b.capacity) b.lists[(size_t)bkt * b.capacity + r] = tile;
  }
}

template <int MaxF>
__global__ void __launch_bounds__(kOrderThreads) k_tile_order(const __grid_constant__ TickWork<MaxF> work,
                                                              TileOrderBuffers b) {
  tile_order_body<MaxF>(work, b);
}

__global__ void __launch_bounds__(kOrderThreads) k_tile_order_dev(const TickWork<kMaxTickFrames>* work,
                                                                  TileOrderBuffers b) {
  tile_order_body<kMaxTickFrames>(*work, b);
}

// Label sink of the wide-frame kernel: device-table lookups on leaf changes, one atomic per
// new label bit.
struct WideEmit {
  const MapView* m;
  uint32_t epoch;
  int plane;
  unsigned long long ckey;
  int cslot;

  __device__ __forceinline__ void operator()(int x, int y, int z, int kind) {
    const unsigned long long key = leaf_key(x >> 3, y >> 3, z >> 3);
    if (key != ckey) {
      ckey = key;
      cslot = map_find_or_insert(*m, key);
      if (cslot >= 0) mark_touched(*m, cslot, epoch, plane);
    }
    if (cslot < 0) return;
    const int l = local_index(x, y, z);
    uint32_t* wp = &m->labels[((size_t)plane * m->capacity + (size_t)cslot) * kLabelWords +
                              (kind == kKindHit ? 0 : 16) + (l >> 5)];
    const uint32_t bit = 1u << (l & 31);
    if (!(__ldcg(wp) & bit)) atomicOr(wp, bit);
  }
};

// Frames whose reach is beyond the leaf code's range: one thread per ray over the work's
// tiles (grid-stride), the same DDA and labels without the shared leaf table.
template <int RM, int MaxF>
__device__ __forceinline__ void traverse_wide_body(const TickWork<MaxF>& work, const MapView& m) {
  const int nrays = work.tile_w * work.tile_h;
  uint32_t visits = 0, rays = 0;
  for (uint32_t tile = blockIdx.x; tile < work.total_tiles; tile += gridDim.x) {
    int fi = 0;
    while (fi + 1 < work.n_frames && work.tile_start[fi + 1] <= tile) ++fi;
    const FrameParams& f = work.fr[fi];
    const uint32_t lt = tile - work.tile_start[fi];
    const int x0 = (int)(lt % (uint32_t)work.tiles_x[fi]) * work.tile_w;
    const int y0 = (int)(lt / (uint32_t)work.tiles_x[fi]) * work.tile_h;
    for (int k = threadIdx.x; k < nrays; k += blockDim.x) {
      const int px = x0 + k % work.tile_w, py = y0 + k / work.tile_w;
      float p[3];
      if (px < f.width && py < f.height && pixel_point(f, px, py, p)) {
        WideEmit em{&m, f.epoch, f.plane, kEmptyKey, -1};
        const int n = trace_point<RM>(f, p[0], p[1], p[2], em);
        if (n >= 0) {
          visits += (uint32_t)n;
          rays += 1;
        }
      }
    }
  }
  unsigned long long vv = visits, rr = rays;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vv += __shfl_xor_sync(kFull, vv, o);
    rr += __shfl_xor_sync(kFull, rr, o);
  }
  if ((threadIdx.x & 31) == 0 && (vv | rr)) {
    atomicAdd(&m.ctr->visits, vv);
    atomicAdd(&m.ctr->rays, rr);
  }
}

// ---- accumulate mode: exact per-voxel hit and miss counts -------------------------------------

// Adds one to a counter, one atomic per group of lanes that hit the same one at the same time.
__device__ __forceinline__ void add_one(const MapView& m, unsigned long long idx) {
  const unsigned act = __activemask();
  const unsigned peers = __match_any_sync(act, idx);
  if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&m.counts[idx], (unsigned)__popc(peers));
}

// Count sink of the table-free walk (accumulate mode).
struct CountEmit {
  const MapView* m;
  uint32_t epoch;
  unsigned long long ckey;
  int cslot;

  __device__ __forceinline__ void operator()(int x, int y, int z, int kind) {
    const unsigned long long key = leaf_key(x >> 3, y >> 3, z >> 3);
    if (key != ckey) {
      ckey = key;
      cslot = map_find_or_insert(*m, key);
      if (cslot >= 0) mark_touched(*m, cslot, epoch, 0);
    }
    if (cslot < 0) return;
    const int l = local_index(x, y, z);
    const unsigned long long idx =
        (unsigned long long)cslot * 1024ull + (kind == kKindHit ? 0u : 512u) + (unsigned)l;
    add_one(*m, idx);
  }
};

// Table-free: a thread per ray of 16 x 16 pixels (8 x 4 a warp), a look-up per leaf change and an atomic per
// group of lanes that are in the same voxel.  For reaches past the leaf codes', and for large images: with
// thousands of CTAs what counts is their throughput, and a table's clearing and copying out, with 4 CTAs a
// SM for it, costs more than it saves.  us a frame, table / table-free: 640x480 at 10 m and 0.05 m (2400 tiles
// of 16 x 8) 127 / 143, 848x480 at 8 m and 0.04 m (3180) 165 / 168, 1280x720 at 6 m and 0.1 m (7200) 174 / 110,
// at 15 m and 0.02 m 787 / 663, 1920x1080 at 5 m and 0.05 m (16200) 579 / 338.
template <int RM>
__global__ void __launch_bounds__(256) k_traverse_count_free(const __grid_constant__ FrameParams f,
                                                             MapView m, int tiles_x) {
  const int tid = threadIdx.x, tile = blockIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int px = (tile % tiles_x) * 16 + (warp & 1) * 8 + (lane & 7);
  const int py = (tile / tiles_x) * 16 + (warp >> 1) * 4 + (lane >> 3);
  uint32_t visits = 0, rays = 0;
  float p[3];
  if (px < f.width && py < f.height && pixel_point(f, px, py, p)) {
    CountEmit em{&m, f.epoch, kEmptyKey, -1};
    const int n = trace_point<RM>(f, p[0], p[1], p[2], em);
    if (n >= 0) {
      visits = (uint32_t)n;
      rays = 1;
    }
  }
  add_ray_counts(m, visits, rays);
}

// A CTA takes 16 x 8 pixels, and its rays' misses are counted in shared memory: a table of leaves by
// code (relative to the eye's leaf), with a byte per voxel, which 128 rays that each visit a voxel
// at most once cannot overflow.  A leaf's voxels then go to the device counters in one coalesced
// pass, and a leaf is looked up there once per CTA.  317x239 pixels at 5 m and 0.05 m 42 us a frame (600 CTAs,
// 592 resident at once; the longest rays bound it), with match, device atomic and probe in every step 80.
// A CTA whose rays fan out over more leaves than pay for the table (count_extent) does it that way.
constexpr int kCountLeaves = 104;                      // 4 CTAs a SM
constexpr int kCountLeafWords = kLeafVoxels / 4;       // voxel l: byte l >> 7 of word l & 127, so
                                                       // neighbours lie in different words
constexpr size_t kCountBytes = (size_t)kCountLeaves * kCountLeafWords * 4;

// A leaf that the walk has entered and not looked up.  (No entry, slot or lost leaf has this number.)
constexpr int kNoEntry = INT_MIN + 1;

// Buckets of four tags, read with one load: a leaf is at its home place or, where others hold that, at the
// first place that was free in the rest of its bucket and then in the next two.  So the look-up of a leaf
// that finds no room ends after three loads; with up to 24 single ones 320x240 pixels at 5 m and 0.01 m
// (500 voxels of reach) took 930 us, 570 now and 606 without a table.
constexpr uint32_t kCountBuckets = kCountLeaves / 4, kCountNear = 3;

__device__ __forceinline__ uint4 count_bucket(const uint32_t* tags, uint32_t b) {
  uint4 t;
  asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(t.x), "=r"(t.y), "=r"(t.z), "=r"(t.w)
               : "r"((uint32_t)__cvta_generic_to_shared(tags + 4 * b)));
  return t;
}

// Place of `code` in a bucket, -1 where it is not.
__device__ __forceinline__ int count_place(const uint4& t, uint32_t code) {
  return t.x == code ? 0 : (t.y == code ? 1 : (t.z == code ? 2 : (t.w == code ? 3 : -1)));
}

// Entry of a leaf in which something is counted, or, where its buckets are full, -(g + 1) for slot g of the
// device table (kLostWord: no room there either).
__device__ __noinline__ int count_leaf_slow(uint32_t* tags, const MapView& m, unsigned long long key,
                                            uint32_t code, uint32_t home, uint32_t epoch) {
  auto bucket = [&](uint32_t q) {
    const uint32_t b = (home >> 2) + q;
    return b < kCountBuckets ? b : b - kCountBuckets;
  };
  for (uint32_t i = 0; i < 4u * kCountNear; ++i) {
    if (i == 2u) {  // both first places are others': the rest at once
      bool room = false;
#pragma unroll
      for (uint32_t q = 0; q < kCountNear; ++q) {
        const uint4 t = count_bucket(tags, bucket(q));
        const int at = count_place(t, code);
        if (at >= 0) return (int)(4u * bucket(q)) + at;
        room |= count_place(t, kNoLeaf) >= 0;
      }
      if (!room) break;
    }
    const uint32_t e = 4u * bucket(i >> 2) + ((i < 4u ? home + i : i) & 3u);
    uint32_t k = ((volatile uint32_t*)tags)[e];
    if (k == kNoLeaf) {
      k = atomicCAS(&tags[e], kNoLeaf, code);
      if (k == kNoLeaf) return (int)e;
    }
    if (k == code) return (int)e;
  }
  const int g = map_find_or_insert(m, key);
  if (g < 0) return kLostWord;
  mark_touched(m, g, epoch, 0);
  return -(g + 1);
}

struct CountExtent {
  uint32_t lo[4][3], hi[4][3];  // per warp and axis: least and greatest component of a unit direction
  uint32_t len[4], n[4];        // sum of the lengths (leaves), rays
};

// Leaves that a CTA's rays fan out over, estimated from their mean length L (in leaves) and the two
// widest spreads a, b of their directions: the integral of (1 + a t)(1 + b t) over [0, L].
__device__ __forceinline__ float count_extent(const FrameParams& f, bool ok, const float p[3],
                                              CountExtent& ext) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float len = sqrtf(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
#pragma unroll
  for (int a = 0; a < 3; ++a) {  // components moved to [1, 3]: floats in the order of their bits
    const uint32_t u = __float_as_uint(2.0f + fminf(fmaxf(__fdividef(p[a], len), -1.0f), 1.0f));
    const uint32_t lo = __reduce_min_sync(kFull, ok ? u : 0xFFFFFFFFu);
    const uint32_t hi = __reduce_max_sync(kFull, ok ? u : 0u);
    if (lane == 0) ext.lo[warp][a] = lo;
    if (lane == 0) ext.hi[warp][a] = hi;
  }
  const float leaves = __fdividef(len, (float)f.res_d * 8.0f);
  const uint32_t sum = __reduce_add_sync(kFull, ok ? (uint32_t)(fminf(leaves, 4096.0f) * 16.0f) : 0u);
  const unsigned have = __ballot_sync(kFull, ok);
  if (lane == 0) ext.len[warp] = sum;
  if (lane == 0) ext.n[warp] = __popc(have);
  __syncthreads();
  float s[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    uint32_t lo = ext.lo[0][a], hi = ext.hi[0][a];
#pragma unroll
    for (int w = 1; w < 4; ++w) lo = min(lo, ext.lo[w][a]), hi = max(hi, ext.hi[w][a]);
    s[a] = __uint_as_float(hi) - __uint_as_float(lo);
  }
  const float L = __fdividef((float)(ext.len[0] + ext.len[1] + ext.len[2] + ext.len[3]) * (1.0f / 16.0f),
                             (float)(ext.n[0] + ext.n[1] + ext.n[2] + ext.n[3]));
  const float least = fminf(fminf(s[0], s[1]), s[2]);
  const float both = s[0] + s[1] + s[2] - least;  // a + b
  const float a = fmaxf(fmaxf(s[0], s[1]), s[2]), b = both - a;
  return L * (1.0f + L * (0.5f * both + L * a * b * (1.0f / 3.0f)));
}

// The limits of count_extent.  Beyond about the table's size the leaves without room cost what the others
// gain: 160x120 pixels at 4 m and 0.02 m 191 us at 48, 134 at 96 and above; 200x150 at 2.5 m and 0.005 m (500
// voxels of reach) 661 at 96, 719 without a limit; 40x30 at 10 m and 0.02 m 494 / 568.  Records packed by the
// voxel filter come from several patches, and their box is far wider than the leaves they visit, the more
// so the shorter they are: 317x239 at 5 m and 0.05 m (100 voxels) 93 us at 96, 69 at 192, 55 at 400 and above;
// 1024 pixels in a row at 12 m and 0.05 m (240) 158 at 400, 114 at 1000; a 64x1024 spinning sensor at 20 m and
// 0.05 m (400) 189 / 170.  Far rays differ: 320x240 at 5 m and 0.01 m (500) 617 at 192, 672 at 400, 719 at 1000,
// 1280x720 at 15 m and 0.02 m (750) 494 / 526 / 547, 40x30 at 10 m and 0.02 m (500) 382 / 424 / 473.  Large images
// of short reach: 1280x720 at 6 m and 0.03 m 183 at 400, 205 at 1000; 1920x1080 at 5 m and 0.05 m 67 at 192 and above.
constexpr float kCountFan = 96.0f, kCountFanPacked = 1000.0f, kCountFanLarge = 400.0f, kCountFanFar = 192.0f;
constexpr float kCountFar = 420.0f;      // voxels of reach
constexpr int64_t kCountTiles = 4096;    // a large image has more tiles of 16 x 8

template <int RM>
__global__ void __launch_bounds__(128) k_traverse_count(const __grid_constant__ FrameParams f,
                                                        MapView m, int tiles_x, float fan) {
  extern __shared__ uint4 s_raw[];
  uint32_t* s_counts = (uint32_t*)s_raw;
  __shared__ __align__(16) uint32_t s_tags[kCountLeaves];
  __shared__ int s_slot[kCountLeaves];
  __shared__ CountExtent s_ext;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tile = blockIdx.x;
  // a warp's rays: a patch of 8 x 4 pixels
  const int px = (tile % tiles_x) * 16 + (warp & 1) * 8 + (lane & 7);
  const int py = (tile / tiles_x) * 8 + (warp >> 1) * 4 + (lane >> 3);
  float p[3] = {0.0f, 0.0f, 0.0f};
  Ray r;
  const bool ok = px < f.width && py < f.height && pixel_point(f, px, py, p) && setup_ray<RM>(f, p, r);
  if (!__syncthreads_or(ok)) return;
  uint32_t visits = 0, rays = 0;
  if (count_extent(f, ok, p, s_ext) > fan) {
    if (ok) {
      CountEmit em{&m, f.epoch, kEmptyKey, -1};
      visits = (uint32_t)trace_point<RM>(f, p[0], p[1], p[2], em);
      rays = 1;
    }
    add_ray_counts(m, visits, rays);
    return;
  }
  for (int i = tid; i < (int)(kCountBytes / 16); i += 128) s_raw[i] = make_uint4(0, 0, 0, 0);
  if (tid < kCountLeaves) s_tags[tid] = kNoLeaf;
  __syncthreads();
  TileTable tt;
  tt.elx = (int)floor(f.eye[0]) >> 3;
  tt.ely = (int)floor(f.eye[1]) >> 3;
  tt.elz = (int)floor(f.eye[2]) >> 3;
  int end_leaf = kLostWord, end_l = 0;
  if (ok) {
    double t0 = r.t0, t1 = r.t1, t2 = r.t2;
    int l = r.l;
    uint32_t code = r.code;
    auto find = [&]() -> int {
      const uint32_t home = __umulhi(code * 0x9E3779B1u, (uint32_t)kCountLeaves);
      if (((volatile uint32_t*)s_tags)[home] == code) return (int)home;
      const uint32_t second = (home & ~3u) + ((home + 1u) & 3u);
      if (((volatile uint32_t*)s_tags)[second] == code) return (int)second;
      return count_leaf_slow(s_tags, m, tt.key(code), code, home, f.epoch);
    };
    int leaf = kNoEntry;  // not looked up yet: only leaves with a label go into the map
    double t;
    for (;;) {
      t = fmin(fmin(t0, t1), t2);
      if (!(t <= r.len)) break;
      if (leaf == kNoEntry) leaf = find();
      ++visits;
      if (leaf >= 0)
        atomicAdd(&s_counts[leaf * kCountLeafWords + (l & 127)], 1u << ((l >> 7) * 8));
      else if (leaf != kLostWord)
        add_one(m, (unsigned long long)(-leaf - 1) * 1024ull + 512u + (unsigned)l);
      int msk, ds;
      dda_step<RM>(t0, t1, t2, r.d0, r.d1, r.d2, r.ds0, r.ds1, r.ds2, msk, ds);
      const int vv = (l & msk) + ds;
      l = (l & ~msk) | (vv & msk);
      if ((unsigned)vv > (unsigned)msk) {
        code += msk == 0x1C0 ? r.hs0 : (msk == 0x38 ? r.hs1 : r.hs2);
        leaf = kNoEntry;
      }
    }
    if (t < (double)f.max_time) {
      end_leaf = leaf == kNoEntry ? find() : leaf;
      end_l = l;
      ++visits;
    }
    rays = 1;
  }
  __syncthreads();
  for (int e = tid; e < kCountLeaves; e += 128) {
    int g = -1;
    if (s_tags[e] != kNoLeaf) {
      g = map_find_or_insert(m, tt.key(s_tags[e]));
      if (g >= 0) mark_touched(m, g, f.epoch, 0);
    }
    s_slot[e] = g;
  }
  __syncthreads();
  if (end_leaf != kLostWord) {
    const int g = end_leaf >= 0 ? s_slot[end_leaf] : -end_leaf - 1;
    if (g >= 0) add_one(m, (unsigned long long)g * 1024ull + (unsigned)end_l);
  }
  for (int e = warp; e < kCountLeaves; e += 4) {
    const int g = s_slot[e];
    if (g < 0) continue;
    unsigned* out = m.counts + (size_t)g * 1024 + 512;
#pragma unroll
    for (int w = 0; w < kCountLeafWords; w += 32) {
      const uint32_t v = s_counts[e * kCountLeafWords + w + lane];
      if (v) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const uint32_t n = (v >> (8 * b)) & 0xFFu;
          if (n) atomicAdd(&out[b * 128 + w + lane], n);
        }
      }
    }
  }
  add_ray_counts(m, visits, rays);
}

// Work list passed by value (single insert, one-shot tick).  MinB resident CTAs per SM: at 4 the
// kernel has 64 registers and spills some of the march's; at 3 it has 80 and spills none.
template <int RM, int MaxF, int MinB>
__global__ void __launch_bounds__(256, MinB) k_traverse(const __grid_constant__ TickWork<MaxF> work,
                                                  MapView m) {
  traverse_body<RM, MaxF>(work, m);
}

// One simulated frame rendered tile by tile inside the traversal (sim render + noise + insert).
template <int RM>
__global__ void __launch_bounds__(256, 4) k_traverse_render(const __grid_constant__ TickWork<1> work,
                                                         MapView m,
                                                         const __grid_constant__ SimRender sr) {
  traverse_body<RM, 1, true>(work, m, &sr);
}

// Work list read from device memory (tick plans replayed as CUDA graphs).
template <int RM>
__global__ void __launch_bounds__(256, 4) k_traverse_dev(const TickWork<kMaxTickFrames>* work,
                                                      MapView m) {
  traverse_body<RM, kMaxTickFrames>(*work, m);
}

template <int RM, int MaxF>
__global__ void __launch_bounds__(256) k_traverse_wide(const __grid_constant__ TickWork<MaxF> work,
                                                       MapView m) {
  traverse_wide_body<RM, MaxF>(work, m);
}

template <int RM>
__global__ void __launch_bounds__(256) k_traverse_wide_dev(const TickWork<kMaxTickFrames>* work,
                                                           MapView m) {
  traverse_wide_body<RM, kMaxTickFrames>(*work, m);
}

// Resident CTAs of a traversal kernel for a block size and dynamic shared memory, queried
// once per (kernel, shape) ahead of any stream capture.
struct GridCache {
  const void* fn = nullptr;
  size_t smem = 0;
  int block = 0;
  int blocks = 0;
};

int g_sm_count = 0;
constexpr int kGridCacheSize = 64;
GridCache g_grid_cache[kGridCacheSize];
int g_grid_next = 0;
std::mutex g_grid_mutex;

cudaError_t resident_grid(const void* fn, size_t smem, int block, int* grid) {
  std::lock_guard<std::mutex> lock(g_grid_mutex);
  for (GridCache& c : g_grid_cache)
    if (c.fn == fn && c.smem == smem && c.block == block) {
      *grid = g_sm_count * c.blocks;
      return cudaSuccess;
    }
  cudaError_t e = cudaSuccess;
  if (g_sm_count == 0) {
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
  }
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
  int blocks = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, block, smem);
  if (e != cudaSuccess) return e;
  if (blocks < 1) blocks = 1;
  GridCache& c = g_grid_cache[g_grid_next];
  g_grid_next = (g_grid_next + 1) % kGridCacheSize;
  c.fn = fn;
  c.smem = smem;
  c.block = block;
  c.blocks = blocks;
  *grid = g_sm_count * blocks;
  return cudaSuccess;
}

bool work_is_wide(const FrameParams* fr, int n) {
  for (int i = 0; i < n; ++i)
    if (!(fr[i].max_time < kNarrowMaxTime)) return true;
  return false;
}

}  // namespace

size_t traverse_smem_bytes(int tile_w, int tile_h, uint32_t smask) {
  const size_t nent = (size_t)smask + 1;
  const size_t nrays = (size_t)tile_w * tile_h;
  const size_t march = march_bytes((int)std::min<size_t>(kMarchRays, nrays / 4));
  return nent * (kLabelWords * 4 + 4 + 4) + std::max<size_t>(nrays * (2 + 1 + 12), march);
}

template <int MaxF>
cudaError_t launch_traverse_labels(const TickWork<MaxF>& w, const MapView& m, int rounding,
                                   cudaStream_t s, bool dependent) {
  const int block = min(kMarchThreads, w.tile_w * w.tile_h);
  const bool down = rounding == NM_ROUND_DOWN;
  int grid = 0;
  if (work_is_wide(w.fr, w.n_frames)) {
    const void* fn = down ? (const void*)k_traverse_wide<NM_ROUND_DOWN, MaxF>
                          : (const void*)k_traverse_wide<NM_ROUND_NEAREST, MaxF>;
    cudaError_t e = resident_grid(fn, 0, block, &grid);
    if (e != cudaSuccess) return e;
    grid = min(grid, (int)w.total_tiles);
    if (down)
      k_traverse_wide<NM_ROUND_DOWN, MaxF><<<grid, block, 0, s>>>(w, m);
    else
      k_traverse_wide<NM_ROUND_NEAREST, MaxF><<<grid, block, 0, s>>>(w, m);
    return cudaGetLastError();
  }
  const size_t smem = traverse_smem_bytes(w.tile_w, w.tile_h, w.smask);
  // Frames that do not fill 3 CTAs per SM gain more from the registers than from a fourth CTA:
  // 320x240 at 0.1 m (300 tiles) 21.5 against 24.2 us, 64x1024 spinning sensor at 20 m (256) 47.4
  // against 51.9, and voxel-filtered 640x480 frames (about 100 tiles of packed points, their
  // number known on the device only) 57.9 against 59.8; 640x480 (1200) 84.8 against 82.3,
  // 1280x720 at 0.02 m (3600) 435 against 412.
  const bool roomy = MaxF == 1 && (w.total_tiles <= 3u * 148u || w.fr[0].input_kind == 2);
  using Kernel = void (*)(TickWork<MaxF>, MapView);
  constexpr int kFew = MaxF == 1 ? 3 : 4;
  const Kernel kernel = roomy ? (down ? (Kernel)k_traverse<NM_ROUND_DOWN, MaxF, kFew>
                                      : (Kernel)k_traverse<NM_ROUND_NEAREST, MaxF, kFew>)
                              : (down ? (Kernel)k_traverse<NM_ROUND_DOWN, MaxF, 4>
                                      : (Kernel)k_traverse<NM_ROUND_NEAREST, MaxF, 4>);
  const void* fn = (const void*)kernel;
  cudaError_t e = resident_grid(fn, smem, block, &grid);
  if (e != cudaSuccess) return e;
  grid = (int)min((long long)grid, (long long)w.total_tiles * (w.split_bucket > 0 ? 4 : 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kernel, w, m);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t launch_traverse_counts(const FrameParams& f, const MapView& m, int rounding,
                                   cudaStream_t s) {
  const bool down = rounding == NM_ROUND_DOWN, packed = f.input_kind == 2;
  const int tiles_x = (f.width + 15) / 16, tiles_y = (f.height + 7) / 8;
  const bool large = (int64_t)tiles_x * tiles_y > kCountTiles;
  if (!(f.max_time < kNarrowMaxTime) || (large && !packed)) {
    auto kernel = down ? k_traverse_count_free<NM_ROUND_DOWN> : k_traverse_count_free<NM_ROUND_NEAREST>;
    kernel<<<tiles_x * ((f.height + 15) / 16), 256, 0, s>>>(f, m, tiles_x);
    return cudaGetLastError();
  }
  const float fan = !packed                  ? kCountFan
                    : f.max_time > kCountFar ? kCountFanFar
                    : large                  ? kCountFanLarge
                                             : kCountFanPacked;
  auto kernel = down ? k_traverse_count<NM_ROUND_DOWN> : k_traverse_count<NM_ROUND_NEAREST>;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCountBytes);
  if (e != cudaSuccess) return e;
  kernel<<<tiles_x * tiles_y, 128, kCountBytes, s>>>(f, m, tiles_x, fan);
  return cudaGetLastError();
}

bool traverse_render_fits(const FrameParams& f) { return f.max_time < kNarrowMaxTime; }

cudaError_t launch_traverse_render(const TickWork<1>& w, const MapView& m, const SimRender& sr,
                                   int rounding, cudaStream_t s) {
  if (!traverse_render_fits(w.fr[0])) return cudaErrorInvalidValue;
  const int block = min(kMarchThreads, w.tile_w * w.tile_h);
  const size_t smem = traverse_smem_bytes(w.tile_w, w.tile_h, w.smask);
  const bool down = rounding == NM_ROUND_DOWN;
  const void* fn = down ? (const void*)k_traverse_render<NM_ROUND_DOWN>
                        : (const void*)k_traverse_render<NM_ROUND_NEAREST>;
  int grid = 0;
  cudaError_t e = resident_grid(fn, smem, block, &grid);
  if (e != cudaSuccess) return e;
  grid = min(grid, (int)w.total_tiles);
  if (down)
    k_traverse_render<NM_ROUND_DOWN><<<grid, block, smem, s>>>(w, m, sr);
  else
    k_traverse_render<NM_ROUND_NEAREST><<<grid, block, smem, s>>>(w, m, sr);
  return cudaGetLastError();
}

namespace {
const void* dev_kernel(int rounding, bool wide) {
  if (wide)
    return rounding == NM_ROUND_DOWN ? (const void*)k_traverse_wide_dev<NM_ROUND_DOWN>
                                     : (const void*)k_traverse_wide_dev<NM_ROUND_NEAREST>;
  return rounding == NM_ROUND_DOWN ? (const void*)k_traverse_dev<NM_ROUND_DOWN>
                                   : (const void*)k_traverse_dev<NM_ROUND_NEAREST>;
}
}  // namespace

cudaError_t prepare_traverse_dev(int tile_w, int tile_h, uint32_t smask, int rounding, bool wide) {
  const int block = min(kMarchThreads, tile_w * tile_h);
  const size_t smem = wide ? 0 : traverse_smem_bytes(tile_w, tile_h, smask);
  int grid = 0;
  return resident_grid(dev_kernel(rounding, wide), smem, block, &grid);
}

cudaError_t launch_traverse_labels_dev(const TickWork<kMaxTickFrames>* d_work, uint32_t total_tiles,
                                       int tile_w, int tile_h, uint32_t smask, const MapView& m,
                                       int rounding, bool wide, cudaStream_t s) {
  const int block = min(kMarchThreads, tile_w * tile_h);
  const size_t smem = wide ? 0 : traverse_smem_bytes(tile_w, tile_h, smask);
  int grid = 0;
  const cudaError_t e = resident_grid(dev_kernel(rounding, wide), smem, block, &grid);
  if (e != cudaSuccess) return e;
  grid = (int)min((long long)grid, (long long)total_tiles * 4);
  const bool down = rounding == NM_ROUND_DOWN;
  if (wide) {
    if (down)
      k_traverse_wide_dev<NM_ROUND_DOWN><<<grid, block, 0, s>>>(d_work, m);
    else
      k_traverse_wide_dev<NM_ROUND_NEAREST><<<grid, block, 0, s>>>(d_work, m);
  } else {
    if (down)
      k_traverse_dev<NM_ROUND_DOWN><<<grid, block, smem, s>>>(d_work, m);
    else
      k_traverse_dev<NM_ROUND_NEAREST><<<grid, block, smem, s>>>(d_work, m);
  }
  return cudaGetLastError();
}

cudaError_t tile_order_reserve(TileOrderBuffers* b, uint32_t tiles, cudaStream_t s) {
  if (tiles <= b->capacity && b->counts) return cudaSuccess;
  // growth frees the old buffers (a device synchronisation): start at 16 K tiles (a 1280x720
  // frame has 7200 tiles of 16x8) and double
  const uint32_t cap = std::max<uint32_t>(tiles, std::max<uint32_t>(1u << 14, 2u * b->capacity));
  tile_order_release(b);
  cudaError_t e = cudaMalloc((void**)&b->counts, kOrderBuckets * 4);
  if (e == cudaSuccess) e = cudaMalloc((void**)&b->lists, (size_t)kOrderBuckets * cap * 4);
  if (e == cudaSuccess) e = cudaMemsetAsync(b->counts, 0, kOrderBuckets * 4, s);
  if (e != cudaSuccess) {
    tile_order_release(b);
    return e;
  }
  b->capacity = cap;
  b->pending = false;
  return cudaSuccess;
}

void tile_order_release(TileOrderBuffers* b) {
  cudaFree(b->counts);
  cudaFree(b->lists);
  *b = TileOrderBuffers{};
}

template <int MaxF>
float tile_order_scale(const TickWork<MaxF>& w) {
  float longest = 0.0f;
  for (int i = 0; i < w.n_frames; ++i) longest = std::max(longest, w.fr[i].max_time);
  return (float)kOrderBuckets / (longest * 1.7320508f + kSetupSteps);
}

template <int MaxF>
int tile_split_bucket(const TickWork<MaxF>& w) {
  // quarters of whole 8 x 4 patches, and of whole rounds
  const int quarter = w.tile_w * w.tile_h / 4;
  if ((w.tile_w & 15) != 0 || (w.tile_h & 7) != 0 || (quarter > kMarchRays && quarter % kMarchRays != 0))
    return 0;
  // (of a filtered frame's tiles only the first few hold points, how many the device knows)
  const float tiles = w.fr[0].input_kind == 2 ? 0.0f : (float)w.total_tiles;
  const float steps = std::max(96.0f, kSplitSteps + kSplitStepsPerTile * tiles);
  const float q = steps * w.order_scale;
  return q < (float)kOrderBuckets ? kOrderBuckets - (int)q : 0;
}

namespace {
cudaError_t clear_pending_counts(TileOrderBuffers* b, cudaStream_t s) {
  if (!b->pending) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(b->counts, 0, kOrderBuckets * 4, s);
  if (e == cudaSuccess) b->pending = false;
  return e;
}
}  // namespace

template <int MaxF>
cudaError_t launch_tile_order(const TickWork<MaxF>& w, TileOrderBuffers* b, cudaStream_t s) {
  if (w.total_tiles == 0) return cudaSuccess;
  if (w.total_tiles > b->capacity) return cudaErrorInvalidValue;
  cudaError_t e = clear_pending_counts(b, s);
  if (e != cudaSuccess) return e;
  k_tile_order<MaxF><<<(int)w.total_tiles, kOrderThreads, 0, s>>>(w, *b);
  e = cudaGetLastError();
  if (e == cudaSuccess) b->pending = true;
  return e;
}

cudaError_t launch_tile_order_dev(const TickWork<kMaxTickFrames>* d_work, uint32_t total_tiles,
                                  TileOrderBuffers* b, cudaStream_t s) {
  if (total_tiles == 0) return cudaSuccess;
  if (total_tiles > b->capacity) return cudaErrorInvalidValue;
  cudaError_t e = clear_pending_counts(b, s);
  if (e != cudaSuccess) return e;
  k_tile_order_dev<<<(int)total_tiles, kOrderThreads, 0, s>>>(d_work, *b);
  e = cudaGetLastError();
  if (e == cudaSuccess) b->pending = true;
  return e;
}

template int tile_split_bucket<1>(const TickWork<1>&);
template int tile_split_bucket<kMaxTickFrames>(const TickWork<kMaxTickFrames>&);
template float tile_order_scale<1>(const TickWork<1>&);
template float tile_order_scale<kMaxTickFrames>(const TickWork<kMaxTickFrames>&);
template cudaError_t launch_tile_order<1>(const TickWork<1>&, TileOrderBuffers*, cudaStream_t);
template cudaError_t launch_tile_order<kMaxTickFrames>(const TickWork<kMaxTickFrames>&,
                                                       TileOrderBuffers*, cudaStream_t);
template cudaError_t launch_traverse_labels<1>(const TickWork<1>&, const MapView&, int, cudaStream_t,
                                               bool);
template cudaError_t launch_traverse_labels<kMaxTickFrames>(const TickWork<kMaxTickFrames>&,
                                                            const MapView&, int, cudaStream_t, bool);

}  // namespace nm
