// Device side of the direct spherical Biot-Savart sum.
//
// One interaction (target x_i, source x_k with circulation G_k = zeta_k A_k):
//     w_ik = G_k / (1 - x_i.x_k + delta^2)
//     u_i  = -1/(4 pi) * x_i  x  sum_k w_ik (x_k - x_i)
// which equals the reference's sum_k (x_i x x_k) w_ik (BVEActiveRHS,
// PanelVelocityParallel.f90:1316-1333) because x_i x x_i = 0; the cross
// product is taken once per target instead of once per pair.
//
// Work decomposition: blockIdx.x = a tile of TB consecutive targets (one of
// up to three target classes), blockIdx.y = a chunk of consecutive sources.
// Each CTA streams its source chunk through shared memory in tiles of TS and
// writes one FP64 partial sum per target and chunk; the stage epilogue adds
// the chunks in a fixed order, so results are deterministic.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "bounds.cuh"

namespace tcb {

constexpr int kNoSelf = INT32_MIN;

// Start of a kernel launched by launch_chained: everything before it in the stream is
// done when this returns, and the next chained kernel may be set up meanwhile. The kernel's
// lifetime overlaps its predecessor's, so its parameters carry no __restrict__ on what a
// predecessor may write: that would promise that nothing else writes it while the kernel
// runs, and allow loads that do not see it. Functions called after this may have it.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct TargetSeg {
  const double* x;  // targets, x[3*i + c]
  const int* perm;  // target at position p in [i0,i1) is perm[p] (null: p itself)
  int i0, i1;       // target range [i0, i1) computed by this launch
  int out_offset;   // partial row of target i is out_offset + i
  int self_offset;  // source index of target i is i + self_offset (ACTIVE), else kNoSelf
  double d2;        // delta^2 for this class
  int compact;      // FP64: are tiles of these targets worth a look for a frame
  int tile_begin;   // first blockIdx.x of this segment
  long long x_len;     // checked build: points in x
  long long perm_len;  // checked build: entries in perm
};

struct PairLaunch {
  TargetSeg seg[3];
  int nseg;
  const double4* src;   // packed sources {x, y, z, G}
  int n;                // number of sources
  int chunk_len;        // sources per blockIdx.y chunk (multiple of the tile; FP64 SHORT
                        // shapes: of 16)
  double* partial;      // partial[(chunk*3 + c)*n_out + row]
  int n_out;
  bool care;            // FP64: a segment with frames has d2 < kCareD
  BoundsRec* bc;        // checked build: violation record (null: release build)
  long long src_len;    // checked build: packed sources in src
  long long partial_len;  // checked build: doubles in partial
};

// Extents a work unit checks its global indices against (checked build).
struct UnitBounds {
  BoundsRec* rec;
  long long x_len, perm_len, src_len;
  long long out_base;  // offset of the unit's out pointer within the partial sums
  long long out_len;   // doubles in the partial sums
};

// ---------------------------------------------------------------------------
// Reciprocals. The hardware seed (rcp.approx.ftz.f64, relative error e0 below
// 1e-6) takes one third-order step, r <- r (1 + e + e^2) with e = 1 - d r: the
// error left is e0^3 < 1e-18, so 3 FMA give a result within an ulp of 1/d
// (measured over [1, 2): 1.1e-16). Two Newton steps would take 4, the
// compiler's IEEE division about 14.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rcp_seed_f64(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  return r;
}

__device__ __forceinline__ double rcp_refine_f64(double d, double r) {
  double e = fma(-d, r, 1.0);
  e = fma(e, e, e);
  return fma(r, e, r);
}

__device__ __forceinline__ double rcp_f64(double d) { return rcp_refine_f64(d, rcp_seed_f64(d)); }

__device__ __forceinline__ float rcp_approx_f32(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}

__device__ __forceinline__ const TargetSeg& find_seg(const PairLaunch& P, int tile) {
  int s = 0;
  if (P.nseg > 1 && tile >= P.seg[1].tile_begin) s = 1;
  if (P.nseg > 2 && tile >= P.seg[2].tile_begin) s = 2;
  return P.seg[s];
}

// ---------------------------------------------------------------------------
// Frames. A CTA with compact targets works in its own frame: an origin c on the
// sphere near the middle of its targets and an orthonormal basis R = (e1, e2, e3)
// with e3 along c. Points become offsets s = R (x - c).
// ---------------------------------------------------------------------------
// Orthonormal basis with e3 = c/|c| (Duff, Burgess, Christensen, Hart, Kensler,
// Liani, Pharr, "Building an Orthonormal Basis, Revisited", JCGT 6(1), 2017).
__device__ __forceinline__ void make_frame(double cx, double cy, double cz, double* f) {
  const double inv = rsqrt(fma(cx, cx, fma(cy, cy, cz * cz)));
  const double nx = cx * inv, ny = cy * inv, nz = cz * inv;
  const double sg = copysign(1.0, nz);
  const double a = -1.0 / (sg + nz);
  const double b = nx * ny * a;
  f[0] = 1.0 + sg * nx * nx * a;
  f[1] = sg * b;
  f[2] = -sg * nx;
  f[3] = b;
  f[4] = sg + ny * ny * a;
  f[5] = -ny;
  f[6] = nx;
  f[7] = ny;
  f[8] = nz;
}

// R v with explicitly fused operations, so a target and the same point as a
// source round identically.
__device__ __forceinline__ double frame_dot(const double* e, double vx, double vy, double vz) {
  return fma(e[0], vx, fma(e[1], vy, __dmul_rn(e[2], vz)));
}

// ---------------------------------------------------------------------------
// FP64 pair kernel.
//
// The kernel is bound by the FP64 pipe, and there by the pair's operation
// count and its register reads (a DFMA of three registers none of which the
// instruction before it read takes 3.1 cycles a warp and scheduler, of two 2.1).
// Two forms, chosen per CTA by how compact its targets are:
//
// * frame form (9 operations a pair), targets within kFrameRho of c: with
//   x_k = c + s_k and x_i = c + t_i,
//       1 + delta^2 - x_i.x_k = a_k (1 - b_i) + b_i' - s_k,1 t_i,1 - s_k,2 t_i,2,
//       a_k = -c.s_k,  b_i = -c.t_i,  b_i' = b_i + delta^2 + (1 - |c|^2)
//   holds for every x on or off the sphere (e3 is along c, so the third products
//   of s.t are a_k b_i), and takes 3 FMA because the targets' part sits in
//   registers. The sum is T' = sum_k r G_k R x_k: staging a source multiplies
//   G_k in once per CTA, so a pair takes 3 FMA here, 3 there and 3 for the
//   reciprocal. The multiple of x_i that T' carries (about sum r G, which
//   u = x_i x T ignores) is taken out in the frame, where x_i is (small, small,
//   about 1), before T' is rotated back. The denominator keeps an absolute error
//   of ulps of |s| |t| where 1 - x.y keeps ulps of 1.
//   A target on a source, or within rounding of one, has a denominator of rounding
//   where delta is 0, r about 1e16, and r G R x_k would leave a rounding as large as G
//   although the pair's velocity is 0. So where a class has delta^2 below kCareD, pairs
//   with a denominator below kCareD are left out of the sums and added as
//   r G (R x_k - R x_i), which is 0 for equal points: their offsets are equal bit for
//   bit. Only source tiles with a source as near to c as the targets can hold such a
//   pair. Those track their largest reciprocal, one integer instruction a pair, and
//   are summed again, with comparisons, if it is that large. This is a kernel of its own
//   (CARE), so that other launches stay as they are. Its source loop is unrolled by 4,
//   by 2 the level-5 Voronoi step takes 0.585 ms instead of 0.561. Without and with it, all
//   classes with delta 0: level-5 Voronoi step 0.559 and 0.561 ms, level-5 vertex sum
//   241.8 and 243.5 us, ten level-4 steps 2.01 and 2.10 ms.
// * wide form (13 operations), for targets all over the sphere: the fused
//   1 - x.y + delta^2 of the global coordinates and sum_k w (x_k - x_i).
//   STRICT variants always take it, with the denominator rounded like the
//   reference's 1.0 - sum(...) + smooth*smooth (six separately rounded
//   operations).
//
// Either way the sums of at most a tile's 256 sources are added to totals in shared
// memory: in one long chain the sums' rounding would outweigh the terms'. The frame
// form's error grows with |t|, by which its largest sum, about sum r G along c, enters
// u. Restated on the CPU with the same fused operations (level-5 panels and vertices, two
// fields, delta 0 and 0.01, 12 frames), its rms error against 80-bit sums is this many
// times that of the plain sum_k w (x_k - x_i): 0.3-0.9 at |t| 0.2, 0.8-1.0 at 0.4, 1.3-3
// at 0.6, 2-6 at 0.85, where it is at most 8e-15 of the largest velocity. The limit is
// where tiles of 1/16 of the sphere's targets still pass; most tiles have |t| of 0.1 to
// 0.5, and whole runs are as far from 64-bit ones as with the plain sum (ten level-4
// steps 2.6e-14 both, level-5 vertex sum 3.5e-14 and 3.8e-14, level 6 2.3e-14 both).
//
// Level 6 refined, 108,923 sources and 199,823 targets in three classes: 1.115e12
// pairs/s with the wide form alone, at 14 operations, and now 1.53e12. 9 DFMA at
// their nominal 2 cycles would allow 18.5e12 / 9 = 2.05e12; the register reads of a
// loop that shares a source among the targets make that 2.3 to 2.5 cycles. Level 8
// reaches 1.60e12.
// ---------------------------------------------------------------------------
constexpr float kFrameRho2 = 0.72f;  // frame form: |t|^2 at most (|t| <= 0.85)
// A tile of 1/16 of the sphere's targets has a radius of 0.5 to 0.8, within that limit;
// classes of fewer tiles are not worth the search for a frame (level 3, 1,280 panels:
// 21.6 us a sum with it, 19.6 without).
constexpr int kCompactTiles = 16;
constexpr int kOwnTiles = 2048;     // bits of the own-tile map
// r at most 1e6, and the rounding of r G R x_k at most 1e-10 G
constexpr double kCareD = 1.0 / (1 << 20);

constexpr int kCareHi = 0x3eb00000;  // high word of kCareD
// high word from which a reciprocal's seed (relative error below 1e-6) may be that of a
// denominator below kCareD: 1/kCareD's, less 2^-19 of it
constexpr unsigned kMostHi = 0x41300000 - 4;

__device__ __forceinline__ bool tiny_denominator(double D) {
  return (__double2hiint(D) & 0x7fffffff) < kCareHi;  // |D| < kCareD
}

template <int NT, int TPT, int TS>
struct Fp64Smem {
  double2 a[TS];              // frame: (s_1, s_2); wide: (x, y)
  double2 b[TS];              // frame: (a_k, G x'_1); wide: (z, G)
  double2 c[TS];              // frame: (G x'_2, G x'_3)
  double acc[3 * TPT * NT];   // totals [c][t][thread]
  double frame[13];           // e1, e2, e3 (rows), c, 1 - |c|^2
  double csum[4][NT / 32];    // per-warp sums of the target positions, and their number
  unsigned own[kOwnTiles / 32];  // source tiles (mod kOwnTiles) that hold own points
  unsigned rho[NT / 32];      // largest |t|^2, per warp
  int framed;                 // a frame was found
};

// 1 - |c|^2 for |c| close to 1, without the rounding of |c|^2 to a double.
__device__ __forceinline__ double one_minus_norm2(double cx, double cy, double cz) {
  const double p[3] = {__dmul_rn(cx, cx), __dmul_rn(cy, cy), __dmul_rn(cz, cz)};
  const double e[3] = {fma(cx, cx, -p[0]), fma(cy, cy, -p[1]), fma(cz, cz, -p[2])};
  double hi = 1.0, lo = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {  // hi + lo = 1 - sum p (TwoSum)
    const double s = __dsub_rn(hi, p[k]);
    const double bb = __dsub_rn(s, hi);
    lo = __dadd_rn(lo, __dadd_rn(__dsub_rn(hi, __dsub_rn(s, bb)), __dsub_rn(-p[k], bb)));
    hi = s;
  }
  return __dadd_rn(hi, __dsub_rn(lo, __dadd_rn(e[0], __dadd_rn(e[1], e[2]))));
}

// The wide form's denominator. STRICT: rounded exactly like the reference's
// 1.0 - sum(...) + smooth*smooth.
template <bool STRICT>
__device__ __forceinline__ double wide_denominator(double qx, double qy, double qz, const double* xi,
                                                   double d2, double one_plus_d2) {
  if (!STRICT) return fma(-qz, xi[2], fma(-qy, xi[1], fma(-qx, xi[0], one_plus_d2)));
  double s = __dmul_rn(qx, xi[0]);
  s = __dadd_rn(s, __dmul_rn(qy, xi[1]));
  s = __dadd_rn(s, __dmul_rn(qz, xi[2]));
  return __dadd_rn(__dsub_rn(1.0, s), d2);
}

// Source j of the staged tile (index k) against the thread's targets. HOW: kSelf skips
// the self pair, needed only in tiles that may hold the CTA's own points; in the frame form
// kTiny skips pairs with a tiny denominator and kMost takes down the high word of the
// largest reciprocal of the others (a negative one counts as larger than any).
enum { kSelf = 1, kTiny = 2, kMost = 4 };
template <int HOW>
struct How {
  static constexpr int value = HOW;
};

template <int TPT, bool FRAME, bool STRICT, int HOW, class Smem>
__device__ __forceinline__ void fp64_source(const Smem& sm, int j, int k, const double (*tg)[4],
                                            const int* self_k, double d2, double one_plus_d2,
                                            double (*f)[3], unsigned& most) {
  const double2 a = sm.a[j], b = sm.b[j];
  double2 c = make_double2(0.0, 0.0);
  if (FRAME) c = sm.c[j];
#pragma unroll
  for (int t = 0; t < TPT; ++t) {
    if (FRAME) {
      double D = fma(b.x, tg[t][2], tg[t][3]);
      D = fma(a.x, tg[t][0], D);
      D = fma(a.y, tg[t][1], D);
      // the seed's low word is 0, and from a seed of 0 the reciprocal comes out as 0
      const bool skip = ((HOW & kSelf) && k == self_k[t]) || ((HOW & kTiny) && tiny_denominator(D));
      double r = rcp_seed_f64(D);
      if (HOW & (kSelf | kTiny)) r = __hiloint2double(skip ? 0 : __double2hiint(r), 0);
      if (HOW & kMost) most = max(most, (unsigned)__double2hiint(r));
      r = rcp_refine_f64(D, r);
      f[t][0] = fma(r, b.y, f[t][0]);
      f[t][1] = fma(r, c.x, f[t][1]);
      f[t][2] = fma(r, c.y, f[t][2]);
    } else {
      const double D = wide_denominator<STRICT>(a.x, a.y, b.x, tg[t], d2, one_plus_d2);
      double w = __dmul_rn(b.y, rcp_f64(D));
      if (HOW & kSelf) w = (k == self_k[t]) ? 0.0 : w;
      f[t][0] = fma(w, a.x - tg[t][0], f[t][0]);
      f[t][1] = fma(w, a.y - tg[t][1], f[t][1]);
      f[t][2] = fma(w, b.x - tg[t][2], f[t][2]);
    }
  }
}

// The pairs that kTiny left out of the tile at ts (sources up to end): as differences
// in the frame. Points with equal offsets are one point, whose denominator is taken as
// the wide form has it: the pair is 0, or NaN where 1 - x.x + delta^2 rounds to 0.
template <int TPT, class Smem>
__device__ __forceinline__ void fp64_tiny_pairs(const Smem& sm, const double4* src, int ts, int end,
                                                const double (*tg)[4], const int* self_k,
                                                double one_plus_d2, double (*f)[3],
                                                const UnitBounds& ub) {
#pragma unroll 1
  for (int j = 0; j < end - ts; ++j) {
    const double2 a = sm.a[j];
    const double ak = sm.b[j].x;
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
      double D = fma(ak, tg[t][2], tg[t][3]);
      D = fma(a.x, tg[t][0], D);
      D = fma(a.y, tg[t][1], D);
      if (!tiny_denominator(D) || ts + j == self_k[t]) continue;
      if (!TC_BC(ub.rec, BC_PAIR_SRC, ts + j, ub.src_len)) continue;
      const double4 q = src[ts + j];
      const double x[3] = {q.x, q.y, q.z};
      const double d[3] = {a.x + tg[t][0], a.y + tg[t][1], (1.0 - ak) - tg[t][2]};
      if (d[0] == 0.0 && d[1] == 0.0 && d[2] == 0.0)
        D = wide_denominator<false>(q.x, q.y, q.z, x, 0.0, one_plus_d2);
      const double w = __dmul_rn(q.w, rcp_f64(D));
#pragma unroll
      for (int c = 0; c < 3; ++c) f[t][c] = fma(w, d[c], f[t][c]);
    }
  }
}

// Sources [c0, c1) against the thread's targets, totals in sm.acc. SHORT: the last
// tile is staged and walked to its end only (a chunk need not be whole tiles);
// otherwise it is padded, and the loop's length is known when it is compiled. CARE
// (frame form): source tiles with |s|^2 <= near2 are looked through for tiny
// denominators, and count as own tiles.
template <int NT, int TPT, int TS, int UNROLL, bool SHORT, bool FRAME, bool CARE, bool STRICT,
          class Smem>
__device__ __forceinline__ void fp64_sum(const double4* __restrict__ src, int c0, int c1, Smem& sm,
                                         const double (*tg)[4], const int* self_k, bool idle,
                                         double d2, double near2, const UnitBounds& ub) {
  const double one_plus_d2 = 1.0 + d2;
  double f[TPT][3];
#pragma unroll
  for (int t = 0; t < TPT; ++t) f[t][0] = f[t][1] = f[t][2] = 0.0;
  for (int ts = c0; ts < c1; ts += TS) {
    __syncthreads();
    const int len = SHORT ? min(TS, (c1 - ts + UNROLL - 1) / UNROLL * UNROLL) : TS;
    const int tile = (ts - c0) / TS % kOwnTiles;
    unsigned most = 0;
    bool near = false;
    for (int j = threadIdx.x; j < len; j += NT) {
      const int k = ts + j;
      // padding: zero weight and (frame) a denominator of at least 1 off the targets
      double4 q = make_double4(0.0, 0.0, 0.0, 0.0);
      const bool in = k < c1 && TC_BC(ub.rec, BC_PAIR_SRC, k, ub.src_len);
      if (in) q = src[k];
      if (FRAME) {
        const double* fr = sm.frame;
        const double dx = q.x - fr[9], dy = q.y - fr[10], dz = q.z - fr[11];
        const double s1 = frame_dot(fr, dx, dy, dz), s2 = frame_dot(fr + 3, dx, dy, dz),
                     ak = -frame_dot(fr + 9, dx, dy, dz);
        sm.a[j] = in ? make_double2(s1, s2) : make_double2(0.0, 0.0);
        sm.b[j] = in ? make_double2(ak, __dmul_rn(q.w, s1)) : make_double2(1.0, 0.0);
        sm.c[j] = in ? make_double2(__dmul_rn(q.w, s2), fma(-q.w, ak, q.w)) : make_double2(0.0, 0.0);
        if (CARE) near |= in && fma(dx, dx, fma(dy, dy, dz * dz)) <= near2;
      } else {
        sm.a[j] = make_double2(q.x, q.y);
        sm.b[j] = make_double2(q.z, q.w);
      }
    }
    if (CARE && near) atomicOr(&sm.own[tile / 32], 1u << (tile % 32));
    __syncthreads();
    if (idle) continue;  // a warp past the last target only stages
    const bool own = (sm.own[tile / 32] >> (tile % 32)) & 1u;
    auto sum = [&](auto how, int n) {
#pragma unroll (CARE ? 4 : UNROLL)
      for (int j = 0; j < n; ++j)
        fp64_source<TPT, FRAME, STRICT, decltype(how)::value>(sm, j, ts + j, tg, self_k, d2,
                                                              one_plus_d2, f, most);
    };
    if (own) {
      sum(How<CARE ? kSelf | kMost : kSelf>{}, len);
      if (CARE && most >= kMostHi) {
#pragma unroll
        for (int t = 0; t < TPT; ++t) f[t][0] = f[t][1] = f[t][2] = 0.0;
#pragma unroll 1
        for (int j = 0; j < len; ++j)
          fp64_source<TPT, FRAME, STRICT, kSelf | kTiny>(sm, j, ts + j, tg, self_k, d2, one_plus_d2, f, most);
        fp64_tiny_pairs<TPT>(sm, src, ts, min(c1, ts + TS), tg, self_k, one_plus_d2, f, ub);
      }
    } else {
      sum(How<0>{}, len);
    }
#pragma unroll
    for (int t = 0; t < TPT; ++t)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sm.acc[(c * TPT + t) * NT + threadIdx.x] += f[t][c];
        f[t][c] = 0.0;
      }
  }
}

// One work unit: the targets at visiting positions [tile0, min(tile0 + NT*TPT,
// i_end)) against the sources [c0, c1); FP64 sums written to out[pos],
// out[stride + pos], out[2*stride + pos]. A target whose index is i has the
// source index i + self_offset and skips itself (self_offset != kNoSelf).
template <int NT, int TPT, int TS, int UNROLL, bool SHORT, bool STRICT, bool CARE>
__device__ __forceinline__ void fp64_unit(const double* __restrict__ x, const int* __restrict__ perm,
                                          int tile0, int i_end, int self_offset, double d2,
                                          bool compact, const double4* __restrict__ src, int c0,
                                          int c1, double* __restrict__ out, size_t stride,
                                          Fp64Smem<NT, TPT, TS>& sm, const UnitBounds& ub) {
  static_assert(TS == 256 && TS % UNROLL == 0, "256 sources between additions to the totals");
  const bool has_self = self_offset != kNoSelf;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  double xi[TPT][3];
  int self_k[TPT];
  double px = 0.0, py = 0.0, pz = 0.0, pn = 0.0;
#pragma unroll
  for (int t = 0; t < TPT; ++t) {
    const int pos = tile0 + (int)threadIdx.x + t * NT;
    const bool valid = pos < i_end;
    const int p = valid ? pos : tile0;
    int ld = p;
    if (perm) ld = TC_BC(ub.rec, BC_PAIR_PERM, p, ub.perm_len) ? perm[p] : 0;
    const bool okx = TC_BC(ub.rec, BC_PAIR_X, ld, ub.x_len);
#pragma unroll
    for (int c = 0; c < 3; ++c) xi[t][c] = okx ? x[3 * (size_t)ld + c] : 0.0;
    self_k[t] = has_self ? ld + self_offset : -1;
    // points far off the sphere (or not finite) have no say in the origin
    const double n2 = fma(xi[t][0], xi[t][0], fma(xi[t][1], xi[t][1], xi[t][2] * xi[t][2]));
    if (!STRICT && compact && valid && n2 > 0.25 && n2 < 4.0) {
      px += xi[t][0];
      py += xi[t][1];
      pz += xi[t][2];
      pn += 1.0;
    }
  }
  if (!STRICT && compact) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      px += __shfl_xor_sync(0xffffffffu, px, o);
      py += __shfl_xor_sync(0xffffffffu, py, o);
      pz += __shfl_xor_sync(0xffffffffu, pz, o);
      pn += __shfl_xor_sync(0xffffffffu, pn, o);
    }
  }
  __syncthreads();  // the previous unit (persistent kernel) is done with the shared memory
  if (!STRICT && lane == 0) {
    sm.csum[0][warp] = px;
    sm.csum[1][warp] = py;
    sm.csum[2][warp] = pz;
    sm.csum[3][warp] = pn;
  }
  for (int k = threadIdx.x; k < kOwnTiles / 32; k += NT) sm.own[k] = 0u;
#pragma unroll
  for (int k = 0; k < 3 * TPT; ++k) sm.acc[k * NT + threadIdx.x] = 0.0;
  __syncthreads();
#pragma unroll
  for (int t = 0; t < TPT; ++t)
    if (self_k[t] >= c0 && self_k[t] < c1) {
      const int tile = (self_k[t] - c0) / TS % kOwnTiles;
      atomicOr(&sm.own[tile / 32], 1u << (tile % 32));
    }
  bool frame = false;
  double near2 = -1.0;
  double tg[TPT][4];  // frame: -t_1, -t_2, 1 - b_i, b_i'; wide: x, y, z
#pragma unroll
  for (int t = 0; t < TPT; ++t) {
    tg[t][0] = xi[t][0];
    tg[t][1] = xi[t][1];
    tg[t][2] = xi[t][2];
    tg[t][3] = 0.0;
  }
  if (!STRICT && compact) {
    if (threadIdx.x == 0) {
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, n = 0.0;
      for (int w = 0; w < NT / 32; ++w) {
        s0 += sm.csum[0][w];
        s1 += sm.csum[1][w];
        s2 += sm.csum[2][w];
        n += sm.csum[3][w];
      }
      const double n2 = fma(s0, s0, fma(s1, s1, s2 * s2));
      sm.framed = n2 > 0.25 * n * n;  // else the targets surround the centre
      if (sm.framed) {
        const double inv = rsqrt(n2);
        const double cx = s0 * inv, cy = s1 * inv, cz = s2 * inv;
        make_frame(cx, cy, cz, sm.frame);
        sm.frame[9] = cx;
        sm.frame[10] = cy;
        sm.frame[11] = cz;
        sm.frame[12] = one_minus_norm2(cx, cy, cz);
      }
    }
    __syncthreads();
    if (sm.framed) {
      const double* fr = sm.frame;
      float rho2 = 0.f;
#pragma unroll
      for (int t = 0; t < TPT; ++t) {
        const double dx = xi[t][0] - fr[9], dy = xi[t][1] - fr[10], dz = xi[t][2] - fr[11];
        const double t1 = frame_dot(fr, dx, dy, dz), t2 = frame_dot(fr + 3, dx, dy, dz),
                     bi = -frame_dot(fr + 9, dx, dy, dz);
        rho2 = fmaxf(rho2, (float)fma(dx, dx, fma(dy, dy, dz * dz)));
        tg[t][0] = -t1;
        tg[t][1] = -t2;
        tg[t][2] = 1.0 - bi;
        tg[t][3] = bi + (d2 + fr[12]);
      }
      const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(rho2));
      if (lane == 0) sm.rho[warp] = m;
      __syncthreads();
      unsigned r = 0;
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) r = max(r, sm.rho[w]);
      frame = __uint_as_float(r) <= kFrameRho2;
      // a denominator below kCareD: |s| <= |t| + 0.0015, (|t| + 0.0015)^2 <= 1.05 |t|^2 + 5e-5
      if (CARE && d2 < kCareD) near2 = 1.05 * (double)__uint_as_float(r) + 5e-5;
      if (!frame) {
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
          tg[t][0] = xi[t][0];
          tg[t][1] = xi[t][1];
          tg[t][2] = xi[t][2];
        }
      }
    }
  }
  const bool idle = tile0 + warp * 32 >= i_end;
  if (frame)
    fp64_sum<NT, TPT, TS, UNROLL, SHORT, true, CARE, false>(src, c0, c1, sm, tg, self_k, idle, d2,
                                                            near2, ub);
  else
    fp64_sum<NT, TPT, TS, 2, SHORT, false, false, STRICT>(src, c0, c1, sm, tg, self_k, idle, d2, 0.0,
                                                          ub);
#pragma unroll
  for (int t = 0; t < TPT; ++t) {
    const int i = tile0 + (int)threadIdx.x + t * NT;
    double T[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) T[c] = sm.acc[(c * TPT + t) * NT + threadIdx.x];
    if (frame) {
      // out with the multiple of x'_i = (t_1, t_2, 1 - b_i), then back: T = R^T T'
      const double* fr = sm.frame;
      const double v0 = -tg[t][0], v1 = -tg[t][1], v2 = tg[t][2];
      const double lam = fma(T[0], v0, fma(T[1], v1, T[2] * v2)) *
                         rcp_f64(fma(v0, v0, fma(v1, v1, v2 * v2)));
      const double a0 = fma(-lam, v0, T[0]), a1 = fma(-lam, v1, T[1]), a2 = fma(-lam, v2, T[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) T[c] = fma(fr[c], a0, fma(fr[3 + c], a1, fr[6 + c] * a2));
    }
    if (i < i_end) {
      if (TC_BC(ub.rec, BC_PAIR_OUT, ub.out_base + i, ub.out_len)) out[i] = T[0];
      if (TC_BC(ub.rec, BC_PAIR_OUT, ub.out_base + (long long)stride + i, ub.out_len))
        out[stride + i] = T[1];
      if (TC_BC(ub.rec, BC_PAIR_OUT, ub.out_base + 2 * (long long)stride + i, ub.out_len))
        out[2 * stride + i] = T[2];
    }
  }
}

template <int NT, int TPT, int TS, int MINB, int UNROLL, bool SHORT, bool STRICT, bool CARE>
__global__ void __launch_bounds__(NT, MINB) pair_fp64_kernel(const PairLaunch P) {
  chain_begin();
  __shared__ Fp64Smem<NT, TPT, TS> sm;
  const TargetSeg& G = find_seg(P, blockIdx.x);
  const int tile0 = G.i0 + (int)(blockIdx.x - G.tile_begin) * (NT * TPT);
  const int c0 = (int)blockIdx.y * P.chunk_len;
  const int c1 = min(P.n, c0 + P.chunk_len);
  const size_t stride = (size_t)P.n_out;
  const long long base = (long long)blockIdx.y * 3 * (long long)stride + G.out_offset;
  double* out = P.partial + base;
  const UnitBounds ub{P.bc, G.x_len, G.perm_len, P.src_len, base, P.partial_len};
  fp64_unit<NT, TPT, TS, UNROLL, SHORT, STRICT, CARE>(
      G.x, G.perm, tile0, G.i1, G.self_offset, G.d2, G.compact != 0, P.src, c0, c1, out, stride, sm,
      ub);
}

// ---------------------------------------------------------------------------
// FP32-compensated pair kernel.
//
// Each CTA takes an origin c - the centroid of its targets projected to the
// sphere - and an orthonormal frame R = (e1, e2, e3) with e3 along c. Sources
// are converted once per CTA and tile from FP64 to FP32 offsets
// s_k = fl32(R(x_k - c)) (FP64 difference and rotation, one rounding),
// targets likewise t_i = fl32(R(x_i - c)). Targets are visited in a spatially
// coherent order (the library's cube-face Hilbert order, sphere_order.cuh, or
// the caller's), so a CTA's targets form a compact patch and every nearby pair
// has small |s_k|, |t_i|: d = s_k - t_i carries an absolute error of a few
// ulps of the patch size instead of ulps of 1. Distances and dot products are
// frame-invariant. The denominator uses the cancellation-free form
//     2(1 - x_i.x_k) + 2 delta^2 = |x_k - x_i|^2 + e_i + e_k,
//     e_i = 1 - |x_i|^2 + 2 delta^2,  e_k = 1 - |x_k|^2
// (evaluated in FP64 once per point, then rounded to FP32), so near pairs
// keep full FP32 relative accuracy although RK4 drifts points off the sphere.
//
// Source pairing: the two f32x2 lanes of every FADD2/FFMA2/FMUL2 carry two
// SOURCES (k, k+1) of one target, so a source tile sits in shared memory once
// (no duplicated values): a warp-wide broadcast 128-bit shared load costs two
// wavefronts of the SM-wide shared pipe, and a far source pair costs 6,
// shared by the T targets of a thread.
//
// Two forms of the pair, chosen per 64-source segment (uniform over the CTA):
// * near (11 FP32 operations): d = s_k - t_i, D = |d|^2 + e_i + e_k,
//   T' += (2G_k / D) d;
// * far (6 FP32 operations), for segments whose every source is farther than
//   kFarRatio times the CTA's target radius rho (the largest |t_i|) from the
//   origin. With a = -c.s_k and b = -c.t_i (minus the offsets' third coordinates,
//   as e3 = c), the identity 1 - x_i.x_k = a + b - a b - s_x t_x - s_y t_y holds
//   on and off the sphere for a unit origin c, so
//       (D/2) / (1 - b_i) = a_k + [(b_i + delta^2) - s_k,x t_i,x - s_k,y t_i,y] / (1 - b_i)
//   takes an addition and 2 FMA with the targets' values, divided by 1 - b_i in
//   FP64, in registers. (Multiplying a_k by 1 - b_i rounded to FP32 would shift
//   all of a target's far terms by the same 2^-25: level 8, 24,575 rows, rms error
//   1.32e-8 where the four products gave 1.12e-8.) T' += r (G_k x'_k) is then 1 - b_i times the sum, taken
//   out at the end, near sums being scaled up to it; x'_k = R x_k = (s_x, s_y, 1 - a) (G x' from FP64,
//   one rounding). In the rotated frame the first two coordinates of x'_k are
//   small tangential offsets and the third is about 1, so the large common part
//   of the sum (about sum r G) sits in the third coordinate only, and u_i = x_i x
//   R^T T' multiplies it by the target's own small offset. With |s| > 3 rho, D >=
//   (|s| - rho)^2 >= 4|s|^2/9, so each rounding of the expansion costs at most a
//   few ulps of D, as in the near form; the self pair never qualifies.
// The far loop is bound by register reads: an FFMA2 of three register pairs takes
// 3.4 cycles a warp and scheduler, 2.5 if the instruction before read one of them,
// 2 only with two. So its instructions go operation by operation over the targets,
// the source's pair staying in the operand cache. Level 7, a launch of 1.61e11 pairs:
// 45.2 ms with 7 operations (the denominator from four products), 42.4 with 6.
// Near and far sums go into the same accumulators: near sum w (x'_k - x'_i)
// and far sum w x'_k differ by multiples of x'_i, which u = x_i x T ignores.
//
// One MUFU reciprocal (rcp.approx.ftz.f32) per pair. The FP32 partials of the
// two source lanes are added and flushed into FP64 accumulators every FLUSH
// sources in mixed tiles (every FLUSH * FARK sources in tiles whose every
// source is far: far terms are small and smooth, and each flush costs F2F
// conversions on the XU pipe that the reciprocals also need), and rotated
// back to the global frame in FP64 once per target.
//
// Self pair (TC_ACTIVE, targets are sources): s_k and t_i are computed by the
// same explicitly fused FP64 operations from the same double, so d = 0
// exactly; e_i carries a +1e-30 bias that keeps D = e_i + e_k away from 0
// and from FP32 subnormals (e is either 0 or at least ~1e-17 in magnitude),
// so w stays finite and w*d adds exactly 0. No per-pair mask is needed.
//
// Form bits (FM): bit 3 always set (the source-paired form; the bit value
// is part of the variant-info ABI); bit 1 keeps the FP64 accumulators in
// shared memory (one slot per thread, target and coordinate: 6 fewer
// registers per target); bit 2 gives near tiles hi/lo offsets; bit 4 lets two targets
// share reciprocals in every second far source pair; bits 8-9 hold log2 FARK.
// HILO (bit 2): near tiles take d = s - t from hi/lo FP32 splits of both
// offsets, (s_hi - t_hi) + (s_lo - t_lo): the rounding of the offsets to FP32
// (an absolute error of ulps of the patch radius, the dominant FP32C error
// for nearest-neighbour pairs) no longer enters, and d keeps a few ulps of its
// own length. Far tiles are unchanged. Both low parts are needed: for the self
// pair s and t are the same point, so (s_hi - t_hi) and (s_lo - t_lo) are
// both exactly 0 and the pair adds w * 0; correcting one side only would
// leave d = s_lo there, a spurious self term.
// ---------------------------------------------------------------------------
constexpr float kSelfBias = 1e-30f;
constexpr float kFarRatio2 = 9.0f;  // kFarRatio = 3
// |s|^2 of a far source: with D/2 >= 2|s|^2/9, products of two denominators lie
// between 5e-34 and 1e33
constexpr float kFarLeast2 = 1e-16f, kFarMost2 = 1e16f;

__device__ __forceinline__ float norm2_f32(float a, float b, float c) {
  return __fmaf_rn(c, c, __fmaf_rn(b, b, __fmul_rn(a, a)));
}

// min (max) of a non-negative float over the CTA: one warp reduction, one
// entry per warp in red[]; the caller synchronises before combine_*.
__device__ __forceinline__ void warp_store_min(float v, unsigned* red) {
  const unsigned m = __reduce_min_sync(0xffffffffu, __float_as_uint(v));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
}
__device__ __forceinline__ void warp_store_max(float v, unsigned* red) {
  const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
}
template <int NW>
__device__ __forceinline__ float combine_min(const unsigned* red) {
  unsigned m = red[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) m = min(m, red[w]);
  return __uint_as_float(m);
}
template <int NW>
__device__ __forceinline__ float combine_max(const unsigned* red) {
  unsigned m = red[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) m = max(m, red[w]);
  return __uint_as_float(m);
}

template <int NT, int TS, int T = 1, bool SMACC = false, bool HILO = false>
struct SpSmem {
  float4 a[TS / 2];        // (sx_k, sx_k+1, sy_k, sy_k+1)
  float4 b[TS / 2];        // (a_k, a_k+1, G x'_k, G x'_k+1)
  float4 c[TS / 2];        // (G y'_k, G y'_k+1, G z'_k, G z'_k+1)
  float4 n[TS / 2];        // near form: (e_k, e_k+1, 2G_k, 2G_k+1)
  double frame[12];        // e1, e2, e3 (rows), origin c
  double csum[3][NT / 32]; // per-warp sums of the target positions
  double acc[SMACC ? 3 * T * NT : 1];  // FP64 accumulators [c][t][thread] (SMACC)
  double om[T * NT];                   // 1 - b of the targets [t][thread]
  float4 lo[HILO ? TS / 2 : 1];        // HILO: low parts (slx_k, slx_k+1, sly_k, sly_k+1)
  float2 loz[HILO ? TS / 2 : 1];       // HILO: low parts of (a_k, a_k+1)
  float tlo[HILO ? 3 * T * NT : 1];    // HILO: low parts of (-t_x, -t_y, -b) [c][t][thread]
  unsigned tmin[NT / 32];
  unsigned rho[NT / 32];
};

__device__ __forceinline__ float2 rcp2(float2 D) {
  return make_float2(rcp_approx_f32(D.x), rcp_approx_f32(D.y));
}

// One far source pair against the thread's T targets. SHARE: targets 0 and 1 share
// their reciprocals, 1/D0 = D1 / (D0 D1): 3 FMUL2 (two registers to read, 2 cycles
// each) in the place of 2 of the MUFU's, 8 cycles each. The far loop shares in every
// second source pair with 3 targets a thread, which evens the two pipes out; always
// sharing, or sharing with 2 targets, measured slower. Level 7, a launch: 41.9 ms
// without, 41.2 with. Errors against FP64 are the same to two digits.
template <int T, bool SHARE>
__device__ __forceinline__ void sp_far_step(const float4 a, const float4 b, const float4 c,
                                            const float2* ftx, const float2* fty, const float2* bd,
                                            float2* fx, float2* fy, float2* fz) {
  const float2 sx = make_float2(a.x, a.y), sy = make_float2(a.z, a.w);
  const float2 ak = make_float2(b.x, b.y), gx = make_float2(b.z, b.w);
  const float2 gy = make_float2(c.x, c.y), gz = make_float2(c.z, c.w);
  float2 D[T];
#pragma unroll
  for (int t = 0; t < T; ++t) D[t] = __fadd2_rn(ak, bd[t]);
#pragma unroll
  for (int t = 0; t < T; ++t) D[t] = __ffma2_rn(sx, ftx[t], D[t]);
#pragma unroll
  for (int t = 0; t < T; ++t) D[t] = __ffma2_rn(sy, fty[t], D[t]);
  if (SHARE && T >= 2) {
    const float2 r = rcp2(__fmul2_rn(D[0], D[1]));
    const float2 r0 = __fmul2_rn(r, D[1]);
    D[1] = __fmul2_rn(r, D[0]);
    D[0] = r0;
  }
#pragma unroll
  for (int t = SHARE && T >= 2 ? 2 : 0; t < T; ++t) D[t] = rcp2(D[t]);
#pragma unroll
  for (int t = 0; t < T; ++t) fx[t] = __ffma2_rn(D[t], gx, fx[t]);
#pragma unroll
  for (int t = 0; t < T; ++t) fy[t] = __ffma2_rn(D[t], gy, fy[t]);
#pragma unroll
  for (int t = 0; t < T; ++t) fz[t] = __ffma2_rn(D[t], gz, fz[t]);
}

// FP64 accumulator of target t, coordinate c: a register, or (SMACC) a
// shared-memory slot of this thread (frees 6 registers per target).
template <int NT, int T, bool SMACC>
struct SpAcc {
  double r[SMACC ? 1 : 3 * T];
  double* sm;
  __device__ __forceinline__ void init(double* base) {
    sm = base + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 3 * T; ++k) {
      if (SMACC)
        sm[k * NT] = 0.0;
      else
        r[k] = 0.0;
    }
  }
  __device__ __forceinline__ void add(int c, int t, double v) {
    if (SMACC)
      sm[(c * T + t) * NT] += v;
    else
      r[c * T + t] += v;
  }
  __device__ __forceinline__ double get(int c, int t) const {
    return SMACC ? sm[(c * T + t) * NT] : r[c * T + t];
  }
};

// Converts the sources of the tile at ts into the CTA's frame: offsets s_k, a_k,
// G_k x'_k, e_k, 2G_k (and the hi/lo low parts), padding past c1; records each
// warp's minimum |s_k|^2.
template <int NT, int TS, bool HILO, class Smem>
__device__ __forceinline__ void sp_stage(const double4* __restrict__ src, int ts, int c1,
                                         const double* fr, Smem& sm, const UnitBounds& ub) {
  constexpr int NP = TS / 2;
  float smin = __int_as_float(0x7f800000);  // +inf
  for (int jp = threadIdx.x; jp < NP; jp += NT) {
    float v[2][11];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = ts + 2 * jp + h;
      // padding sources: zero weight, denominators of about 1
      v[h][0] = v[h][1] = 0.f;
      v[h][2] = 1.f;
      v[h][3] = v[h][4] = v[h][5] = 0.f;
      v[h][6] = 1.f;
      v[h][7] = 0.f;
      v[h][8] = v[h][9] = v[h][10] = 0.f;
      if (k < c1 && TC_BC(ub.rec, BC_PAIR_SRC, k, ub.src_len)) {
        const double4 q = src[k];
        const double dx = q.x - fr[9], dy = q.y - fr[10], dz = q.z - fr[11];
        const double sxd = frame_dot(fr, dx, dy, dz), syd = frame_dot(fr + 3, dx, dy, dz),
                     akd = -frame_dot(fr + 6, dx, dy, dz);
        const float sx = (float)sxd, sy = (float)syd, ak = (float)akd;
        if (HILO) {
          v[h][8] = (float)(sxd - (double)sx);
          v[h][9] = (float)(syd - (double)sy);
          v[h][10] = (float)(akd - (double)ak);
        }
        const double ek = 1.0 - (q.x * q.x + q.y * q.y + q.z * q.z);
        // a source far off the sphere (or not finite) counts as near: products of two
        // far denominators stay in range
        const float s2 = norm2_f32(sx, sy, ak);
        smin = fminf(smin, s2 < kFarMost2 ? s2 : 0.f);
        v[h][0] = sx;
        v[h][1] = sy;
        v[h][2] = ak;
        v[h][3] = (float)(q.w * sxd);
        v[h][4] = (float)(q.w * syd);
        v[h][5] = (float)fma(-q.w, akd, q.w);
        v[h][6] = (float)ek;
        v[h][7] = (float)(2.0 * q.w);
      }
    }
    sm.a[jp] = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
    sm.b[jp] = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
    sm.c[jp] = make_float4(v[0][4], v[1][4], v[0][5], v[1][5]);
    sm.n[jp] = make_float4(v[0][6], v[1][6], v[0][7], v[1][7]);
    if (HILO) {
      sm.lo[jp] = make_float4(v[0][8], v[1][8], v[0][9], v[1][9]);
      sm.loz[jp] = make_float2(v[0][10], v[1][10]);
    }
  }
  warp_store_min(smin, sm.tmin);
}

// Far source pairs [j0, j1) of the staged tile against the thread's targets.
template <int T, int UNROLL, bool SHARE, class Smem>
__device__ __forceinline__ void sp_far_run(const Smem& sm, int j0, int j1, const float2 (&ftx)[T],
                                           const float2 (&fty)[T], const float2 (&bd)[T],
                                           float2 (&fx)[T], float2 (&fy)[T], float2 (&fz)[T]) {
  static_assert(UNROLL % 2 == 0, "an even number of source pairs per loop body");
#pragma unroll UNROLL / 2
  for (int j = j0; j < j1; j += 2) {
    sp_far_step<T, SHARE>(sm.a[j], sm.b[j], sm.c[j], ftx, fty, bd, fx, fy, fz);
    sp_far_step<T, false>(sm.a[j + 1], sm.b[j + 1], sm.c[j + 1], ftx, fty, bd, fx, fy, fz);
  }
}

// Sums the staged tile into the thread's T targets: a tile whose
// every source is far in one tight far loop flushed every FARK segments; else
// per 64-source segment, far or near. With NT = TS/2 source pairs and FP = 32
// every warp staged exactly one segment, so segment g's minimum |s|^2 is warp
// g's and only the segments that hold near sources take the near form;
// otherwise one far test for the whole tile.
template <int NT, int T, int TS, int FLUSH, int UNROLL, bool SMACC, bool HILO, int FARK, bool SHARE,
          class Smem>
__device__ __forceinline__ void sp_sum(const Smem& sm, const float2 (&ftx)[T],
                                       const float2 (&fty)[T], const float2 (&bd)[T],
                                       const float (&ntx)[T], const float (&nty)[T],
                                       const float (&nb)[T], const float (&ei)[T],
                                       float2 (&fx)[T], float2 (&fy)[T], float2 (&fz)[T],
                                       SpAcc<NT, T, SMACC>& acc) {
  constexpr int NP = TS / 2;
  constexpr int FP = FLUSH / 2;
  constexpr int FPF = FP * FARK;  // source pairs between flushes in all-far tiles
  constexpr bool PERSEG = (NT == TS / 2) && (FP == 32);
  const float lim = fmaxf(kFarRatio2 * combine_max<NT / 32>(sm.rho), kFarLeast2);
  const bool tile_far = combine_min<NT / 32>(sm.tmin) > lim;
  if (tile_far) {
    for (int jf = 0; jf < NP; jf += FPF) {
      sp_far_run<T, UNROLL, SHARE>(sm, jf, jf + FPF, ftx, fty, bd, fx, fy, fz);
#pragma unroll
      for (int t = 0; t < T; ++t) {
        acc.add(0, t, (double)__fadd_rn(fx[t].x, fx[t].y));
        acc.add(1, t, (double)__fadd_rn(fy[t].x, fy[t].y));
        acc.add(2, t, (double)__fadd_rn(fz[t].x, fz[t].y));
        fx[t] = fy[t] = fz[t] = make_float2(0.f, 0.f);
      }
    }
    return;
  }
  for (int jf = 0; jf < NP; jf += FP) {
    const bool far = PERSEG && __uint_as_float(sm.tmin[jf / FP]) > lim;
    if (far) {
      sp_far_run<T, UNROLL, SHARE>(sm, jf, jf + FP, ftx, fty, bd, fx, fy, fz);
    } else {
      // HILO: d = (s_hi - t_hi) + (s_lo - t_lo), accurate to a few ulps of d itself
      float ntl[HILO ? 3 * T : 1];
      if (HILO) {
#pragma unroll
        for (int k = 0; k < 3 * T; ++k) ntl[k] = sm.tlo[k * NT + threadIdx.x];
      }
#pragma unroll 4
      for (int j = jf; j < jf + FP; ++j) {
        const float4 a = sm.a[j];
        const float4 b = sm.b[j];
        const float4 n = sm.n[j];
        const float2 sx = make_float2(a.x, a.y), sy = make_float2(a.z, a.w);
        const float2 ak = make_float2(b.x, b.y);
        const float2 ee = make_float2(n.x, n.y), gg = make_float2(n.z, n.w);
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 loz = make_float2(0.f, 0.f);
        if (HILO) {
          lo = sm.lo[j];
          loz = sm.loz[j];
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
          float2 dx = __fadd2_rn(sx, make_float2(ntx[t], ntx[t]));
          float2 dy = __fadd2_rn(sy, make_float2(nty[t], nty[t]));
          float2 dz = __fadd2_rn(ak, make_float2(nb[t], nb[t]));  // -(s_z - t_z)
          if (HILO) {
            dx = __fadd2_rn(dx, __fadd2_rn(make_float2(lo.x, lo.y), make_float2(ntl[t], ntl[t])));
            dy = __fadd2_rn(dy, __fadd2_rn(make_float2(lo.z, lo.w), make_float2(ntl[T + t], ntl[T + t])));
            dz = __fadd2_rn(dz, __fadd2_rn(loz, make_float2(ntl[2 * T + t], ntl[2 * T + t])));
          }
          float2 D = __fadd2_rn(ee, make_float2(ei[t], ei[t]));
          D = __ffma2_rn(dx, dx, D);
          D = __ffma2_rn(dy, dy, D);
          D = __ffma2_rn(dz, dz, D);
          const float2 w = __fmul2_rn(gg, rcp2(D));
          fx[t] = __ffma2_rn(w, dx, fx[t]);
          fy[t] = __ffma2_rn(w, dy, fy[t]);
          fz[t] = __ffma2_rn(w, dz, fz[t]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
      // near: scaled up to the far sums, and z was summed with the other sign
      const double up = far ? 1.0 : sm.om[t * NT + threadIdx.x];
      acc.add(0, t, up * (double)__fadd_rn(fx[t].x, fx[t].y));
      acc.add(1, t, up * (double)__fadd_rn(fy[t].x, fy[t].y));
      acc.add(2, t, (far ? up : -up) * (double)__fadd_rn(fz[t].x, fz[t].y));
      fx[t] = fy[t] = fz[t] = make_float2(0.f, 0.f);
    }
  }
}

// One work unit: targets at visiting positions [tile0, min(tile0 + NT*T,
// i_end)) against sources [c0, c1); FP64 sums in the global frame written to
// out[pos], out[stride + pos], out[2*stride + pos].
template <int NT, int T, int TS, int FLUSH, int UNROLL, bool SMACC, bool HILO, int FARK, bool SHARE>
__device__ __forceinline__ void fp32c_sp_unit(const double* __restrict__ x, const int* __restrict__ perm,
                                              int tile0, int i_end, double d2,
                                              const double4* __restrict__ src, int c0, int c1,
                                              double* __restrict__ out, size_t stride,
                                              SpSmem<NT, TS, T, SMACC, HILO>& sm,
                                              const UnitBounds& ub) {
  static_assert(TS % FLUSH == 0 && FLUSH % 2 == 0, "flush interval: even, divides the tile");
  static_assert(NT % 32 == 0, "whole warps");
  static_assert(TS % (FLUSH * FARK) == 0, "far-tile flush interval divides the tile");
  constexpr int TB = NT * T;

  const int mid_pos = min(tile0 + TB / 2, i_end - 1);
  int mid = mid_pos;
  if (perm) mid = TC_BC(ub.rec, BC_PAIR_PERM, mid_pos, ub.perm_len) ? perm[mid_pos] : 0;
  // checked build: an out-of-range target index reads point 0 instead (and is recorded)
  auto target = [&](int p) -> int {
    int ld = p;
    if (perm) ld = TC_BC(ub.rec, BC_PAIR_PERM, p, ub.perm_len) ? perm[p] : 0;
    return TC_BC(ub.rec, BC_PAIR_X, ld, ub.x_len) ? ld : 0;
  };
  // Origin: the CTA's targets' centroid, projected to the sphere (a smaller
  // patch radius than any one target gives: fewer near tiles, smaller FP32
  // offsets); the middle target's direction when the targets surround the centre.
  double px = 0.0, py = 0.0, pz = 0.0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int pos = tile0 + (int)threadIdx.x + t * NT;
    if (pos < i_end) {
      const int ld = target(pos);
      px += x[3 * (size_t)ld];
      py += x[3 * (size_t)ld + 1];
      pz += x[3 * (size_t)ld + 2];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    px += __shfl_xor_sync(0xffffffffu, px, o);
    py += __shfl_xor_sync(0xffffffffu, py, o);
    pz += __shfl_xor_sync(0xffffffffu, pz, o);
  }
  __syncthreads();  // the previous unit (persistent kernel) is done with sm.frame, sm.csum
  if ((threadIdx.x & 31) == 0) {
    sm.csum[0][threadIdx.x >> 5] = px;
    sm.csum[1][threadIdx.x >> 5] = py;
    sm.csum[2][threadIdx.x >> 5] = pz;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int w = 0; w < NT / 32; ++w) {
      sx += sm.csum[0][w];
      sy += sm.csum[1][w];
      sz += sm.csum[2][w];
    }
    const double count = (double)min(TB, i_end - tile0);
    const double n2 = sx * sx + sy * sy + sz * sz;
    double cx = sx, cy = sy, cz = sz, m2 = n2;
    if (!(n2 > 0.25 * count * count && n2 < 1e6 * count * count)) {
      const int c = TC_BC(ub.rec, BC_PAIR_X, mid, ub.x_len) ? mid : 0;
      cx = x[3 * (size_t)c];
      cy = x[3 * (size_t)c + 1];
      cz = x[3 * (size_t)c + 2];
      m2 = cx * cx + cy * cy + cz * cz;
      if (!(m2 > 1e-6 && m2 < 1e6)) {  // not finite or far off the sphere: any unit origin serves
        cx = cy = 0.0;
        cz = m2 = 1.0;
      }
    }
    const double inv = 1.0 / sqrt(m2);
    cx *= inv;
    cy *= inv;
    cz *= inv;
    make_frame(cx, cy, cz, sm.frame);
    sm.frame[9] = cx;
    sm.frame[10] = cy;
    sm.frame[11] = cz;
  }
  __syncthreads();
  const double* fr = sm.frame;
  const double cx = fr[9], cy = fr[10], cz = fr[11];

  float2 ftx[T], fty[T], bd[T];  // far: (-t_x, -t_y, b + delta^2) / (1 - b)
  float ntx[T], nty[T], nb[T], ei[T];  // near, paired on use: -t_x, -t_y, -b, e
  float2 fx[T], fy[T], fz[T];
  SpAcc<NT, T, SMACC> acc;
  acc.init(sm.acc);
  float rho2 = 0.f;
  unsigned bad = 0u;  // SHARE: targets that are not finite
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int pos = tile0 + (int)threadIdx.x + t * NT;
    const int ld = pos < i_end ? target(pos) : (TC_BC(ub.rec, BC_PAIR_X, mid, ub.x_len) ? mid : 0);
    double px = x[3 * (size_t)ld], py = x[3 * (size_t)ld + 1], pz = x[3 * (size_t)ld + 2];
    // a target that is not finite must not reach its neighbour's reciprocals: it takes
    // the origin's place, and NaN at the end
    if (SHARE && !isfinite(px + py + pz)) {
      bad |= 1u << t;
      px = cx;
      py = cy;
      pz = cz;
    }
    const double dx = px - cx, dy = py - cy, dz = pz - cz;
    const double txd = frame_dot(fr, dx, dy, dz), tyd = frame_dot(fr + 3, dx, dy, dz),
                 bid = -frame_dot(fr + 6, dx, dy, dz);
    const float tx = (float)txd, ty = (float)tyd, b = (float)bid;
    if (HILO) {
      sm.tlo[(0 * T + t) * NT + threadIdx.x] = -(float)(txd - (double)tx);
      sm.tlo[(1 * T + t) * NT + threadIdx.x] = -(float)(tyd - (double)ty);
      sm.tlo[(2 * T + t) * NT + threadIdx.x] = -(float)(bid - (double)b);
    }
    const double E = (1.0 - (px * px + py * py + pz * pz)) + 2.0 * d2;
    rho2 = fmaxf(rho2, norm2_f32(tx, ty, b));
    double om = 1.0 - bid;
    if (!(om > 0.5)) {  // more than 60 degrees from the origin: no tile of this CTA is far
      om = 1.0;
      rho2 = __int_as_float(0x7f800000);
    }
    const double sc = rcp_f64(om);
    const float fx0 = (float)(-txd * sc), fy0 = (float)(-tyd * sc), b0 = (float)((bid + d2) * sc);
    ftx[t] = make_float2(fx0, fx0);
    fty[t] = make_float2(fy0, fy0);
    bd[t] = make_float2(b0, b0);
    sm.om[t * NT + threadIdx.x] = om;
    ntx[t] = -tx;
    nty[t] = -ty;
    nb[t] = -b;
    ei[t] = (float)E + kSelfBias;
    fx[t] = fy[t] = fz[t] = make_float2(0.f, 0.f);
  }
  warp_store_max(rho2, sm.rho);
  for (int ts = c0; ts < c1; ts += TS) {
    __syncthreads();
    sp_stage<NT, TS, HILO>(src, ts, c1, fr, sm, ub);
    __syncthreads();
    sp_sum<NT, T, TS, FLUSH, UNROLL, SMACC, HILO, FARK, SHARE>(
        sm, ftx, fty, bd, ntx, nty, nb, ei, fx, fy, fz, acc);
  }
  // back to the global frame: T = R^T T'
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int pos = tile0 + (int)threadIdx.x + t * NT;
    if (pos < i_end) {
      const double sc = rcp_f64(sm.om[t * NT + threadIdx.x]);
      double ax = acc.get(0, t) * sc;
      const double ay = acc.get(1, t) * sc, az = acc.get(2, t) * sc;
      if (SHARE && ((bad >> t) & 1u)) ax = __longlong_as_double(0x7ff8000000000000ll);
      if (TC_BC(ub.rec, BC_PAIR_OUT, ub.out_base + pos, ub.out_len))
        out[pos] = fma(fr[0], ax, fma(fr[3], ay, fr[6] * az));
      if (TC_BC(ub.rec, BC_PAIR_OUT, ub.out_base + (long long)stride + pos, ub.out_len))
        out[stride + pos] = fma(fr[1], ax, fma(fr[4], ay, fr[7] * az));
      if (TC_BC(ub.rec, BC_PAIR_OUT, ub.out_base + 2 * (long long)stride + pos, ub.out_len))
        out[2 * stride + pos] = fma(fr[2], ax, fma(fr[5], ay, fr[8] * az));
    }
  }
}

// Template parameters of fp32c_sp_unit from a form bit set FM.
template <int FM>
struct SpForm {
  static constexpr bool smacc = (FM & 2) != 0;
  static constexpr bool hilo = (FM & 4) != 0;
  static constexpr int fark = 1 << ((FM >> 8) & 3);
  static constexpr bool share = (FM & 16) != 0;
};

template <int NT, int T, int TS, int FLUSH, int MINB, int UNROLL, int FM>
__global__ void __launch_bounds__(NT, MINB) pair_fp32c_kernel(const PairLaunch P) {
  chain_begin();
  using F = SpForm<FM>;
  const TargetSeg& G = find_seg(P, blockIdx.x);
  const int tile0 = G.i0 + (int)(blockIdx.x - G.tile_begin) * (NT * T);
  const int c0 = (int)blockIdx.y * P.chunk_len;
  const int c1 = min(P.n, c0 + P.chunk_len);
  const size_t stride = (size_t)P.n_out;
  const long long base = (long long)blockIdx.y * 3 * (long long)stride + G.out_offset;
  double* out = P.partial + base;
  const UnitBounds ub{P.bc, G.x_len, G.perm_len, P.src_len, base, P.partial_len};
  __shared__ SpSmem<NT, TS, T, F::smacc, F::hilo> sm;
  fp32c_sp_unit<NT, T, TS, FLUSH, UNROLL, F::smacc, F::hilo, F::fark, F::share>(G.x, G.perm, tile0, G.i1,
                                                                      G.d2, P.src, c0, c1, out,
                                                                      stride, sm, ub);
}

// ---------------------------------------------------------------------------
// Batched (ensemble) form: many independent particle sets concatenated in one
// RK4 state. A work item is (target tile of one class of one instance, one
// chunk of that instance's sources); a persistent grid of one wave of CTAs
// takes items from an atomic counter until none is left (no CTA ever waits
// on another). Items are queued longest first, so the uneven instance sizes
// even out across the SMs.
// ---------------------------------------------------------------------------
struct BatchSeg {
  const double* x;   // target positions of the class (concatenated instances)
  const int* perm;   // visiting order (null: as stored)
  int out_offset;    // partial row of target position p is out_offset + p
  int self_offset;   // TC_ACTIVE: source index of target i is i + self_offset
  double d2;
  int targets;       // targets of the class in the instance
  long long x_len;     // checked build: points in x
  long long perm_len;  // checked build: entries in perm
};

struct BatchItem {
  int seg;           // index into the segment table
  int tile0, i1;     // target positions [tile0, min(tile0 + TB, i1))
  int c0, c1;        // sources [c0, c1) (absolute rows of the packed sources)
  int chunk;         // chunk index within the instance (partial slab)
};

struct BatchLaunch {
  const BatchItem* items;
  int n_items;
  int* counter;      // zeroed before each launch
  const BatchSeg* segs;
  const double4* src;
  double* partial;   // partial[(chunk*3 + c)*stride + row]
  size_t stride;
  bool care;              // FP64: a segment has d2 < kCareD
  BoundsRec* bc;          // checked build: violation record (null: release build)
  int n_segs;             // checked build: entries in segs
  long long src_len;      // checked build: packed sources in src
  long long partial_len;  // checked build: doubles in partial
};

__device__ __forceinline__ int next_item(int* counter, int* slot) {
  __syncthreads();  // every thread is done with the previous item's slot value
  if (threadIdx.x == 0) *slot = atomicAdd(counter, 1);
  __syncthreads();
  return *slot;
}

template <int NT, int T, int TS, int FLUSH, int MINB, int UNROLL, int FM>
__global__ void __launch_bounds__(NT, MINB) pair_fp32c_batch_kernel(const BatchLaunch B) {
  chain_begin();
  using F = SpForm<FM>;
  __shared__ int slot;
  __shared__ SpSmem<NT, TS, T, F::smacc, F::hilo> sm;
  for (int it = next_item(B.counter, &slot); it < B.n_items; it = next_item(B.counter, &slot)) {
    const BatchItem I = B.items[it];
    if (!TC_BC(B.bc, BC_BATCH_SEG, I.seg, B.n_segs)) continue;
    const BatchSeg S = B.segs[I.seg];
    const long long base = (long long)I.chunk * 3 * (long long)B.stride + S.out_offset;
    double* out = B.partial + base;
    const UnitBounds ub{B.bc, S.x_len, S.perm_len, B.src_len, base, B.partial_len};
    fp32c_sp_unit<NT, T, TS, FLUSH, UNROLL, F::smacc, F::hilo, F::fark, F::share>(
        S.x, S.perm, I.tile0, I.i1, S.d2, B.src, I.c0, I.c1, out, B.stride, sm, ub);
  }
}

template <int NT, int TPT, int TS, int MINB, int UNROLL, bool SHORT, bool STRICT, bool CARE>
__global__ void __launch_bounds__(NT, MINB) pair_fp64_batch_kernel(const BatchLaunch B) {
  chain_begin();
  __shared__ Fp64Smem<NT, TPT, TS> sm;
  __shared__ int slot;
  for (int it = next_item(B.counter, &slot); it < B.n_items; it = next_item(B.counter, &slot)) {
    const BatchItem I = B.items[it];
    if (!TC_BC(B.bc, BC_BATCH_SEG, I.seg, B.n_segs)) continue;
    const BatchSeg S = B.segs[I.seg];
    const long long base = (long long)I.chunk * 3 * (long long)B.stride + S.out_offset;
    double* out = B.partial + base;
    const UnitBounds ub{B.bc, S.x_len, S.perm_len, B.src_len, base, B.partial_len};
    fp64_unit<NT, TPT, TS, UNROLL, SHORT, STRICT, CARE>(
        S.x, S.perm, I.tile0, I.i1, S.self_offset, S.d2,
        S.targets >= kCompactTiles * NT * TPT, B.src, I.c0, I.c1, out,
        B.stride, sm, ub);
  }
}

}  // namespace tcb
