// Spatially coherent visiting order of targets for the pair kernels: each target is
// keyed by its cube face and its position along a 2-D
// Hilbert curve over that face (sphere_order.cuh) and the keys are sorted with
// a stable sort, so a CTA's consecutive targets form a compact patch of
// the sphere whatever order the caller stores them in (the reference numbers
// particles in creation order, level by level). The sort is stable and the
// keys are a pure function of the positions, so the order - and with it every
// result - is deterministic.
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>

#include "sphere_order.cuh"
#include "tc_ctx.h"

namespace tcb {
namespace {

// Checked build: extents of the key kernel's arrays.
struct KeyBounds {
  BoundsRec* rec;
  long long x_len, key_len;  // points in x; entries in keys and idx
};

__global__ void hilbert_keys_kernel(const double* __restrict__ x, int i0, int n,
                                    unsigned* __restrict__ keys, int* __restrict__ idx,
                                    const KeyBounds kb) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  if (!TC_BC(kb.rec, BC_ORDER_KEYS, j, kb.key_len)) return;
  const size_t b = 3 * (size_t)(i0 + j);
  keys[j] = TC_BC(kb.rec, BC_ORDER_X, i0 + j, kb.x_len) ? sphere_key(x[b], x[b + 1], x[b + 2]) : 0u;
  idx[j] = i0 + j;
}

// Orders of up to three target classes whose points each fit one CTA's shared
// memory (kSmallOrder): one key launch and one sorting launch for all of them,
// where keys and the device-wide radix sort take seven or more launches a class.
// Both are bound by latency, the sort's by its chain of launches. Level 4 refined,
// 7,451 panels and 3,768 particles: 15 us for the two launches, and a five-step
// FP32C run on that grid 1.36 ms -> 1.10 ms on the device. The result is the radix sort's, entry
// for entry.
struct SmallOrder {
  const double* x;
  int* perm;       // perm[i0 .. i0 + n)
  unsigned* keys;  // n entries
  int i0, n;
  KeyBounds kb;
};
struct SmallOrders {
  SmallOrder s[3];
};

constexpr int kSmallOrder = 16384;     // points: 6 bytes each in shared memory
constexpr int kOrderThreads = 1024;
constexpr int kOrderWarps = kOrderThreads / 32;
constexpr int kOrderCellBits = 13;     // cells = leading key bits, six faces of 1,024
constexpr int kOrderCells = 1 << kOrderCellBits;
constexpr int kOrderShift = kSphereKeyBits - kOrderCellBits;
constexpr int kFullCell = 64;          // points of a cell that are still ranked by comparing
constexpr int kDigitBits = 8, kDigits = 1 << kDigitBits;
constexpr int kDigitPasses = (kSphereKeyBits + kDigitBits - 1) / kDigitBits;
constexpr int kOrderSteps = kSmallOrder / kOrderThreads;  // points of a lane, at most
// the cells' counts, or a padded column of digit counts for each warp
constexpr int kOrderCounts = kDigits * (kOrderWarps + 1);
static_assert(kOrderCounts >= kOrderCells && kDigits * kOrderWarps == kOrderCells, "one array for both");

__global__ void small_keys_kernel(const SmallOrders P) {
  chain_begin();
  const SmallOrder& S = P.s[blockIdx.y];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= S.n) return;
  if (!TC_BC(S.kb.rec, BC_ORDER_KEYS, j, S.kb.key_len)) return;
  const size_t b = 3 * (size_t)(S.i0 + j);
  S.keys[j] = TC_BC(S.kb.rec, BC_ORDER_X, S.i0 + j, S.kb.x_len)
                  ? sphere_key(S.x[b], S.x[b + 1], S.x[b + 2])
                  : 0u;
}

// Exclusive prefix sum, over the CTA's threads in order, of eight counts each; the
// thread's largest count.
constexpr int kPer = kOrderCells / kOrderThreads;
__device__ __forceinline__ int order_prefix(int* mine, int* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int n[kPer], total = 0, most = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    n[q] = mine[q];
    total += n[q];
    most = max(most, n[q]);
  }
  int incl = total;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int base = incl - total;
  for (int w = 0; w < warp; ++w) base += wsum[w];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    mine[q] = base;
    base += n[q];
  }
  return most;
}

// The order of n keys by a stable counting sort of idx, 8 key bits at a time, the lowest
// first: its time does not depend on where the points are. In each pass a warp takes a
// stretch of the indices in their present order, finds the lanes of equal digit by ballots
// and counts digits as it goes, so a point's rank among its warp's points of that digit
// is known at once; the counts' prefix sum, digits before warps, gives every point its
// place.
__device__ __noinline__ void order_by_digits(const SmallOrder& S, const unsigned* keys,
                                                unsigned short* idx, int* counts, int* wsum) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int(*count)[kOrderWarps + 1] = reinterpret_cast<int(*)[kOrderWarps + 1]>(counts);
  for (int j = tid; j < S.n; j += kOrderThreads) idx[j] = (unsigned short)j;
  const int steps = (S.n + kOrderThreads - 1) / kOrderThreads;  // of 32 points a warp
  for (int pass = 0; pass < kDigitPasses; ++pass) {
    const int shift = pass * kDigitBits;
    for (int c = tid; c < kOrderCounts; c += kOrderThreads) counts[c] = 0;
    __syncthreads();
    int point[kOrderSteps], rank[kOrderSteps];
#pragma unroll
    for (int q = 0; q < kOrderSteps; ++q) {
      if (q >= steps) break;
      const int p = 32 * (warp * steps + q) + lane;
      const bool in = p < S.n;
      point[q] = in ? idx[p] : -1;
      const unsigned d = in ? (keys[point[q]] >> shift) & (kDigits - 1) : kDigits;
      unsigned same = 0xffffffffu;
#pragma unroll
      for (int b = 0; b <= kDigitBits; ++b) {
        const bool set = (d >> b) & 1u;
        const unsigned with = __ballot_sync(0xffffffffu, set);
        same &= set ? with : ~with;
      }
      const int before = __popc(same & ((1u << lane) - 1u));
      const int seen = in ? count[d][warp] : 0;
      __syncwarp();
      if (in && before == 0) count[d][warp] = seen + __popc(same);
      __syncwarp();
      rank[q] = seen + before;
    }
    __syncthreads();
    order_prefix(&count[tid * kPer / kOrderWarps][tid * kPer % kOrderWarps], wsum);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kOrderSteps; ++q) {
      if (q >= steps || point[q] < 0) break;
      const int j = point[q];
      const int to = count[(keys[j] >> shift) & (kDigits - 1)][warp] + rank[q];
      if (pass < kDigitPasses - 1)
        idx[to] = (unsigned short)j;
      else if (TC_BC(S.kb.rec, BC_ORDER_KEYS, j, S.kb.key_len))
        S.perm[S.i0 + to] = S.i0 + j;
    }
    __syncthreads();
  }
}

// One CTA per class: a counting sort by cell, then each point's rank among its
// cell's points by (key, index). The order inside a cell that the atomics leave
// is not used, so the result is deterministic. The ranks take a comparison for every
// pair of a cell, 10 ns for 1,024 points at a time: where a cell holds more than kFullCell
// points (a dense local set) the keys are sorted by digits instead, which would take
// 37 us longer over points all over the sphere. 16,384 targets against 20 sources, all
// over the sphere: 42 us a call; in one cell 2.53 ms by comparing, 72 us by digits.
__global__ void __launch_bounds__(kOrderThreads) small_order_kernel(const SmallOrders P) {
  chain_begin();
  extern __shared__ unsigned order_smem[];
  const SmallOrder& S = P.s[blockIdx.x];
  unsigned* keys = order_smem;                                       // n
  int* cell = reinterpret_cast<int*>(order_smem + S.n);              // kOrderCounts
  unsigned short* slot = reinterpret_cast<unsigned short*>(cell + kOrderCounts);  // n
  __shared__ int wsum[kOrderWarps];
  const int tid = threadIdx.x;
  for (int c = tid; c < kOrderCells; c += kOrderThreads) cell[c] = 0;
  __syncthreads();
  for (int j = tid; j < S.n; j += kOrderThreads) {
    const unsigned k = TC_BC(S.kb.rec, BC_ORDER_KEYS, j, S.kb.key_len)
                           ? S.keys[j] & ((1u << kSphereKeyBits) - 1u)
                           : 0u;
    keys[j] = k;
    atomicAdd(&cell[k >> kOrderShift], 1);
  }
  __syncthreads();
  if (__syncthreads_or(order_prefix(cell + tid * kPer, wsum) > kFullCell)) {
    order_by_digits(S, keys, slot, cell, wsum);
    return;
  }
  for (int j = tid; j < S.n; j += kOrderThreads)
    slot[atomicAdd(&cell[keys[j] >> kOrderShift], 1)] = (unsigned short)j;
  __syncthreads();
  // cell[c] is now the end of cell c
  for (int p = tid; p < S.n; p += kOrderThreads) {
    const int j = slot[p];
    const unsigned k = keys[j];
    const int c = (int)(k >> kOrderShift);
    const int lo = c ? cell[c - 1] : 0, hi = cell[c];
    int rank = lo;
    for (int q = lo; q < hi; ++q) {
      const int o = slot[q];
      rank += (keys[o] < k || (keys[o] == k && o < j)) ? 1 : 0;
    }
    if (TC_BC(S.kb.rec, BC_ORDER_KEYS, j, S.kb.key_len)) S.perm[S.i0 + rank] = S.i0 + j;
  }
}

size_t small_order_smem(int n) {
  return (size_t)n * (sizeof(unsigned) + sizeof(unsigned short)) + kOrderCounts * sizeof(int) + 16;
}

int launch_small_orders(tc_ctx* ctx, const SmallOrders& P, int count) {
  int most = 0;
  for (int c = 0; c < count; ++c) most = std::max(most, P.s[c].n);
  const size_t smem = small_order_smem(most);
  TC_CUDA_TRY(cudaFuncSetAttribute(small_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)small_order_smem(kSmallOrder)));
  launch_chained(small_keys_kernel, dim3((most + 127) / 128, count), dim3(128), 0, ctx->stream, P);
  TC_CUDA_TRY(cudaGetLastError());
  launch_chained(small_order_kernel, dim3(count), dim3(kOrderThreads), smem, ctx->stream, P);
  TC_CUDA_TRY(cudaGetLastError());
  ctx->launches += 2;
  return TC_OK;
}

}  // namespace

// Bytes of sort scratch (CUB's temporary storage) for an order over n targets.
int order_sort_bytes(int n, size_t* bytes) {
  *bytes = 0;
  if (n <= 0) return TC_OK;
  TC_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, *bytes, (const unsigned*)nullptr,
                                              (unsigned*)nullptr, (const int*)nullptr, (int*)nullptr,
                                              n, 0, kSphereKeyBits));
  return TC_OK;
}

// perm[i0 .. i1) <- the indices i0..i1-1 sorted by the sphere key of x[i], in
// caller-provided scratch: keys k_in, k_out and indices v_in of i1 - i0 entries
// each, and `temp` of at least order_sort_bytes(i1 - i0) bytes.
int compute_order_into(tc_ctx* ctx, const double* x, int i0, int i1, int* perm, unsigned* k_in,
                       unsigned* k_out, int* v_in, void* temp, size_t temp_bytes,
                       const OrderExtents& ext) {
  const int n = i1 - i0;
  if (n <= 0) return TC_OK;
  if ((long long)i1 > ext.perm_len || (long long)n > ext.key_len || (long long)i1 > ext.x_len) {
    tc_record_error("visiting order of [%d,%d): %lld points, %lld order entries, %lld keys", i0, i1,
                    ext.x_len, ext.perm_len, ext.key_len);
    return TC_ERR_ARG;
  }
  const KeyBounds kb{ctx->bc_rec, bc_extent(ctx, BC_ORDER_X, ext.x_len),
                     bc_extent(ctx, BC_ORDER_KEYS, ext.key_len)};
  if (n <= kSmallOrder) {
    SmallOrders P{};
    P.s[0] = SmallOrder{x, perm, k_in, i0, n, kb};
    return launch_small_orders(ctx, P, 1);
  }
  hilbert_keys_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(x, i0, n, k_in, v_in, kb);
  TC_CUDA_TRY(cudaGetLastError());
  ctx->launches += 1;
  TC_CUDA_TRY(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, k_in, k_out, v_in, perm + i0, n, 0,
                                              kSphereKeyBits, ctx->stream));
  return TC_OK;
}

// The orders of up to three classes; those that fit one CTA share two launches.
int compute_orders(tc_ctx* ctx, const OrderJob* jobs, int count) {
  if (count < 0 || count > 3) {
    tc_record_error("internal: %d visiting orders (at most 3)", count);
    return TC_ERR_ARG;
  }
  size_t small = 0, large = 0, temp = 0;
  int rc;
  for (int c = 0; c < count; ++c) {
    const OrderJob& J = jobs[c];
    const int n = J.i1 - J.i0;
    if (n <= 0) continue;
    if ((long long)J.i1 > J.perm_len || (long long)J.i1 > J.x_len) {
      tc_record_error("visiting order of [%d,%d): %lld points, %lld order entries", J.i0, J.i1,
                      J.x_len, J.perm_len);
      return TC_ERR_ARG;
    }
    if (n <= kSmallOrder) {
      small += (size_t)n;
    } else {
      size_t t = 0;
      if ((rc = order_sort_bytes(n, &t))) return rc;
      temp = std::max(temp, t);
      large = std::max(large, (size_t)n);
    }
  }
  if ((rc = ctx->order_buf[0].ensure(std::max(small, large) * sizeof(unsigned)))) return rc;
  if (large && ((rc = ctx->order_buf[1].ensure(large * sizeof(unsigned))) ||
                (rc = ctx->order_buf[2].ensure(large * sizeof(int))) ||
                (rc = ctx->order_buf[3].ensure(temp))))
    return rc;
  SmallOrders P{};
  int smalls = 0;
  long long used = 0;
  const long long cap = (long long)(ctx->order_buf[0].bytes / sizeof(unsigned));
  for (int c = 0; c < count; ++c) {
    const OrderJob& J = jobs[c];
    const int n = J.i1 - J.i0;
    if (n <= 0 || n > kSmallOrder) continue;
    const KeyBounds kb{ctx->bc_rec, bc_extent(ctx, BC_ORDER_X, J.x_len),
                       bc_extent(ctx, BC_ORDER_KEYS, cap - used)};
    P.s[smalls++] =
        SmallOrder{J.x, J.perm, ctx->order_buf[0].as<unsigned>() + used, J.i0, n, kb};
    used += n;
  }
  if (smalls && (rc = launch_small_orders(ctx, P, smalls))) return rc;
  // one class after the other: they share the keys' and the sort's buffers
  for (int c = 0; c < count; ++c) {
    const OrderJob& J = jobs[c];
    if (J.i1 - J.i0 <= kSmallOrder) continue;
    const long long key_len = (long long)std::min(
        {ctx->order_buf[0].bytes / sizeof(unsigned), ctx->order_buf[1].bytes / sizeof(unsigned),
         ctx->order_buf[2].bytes / sizeof(int)});
    if ((rc = compute_order_into(ctx, J.x, J.i0, J.i1, J.perm, ctx->order_buf[0].as<unsigned>(),
                                 ctx->order_buf[1].as<unsigned>(), ctx->order_buf[2].as<int>(),
                                 ctx->order_buf[3].ptr, temp,
                                 OrderExtents{J.x_len, J.perm_len, key_len})))
      return rc;
  }
  return TC_OK;
}

// FP64 targets are visited in order where that pays. The refinement's panel order
// is compact already, the particles' creation order is not, and a CTA whose targets
// lie all over the sphere runs the 13-operation wide form instead of the 9-operation
// frame form. Pair launches in the given order and sorted: level 4 (3.9e7 pairs)
// 45.5 and 43.3 us, level 4 refined (6.7e7) 61.7 and 54.5, level 5 (6.3e8) 515 and
// 455; the sort's two launches take 13 to 18 us once in a step of four. So: from
// 2e8 pairs a call, and 2,048 targets, below which a tile covers too much of the
// sphere for the frame form.
bool wants_order(const tc_ctx* ctx, long long most_targets, double pairs) {
  if (ctx->target_order != TC_ORDER_HILBERT) return false;
  if (ctx->precision == TC_FP32C) return true;
  return most_targets >= 2048 && pairs >= 2e8;
}

}  // namespace tcb
