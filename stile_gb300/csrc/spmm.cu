// SpMM kernels for sm_103a.
//
//  * csr_spmm_kernel     plain CSR-row SpMM (the comparator)
//  * zero_rows_kernel    zeroes output rows that no owned tile stores
//  * spmm_tc_kernel      dense 16-row block tiles on the tensor cores
//                        (tcgen05.mma, accumulator in TMEM): gathering warps
//                        that hold the rows in registers + an MMA warp (bf16 /
//                        fp16 / fp8, and split-bf16 hi+lo products with
//                        periodic accumulator drains for fp32-level accuracy)
//  * spmm_ell_seg_kernel ELL row-bucket tiles on CUDA cores, as a stream of
//                        live entries cut into groups at row boundaries
//                        The two launches together are the reference's
//                        horizontally fused kernel (my_fuse_formats.py:2437):
//                        the same tiles, split by template into two grids so
//                        that each gets its own block shape and shared memory.
//  * dvals               value gradient <dY[row], B[col]> for every nonzero,
//                        over an entry list built from the same tiles (the
//                        SDDMM entry-list kernel of sddmm.cu)
//  * pack_values_kernel  the tile values from CSR-ordered values (refresh, batched sets)
#include "common.cuh"
#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <type_traits>

#include "spmm.cuh"

namespace stile {

// ===========================================================================
// plain CSR SpMM (the comparator)
// ===========================================================================
// Nonzero-balanced CSR: every LPR-lane group owns kCsrNnz consecutive
// nonzeros, takes its first row from group_rows (or, when that is NULL,
// from a binary search in indptr) and walks the
// rows it touches (4 B rows in flight per lane).  A row lying wholly inside
// the range is stored; a row that straddles a range boundary is accumulated
// with atomics into a row that csr_prezero_kernel zeroed first.
constexpr int kCsrNnz = kCsrGroupNnz;

__device__ __forceinline__ int row_of_nnz(const int* __restrict__ indptr, int M, long t) {
  // largest r with indptr[r] <= t
  int lo = 0, hi = M;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (indptr[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void csr_prezero_kernel(int M, const int* __restrict__ indptr, float* __restrict__ C, long ldc,
                                   int N) {
  // one thread per row: rows without nonzeros and rows that straddle a
  // range boundary (accumulated with atomics) start at zero
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= M) return;
  const long rb = indptr[r], re = indptr[r + 1];
  const bool empty = rb == re;
  const bool split = !empty && (rb / kCsrNnz) != ((re - 1) / kCsrNnz);
  if (!empty && !split) return;
  float* row = C + (long)r * ldc;
  for (int f = 0; f < N; f += 4) st_row4(row, f, N, make_float4(0.f, 0.f, 0.f, 0.f));
}

template <int LPR>
__global__ void __launch_bounds__(256) csr_spmm_kernel(int M, const int* __restrict__ indptr,
                                                       const int* __restrict__ indices,
                                                       const float* __restrict__ vals,
                                                       const float* __restrict__ B, long ldb,
                                                       float* __restrict__ C, long ldc, int N,
                                                       int n_groups, const int* __restrict__ group_rows) {
  const int lane = threadIdx.x & 31;
  const int sub = lane / LPR, sl = lane % LPR;
  const int g = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (kWarp / LPR) + sub;
  if (g >= n_groups) return;
  const long nnz = indptr[M];
  const long t0 = (long)g * kCsrNnz;
  const long t1 = min(t0 + kCsrNnz, nnz);
  int r = group_rows ? __ldg(group_rows + g) : row_of_nnz(indptr, M, t0);
  long t = t0;
  while (r < M && t < t1) {
    const long rb = indptr[r], re = indptr[r + 1];
    const long a = max(rb, t0), b = min(re, t1);
    if (a >= b) {  // empty row (already zero)
      t = re;
      ++r;
      continue;
    }
    const bool whole = (rb >= t0) && (re <= t1);
    for (int fc = 0; fc < N; fc += 4 * LPR) {
      const int f = fc + 4 * sl;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      long k = a;
      for (; k + 4 <= b; k += 4) {
        const int c0 = __ldg(indices + k), c1 = __ldg(indices + k + 1), c2 = __ldg(indices + k + 2),
                  c3 = __ldg(indices + k + 3);
        const float v0 = __ldg(vals + k), v1 = __ldg(vals + k + 1), v2 = __ldg(vals + k + 2),
                    v3 = __ldg(vals + k + 3);
        const float4 b0 = ld_row4(B + (long)c0 * ldb, f, N);
        const float4 b1 = ld_row4(B + (long)c1 * ldb, f, N);
        const float4 b2 = ld_row4(B + (long)c2 * ldb, f, N);
        const float4 b3 = ld_row4(B + (long)c3 * ldb, f, N);
        fma4(acc, v0, b0);
        fma4(acc, v1, b1);
        fma4(acc, v2, b2);
        fma4(acc, v3, b3);
      }
      for (; k < b; ++k) fma4(acc, __ldg(vals + k), ld_row4(B + (long)__ldg(indices + k) * ldb, f, N));
      if (whole) st_row4(C + (long)r * ldc, f, N, acc); else red_row4(C + (long)r * ldc, f, N, acc);
    }
    t = re;
    ++r;
  }
}

// ===========================================================================
// zero rows
// ===========================================================================
__global__ void zero_rows_kernel(const int* __restrict__ rows, int n_rows, float* __restrict__ C,
                                 long ldc, int N, long c_head_stride) {
  // one warp per row, float4 stores.  Launched dependent on the previous
  // kernel, whose reads of C must be done first; the ELL kernel may launch
  // meanwhile (it waits for this grid before adding into these rows)
  griddep_wait();
  griddep_launch_dependents();
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp_global >= n_rows) return;
  float* row = C + blockIdx.y * c_head_stride + (long)rows[warp_global] * ldc;
  for (int f = 4 * lane; f < N; f += 128) st_row4(row, f, N, make_float4(0.f, 0.f, 0.f, 0.f));
}

// ===========================================================================
// hybrid SpMM: tensor-core kernel + ELL kernel (launched back to back)
// ===========================================================================
// Tensor-core chunks.  A chunk is a run of at most kChunkSteps k-steps of
// one item (items longer than that are split; the parts add into rows that
// another writer initialises).  Per k-step the kernel gathers the 16
// referenced B rows (fp32, 128 features) and the step's 16x16 value image,
// converts the rows to the bf16 / fp16 A-operand image and one thread
// issues the tcgen05.mma.
//
// Shared-memory operand layouts (checked by the layout probe):
//   A: [128 features (M) x 16 k (K)], MN-major, 128-byte swizzle: two
//      64-feature atoms (LBO 2048 B), two 8-row k groups (SBO 1024 B)
//   B: the 16x16 block values (N = 16 rows x K = 16), K-major, no swizzle:
//      core matrices 8 rows x 16 B, LBO 128 B (k), SBO 256 B (rows); the
//      plan stores this image and it is used in place.
constexpr uint32_t kAStage = 4096;   // bytes of one A image (16-bit)
constexpr uint32_t kBStage = 512;    // bytes of one B image (16-bit)
constexpr uint32_t kALbo = 2048, kASbo = 1024;
constexpr uint32_t kBLbo = 128, kBSbo = 256;
// fp8 operands (K = 32 bytes, K-major, no swizzle): core matrices of 8 rows
// x 16 bytes, the two k halves 128 B apart (LBO), 8-row groups 256 B apart
// (SBO); the A image is 4 KB, a k-step's value image 512 B
constexpr uint32_t kF8Lbo = 128, kF8Sbo = 256;
constexpr float kE4m3Max = 448.f;

__device__ __forceinline__ uint32_t a_img_off(int m, int k) {
  // m: feature (0..127), k: column within the k-step (0..15)
  const int atom = m >> 6, grp = k >> 3, r = k & 7, chunk = (m & 63) >> 3;
  return (uint32_t)(atom * kALbo + grp * kASbo + r * 128 + ((chunk ^ r) << 4) + (m & 7) * 2);
}

// Tensor-core kernel.
//
// The upload assigns chunks to the kernel's CTAs (longest first, each to the
// least loaded CTA) and stores every CTA's k-steps contiguously, so a CTA's
// work is the step range [s_beg, s_beg + S), walked once per 128-feature
// slice; its units are (slice, accumulation unit) pairs in that order.
//  * Four gathering warps.  A stage is kSpw consecutive k-steps: 1 at 128
//    fp32 features a row, 2 or 4 where 64 or 32 features (or 16-bit rows)
//    leave a warp-wide 16-byte load room for 2 or 4 rows, so every stage is 16
//    loads of 512 bytes.  Warp w takes the stages w, w + 4, ...  It holds a
//    stage's rows in registers, converts them into its operand slot (A: the
//    features are M = 128) and at once loads its next stage's rows, which are
//    in flight while the MMA warp and the epilogue work.  The rows never pass
//    through a shared-memory stage: a gathered row costs the L1 / shared
//    memory pipe its load, half its bytes as operand image and the MMA's read
//    of that, where the cp.async stage of an earlier build added a write and a
//    read of the whole fp32 row.  Column ids and value images come by cp.async
//    two and one stages ahead.
//    16 gathering warps per SM at 96 registers spilled; 16 warps that each
//    owned accumulators made the sums depend on the split.
//  * The MMA warp takes the stages in order and accumulates the
//    k-steps of a unit one after another into one of kAccBufs 16-column
//    accumulators, so the sums do not depend on the warps' timing.
//  * Epilogue, by the gathering warps: before its stage in unit y a warp
//    writes its quarter of the features of every unit up to y - kLag - 1,
//    whose MMAs are long done.
// Bound by two chains, not by L2 or the tensor pipe: a stage's (wait, convert,
// issue, fence: about 1,400 cycles without contention) and the MMA warp's
// (about 350 cycles a stage, most of it barrier latency).  Three CTAs of 4 + 1
// warps per SM give the second chain three times; two of 7 + 1 warps left the
// gathering warps waiting 60% of their time for slots over wide B (pruned
// weight, N = 4096 in bf16: 133 against 119 us).  Forward of a graph (row tiles
// included), before -> after: 169,343 nodes, 1.17M nonzeros: N = 128 64 -> 58
// us, N = 41 80 -> 61 us, N = 256 in bf16 121 -> 97 us; 50,000 nodes, 2.4M
// nonzeros: N = 128 73 -> 63 us, N = 41 70 -> 50 us; a 4096^2 matrix in
// split-bf16 22 -> 13 us; a pruned 3072 x 768 weight at N = 4096 in bf16
// 223 -> 119 us, 768 x 3072 in fp32 156 -> 109 us.
// Every wait is bounded; a wait that gives up sets the error flag and ends
// that warp's work, and the others then end at their next (bounded) wait.
constexpr int kTcWarps = 4;                        // gathering warps
constexpr int kTcThreads = (kTcWarps + 1) * kWarp; // and the MMA warp
constexpr int kTcCtas = 3;                         // resident CTAs per SM (128 registers a thread)
constexpr int kAccBufs = 8;                        // accumulators of 16 TMEM columns
// units between a warp's stage and the ones it writes; a warp whose next stage
// is in unit y has written every unit below y - kLag, so the MMA of unit y or
// an earlier one finds its accumulator read
constexpr int kLag = 4;

// Split-bf16 (fp32-level accuracy) keeps hi and lo images of both operands:
// A = hi(B rows) | lo(B rows), values = hi | lo, and issues three MMAs per
// step (hi*hi + hi*lo + lo*hi); its units are 4 k-steps, summed in the
// epilogue's registers, which bounds the tensor core's accumulation chain: it
// truncates, so sums of one sign come out small by half a unit of the last
// place a step.  (8 k-steps a unit: 12.9 against 13.4 us on a 4096^2 matrix of
// 160k nonzeros at N = 64, but 3.1e-7 against 1.9e-7 of such a sum lost.)
template <int MODE, bool kIn16, int kRowF>
struct TcCfg {
  static constexpr bool kSplit = MODE == STILE_TC_SPLIT_BF16;
  static constexpr int kLanes = kRowF * (kIn16 ? 2 : 4) / 16;  // lanes that cover a gathered row
  static constexpr int kSpw = kWarp / kLanes;                  // k-steps per stage, rows per load
  static constexpr uint32_t kVals = kSplit ? 2 * kBStage : kBStage;  // value image(s) of a step
  // A image of a step: both 64-feature atoms, or only the one that narrow
  // rows fill (the MMA then reads what follows it as its upper 64 features,
  // whose accumulator rows nobody reads; kTail keeps that inside the slots)
  static constexpr uint32_t kAOne = kRowF == 128 ? kAStage : kALbo;
  static constexpr uint32_t kAImg = kSplit ? 2 * kAOne : kAOne;
  static constexpr uint32_t kSlot = kSpw * kAImg;
  static constexpr int kNs = kSlot <= 4096 ? 2 : 1;  // operand slots per warp
  static constexpr int kNv = kNs + 1;                // value buffers per warp (one is being filled)
  static constexpr uint32_t kTail = kAStage - kAOne;
  static constexpr uint32_t kVBuf = kSpw * kVals;
  static constexpr uint32_t kCBuf = kSpw * 64;       // column ids of a stage; two per warp
  static constexpr uint32_t kVOff = kTcWarps * kNs * kSlot + kTail;
  static constexpr uint32_t kCOff = kVOff + kTcWarps * kNv * kVBuf;
  static constexpr uint32_t kBars = kCOff + kTcWarps * 2 * kCBuf;
  // full and empty per slot, full and empty per accumulator, drain, TMEM address
  static constexpr uint32_t kBytes = 1024 + kBars + 16 * kTcWarps * kNs + 16 * kAccBufs + 16;
  static_assert(kSpw == 1 || kSpw == 2 || kSpw == 4, "a stage is 16 loads");
  // a stage holds k-steps of up to kSpw units: a warp that waits with a stage
  // which begins in unit y has not written unit y - kLag, and the MMA warp may
  // wait for that stage in unit y + kSpw - 1
  static_assert(kLag + kSpw - 1 < kAccBufs, "the MMA warp waits for accumulators that every warp has passed");
  static_assert(!(kIn16 && MODE != STILE_TC_BF16), "a bf16 B feeds bf16 MMAs");
  static_assert(MODE != STILE_TC_FP8 || kSpw == 1, "fp8 converts whole 16-row stages");
  static_assert(kTcCtas * (kBytes + 1024) <= 228 * 1024, "resident CTAs");
};

// one warp's bounded wait; the same answer in every lane
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, uint32_t polls) {
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, polls));
}

// kFull: every feature slice is complete (N % kRowF == 0)
// kBig: a row of B or C is 4 GB or longer (64-bit row strides)
template <int MODE, bool kFull, bool kIn16, int kRowF, bool kBig>
__global__ void __launch_bounds__(kTcThreads, kTcCtas) spmm_tc_kernel(SpmmArgs p) {
  using W = TcCfg<MODE, kIn16, kRowF>;
  constexpr int kSpw = W::kSpw, kNs = W::kNs, kNv = W::kNv;
  griddep_launch_dependents();  // the next kernel waits for this grid before using its results
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  // slot s of warp w: image at base + (kNs w + s) kSlot, barriers full and
  // empty at bars + 8 (kNs w + s) and kNs kTcWarps further
  const uint32_t bars = base + W::kBars;
  const uint32_t full0 = bars, empty0 = bars + 8 * kTcWarps * kNs;
  const uint32_t accf0 = empty0 + 8 * kTcWarps * kNs, acce0 = accf0 + 8 * kAccBufs;
  const uint32_t drain = acce0 + 8 * kAccBufs, tmem_slot = drain + 8;

  // this CTA's first unit, units, first k-step and k-steps
  const int4 cta = __ldg(p.tc_cta_info + blockIdx.y);
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * kTcWarps * kNs; ++s) mbar_init(full0 + 8 * s, 1);
    for (int b = 0; b < kAccBufs; ++b) {
      mbar_init(accf0 + 8 * b, 1);
      mbar_init(acce0 + 8 * b, kTcWarps);
    }
    mbar_init(drain, 1);
    fence_mbar_init();
  }
  if constexpr (MODE == STILE_TC_FP8) {
    // the A images' upper k halves stay zero (each k-step fills the lower
    // half of a K = 32 operand); made visible to the tensor core's proxy
    for (int i = threadIdx.x; i < (int)(kTcWarps * kNs * W::kSlot / 16); i += kTcThreads)
      st_shared_v4(base + 16 * i, make_uint4(0u, 0u, 0u, 0u));
    fence_proxy_async_smem();
  }
  if (warp == kTcWarps) {
    __syncwarp();
    tmem_alloc(tmem_slot, 16 * kAccBufs);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");

  const int ub = cta.x, nu = cta.y, s_beg = cta.z, S = cta.w;
  // feature slices of this CTA: blockIdx.x takes [sl0, sl0 + nf) (a wide B
  // spreads its slices over more CTAs than the schedule has)
  const int sl0 = blockIdx.x * p.tc_slice_per;
  const int nf = nu > 0 ? min(p.tc_slice_per, p.n_fchunks - sl0) : 0;
  const int Q = (S + kSpw - 1) / kSpw;  // stages per slice
  const int n_units = nu * nf;
  const int N = p.N;
  const uint32_t polls = p.poll_limit ? p.poll_limit : kDefaultPolls;  // pipeline waits
  bool ok = true;

  if (warp == kTcWarps) {
    // ---------------- MMA warp ----------------
    {
      const bool on = elect_one();
      // kind::f16 with MN-major A; fp8: e4m3 x e4m3, both operands K-major
      constexpr uint32_t idesc = (MODE == STILE_TC_F16)   ? make_idesc(0, 0, 1, 0, 128, 16)
                                 : (MODE == STILE_TC_FP8) ? make_idesc(0, 0, 0, 0, 128, 16)
                                                          : make_idesc(1, 1, 1, 0, 128, 16);
      // failure-detection test: nothing arrives on `drain` before the commit
      // below, so this wait runs out
      if (p.stall_test && !warp_wait(drain, 0u, polls)) ok = false;
      int w = 0, round = 0, rv = 0;  // the stage's warp; its how-manieth stage (and that modulo kNv)
      int l = 0, u1 = 0;             // step in the slice, unit in the slice
      int n = n_units > 0 ? __ldg(p.tc_unit_meta + ub) & 0xffff : 0;
#pragma unroll 1
      for (int t = 0; t < n_units && ok; ++t) {
        const int b = t % kAccBufs;
        u1 = u1 + 1 < nu ? u1 + 1 : 0;
        const int n1 = __ldg(p.tc_unit_meta + ub + u1) & 0xffff;
        if (t >= kAccBufs && !warp_wait(acce0 + 8 * b, (uint32_t)(t / kAccBufs - 1) & 1u, polls)) {
          ok = false;
          break;
        }
        const uint32_t d = tmem + (uint32_t)(16 * b);
#pragma unroll 1
        for (int s = 0; s < n; ++s) {
          const int j = l % kSpw;
          const int slot = kNs * w + (kNs == 2 ? round & 1 : 0);
          if (j == 0 && !warp_wait(full0 + 8 * slot, (uint32_t)(round / kNs) & 1u, polls)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = base + slot * W::kSlot + j * W::kAImg;
          const uint32_t sv = base + W::kVOff + (kNv * w + rv) * W::kVBuf + j * W::kVals;
          if constexpr (MODE == STILE_TC_FP8) {
            umma_f8_if(on, d, smem_desc(sa, kF8Lbo, kF8Sbo, kSwizzleNone), smem_desc(sv, kF8Lbo, kF8Sbo, kSwizzleNone),
                    idesc, s > 0 ? 1u : 0u);
          } else {
            const uint64_t a_hi = smem_desc(sa, kALbo, kASbo, kSwizzle128B);
            const uint64_t v_hi = smem_desc(sv, kBLbo, kBSbo, kSwizzleNone);
            umma_f16_if(on, d, a_hi, v_hi, idesc, s > 0 ? 1u : 0u);
            if constexpr (W::kSplit) {
              umma_f16_if(on, d, a_hi, smem_desc(sv + kBStage, kBLbo, kBSbo, kSwizzleNone), idesc, 1u);
              umma_f16_if(on, d, smem_desc(sa + W::kAOne, kALbo, kASbo, kSwizzle128B), v_hi, idesc, 1u);
            }
          }
          ++l;
          if (j == kSpw - 1 || l == S) {  // the stage's last k-step
            umma_commit_if(on, empty0 + 8 * slot);
            if (++w == kTcWarps) {
              w = 0;
              ++round;
              rv = rv + 1 < kNv ? rv + 1 : 0;
            }
          }
          if (l == S) l = 0;
        }
        if (ok) umma_commit_if(on, accf0 + 8 * b);
        n = n1;
      }
      // every MMA this thread issued has completed before TMEM is freed
      umma_commit_if(on, drain);
      if (!warp_wait(drain, 0u, kDefaultPolls)) ok = false;
      if (!ok && lane == 0) atomicOr(p.err_flag, 1);
    }
    __syncwarp();
    griddep_wait();
  } else {
    // ---------------- gathering warps ----------------
    // lane -> k-step rsub of the stage, features fl .. of the slice
    using T = typename std::conditional<kIn16, uint16_t, float>::type;
    const int rsub = lane / W::kLanes, fl = (lane % W::kLanes) * (kIn16 ? 8 : 4);
    // row strides in bytes (one 32 x 32 + 64 bit multiply-add a row)
    using Stride = typename std::conditional<kBig, unsigned long long, unsigned>::type;
    const Stride ldb = (Stride)(p.ldb * (long)sizeof(T)), ldc = (Stride)(p.ldc * 4);
    auto at = [](const char* from, Stride ld, int row) {
      return kBig ? from + (unsigned long long)row * ld : from + (unsigned long long)(unsigned)row * (unsigned)ld;
    };
    const char* Bl = reinterpret_cast<const char*>(reinterpret_cast<const T*>(p.B) + blockIdx.z * p.b_head_stride + fl);
    const uint32_t cbuf = base + W::kCOff + warp * 2 * W::kCBuf;
    const uint32_t vbuf = base + W::kVOff + warp * kNv * W::kVBuf;
    // column ids of stage q into buffer b (past the slice's k-steps: column
    // 0, a valid row that no MMA reads)
    const int* my_cols = p.tc_cols + (long)s_beg * 16 + lane * 4;
    auto copy_cols = [&](int b, int q) {
      if (lane < 4 * kSpw) {
        const bool in = kSpw == 1 || q * kSpw + (lane >> 2) < S;
        cp_async16(cbuf + b * W::kCBuf + lane * 16, in ? my_cols + (long)q * kSpw * 16 : p.tc_cols, in ? 16u : 0u);
      }
    };
    uint4 v[16];  // row i of k-step rsub
    // loads the rows of the stage whose ids are in buffer b; from: this
    // lane's features of the slice in row 0
    auto load_rows = [&](int b, const char* from, bool live) {
      int c[16];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 x = ld_shared_v4(cbuf + b * W::kCBuf + rsub * 64 + 16 * j);
        c[4 * j] = (int)x.x;
        c[4 * j + 1] = (int)x.y;
        c[4 * j + 2] = (int)x.z;
        c[4 * j + 3] = (int)x.w;
      }
      // features past N inside the last 16 bytes are the row's padding: they
      // only reach accumulator rows that are never stored
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = (kFull || live) ? ldg_u4(at(from, ldb, c[i])) : make_uint4(0u, 0u, 0u, 0u);
    };
    const uint8_t* my_vals = reinterpret_cast<const uint8_t*>(p.tc_vals) + blockIdx.z * p.tc_vals_head_stride +
                             (long)s_beg * W::kVals + lane * 16;
    auto copy_vals = [&](uint32_t to, int q) {
      const uint8_t* src = my_vals + (long)q * W::kVBuf;
#pragma unroll
      for (int c = 0; c < (int)(W::kVBuf / 512); ++c)
        if (kSpw == 1 || q * kSpw + c * 512 / (int)W::kVals < S)
          cp_async16(to + lane * 16 + c * 512, src + c * 512, 16u);
    };
    // fp8: B's e4m3 scale comes from the run's amax pass, which finished
    // before this kernel started (an ordinary launch never lets a dependent
    // start early)
    float xinv = 1.f;
    if constexpr (MODE == STILE_TC_FP8) {
      const float amax = __uint_as_float(*p.tc_xamax);
      xinv = amax > 0.f ? kE4m3Max / amax : 0.f;
    }

    // ---- epilogue: the next unit to write, its slice, its meta and output
    // rows (those of the one after it are loaded while it is written)
    const int quarter = warp & 3;
    const int* my_rows = p.tc_unit_rows + (long)ub * 16 + (lane & 15);
    int e = 0, eu = 0, esl = 0;
    int meta = n_units > 0 ? __ldg(p.tc_unit_meta + ub) : 0, rows = n_units > 0 ? __ldg(my_rows) : -1;
    bool waited = false;  // griddep_wait done
    constexpr int kKeep = W::kSplit ? 2 : 1;  // split-bf16 keeps the sums over the units of a chunk
    float acc[kKeep][8];
    // writes units up to and without `upto`
    auto write_units = [&](int upto) {
#pragma unroll 1
      while (e < upto) {
        if (!waited) {
          // launched dependent on the ELL kernel: the gathers and MMAs start
          // while it drains, the C writes (adds to rows it stores) wait for it
          griddep_wait();
          waited = true;
        }
        const int b = e % kAccBufs;
        const int eu1 = eu + 1 < nu ? eu + 1 : 0;
        const int meta1 = __ldg(p.tc_unit_meta + ub + eu1), rows1 = __ldg(my_rows + (long)eu1 * 16);
        if (!warp_wait(accf0 + 8 * b, (uint32_t)(e / kAccBufs) & 1u, polls)) {
          ok = false;
          return;
        }
        tc_fence_after();
        const bool live = 32 * quarter < kRowF;  // narrow rows: the upper quarters' features do not exist
        const int f = (sl0 + esl) * 128 + 32 * quarter + lane;
        const char* Cf = reinterpret_cast<const char*>(p.C + blockIdx.z * p.c_head_stride + f);
        const bool in = (kFull && kRowF == 128) || f < N;
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // rows 0-7, 8-15 of the tile
          if (!live) continue;
          uint32_t r[8];
          tmem_ld8(tmem + (uint32_t)(16 * b + 8 * h) + ((uint32_t)(32 * quarter) << 16), r);
          tmem_wait_ld();
          float(&a)[8] = acc[W::kSplit ? h : 0];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            a[i] = W::kSplit ? ((meta & kUnitFirst) ? 0.f : a[i]) + __uint_as_float(r[i]) : __uint_as_float(r[i]);
          if (W::kSplit && !(meta & kUnitLast)) continue;
          if constexpr (MODE == STILE_TC_FP8) {
            // undo the scales: B's (per tensor) and the tile row's
            const float sx = __uint_as_float(*p.tc_xamax) / kE4m3Max;
            const int item = __ldg(p.tc_unit_item + ub + eu);
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] *= sx * __ldg(p.tc_row_scale + (long)item * 16 + 8 * h + i);
          }
          int row[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) row[i] = __shfl_sync(0xffffffffu, rows, 8 * h + i);
          if (meta & kUnitAdds) {
#pragma unroll
            for (int i = 0; i < 8; ++i) red_if(row[i] >= 0 && in, const_cast<char*>(at(Cf, ldc, row[i])), a[i]);
          } else {
            // C is not read again: evict first
#pragma unroll
            for (int i = 0; i < 8; ++i) st_if(row[i] >= 0 && in, const_cast<char*>(at(Cf, ldc, row[i])), a[i]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acce0 + 8 * b);
        ++e;
        eu = eu1;
        if (eu == 0) ++esl;
        meta = meta1;
        rows = rows1;
      }
    };

    // stage cursors: (sl, q) the stage in registers, (sl1, q1) the next one
    auto advance = [&](int& sl, int& q) {
      q += kTcWarps;
      while (q >= Q) {
        q -= Q;
        ++sl;
      }
    };
    const int* my_unit = p.tc_step_unit + s_beg;  // unit (in the slice) of a k-step
    int sl = nf, q = warp;
    if (n_units > 0) {
      sl = 0;
      while (q >= Q) {
        q -= Q;
        ++sl;
      }
    }
    int sl1 = sl, q1 = q, unit = 0, vb = 0, done = 0;
    if (sl < nf) {
      copy_cols(0, q);
      cp_async_commit();
      advance(sl1, q1);
      unit = sl * nu + __ldg(my_unit + q * kSpw);
      cp_async_wait<0>();
      __syncwarp();
      copy_vals(vbuf, q);
      if (sl1 < nf) copy_cols(1, q1);
      cp_async_commit();
      load_rows(0, Bl + (sl0 + sl) * 128 * (long)sizeof(T), (sl0 + sl) * 128 + fl < N);
    }
    const uint32_t a0 = base + kNs * warp * W::kSlot + (uint32_t)rsub * W::kAImg + a_img_off(fl, 0);
#pragma unroll 1
    for (;;) {
      // write the units well behind this warp's next stage (all of them after
      // its last one) while the stage's rows arrive
      write_units(sl < nf ? unit - kLag : n_units);
      if (!ok || sl >= nf) break;
      cp_async_wait<0>();
      __syncwarp();  // this stage's values and the next one's column ids are there
      // the MMAs of the slot's last stage have read it and its values
      const int slot = kNs * warp + (kNs == 2 ? done & 1 : 0);
      if (done >= kNs && !warp_wait(empty0 + 8 * slot, (uint32_t)(done / kNs - 1) & 1u, polls)) {
        ok = false;
        break;
      }
      const bool more = sl1 < nf;
      int sl2 = sl1, q2 = q1, unit1 = 0;
      vb = vb + 1 < kNv ? vb + 1 : 0;  // the next stage's value buffer
      if (more) {
        unit1 = __ldg(my_unit + q1 * kSpw);
        copy_vals(vbuf + vb * W::kVBuf, q1);
        advance(sl2, q2);
        if (sl2 < nf) copy_cols(done & 1, q2);
      }
      cp_async_commit();
      const uint32_t to0 = a0 + (kNs == 2 ? (done & 1) * W::kSlot : 0u);
      if constexpr (MODE == STILE_TC_FP8) {
        // this lane's 4 features x the step's 16 rows -> four K-major 16-byte
        // rows of the A image (feature m: the e4m3 bytes of x / s_x for
        // k = 0..15), core matrices of 8 features x 16 bytes
        uint32_t wd[4][4];
#pragma unroll
        for (int r = 0; r < 16; r += 2) {
          const uint32_t ua[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
          const uint32_t ub4[4] = {v[r + 1].x, v[r + 1].y, v[r + 1].z, v[r + 1].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t h = pack_e4m3x2(__uint_as_float(ua[j]) * xinv, __uint_as_float(ub4[j]) * xinv);
            if ((r & 2) == 0) wd[j][r >> 2] = h; else wd[j][r >> 2] |= h << 16;
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int m = 4 * lane + j;
          st_shared_v4(base + slot * W::kSlot + (uint32_t)((m >> 3) * kF8Sbo + (m & 7) * 16),
                       make_uint4(wd[j][0], wd[j][1], wd[j][2], wd[j][3]));
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          // the swizzle XORs the row's low bits into the 16-byte chunk; what
          // else a row adds to the address is a constant
          const uint32_t to = (to0 ^ (uint32_t)((i & 7) << 4)) + (uint32_t)((i >> 3) * kASbo + (i & 7) * 128);
          if constexpr (kIn16) {
            st_shared_v4(to, v[i]);
          } else {
            const float4 x = make_float4(__uint_as_float(v[i].x), __uint_as_float(v[i].y), __uint_as_float(v[i].z),
                                         __uint_as_float(v[i].w));
            if constexpr (MODE == STILE_TC_F16) {
              st_shared_v2(to, pack_f16x2(x.x, x.y), pack_f16x2(x.z, x.w));
            } else {
              const uint32_t h01 = pack_bf16x2(x.x, x.y), h23 = pack_bf16x2(x.z, x.w);
              st_shared_v2(to, h01, h23);
              if constexpr (W::kSplit) {
                // lo = x - float(hi): exact in fp32, then rounded to bf16
                st_shared_v2(to + W::kAOne,
                             pack_bf16x2(x.x - __uint_as_float(h01 << 16), x.y - __uint_as_float(h01 & 0xffff0000u)),
                             pack_bf16x2(x.z - __uint_as_float(h23 << 16), x.w - __uint_as_float(h23 & 0xffff0000u)));
              }
            }
          }
        }
      }
      if (more) {
        const char* from = Bl + (sl0 + sl1) * 128 * (long)sizeof(T);
        load_rows((done + 1) & 1, from, (sl0 + sl1) * 128 + fl < N);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full0 + 8 * slot);
      ++done;
      unit = sl1 * nu + unit1;
      sl = sl1;
      q = q1;
      sl1 = sl2;
      q1 = q2;
    }
    cp_async_wait<0>();
    if (!waited) griddep_wait();
    if (!ok && lane == 0) atomicOr(p.err_flag, 1);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kTcWarps) tmem_dealloc(tmem, 16 * kAccBufs);
}

// ELL tiles as a stream of live entries in row order: records {column,
// 2 * row code + run end} and, apart from them, the values (a refresh of the
// values then writes 4 contiguous bytes an entry).  An LPR-lane
// sub-group owns one group of <= kSegNnz entries; each lane covers 4 * VEC
// features of a row, float4 w at features 4 (w LPR + lane), so that every
// load instruction of the sub-group reads 16 LPR contiguous bytes (whole
// 128-byte lines: the L1 tag stage, not DRAM, limits these gathers, and an
// interleaved 8-features-per-lane split touched twice the lines per
// instruction).  The sub-group holds the group's records LPR at a time
// (one per lane, the next LPR loaded while these are consumed), broadcasts
// them by shuffle, keeps 4 float4 B-row gathers in flight per lane and
// flushes the running sum after every entry that ends its row's run (store
// for a row the ELL kernel initialises, atomic add otherwise).  With
// VEC = 2 two sub-groups share every warp-wide shuffle and branch, so the
// instructions per gathered byte halve; no gather waits on a metadata load,
// and few registers leave room for many warps per SM.
// kFull: N % (4 * VEC * LPR) == 0, every lane's features are in range
// (otherwise a float4 that starts past N reads as zero).
// kAddr: how a B row's address is formed: kOff32, every row offset col * ldb
// fits in 31 bits; kRow32, a row is shorter than 4 GB (one 32 x 32 + 64 bit
// multiply-add a row: a graph at N = 200 117 us where the 64-bit product took
// 126; full rows gain another 2 to 10% from the 31-bit offset, which leaves a
// register free); kRow64, any.
// kSpanY: blockIdx.y takes features [y span, (y + 1) span) (a wide B over
// few groups; span = p.ell_fc_span, a multiple of the pass width).
// kHeads: a batched run (blockIdx.z = head offsets B, C and the values).
//
// entry i of a group of n as {column, value bits, 2 * row code + run end};
// past the group: column 0, value 0, no run end
__device__ __forceinline__ int3 ell_record(const int2* __restrict__ ent, const float* __restrict__ val, int i, int n) {
  if (i >= n) return make_int3(0, 0, 0);
  const int2 e = __ldcs(ent + i);
  return make_int3(e.x, __float_as_int(__ldcs(val + i)), e.y);
}

template <int LPR, int VEC, bool kFull, int kAddr, bool kSpanY = false, bool kHeads = false>
__global__ void __launch_bounds__(256, 5) spmm_ell_seg_kernel(SpmmArgs p) {
  constexpr int kBatch = 4 / VEC;  // entries per batch: 4 float4 in flight per lane
  // Launched dependent on the previous kernel.  When that is the zero-rows
  // kernel (p.ell_lazy_wait), only the atomic adds (into rows it zeroes)
  // wait for it, and every thread waits before it exits, so that this
  // grid's completion implies that kernel's; otherwise (B may come from the
  // previous kernel) everything waits.  The tensor-core kernel may launch
  // once this grid is running.
  if (!p.ell_lazy_wait) griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 31, sub = lane / LPR, sl = lane % LPR;
  const unsigned mask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << (sub * LPR));
  const int g = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (kWarp / LPR) + sub;
  if (g >= p.ell_n_groups) {  // the whole sub-group leaves together
    if (p.ell_lazy_wait) griddep_wait();
    return;
  }
  const int p0 = __ldg(p.ell_group_ptr + g);
  const int n = __ldg(p.ell_group_ptr + g + 1) - p0;
  const long head = kHeads ? blockIdx.z : 0;
  const int2* __restrict__ ent = p.ell_entry + p0;
  const float* __restrict__ val = p.ell_val + head * p.ell_n_pos + p0;
  const int N = p.N;
  // records are read once: streaming loads leave L2 to the B rows
  auto rec = [&](int i) { return ell_record(ent, val, i, n); };
  for (int fc = kSpanY ? blockIdx.y * p.ell_fc_span : 0;
       fc < (kSpanY ? min(N, (int)(blockIdx.y + 1) * p.ell_fc_span) : N); fc += 4 * VEC * LPR) {
    // float4 w of this lane holds features f + 4 LPR w: each load
    // instruction of the group reads 16 LPR contiguous bytes of a row
    const int f = fc + 4 * sl;
    const float* Bf = p.B + head * p.b_head_stride + f;
    float4 acc[VEC];
#pragma unroll
    for (int w = 0; w < VEC; ++w) acc[w] = make_float4(0.f, 0.f, 0.f, 0.f);
    int3 mcur = rec(sl);
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += LPR) {
      const int3 mnext = rec(c0 + LPR + sl);
#pragma unroll 1
      for (int b0 = c0; b0 < min(n, c0 + LPR); b0 += kBatch) {
        float4 bv[kBatch][VEC];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int c = __shfl_sync(mask, mcur.x, b0 - c0 + u, LPR);
          // records past n hold column 0: a valid row, multiplied by 0
          if (kFull) {
            const float* row = row_at<kAddr>(Bf, p.ldb, c);
#pragma unroll
            for (int w = 0; w < VEC; ++w) bv[u][w] = ldg4(row + 4 * LPR * w);
          } else {
            // float4 past N read as zero; padding features inside the last
            // live float4 only reach features that are never stored
            const float* row = row_at<kAddr>(p.B + head * p.b_head_stride, p.ldb, c);
#pragma unroll
            for (int w = 0; w < VEC; ++w) bv[u][w] = ld4_pad(row, f + 4 * LPR * w, N);
          }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const float v = __int_as_float(__shfl_sync(mask, mcur.y, b0 - c0 + u, LPR));
          const int ce = __shfl_sync(mask, mcur.z, b0 - c0 + u, LPR);
#pragma unroll
          for (int w = 0; w < VEC; ++w) fma4(acc[w], v, bv[u][w]);  // records past n: value 0, no run end
          if (ce & 1) {
            const int code = ce >> 1;
            float* row = p.C + head * p.c_head_stride + (long)(code >= 0 ? code : -code - 1) * p.ldc;
#pragma unroll
            for (int w = 0; w < VEC; ++w) {
              const int fw = f + 4 * LPR * w;
              if (code < 0 && p.ell_lazy_wait) griddep_wait();
              if (kFull) {
                if (code >= 0) __stcs(reinterpret_cast<float4*>(row + fw), acc[w]);  // evict first
                else atomicAdd(reinterpret_cast<float4*>(row + fw), acc[w]);
              } else {
                if (code >= 0) st_row4(row, fw, N, acc[w]); else red_row4(row, fw, N, acc[w]);
              }
              acc[w] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
          }
        }
      }
      mcur = mnext;
    }
  }
  if (p.ell_lazy_wait) griddep_wait();
}

// The fused backward's ELL pass, run over the transposed operator's tiles
// with B = dC: the stream kernel above for VEC = 2 in one feature pass
// (N <= 8 LPR), and for every entry (row r, column c) of A^T also
//   dv_out[id] = <dC[c], dvx[r]>,
// the value gradient of the forward's nonzero (c, r); id, in the forward's
// numbering, comes with the entry (ell_fid).  The dC row gathered
// for the product is the one the gradient needs; dvx[r] (the forward's
// dense operand) is loaded where a row run starts, for both entries of a
// batch before either is used, so those loads overlap the dC gathers.  The
// two entries reduce their dot products together with the transposing
// butterfly (lanes whose high bit spells the entry hold its sum).
// kFull: N == 8 LPR.
template <int LPR, bool kFull>
__global__ void __launch_bounds__(256, 4) spmm_ell_bwd_kernel(SpmmArgs p) {
  static_assert(LPR >= 2, "two entries per batch");
  if (!p.ell_lazy_wait) griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 31, sub = lane / LPR, sl = lane % LPR;
  const unsigned mask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << (sub * LPR));
  const int g = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (kWarp / LPR) + sub;
  if (g >= p.ell_n_groups) {  // the whole sub-group leaves together
    if (p.ell_lazy_wait) griddep_wait();
    return;
  }
  const int p0 = __ldg(p.ell_group_ptr + g);
  const int n = __ldg(p.ell_group_ptr + g + 1) - p0;
  const int2* __restrict__ ent = p.ell_entry + p0;
  const float* __restrict__ val = p.ell_val + p0;
  const int* __restrict__ fid = p.ell_fid + p0;
  const int N = p.N;
  // this lane's features: f .. f + 3 and f + 4 LPR .. f + 4 LPR + 3 (each
  // load instruction of the group reads 16 LPR contiguous bytes of a row)
  const int f = 4 * sl, f2 = f + 4 * LPR;
  auto rec = [&](int i) {
    const int3 r = ell_record(ent, val, i, n);
    return make_int4(r.x, r.y, r.z, i < n ? __ldcs(fid + i) : -1);
  };
  auto row_of = [](int ce) { const int code = ce >> 1; return code >= 0 ? code : -code - 1; };
  auto ld8 = [&](const float* row, float4& a, float4& b) {
    a = kFull ? ldg4(row + f) : ld4_live(row, f, N);
    b = kFull ? ldg4(row + f2) : ld4_live(row, f2, N);
  };
  float4 acc0 = make_float4(0.f, 0.f, 0.f, 0.f), acc1 = acc0;
  float4 xa0 = acc0, xa1 = acc0;  // dvx row of the last entry handled
  int xrow = -1;
  int4 mcur = rec(sl);
#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += LPR) {
#pragma unroll 1
    for (int b0 = c0; b0 < min(n, c0 + LPR); b0 += 2) {
      const int j = b0 - c0;
      const int col0 = __shfl_sync(mask, mcur.x, j, LPR), col1 = __shfl_sync(mask, mcur.x, j + 1, LPR);
      const int ce0 = __shfl_sync(mask, mcur.z, j, LPR), ce1 = __shfl_sync(mask, mcur.z, j + 1, LPR);
      const float v0 = __int_as_float(__shfl_sync(mask, mcur.y, j, LPR));
      const float v1 = __int_as_float(__shfl_sync(mask, mcur.y, j + 1, LPR));
      const int id0 = __shfl_sync(mask, mcur.w, j, LPR), id1 = __shfl_sync(mask, mcur.w, j + 1, LPR);
      const int r0 = row_of(ce0), r1 = row_of(ce1);
      // records past n: row 0, column 0, value 0, no run end, id -1
      float4 b00, b01, b10, b11;
      ld8(p.B + (long)col0 * p.ldb, b00, b01);
      ld8(p.B + (long)col1 * p.ldb, b10, b11);
      float4 x00 = xa0, x01 = xa1;
      if (r0 != xrow) ld8(p.dvx + (long)r0 * p.dvx_ld, x00, x01);
      float4 x10 = x00, x11 = x01;
      if (r1 != r0) ld8(p.dvx + (long)r1 * p.dvx_ld, x10, x11);
      xa0 = x10;
      xa1 = x11;
      xrow = r1;
      const float s0 = dot4(x00, b00) + dot4(x01, b01);
      const float s1 = dot4(x10, b10) + dot4(x11, b11);
      fma4(acc0, v0, b00);
      fma4(acc1, v0, b01);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int ce = u ? ce1 : ce0;
        if (u) {
          fma4(acc0, v1, b10);
          fma4(acc1, v1, b11);
        }
        if (ce & 1) {
          const int code = ce >> 1;
          float* crow = p.C + (long)(u ? r1 : r0) * p.ldc;
          if (code < 0 && p.ell_lazy_wait) griddep_wait();
          if (kFull) {
            if (code >= 0) {
              __stcs(reinterpret_cast<float4*>(crow + f), acc0);
              __stcs(reinterpret_cast<float4*>(crow + f2), acc1);
            } else {
              atomicAdd(reinterpret_cast<float4*>(crow + f), acc0);
              atomicAdd(reinterpret_cast<float4*>(crow + f2), acc1);
            }
          } else if (code >= 0) {
            st_row4(crow, f, N, acc0);
            st_row4(crow, f2, N, acc1);
          } else {
            red_row4(crow, f, N, acc0);
            red_row4(crow, f2, N, acc1);
          }
          acc0 = make_float4(0.f, 0.f, 0.f, 0.f);
          acc1 = acc0;
        }
      }
      // transposing butterfly over the pair: the upper half keeps entry 1
      const bool up = (sl & (LPR / 2)) != 0;
      float t = (up ? s1 : s0) + __shfl_xor_sync(mask, up ? s0 : s1, LPR / 2);
#pragma unroll
      for (int o = LPR / 4; o > 0; o >>= 1) t += __shfl_xor_sync(mask, t, o);
      const int id = up ? id1 : id0;
      if ((sl & (LPR / 2 - 1)) == 0 && id >= 0) __stcs(p.dv_out + id, t);
    }
    if (c0 + LPR < n) mcur = rec(c0 + LPR + sl);
  }
  if (p.ell_lazy_wait) griddep_wait();
}

__global__ void permute_ids_kernel(const int* __restrict__ in, long n, const int* __restrict__ perm,
                                   int* __restrict__ out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int v = in[i];
  out[i] = v >= 0 ? perm[v] : -1;
}

cudaError_t launch_permute_ids(const int* in, long n, const int* perm, int* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  permute_ids_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, n, perm, out);
  return cudaGetLastError();
}

// The same entry stream over a bf16 B: each lane covers 8 features with one
// 16-byte load (half the gathered bytes of fp32 rows), converts them to
// fp32 and accumulates in fp32; 4 entries' rows in flight per lane.
template <int LPR, bool kFull, int kAddr, bool kSpanY = false>
__global__ void __launch_bounds__(256, 4) spmm_ell_seg_bf16_kernel(SpmmArgs p) {
  constexpr int kBatch = 4;
  static_assert(LPR % kBatch == 0, "batches stay inside one record block");
  // Launched dependent on the previous kernel.  When that is the zero-rows
  // kernel (p.ell_lazy_wait), only the atomic adds (into rows it zeroes)
  // wait for it, and every thread waits before it exits, so that this
  // grid's completion implies that kernel's; otherwise (B may come from the
  // previous kernel) everything waits.  The tensor-core kernel may launch
  // once this grid is running.
  if (!p.ell_lazy_wait) griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 31, sub = lane / LPR, sl = lane % LPR;
  const unsigned mask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << (sub * LPR));
  const int g = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (kWarp / LPR) + sub;
  if (g >= p.ell_n_groups) {  // the whole sub-group leaves together
    if (p.ell_lazy_wait) griddep_wait();
    return;
  }
  const int p0 = __ldg(p.ell_group_ptr + g);
  const int n = __ldg(p.ell_group_ptr + g + 1) - p0;
  const int2* __restrict__ ent = p.ell_entry + p0;
  const float* __restrict__ val = p.ell_val + blockIdx.z * p.ell_n_pos + p0;
  const uint16_t* __restrict__ B16 = reinterpret_cast<const uint16_t*>(p.B) + blockIdx.z * p.b_head_stride;
  float* __restrict__ Ch = p.C + blockIdx.z * p.c_head_stride;
  const int N = p.N;
  // records are read once: streaming loads leave L2 to the B rows
  auto rec = [&](int i) { return ell_record(ent, val, i, n); };
  for (int fc = kSpanY ? blockIdx.y * p.ell_fc_span : 0;
       fc < (kSpanY ? min(N, (int)(blockIdx.y + 1) * p.ell_fc_span) : N); fc += 8 * LPR) {
    const int f = fc + 8 * sl;
    float4 acc0 = make_float4(0.f, 0.f, 0.f, 0.f), acc1 = acc0;
    int3 mcur = rec(sl);
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += LPR) {
      const int3 mnext = rec(c0 + LPR + sl);
#pragma unroll 1
      for (int b0 = c0; b0 < min(n, c0 + LPR); b0 += kBatch) {
        uint4 bv[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int c = __shfl_sync(mask, mcur.x, b0 - c0 + u, LPR);
          // records past n hold column 0: a valid row, multiplied by 0
          const uint16_t* row = row_at<kAddr>(B16, p.ldb, c);
          bv[u] = kFull ? ldg_u4(row + f) : ld_row8_bf16(row, f, N);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const float v = __int_as_float(__shfl_sync(mask, mcur.y, b0 - c0 + u, LPR));
          const int ce = __shfl_sync(mask, mcur.z, b0 - c0 + u, LPR);
          float4 lo, hi;
          bf16x8_to_f32(bv[u], lo, hi);
          fma4(acc0, v, lo);
          fma4(acc1, v, hi);
          if (ce & 1) {
            const int code = ce >> 1;
            float* row = Ch + (long)(code >= 0 ? code : -code - 1) * p.ldc;
            if (code < 0 && p.ell_lazy_wait) griddep_wait();
            if (kFull) {
              if (code >= 0) {
                __stcs(reinterpret_cast<float4*>(row + f), acc0);
                __stcs(reinterpret_cast<float4*>(row + f + 4), acc1);
              } else {
                atomicAdd(reinterpret_cast<float4*>(row + f), acc0);
                atomicAdd(reinterpret_cast<float4*>(row + f + 4), acc1);
              }
            } else if (code >= 0) {
              st_row4(row, f, N, acc0);
              st_row4(row, f + 4, N, acc1);
            } else {
              red_row4(row, f, N, acc0);
              red_row4(row, f + 4, N, acc1);
            }
            acc0 = make_float4(0.f, 0.f, 0.f, 0.f);
            acc1 = acc0;
          }
        }
      }
      mcur = mnext;
    }
  }
  if (p.ell_lazy_wait) griddep_wait();
}

// ===========================================================================
// value gradient: dvals[t] = <dY[row(t)], B[col(t)]> over the plan's entry
// list (launch_dvals -> launch_sddmm_list)
// ===========================================================================

// ===========================================================================
// value refresh: the plan's tile values from CSR-ordered value arrays (new
// values on the same pattern; the value sets of a batched run)
// ===========================================================================
// Bound by memory: it reads every value once (a 32-byte sector per value,
// their order is the tiles', not the CSR's) and writes every tile value.  A
// warp takes kPackSteps k-steps of a tensor tile at a time: lane l owns the 8
// image elements 8l .. 8l + 7 of each, a byte of the k-step's mask says which
// of them hold a nonzero, their ids lie one after another, and the lane writes
// its 16 bytes of the image at once (the other elements are zero).  The ids of
// the dead elements are never read: a k-step of the 233k-node graph holds 41
// nonzeros of 256, 196 bytes of mask and ids in place of 1 KB.  The row-tile
// values are an array of their own, 4 entries a thread.  One launch takes the
// plan, the plan of the transposed operator (ids in the forward's numbering)
// and the operator's own copy of the values: blocks [0, a.blocks) the first,
// [a.blocks, a.blocks + b.blocks) the second, the rest copy.
// (233k-node graph, 11.4M nonzeros, both plans and the copy: 119 us; a launch
// each, one k-step a warp and a copy by torch 136 us.)
constexpr int kPackThreads = 256;
constexpr int kPackSteps = 2;

// one plan's part: k-steps by the first tc_blocks blocks, row-tile values by
// the others
template <int MODE>
__device__ __forceinline__ void pack_plan(const PackPlan& p, int block, const float* __restrict__ hv, long h,
                                          long tc_head_bytes) {
  if (block < p.tc_blocks) {
    constexpr uint32_t kBytes = MODE == STILE_TC_SPLIT_BF16 ? 2 * kBStage : kBStage;
    const int lane = threadIdx.x & 31;
    const int ks0 = (block * (kPackThreads / kWarp) + (threadIdx.x >> 5)) * kPackSteps;
    unsigned m[kPackSteps];
    const int* ids[kPackSteps];
#pragma unroll
    for (int s = 0; s < kPackSteps; ++s) {
      const bool in = ks0 + s < p.n_ks;
      m[s] = in ? __ldg(p.mask + (long)(ks0 + s) * 32 + lane) : 0u;
      ids[s] = p.ids + (in ? __ldg(p.ptr + ks0 + s) : 0);
    }
#pragma unroll
    for (int s = 0; s < kPackSteps; ++s) {
      int before = __popc(m[s]);  // inclusive scan of the lanes' counts
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += v;
      }
      ids[s] += before - __popc(m[s]);
    }
    float v[kPackSteps][8];
#pragma unroll
    for (int s = 0; s < kPackSteps; ++s) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool live = (m[s] >> j) & 1u;
        v[s][j] = live ? __ldg(hv + __ldcs(ids[s] + __popc(m[s] & ((1u << j) - 1u)))) : 0.f;
      }
    }
#pragma unroll
    for (int s = 0; s < kPackSteps; ++s) {
      if (ks0 + s >= p.n_ks) continue;
      uint4* out = reinterpret_cast<uint4*>(p.tc_out + h * tc_head_bytes + (long)(ks0 + s) * kBytes) + lane;
      const float(&x)[8] = v[s];
      if constexpr (MODE == STILE_TC_F16) {
        *out = make_uint4(pack_f16x2(x[0], x[1]), pack_f16x2(x[2], x[3]), pack_f16x2(x[4], x[5]),
                          pack_f16x2(x[6], x[7]));
      } else {
        uint32_t hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) hi[j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
        *out = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if constexpr (MODE == STILE_TC_SPLIT_BF16) {
          uint32_t lo[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            lo[j] = pack_bf16x2(x[2 * j] - __uint_as_float(hi[j] << 16),
                                x[2 * j + 1] - __uint_as_float(hi[j] & 0xffff0000u));
          out[kBStage / 16] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
    }
    return;
  }
  const long i = 4 * ((long)(block - p.tc_blocks) * kPackThreads + threadIdx.x);
  float* __restrict__ out = p.ell_out + h * p.n_ell;
  auto value = [&](int id) { return id >= 0 ? __ldg(hv + id) : 0.f; };
  if (i + 4 <= p.n_ell) {
    // the ids are 16-byte aligned; a head's values only when n_ell % 4 == 0
    const int4 id = __ldcs(reinterpret_cast<const int4*>(p.ell_ids + i));
    const float4 v = make_float4(value(id.x), value(id.y), value(id.z), value(id.w));
    if (((h * p.n_ell) & 3) == 0) {
      *reinterpret_cast<float4*>(out + i) = v;
    } else {
      out[i] = v.x;
      out[i + 1] = v.y;
      out[i + 2] = v.z;
      out[i + 3] = v.w;
    }
  } else {
    for (long j = i; j < p.n_ell; ++j) out[j] = value(__ldg(p.ell_ids + j));
  }
}

template <int MODE>
__global__ void __launch_bounds__(kPackThreads) pack_values_kernel(PackPlan a, PackPlan b,
                                                                   const float* __restrict__ vals, long nnz,
                                                                   long tc_head_bytes, float* __restrict__ copy) {
  const long h = blockIdx.y;
  const float* __restrict__ hv = vals + h * nnz;
  const int block = blockIdx.x;
  if (block < a.blocks) {
    pack_plan<MODE>(a, block, hv, h, tc_head_bytes);
  } else if (block < a.blocks + b.blocks) {
    pack_plan<MODE>(b, block - a.blocks, hv, h, tc_head_bytes);
  } else {
    // 4 values a thread, one every kPackThreads
    const long i0 = (long)(block - a.blocks - b.blocks) * 4 * kPackThreads + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long i = i0 + k * kPackThreads;
      if (i < nnz) copy[i] = __ldg(vals + i);
    }
  }
}

// bits of max |B| over K rows x N features into *out (atomicMax on the bits
// of non-negative floats, which order like the floats)
__global__ void amax_kernel(const float* __restrict__ B, long ldb, int K, int N, unsigned* __restrict__ out) {
  float m = 0.f;
  const long total = (long)K * N;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x)
    m = fmaxf(m, fabsf(B[(i / N) * ldb + i % N]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(out, __float_as_uint(m));
}

// Rows of `cols` elements (any row stride, any alignment) into rows of ld
// elements, zeros past cols: the operand rows of the gathering kernels are
// 16-byte vectors.  Bound by memory: a thread writes one 16-byte vector; its
// element loads share sectors with its neighbours' in L1.
template <typename T>
__global__ void __launch_bounds__(256) pad_rows_kernel(const T* __restrict__ src, long rows, int cols, long src_ld,
                                                       uint4* __restrict__ dst, unsigned vecs) {
  constexpr int kPer = 16 / sizeof(T);
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  const long r = i / vecs;
  if (r >= rows) return;
  const int c = (int)(i - r * vecs) * kPer;
  const T* from = src + r * src_ld + c;
  union {
    T e[kPer];
    uint4 v;
  } x;
#pragma unroll
  for (int k = 0; k < kPer; ++k) x.e[k] = c + k < cols ? __ldg(from + k) : T(0);
  dst[i] = x.v;
}

cudaError_t launch_pad_rows(const void* src, long rows, int cols, long src_ld, int elem_bytes, void* dst, long dst_ld,
                            cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const long vecs = dst_ld * elem_bytes / 16;
  const unsigned grid = (unsigned)((rows * vecs + 255) / 256);
  if (elem_bytes == 4)
    pad_rows_kernel<<<grid, 256, 0, st>>>(static_cast<const unsigned*>(src), rows, cols, src_ld,
                                          static_cast<uint4*>(dst), (unsigned)vecs);
  else
    pad_rows_kernel<<<grid, 256, 0, st>>>(static_cast<const unsigned short*>(src), rows, cols, src_ld,
                                          static_cast<uint4*>(dst), (unsigned)vecs);
  return cudaGetLastError();
}

cudaError_t launch_amax(const float* B, long ldb, int K, int N, unsigned* amax_bits, cudaStream_t st) {
  const long total = (long)K * N;
  if (total == 0) return cudaSuccess;
  const long cap = (long)device_sm_count() * 8;
  const long grid = std::min((total + 255) / 256, cap);
  amax_kernel<<<(unsigned)grid, 256, 0, st>>>(B, ldb, K, N, amax_bits);
  return cudaGetLastError();
}

PackPlan pack_of(const SpmmArgs& p, long n_ell, float* ell_out, void* tc_out, bool forward_ids) {
  constexpr int kPer = kPackThreads / kWarp * kPackSteps;
  PackPlan r{};
  r.mask = p.tc_live_mask;
  r.ptr = p.tc_live_ptr;
  r.ids = forward_ids ? p.tc_live_fid : p.tc_live_id;
  r.tc_out = static_cast<uint8_t*>(tc_out);
  r.n_ks = p.tc_n_ksteps;
  r.ell_ids = forward_ids ? p.ell_fid : p.ell_nnz_id;
  r.ell_out = ell_out;
  r.n_ell = n_ell;
  r.tc_blocks = (p.tc_n_ksteps + kPer - 1) / kPer;
  r.blocks = r.tc_blocks + (int)((n_ell + 4 * kPackThreads - 1) / (4 * kPackThreads));
  return r;
}

cudaError_t launch_pack_values(int tc_mode, const PackPlan& a, const PackPlan& b, const float* vals, long nnz,
                               int heads, long tc_head_bytes, float* copy, cudaStream_t st) {
  const long copy_blocks = copy ? (nnz + 4 * kPackThreads - 1) / (4 * kPackThreads) : 0;
  const long blocks = (long)a.blocks + b.blocks + copy_blocks;
  if (blocks == 0 || heads == 0) return cudaSuccess;
  auto k = tc_mode == STILE_TC_F16            ? pack_values_kernel<STILE_TC_F16>
           : tc_mode == STILE_TC_SPLIT_BF16 ? pack_values_kernel<STILE_TC_SPLIT_BF16>
                                            : pack_values_kernel<STILE_TC_BF16>;
  k<<<dim3((unsigned)blocks, (unsigned)heads), kPackThreads, 0, st>>>(a, b, vals, nnz, tc_head_bytes, copy);
  return cudaGetLastError();
}

// ===========================================================================
// host-side launchers
// ===========================================================================
static int lpr_for(int N) {
  const int lanes = (N + 3) / 4;
  if (lanes >= 32) return 32;
  int l = 1;
  while (l < lanes) l <<= 1;
  return l < 4 ? 4 : l;
}

template <template <int> class F, typename... Args>
static cudaError_t dispatch_lpr(int lpr, Args... args) {
  switch (lpr) {
    case 4: return F<4>::run(args...);
    case 8: return F<8>::run(args...);
    case 16: return F<16>::run(args...);
    default: return F<32>::run(args...);
  }
}

template <int LPR>
struct CsrLaunch {
  static cudaError_t run(int M, const int* indptr, const int* indices, const float* vals, const float* B,
                         long ldb, float* C, long ldc, int N, long nnz, const int* group_rows, cudaStream_t st) {
    const int n_groups = (int)((nnz + kCsrNnz - 1) / kCsrNnz);
    csr_prezero_kernel<<<(M + 255) / 256, 256, 0, st>>>(M, indptr, C, ldc, N);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    constexpr int GPB = 256 / LPR;
    const int grid = (n_groups + GPB - 1) / GPB;
    if (grid == 0) return cudaSuccess;
    csr_spmm_kernel<LPR><<<grid, 256, 0, st>>>(M, indptr, indices, vals, B, ldb, C, ldc, N, n_groups, group_rows);
    return cudaGetLastError();
  }
};

cudaError_t launch_csr_spmm(int M, const int* indptr, const int* indices, const float* vals,
                            const float* B, long ldb, float* C, long ldc, int N, long nnz,
                            const int* group_rows, cudaStream_t st) {
  return dispatch_lpr<CsrLaunch>(lpr_for(N), M, indptr, indices, vals, B, ldb, C, ldc, N, nnz, group_rows, st);
}

cudaError_t launch_zero_rows(const int* rows, int n, float* C, long ldc, int N, cudaStream_t st, int heads,
                             long c_head_stride) {
  if (n == 0 || heads == 0) return cudaSuccess;
  const int grid = (n + 7) / 8;
  return launch_dependent(zero_rows_kernel, dim3(grid, heads), dim3(256), 0, st, rows, n, C, ldc, N, c_head_stride);
}

// CTAs of `kernel` resident per SM at `threads` threads and `smem` bytes of
// dynamic shared memory, from the device's limits (shared memory with the
// per-block reservation, registers, threads, blocks); at least 1.
template <typename K>
static cudaError_t resident_ctas(K kernel, int threads, size_t smem, int* sms, int* per_sm) {
  int dev = 0, smem_sm = 0, reserved = 0, regs_sm = 0, thr_sm = 0, blk_sm = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess)
    return e;
  if ((e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess)
    return e;
  if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess)
    return e;
  if ((e = cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&blk_sm, cudaDevAttrMaxBlocksPerMultiprocessor, dev)) != cudaSuccess) return e;
  cudaFuncAttributes fa;
  if ((e = cudaFuncGetAttributes(&fa, kernel)) != cudaSuccess) return e;
  const int warps = (threads + 31) / 32;
  const int regs_warp = ((fa.numRegs * 32 + 255) / 256) * 256;
  const long by_smem = (long)smem_sm / (long)(smem + fa.sharedSizeBytes + reserved);
  const long by_regs = regs_warp > 0 ? (long)(regs_sm / regs_warp) / warps : blk_sm;
  const long by_thr = thr_sm / (warps * 32);
  long n = std::min(std::min(by_smem, by_regs), std::min(by_thr, (long)blk_sm));
  *per_sm = (int)std::max(1L, n);
  return cudaSuccess;
}

template <int MODE, bool kFull, bool kIn16 = false, int kRowF = 128, bool kBig = false>
static cudaError_t launch_tc_t(const SpmmArgs& p, cudaStream_t st) {
  // (the slice groups of a CTA's chunks are neighbours in the launch: the CTAs
  // with the longest chunks, the schedule's first ones, all start first)
  auto k = spmm_tc_kernel<MODE, kFull, kIn16, kRowF, kBig>;
  constexpr uint32_t kBytes = TcCfg<MODE, kIn16, kRowF>::kBytes;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBytes);
  if (e != cudaSuccess) return e;
  // shared memory for the resident CTAs (1 KB reserved each) out of 228 KB;
  // the rest of the unified L1 / shared storage stays L1
  constexpr int kCarveout = (int)((kTcCtas * (kBytes + 1024) * 100 + 228 * 1024 - 1) / (228 * 1024));
  e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveout > 100 ? 100 : kCarveout);
  if (e != cudaSuccess) return e;
  if (p.tc_n_chunks == 0 || p.tc_grid == 0) return cudaSuccess;
  return launch_dependent(k, dim3((p.n_fchunks + p.tc_slice_per - 1) / p.tc_slice_per, p.tc_grid, std::max(1, p.heads)),
                          dim3(kTcThreads), kBytes, st, p);
}

// The gathered row of a narrow B: the 32 or 64 features that cover it, so
// that a load takes 4 or 2 rows (N <= 64 in 16 bits: 4).  The split-bf16 tiles
// start at 64: four steps' hi and lo images would leave room for one CTA.
template <int MODE, bool kIn16>
static cudaError_t launch_tc_rows(const SpmmArgs& p, cudaStream_t st) {
  if (p.ldb * (kIn16 ? 2 : 4) >= (1L << 32) || p.ldc * 4 >= (1L << 32))
    return launch_tc_t<MODE, false, kIn16, 128, true>(p, st);
  if constexpr (!kIn16 && (MODE == STILE_TC_BF16 || MODE == STILE_TC_F16)) {
    if (p.N == 32) return launch_tc_t<MODE, true, false, 32>(p, st);
    if (p.N < 32) return launch_tc_t<MODE, false, false, 32>(p, st);
  }
  if constexpr (MODE != STILE_TC_FP8) {
    if (p.N == 64) return launch_tc_t<MODE, true, kIn16, 64>(p, st);
    if (p.N < 64) return launch_tc_t<MODE, false, kIn16, 64>(p, st);
  }
  return p.N % 128 == 0 ? launch_tc_t<MODE, true, kIn16>(p, st) : launch_tc_t<MODE, false, kIn16>(p, st);
}

// resident CTAs of the tensor-core kernel on the current device, computed
// once per (device, split mode)
int tc_persistent_ctas(int mode) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const std::pair<int, int> key{dev, mode == STILE_TC_SPLIT_BF16 ? 1 : 0};
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
  }
  int sms = 0, per_sm = 0;
  const cudaError_t e =
      mode == STILE_TC_SPLIT_BF16
          ? resident_ctas(spmm_tc_kernel<STILE_TC_SPLIT_BF16, true, false, 128, false>, kTcThreads,
                          TcCfg<STILE_TC_SPLIT_BF16, false, 128>::kBytes, &sms, &per_sm)
          : resident_ctas(spmm_tc_kernel<STILE_TC_BF16, true, false, 128, false>, kTcThreads,
                          TcCfg<STILE_TC_BF16, false, 128>::kBytes, &sms, &per_sm);
  if (e != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  cache[key] = sms * std::min(per_sm, kTcCtas);
  return cache[key];
}

// Feature slices per CTA of the tensor-core grid.  The chunk schedule
// balances k-steps over tc_grid CTAs; with nf slices a CTA's work is its
// k-steps times nf.  When that makes the longest CTA much longer than the
// average over all resident CTAs (a wide B over few chunks), the slices are
// split over grid.x so that no CTA holds more than about the average.
static int tc_slices_per_cta(const SpmmArgs& p) {
  const int nf = p.n_fchunks;
  if (nf <= 1 || p.tc_max_cta_steps <= 0) return nf;
  const int resident = tc_persistent_ctas(p.tc_mode);
  if (resident <= 0) return nf;
  const long avg = ((long)p.tc_n_ksteps * nf + resident - 1) / resident;  // step-slices per CTA
  const long per = avg / p.tc_max_cta_steps;
  return (int)std::max(1L, std::min<long>(per, nf));
}

cudaError_t launch_tc(const SpmmArgs& args, cudaStream_t st) {
  SpmmArgs p = args;
  p.tc_slice_per = tc_slices_per_cta(p);
  if (p.b_bf16) {
    if (p.tc_mode != STILE_TC_BF16) return cudaErrorNotSupported;
    return launch_tc_rows<STILE_TC_BF16, true>(p, st);
  }
  switch (p.tc_mode) {
    case STILE_TC_F16: return launch_tc_rows<STILE_TC_F16, false>(p, st);
    case STILE_TC_FP8: return launch_tc_rows<STILE_TC_FP8, false>(p, st);
    case STILE_TC_SPLIT_BF16: return launch_tc_rows<STILE_TC_SPLIT_BF16, false>(p, st);
    default: return launch_tc_rows<STILE_TC_BF16, false>(p, st);
  }
}

// Streaming multiprocessors of the current device (cached per device; 1 if
// the query fails, which only shrinks grids).
int device_sm_count() {
  static std::mutex mu;
  static std::map<int, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(dev);
  if (it != cache.end()) return it->second;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
  cache[dev] = sms;
  return sms;
}

// Blocks of the ELL kernels: x over groups; when that leaves the GPU short
// of blocks (a wide B over few groups), y splits the feature passes, up to
// about ten blocks per SM in all.
// (sets p.ell_fc_span to the features of one block row)
static dim3 ell_grid(SpmmArgs& p, int groups_per_block, int pass) {
  const long gx = (p.ell_n_groups + groups_per_block - 1) / groups_per_block;
  const int n_pass = (p.N + pass - 1) / pass;
  const long want = (long)device_sm_count() * 10;
  long gy = gx >= want ? 1 : (want + gx - 1) / gx;
  gy = std::max(1L, std::min<long>(gy, n_pass));
  const int per = (int)((n_pass + gy - 1) / gy);
  gy = (n_pass + per - 1) / per;
  p.ell_fc_span = per * pass;
  return dim3((unsigned)gx, (unsigned)gy, (unsigned)std::max(1, p.heads));
}

// every row offset of B in 31 bits; a row's bytes in 32
static bool b_off32(const SpmmArgs& p) { return (long)p.K * p.ldb < (1L << 31); }
static bool b_row32(const SpmmArgs& p) { return p.ldb * (p.b_bf16 ? 2 : 4) < (1L << 32); }

template <int LPR, int VEC, bool kFull, int kAddr>
static cudaError_t launch_ell_addr(const SpmmArgs& p, dim3 grid, cudaStream_t st) {
  if (grid.z > 1)
    return launch_dependent(spmm_ell_seg_kernel<LPR, VEC, kFull, kAddr, true, true>, grid, dim3(256), 0, st, p);
  if (grid.y > 1)
    return launch_dependent(spmm_ell_seg_kernel<LPR, VEC, kFull, kAddr, true>, grid, dim3(256), 0, st, p);
  return launch_dependent(spmm_ell_seg_kernel<LPR, VEC, kFull, kAddr>, grid, dim3(256), 0, st, p);
}

// (the 64-bit row stride: one general variant per group width)
template <int LPR, int VEC, bool kFull>
static cudaError_t launch_ell_seg(const SpmmArgs& p, dim3 grid, cudaStream_t st) {
  if (!b_row32(p))
    return launch_dependent(spmm_ell_seg_kernel<LPR, VEC, false, kRow64, true, true>, grid, dim3(256), 0, st, p);
  if (kFull && b_off32(p)) return launch_ell_addr<LPR, VEC, kFull, kFull ? kOff32 : kRow32>(p, grid, st);
  return launch_ell_addr<LPR, VEC, kFull, kRow32>(p, grid, st);
}

template <int LPR>
struct EllLaunch {
  static cudaError_t run(SpmmArgs p, cudaStream_t st) {
    if (p.ell_n_groups == 0) return cudaSuccess;
    const dim3 grid = ell_grid(p, 256 / LPR, 4 * LPR);
    return launch_ell_seg<LPR, 1, false>(p, grid, st);
  }
};

// fp32 B of two float4 a lane: N < 128 in LPR-lane sub-groups, LPR the power of
// two covering N, so a 41-wide row takes 6 of 8 lanes instead of 11 of 16
// single-float4 lanes; wider rows in passes of 256 (launch_ell).
template <int LPR>
struct EllNarrowLaunch {
  static cudaError_t run(SpmmArgs p, cudaStream_t st) {
    const dim3 grid = ell_grid(p, 256 / LPR, 8 * LPR);
    // (4 entries per batch at 4 blocks per SM measured slower at N = 41,
    // 159 against 154 us on the GCN graph)
    return p.N % (8 * LPR) == 0 ? launch_ell_seg<LPR, 2, true>(p, grid, st) : launch_ell_seg<LPR, 2, false>(p, grid, st);
  }
};

template <int LPR, bool kFull>
static cudaError_t launch_ell_seg_bf16(const SpmmArgs& p, dim3 grid, cudaStream_t st) {
  if (!b_row32(p))
    return launch_dependent(spmm_ell_seg_bf16_kernel<LPR, false, kRow64, true>, grid, dim3(256), 0, st, p);
  if (grid.y > 1) return launch_dependent(spmm_ell_seg_bf16_kernel<LPR, kFull, kRow32, true>, grid, dim3(256), 0, st, p);
  return launch_dependent(spmm_ell_seg_bf16_kernel<LPR, kFull, kRow32>, grid, dim3(256), 0, st, p);
}

template <int LPR>
struct EllBf16Launch {
  static cudaError_t run(SpmmArgs p, cudaStream_t st) {
    const dim3 grid = ell_grid(p, 256 / LPR, 8 * LPR);
    return launch_ell_seg_bf16<LPR, false>(p, grid, st);
  }
};

static int lpr_for_bf16(int N) {
  const int lanes = (N + 7) / 8;
  if (lanes >= 32) return 32;
  int l = 4;
  while (l < lanes) l <<= 1;
  return l;
}

cudaError_t launch_ell(const SpmmArgs& args, cudaStream_t st) {
  if (args.ell_n_groups == 0) return cudaSuccess;
  SpmmArgs p = args;
  if (p.b_bf16) {
    // 16-lane sub-groups of 8 features per lane (two groups per warp)
    if (p.N % 128 == 0) return launch_ell_seg_bf16<16, true>(p, ell_grid(p, 16, 128), st);
    return dispatch_lpr<EllBf16Launch>(lpr_for_bf16(p.N), p, st);
  }
  // 16-lane sub-groups of 8 features per lane (two groups per warp)
  if (p.N % 128 == 0) return launch_ell_seg<16, 2, true>(p, ell_grid(p, 16, 128), st);
  if (p.N < 128) {
    int lpr = 4;
    while (lpr < (p.N + 7) / 8) lpr <<= 1;
    return dispatch_lpr<EllNarrowLaunch>(lpr, p, st);
  }
  // wider rows that are no multiple of 128: 256 features a pass (two float4 a
  // lane) where that covers no more than passes of 128 do (one float4): N = 150
  // on the 50,000-node graph 133 -> 121 us; N = 300 on the 169k-node graph would
  // go from 179 to 186.  Not where the passes of 128, a block each, leave SMs
  // idle: a block then lasts as long as its longest group times its features
  // (N = 150, 21,198 entries: 5.8 against 7.5 us; 47,232 entries fill the
  // device: 8.7 against 7.9).
  const long blocks = (p.ell_n_groups + 7L) / 8 * ((p.N + 127) / 128);
  if ((p.N + 255) / 256 * 2 == (p.N + 127) / 128 && blocks >= 5L * device_sm_count())
    return EllNarrowLaunch<32>::run(p, st);
  return EllLaunch<32>::run(p, st);
}

// dvals[t] = <dY[row(t)], B[col(t)]> over the plan's entry list, as runs of
// one row (the row-run SDDMM kernel holds the dY row and gathers B rows)
template <int LPR>
static cudaError_t launch_ell_bwd_t(SpmmArgs p, cudaStream_t st) {
  const long gx = (p.ell_n_groups + (256 / LPR) - 1) / (256 / LPR);
  const dim3 grid((unsigned)gx, 1, 1);
  return p.N == 8 * LPR ? launch_dependent(spmm_ell_bwd_kernel<LPR, true>, grid, dim3(256), 0, st, p)
                        : launch_dependent(spmm_ell_bwd_kernel<LPR, false>, grid, dim3(256), 0, st, p);
}

cudaError_t launch_ell_bwd(const SpmmArgs& p, cudaStream_t st) {
  if (p.ell_n_groups == 0) return cudaSuccess;
  if (p.N > 128 || p.b_bf16 || p.heads > 1) return cudaErrorNotSupported;
  int lpr = 4;
  while (8 * lpr < p.N) lpr <<= 1;
  switch (lpr) {
    case 4: return launch_ell_bwd_t<4>(p, st);
    case 8: return launch_ell_bwd_t<8>(p, st);
    default: return launch_ell_bwd_t<16>(p, st);
  }
}

// Value gradients of the tensor-tile nonzeros on the tensor cores.
//
// A unit is up to 8 k-steps of one chunk (one item): its 128 k-step columns
// (16 per k-step) are the M = 128 rows of the MMA's A operand, the item's 16
// rows its N = 16 B operand, the features its K, so
//   D[16 j + k][r] = <Y[col(j, k)], X[row r]>
// is the gradient of the nonzero (r, k) of k-step j.  The item's 16 X rows
// are gathered once per unit, the columns once per k-step (the row-run
// kernel gathers one row per nonzero: ~41 per k-step on the GCN graph).
// Per 64-feature chunk each of the 16 half-warps (256 threads) issues the
// loads of its 8 columns and 1 item row at once (a float4 a lane, 256
// contiguous bytes a row), then splits every row into hi = bf16(x) and
// lo = bf16(x - hi), and stores both into K-major images with the 128-byte
// swizzle (128-byte rows of 64 features, the 16-byte chunk q of row m at
// q ^ (m % 8), 8-row atoms 1 KB apart), so each half-warp writes one
// 128-byte row: no bank conflicts.  One thread issues hi.hi + hi.lo + lo.hi
// per 16-feature slice (the K advance is 32 bytes inside the atom row) into
// a 16-column TMEM accumulator; the epilogue reads lane m = 16 j + k and
// writes the live entries through the k-step's id table.  The wait for the
// MMAs is bounded; a wait that runs out sets the error flag and ends the
// kernel's work.
constexpr uint32_t kDvYImg = 16384;  // 128 rows x 64 bf16
constexpr uint32_t kDvXImg = 2048;   // 16 rows x 64 bf16
constexpr uint32_t kDvBytes = 1024 + 2 * kDvYImg + 2 * kDvXImg + 64 + 64;

constexpr int kDvThreads = 256;

__global__ void __launch_bounds__(kDvThreads, 3) spmm_tc_dvals_kernel(SpmmArgs p, const float* __restrict__ X, long ldx,
                                                              const float* __restrict__ Y, long ldy,
                                                              float* __restrict__ out, int F) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t yhi = base, ylo = base + kDvYImg, xhi = base + 2 * kDvYImg, xlo = xhi + kDvXImg;
  const uint32_t orow_s = xlo + kDvXImg, bar = orow_s + 64, tmem_slot = bar + 8;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hw = lane >> 4, sl = lane & 15;
  griddep_wait();  // X and Y may come from the previous kernel
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 32);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
  // kind::f16, bf16 x bf16, M = 128, N = 16, both operands K-major
  constexpr uint32_t idesc = make_idesc(1, 1, 0, 0, 128, 16);
  uint32_t phase = 0;
  bool ok = true;
  // one float4 of a gathered row -> hi and lo bf16 halves of its 16-byte chunk
  auto put = [&](uint32_t hi_img, uint32_t lo_img, int row, float4 v) {
    const uint32_t o = sw128_off(row, sl >> 1) + (sl & 1) * 8;
    const uint32_t h01 = pack_bf16x2(v.x, v.y), h23 = pack_bf16x2(v.z, v.w);
    st_shared_v2(hi_img + o, h01, h23);
    st_shared_v2(lo_img + o, pack_bf16x2(v.x - __uint_as_float(h01 << 16), v.y - __uint_as_float(h01 & 0xffff0000u)),
                 pack_bf16x2(v.z - __uint_as_float(h23 << 16), v.w - __uint_as_float(h23 & 0xffff0000u)));
  };
#pragma unroll 1
  for (int u = blockIdx.x; u < p.tcdv_n_units && ok; u += gridDim.x) {
    const int ks0 = __ldg(p.tcdv_unit_ks + u);
    const int meta = __ldg(p.tcdv_unit_meta + u);
    const int item = meta >> 3, nks = (meta & 7) + 1;
    // this half-warp (hg = 0..15) gathers columns m = 16 i + hg (i < 8) and
    // item row hg
    const int hg = 2 * warp + hw;
    int ycol[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = 16 * i + hg, j = m >> 4;
      ycol[i] = j < nks ? __ldg(p.tc_cols + (long)(ks0 + j) * 16 + (m & 15)) : -1;
    }
    const int xrow = __ldg(p.tc_out_rows + (long)item * 16 + hg);
    if (sl == 0) asm volatile("st.shared.b32 [%0], %1;" ::"r"(orow_s + 4 * hg), "r"(xrow) : "memory");
#pragma unroll 1
    for (int fc = 0; fc < F; fc += 64) {
      const int f = fc + 4 * sl;
      // every load of the chunk in flight at once, then the conversions
      float4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = ycol[i] >= 0 ? ld4_live(Y + (long)ycol[i] * ldy, f, F) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xv = xrow >= 0 ? ld4_live(X + (long)xrow * ldx, f, F) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; ++i) put(yhi, ylo, 16 * i + hg, v[i]);
      put(xhi, xlo, hg, xv);
      fence_proxy_async_smem();
      tc_fence_before();
      __syncthreads();
      tc_fence_after();
      if (tid == 0) {
        const int ns = min(4, (F - fc + 15) / 16);
        for (int s = 0; s < ns; ++s) {
          const uint64_t ah = smem_desc(yhi + 32 * s, 16, 1024, kSwizzle128B);
          const uint64_t bh = smem_desc(xhi + 32 * s, 16, 1024, kSwizzle128B);
          umma_f16(tmem, ah, bh, idesc, (fc > 0 || s > 0) ? 1u : 0u);
          umma_f16(tmem, ah, smem_desc(xlo + 32 * s, 16, 1024, kSwizzle128B), idesc, 1u);
          umma_f16(tmem, smem_desc(ylo + 32 * s, 16, 1024, kSwizzle128B), bh, idesc, 1u);
        }
        umma_commit(bar);
      }
      // the MMAs read the images: nobody rewrites them, or reads TMEM, first
      const bool done = __syncthreads_and(tid == 0 ? mbar_wait_bounded(bar, phase) : true) != 0;
      phase ^= 1u;
      if (!done) {
        ok = false;
        break;
      }
      if (tid != 0) mbar_wait_bounded(bar, phase ^ 1u);  // completed: returns at once
      tc_fence_after();
    }
    if (!ok) break;
    // epilogue (warps 0-3): warp w holds TMEM lanes m = 32 w .. 32 w + 31
    // (k-steps 2 w and 2 w + 1), columns r = 0..15
    const int m = 32 * warp + lane, j = m >> 4, k = m & 15;
    uint32_t v[16];
    if (warp < 4) {
      tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16), v);
      tmem_wait_ld();
    }
    if (warp < 4 && j < nks) {
      const int* ids = p.tcdv_id + (long)(ks0 + j) * 256 + k;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        int orow;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(orow) : "r"(orow_s + 4 * r) : "memory");
        const int id = __ldcs(ids + 16 * r);
        if (id >= 0 && orow >= 0) __stcs(out + id, __uint_as_float(v[r]));
      }
    }
    tc_fence_before();
    __syncthreads();
  }
  if (!ok && tid == 0 && p.err_flag) atomicOr(p.err_flag, 1);
  // every MMA this CTA issued has completed before TMEM is freed
  if (!ok && tid == 0) mbar_wait_bounded(bar, phase ^ 1u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 32);
}

cudaError_t launch_tc_dvals(const SpmmArgs& p, const float* X, long ldx, const float* Y, long ldy, float* out, int F,
                            cudaStream_t st) {
  if (p.tcdv_n_units == 0) return cudaSuccess;
  if (!p.tcdv_id) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(spmm_tc_dvals_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kDvBytes);
  if (e != cudaSuccess) return e;
  // 37 KB of shared memory, 256 threads at 80 registers and 32 TMEM columns
  // per CTA: 3 CTAs per SM
  const int grid = std::min(p.tcdv_n_units, device_sm_count() * 3);
  return launch_dependent(spmm_tc_dvals_kernel, dim3((unsigned)grid), dim3(kDvThreads), kDvBytes, st, p, X, ldx, Y,
                          ldy, out, F);
}

cudaError_t launch_dvals(const SpmmArgs& p, const float* dY, long lddy, float* dvals, cudaStream_t st) {
  return launch_sddmm_runs(p.dv_n_groups, p.dv_n, p.dv_gptr, p.dv_grow, p.dv_col, p.dv_id, dY, false, lddy, p.B,
                           p.b_bf16 != 0, p.ldb, dvals, p.N, st);
}

}  // namespace stile
