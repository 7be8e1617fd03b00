// Fused sparse attention for sm_103a:
//   out[h][r] = sum_t softmax_t(scale * <Q[h][r], K[h][c_t]>) * V[h][c_t]
// over the stored entries c_t of row r of a CSR pattern (entries outside the
// pattern count as -inf), every head in one launch (blockIdx.y = head).
//
// This is the sparse-attention step the reference's LogSparse / Strided
// operators come from (MY_sparse/gen_formats_v2.py:2926-3003): the SDDMM of
// the scores on the pattern, the row softmax of the sparse transformer
// (my_3rdparty/Magicube/Magicube1/end2end_eval/sparse_transformer_magicube/
// src/cuda/softmax_kernel.cu) and the SpMM with the probabilities as values,
// here in one pass per row: an LPR-lane group holds its query row (8 features
// a lane, as two float4 4 LPR features apart), takes the row's entries kU at a
// time with their K and V rows in flight, and reduces the kU scores with a
// transposing butterfly, so that each lane holds one entry's score and takes
// one exponential for it.  An online softmax -- running maximum m, a sum l per
// entry slot, and an output accumulator rescaled by exp(m_old - m_new) -- keeps
// the scores and the probabilities out of memory.
//
// Bound by instruction issue before and by the L1 data pipe now (a strided
// mask's neighbouring rows share their columns: two thirds of the loads hit
// L1, and 3.1 GB of K and V rows pass the pipe): the multiply-adds are paired
// (fma.rn.f32x2), the column ids come LPR at a time, rows load without
// predicates and one exponential a batch serves its kU entries.  4096 tokens, 8
// heads, 64 features, strided mask (766k entries a head): 188 us with pairs of
// entries and scalar multiply-adds, 152 us now; 4 heads of 41 / 80 / 127
// features: 114 / 188 / 188 us, with predicated loads of kU entries (which
// spilled) 128 / 182 / 205 us, now 104 / 150 / 181 us.
#include "common.cuh"
#include "spmm.cuh"

namespace stile {

struct Feat8 {  // this lane's 8 features of a row: f .. f + 3 and f2 .. f2 + 3
  f32x2 v[4];
};

// the row's float4 at a and b (both inside the row)
__device__ __forceinline__ Feat8 load8(const float* row, int a, int b) {
  const float4 x = ldg4(row + a), y = ldg4(row + b);
  return {{pack2(x.x, x.y), pack2(x.z, x.w), pack2(y.x, y.y), pack2(y.z, y.w)}};
}

// the pair with its components past the first `live` features zero
__device__ __forceinline__ f32x2 keep2(f32x2 v, int live) {
  const float2 x = unpack2(v);
  return pack2(live > 0 ? x.x : 0.f, live > 1 ? x.y : 0.f);
}

constexpr int kAttThreads = 128;

// kMask 0: F and Fv are 8 LPR; 1: F is a multiple of 4; 2: any F.  A lane whose
// float4 starts past a row's features loads the row's last one instead (no
// predicates, no zeroed registers); K's products of such a float4 are left out
// of the score by selects (a product with a zeroed q would turn an infinite K
// into NaN), and V's features past Fv are never stored.
template <int LPR, int kMask>
__global__ void __launch_bounds__(kAttThreads, 5) sparse_attention_kernel(
    int n_rows, const int* __restrict__ indptr, const int* __restrict__ indices, const float* __restrict__ Q,
    const float* __restrict__ K, const float* __restrict__ V, long ldq, long ldk, long ldv, long q_head, long k_head,
    long v_head, float* __restrict__ out, long ldo, long o_head, int F, int Fv, float scale) {
  constexpr int kU = LPR < 4 ? LPR : 4;  // entries per batch
  const int lane = threadIdx.x & 31, sub = lane / LPR, sl = lane % LPR;
  const unsigned mask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << (sub * LPR));
  const long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
  if (r >= n_rows) return;  // the whole group leaves together
  const long h = blockIdx.y;
  const float* Kh = K + h * k_head;
  const float* Vh = V + h * v_head;
  // each load instruction of the group reads 16 LPR contiguous bytes of a row
  const int f = 4 * sl, f2 = f + 4 * LPR;
  const int last = (F - 1) & ~3, lastv = (Fv - 1) & ~3;
  const int ka = kMask ? min(f, last) : f, kb = kMask ? min(f2, last) : f2;
  const int va = kMask ? min(f, lastv) : f, vb = kMask ? min(f2, lastv) : f2;
  Feat8 q = load8(Q + h * q_head + r * ldq, ka, kb);
  if constexpr (kMask == 2) {
    // q's padding; K's, which meets it, is cleared as it comes
    q.v[0] = keep2(q.v[0], F - ka);
    q.v[1] = keep2(q.v[1], F - ka - 2);
    q.v[2] = keep2(q.v[2], F - kb);
    q.v[3] = keep2(q.v[3], F - kb - 2);
  }
  const int rb = __ldg(indptr + r), n = __ldg(indptr + r + 1) - rb;
  // this lane's entry of a batch: the halving strides' bits of its index
  int e = 0;
#pragma unroll
  for (int m = kU, hw = LPR / 2; m > 1; m >>= 1, hw >>= 1)
    if (sl & hw) e += m / 2;
  float m = -INFINITY, l = 0.f;
  f32x2 acc[4] = {0, 0, 0, 0};
  auto col_at = [&](int i) { return __ldg(indices + rb + min(i, n - 1)); };  // past the row: a valid entry, weight 0
  int cl = n > 0 ? col_at(sl) : 0;
#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += LPR) {
    const int cl1 = col_at(c0 + LPR + sl);
#pragma unroll 1
    for (int b0 = 0; b0 < min(LPR, n - c0); b0 += kU) {
      Feat8 k[kU], v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const long c = __shfl_sync(mask, cl, b0 + u, LPR);
        k[u] = load8(Kh + c * ldk, ka, kb);
        v[u] = load8(Vh + c * ldv, va, vb);
      }
      float s[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if constexpr (kMask == 2) {
          k[u].v[0] = keep2(k[u].v[0], F - ka);
          k[u].v[1] = keep2(k[u].v[1], F - ka - 2);
          k[u].v[2] = keep2(k[u].v[2], F - kb);
          k[u].v[3] = keep2(k[u].v[3], F - kb - 2);
        }
        const f32x2 da = fma2(q.v[1], k[u].v[1], mul2(q.v[0], k[u].v[0]));
        const f32x2 d = fma2(q.v[3], k[u].v[3], fma2(q.v[2], k[u].v[2], da));
        const float2 p = unpack2(kMask == 0 || f2 < F ? d : da);
        s[u] = kMask == 0 || f < F ? p.x + p.y : 0.f;
      }
      // transposing butterfly: this lane keeps entry e's score
#pragma unroll
      for (int w = kU, hw = LPR / 2; w > 1; w >>= 1, hw >>= 1) {
        const bool up = (sl & hw) != 0;
#pragma unroll
        for (int i = 0; i < w / 2; ++i) {
          const float send = up ? s[i] : s[i + w / 2];
          const float keep = up ? s[i + w / 2] : s[i];
          s[i] = keep + __shfl_xor_sync(mask, send, hw);
        }
      }
#pragma unroll
      for (int o = LPR / (2 * kU); o > 0; o >>= 1) s[0] += __shfl_xor_sync(mask, s[0], o);
      const float t = c0 + b0 + e < n ? scale * s[0] : -INFINITY;
      float mn = fmaxf(m, t);
#pragma unroll
      for (int w = kU, hw = LPR / 2; w > 1; w >>= 1, hw >>= 1) mn = fmaxf(mn, __shfl_xor_sync(mask, mn, hw));
      const float ref = mn == -INFINITY ? 0.f : mn;  // only -inf scores so far: weights 0
      const float alpha = expf(m - ref);             // 0 for the first batch (m = -inf)
      const float p = expf(t - ref);
      l = fmaf(l, alpha, p);
      m = mn;
      const f32x2 a2 = pack2(alpha, alpha);
#pragma unroll
      for (int w = 0; w < 4; ++w) acc[w] = mul2(acc[w], a2);
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        // a lane that holds entry u: its index's halving bits spell u
        int src = 0;
#pragma unroll
        for (int w = kU, hw = LPR / 2, x = u; w > 1; w >>= 1, hw >>= 1) {
          if (x >= w / 2) {
            src += hw;
            x -= w / 2;
          }
        }
        const float pu = __shfl_sync(mask, p, src, LPR);
        const f32x2 p2 = pack2(pu, pu);
        // entries past the row add nothing (a weight of 0 would still turn an
        // infinite V into NaN; predicates on their loads cost a third of the
        // kernel's rate)
        if (u == 0 || c0 + b0 + u < n) {
#pragma unroll
          for (int w = 0; w < 4; ++w) acc[w] = fma2(p2, v[u].v[w], acc[w]);
        }
      }
    }
    cl = cl1;
  }
  // the entry slots' sums
#pragma unroll
  for (int w = kU, hw = LPR / 2; w > 1; w >>= 1, hw >>= 1) l += __shfl_xor_sync(mask, l, hw);
  // a row without entries attends to nothing: zeros
  const float inv = n > 0 ? 1.f / l : 0.f;
  float* orow = out + h * o_head + r * ldo;
  float2 o[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) o[w] = unpack2(acc[w]);
  st_row4(orow, f, Fv, make_float4(o[0].x * inv, o[0].y * inv, o[1].x * inv, o[1].y * inv));
  st_row4(orow, f2, Fv, make_float4(o[2].x * inv, o[2].y * inv, o[3].x * inv, o[3].y * inv));
}

template <int LPR>
static cudaError_t launch_att_t(dim3 grid, cudaStream_t st, int n_rows, const int* indptr, const int* indices,
                                const float* Q, const float* K, const float* V, long ldq, long ldk, long ldv,
                                long q_head, long k_head, long v_head, float* out, long ldo, long o_head, int F, int Fv,
                                float scale) {
#define STILE_ATT(MASK)                                                                                        \
  sparse_attention_kernel<LPR, MASK><<<grid, kAttThreads, 0, st>>>(n_rows, indptr, indices, Q, K, V, ldq, ldk, ldv, \
                                                                   q_head, k_head, v_head, out, ldo, o_head, F, Fv, scale)
  if (F == 8 * LPR && Fv == 8 * LPR) STILE_ATT(0);
  else if (F % 4 == 0) STILE_ATT(1);
  else STILE_ATT(2);
#undef STILE_ATT
  return cudaGetLastError();
}

cudaError_t launch_sparse_attention(int n_rows, const int* indptr, const int* indices, const float* Q,
                                    const float* K, const float* V, long ldq, long ldk, long ldv, long q_head,
                                    long k_head, long v_head, float* out, long ldo, long o_head, int F, int Fv,
                                    float scale, int heads, cudaStream_t st) {
  if (n_rows == 0 || heads == 0) return cudaSuccess;
  const int width = F > Fv ? F : Fv;  // features per lane: 8; lanes: the power of two covering the wider row
  int lpr = 2;
  while (8 * lpr < width) lpr <<= 1;
  const dim3 grid((unsigned)(((long)n_rows * lpr + kAttThreads - 1) / kAttThreads), (unsigned)heads);
#define STILE_ATT_ARGS grid, st, n_rows, indptr, indices, Q, K, V, ldq, ldk, ldv, q_head, k_head, v_head, out, ldo, \
                       o_head, F, Fv, scale
  switch (lpr) {
    case 2: return launch_att_t<2>(STILE_ATT_ARGS);
    case 4: return launch_att_t<4>(STILE_ATT_ARGS);
    case 8: return launch_att_t<8>(STILE_ATT_ARGS);
    default: return launch_att_t<16>(STILE_ATT_ARGS);
  }
#undef STILE_ATT_ARGS
}

}  // namespace stile
