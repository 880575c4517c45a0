// Exact forward kernel: fp32 FFMA arithmetic for every composition and any head_dim <= 256.
//
// Serves the compositions the tcgen05 kernel does not instantiate: fp32 inputs (whose parity
// bound of 1e-4 rules out single-pass TF32), head dims other than 64/128, additive bias,
// ReLU normalisation and block lists whose block size is not a multiple of 128.  The
// arithmetic follows the reference forward kernel step by step
// (attnfuse/compiler/codegen.py:98-381): scores in fp32, scale, ALiBi / additive bias,
// causal / window / out-of-range masking with -inf, online softmax (or ReLU row sums),
// O = acc / l with l == 0 mapped to 1, L = m + log(l).
//
// Tiling: one CTA owns 32 query rows of one (batch, head) and walks 64-key tiles, with one group of
// 128 threads (head dims above 128) or two that take the tiles in turn, each with K / V / P buffers
// and online-softmax state of its own, merged at the end.  Thread (ty, tx) = (tid / 16, tid % 16) of a
// group owns rows 4*ty..4*ty+3, keys tx + 16*j and output columns 64*c + 4*tx .. +3, so row reductions
// stay inside 16-lane groups.
//
// Bound: FP32 FMA issue, and latency where a problem is a few hundred CTAs.  Shared-memory operands are
// read 16 bytes at a time and products run on packed fp32 pairs (fma.rn.f32x2: even and odd d, or two
// output columns).  [2,12,512,64] causal + RoPE + ALiBi, 0.82 GFLOP: 150 us with 4-byte reads and
// scalar FMAs, 70 us with 16-byte reads (30 % of the issue slots: 1.9 warps per scheduler on average,
// the longest CTA's eight tiles one after the other), 47 us with two groups and packed FMAs.
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace af {
namespace {

constexpr int TM = 32;
constexpr int TN = 64;
constexpr int NT = 128;       // threads of a group
constexpr int PAD = 4;        // row pitch D + 4 floats: 16-byte rows, 8 consecutive rows on distinct banks
constexpr int LDP = 2 * TN + PAD;   // P is stored twice over, (p, p): the broadcast operand of a packed FMA

using namespace ptx;          // packed fp32 pairs

// Barrier of one group's 128 threads (group 0 or 1; number 0 is __syncthreads).
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(NT) : "memory"); }

template <typename T>
__device__ __forceinline__ float ld_elem(const void* base, int64_t off) {
  return Elem<T>::to_f32(reinterpret_cast<const T*>(base)[off]);
}

__device__ __forceinline__ void copy16_async(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Rotate-half on a tile held as fp32 in shared memory, then round through T -- the reference
// rotates in fp32 and casts back to the input dtype before the matmul
// (attnfuse/compiler/codegen.py:126-135, 332-341).
template <typename T, int LD>
__device__ __forceinline__ void rope_tile(float* tile, int rows, int pos0, int pos_end, int D,
                                          const void* cos_, const void* sin_, int64_t stride_n) {
  const int half = D / 2;
  for (int idx = threadIdx.x % NT; idx < rows * half; idx += NT) {
    const int r = idx / half, d = idx - r * half;
    const int pos = pos0 + r;
    if (pos >= pos_end) continue;
    const int64_t base = (int64_t)pos * stride_n;
    const float c1 = ld_elem<T>(cos_, base + d), s1 = ld_elem<T>(sin_, base + d);
    const float c2 = ld_elem<T>(cos_, base + d + half), s2 = ld_elem<T>(sin_, base + d + half);
    const float x1 = tile[r * LD + d], x2 = tile[r * LD + d + half];
    tile[r * LD + d] = round_through<T>(x1 * c1 - x2 * s1);
    tile[r * LD + d + half] = round_through<T>(x2 * c2 + x1 * s2);
  }
}

// Rows [row0, row0 + ROWS) of `src` (already at its (batch, head)) into a tile; rows at or past
// `row_end` and columns past D are zero.  VEC (fp32, 16-byte aligned rows, D a multiple of 4, or of 8
// with rotation): 16-byte accesses -- asynchronous, the caller commits and waits -- and a rotated
// tile is rotated on the way in, so that it goes through shared memory once.
template <typename T, int DMAX, bool VEC, int ROWS>
__device__ __forceinline__ void load_tile(float* tile, const T* src, const int64_t s_n, const int64_t s_d, const int row0,
                                          const int row_end, const AfProblem& p, const bool rope, const int pos_off) {
  constexpr int LD = DMAX + PAD;
  const int tid = threadIdx.x % NT, D = p.D;
  if constexpr (VEC) {
    const float* base = reinterpret_cast<const float*>(src);
    if (!rope) {
#pragma unroll 8
      for (int idx = tid; idx < ROWS * (DMAX / 4); idx += NT) {
        const int r = idx / (DMAX / 4), c = (idx % (DMAX / 4)) * 4;
        const bool ok = row0 + r < row_end && c < D;
        copy16_async(tile + r * LD + c, base + (ok ? (int64_t)(row0 + r) * s_n + c : 0), ok);
      }
      return;
    }
    const int half = D / 2;
#pragma unroll 2
    for (int idx = tid; idx < ROWS * (DMAX / 8); idx += NT) {
      const int r = idx / (DMAX / 8), c = (idx % (DMAX / 8)) * 4;
      if (c >= half) continue;
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      if (row0 + r < row_end) {
        const float* x = base + (int64_t)(row0 + r) * s_n + c;
        const int64_t tab = (int64_t)(row0 + r + pos_off) * p.rope_stride_n + c;
        const float* cos_ = reinterpret_cast<const float*>(p.cos) + tab;
        const float* sin_ = reinterpret_cast<const float*>(p.sin) + tab;
        const float4 x1 = __ldg(reinterpret_cast<const float4*>(x)), x2 = __ldg(reinterpret_cast<const float4*>(x + half));
        const float4 c1 = __ldg(reinterpret_cast<const float4*>(cos_)), c2 = __ldg(reinterpret_cast<const float4*>(cos_ + half));
        const float4 s1 = __ldg(reinterpret_cast<const float4*>(sin_)), s2 = __ldg(reinterpret_cast<const float4*>(sin_ + half));
        lo = make_float4(x1.x * c1.x - x2.x * s1.x, x1.y * c1.y - x2.y * s1.y, x1.z * c1.z - x2.z * s1.z, x1.w * c1.w - x2.w * s1.w);
        hi = make_float4(x2.x * c2.x + x1.x * s2.x, x2.y * c2.y + x1.y * s2.y, x2.z * c2.z + x1.z * s2.z, x2.w * c2.w + x1.w * s2.w);
      }
      *reinterpret_cast<float4*>(tile + r * LD + c) = lo;
      *reinterpret_cast<float4*>(tile + r * LD + half + c) = hi;
    }
  } else {
    for (int idx = tid; idx < ROWS * DMAX; idx += NT) {
      const int r = idx / DMAX, d = idx - r * DMAX;
      float x = 0.f;
      if (row0 + r < row_end && d < D) x = Elem<T>::to_f32(src[(int64_t)(row0 + r) * s_n + (int64_t)d * s_d]);
      tile[r * LD + d] = x;
    }
    if (rope) {
      group_sync(threadIdx.x / NT);
      rope_tile<T, LD>(tile, ROWS, row0 + pos_off, row_end + pos_off, D, p.cos, p.sin, p.rope_stride_n);
    }
  }
}

template <int DMAX> struct Groups { static constexpr int value = DMAX <= 128 ? 2 : 1; };   // shared memory holds two up to 128

template <typename T, int DMAX, bool VEC>
__global__ void __launch_bounds__(NT * Groups<DMAX>::value, DMAX == 64 ? 2 : 1) fwd_ffma_kernel(const AfFwdParams a, const int subs_per_block) {
  constexpr int LD = DMAX + PAD;
  constexpr int NCH = DMAX / 64;       // chunks of 64 output columns; a thread owns 4 columns of each
  constexpr int G = Groups<DMAX>::value;
  constexpr int GROUP_FLOATS = 2 * TN * LD + TM * LDP;
  const AfProblem& p = a.p;
  extern __shared__ __align__(16) float smem[];
  const int grp = G == 1 ? 0 : threadIdx.x / NT;
  float* sQ = smem;
  float* sK = sQ + TM * LD + grp * GROUP_FLOATS;
  float* sV = sK + TN * LD;
  float* sP = sV + TN * LD;  // [TM][LDP]

  const int tid = threadIdx.x % NT, tx = tid & 15, ty = tid >> 4;
  const int bh_count = p.B * p.H_q, bh = (int)(blockIdx.x % bh_count);
  const int b = bh / p.H_q, h = bh % p.H_q;
  const int h_kv = h / (p.H_q / p.H_kv);
  const int D = p.D;
  // Row tiles run slowest over the grid and, under a causal mask, from the last (longest) to the
  // first, so that the short ones fill in at the end.
  int row_tile = (int)(blockIdx.x / bh_count);
  if (p.mask_kind == AF_MASK_CAUSAL) row_tile = (int)(gridDim.x / bh_count) - 1 - row_tile;

  int r0, r_end, qb = 0;
  if (p.mask_kind == AF_MASK_BLOCKS) {
    qb = row_tile / subs_per_block;
    r0 = qb * p.block_m + (row_tile % subs_per_block) * TM;
    r_end = min(qb * p.block_m + p.block_m, p.N_q);
  } else {
    r0 = row_tile * TM;
    r_end = min(r0 + TM, p.N_q);
  }
  if (r0 >= r_end) return;

  const T* q_base = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride[0] + (int64_t)h * p.q_stride[1];
  const T* k_base = reinterpret_cast<const T*>(p.k) + (int64_t)b * p.k_stride[0] + (int64_t)h_kv * p.k_stride[1];
  const T* v_base = reinterpret_cast<const T*>(p.v) + (int64_t)b * p.v_stride[0] + (int64_t)h_kv * p.v_stride[1];

  // The key tiles this CTA visits: keys [k0, k_end); block lists carry the bit matrix of a partially
  // active tile whose first key is key_base (rows = queries from the block's first row), or nullptr
  // when every element of the tile is active.
  const int bit_words = (p.block_n + 63) / 64;
  int lo = 0, hi = p.N_kv, list_n = 0, list_at = -1;
  const int32_t* list = nullptr;
  const int32_t* slots = nullptr;
  if (p.mask_kind == AF_MASK_BLOCKS) {
    list_n = p.kv_num[(int64_t)h * p.kv_num_stride_h + qb];
    list = p.kv_idx + (int64_t)h * p.kv_idx_stride_h + (int64_t)qb * p.kv_idx_stride_q;
    slots = p.kv_slot ? p.kv_slot + (int64_t)h * p.kv_idx_stride_h + (int64_t)qb * p.kv_idx_stride_q : nullptr;
    hi = lo = 0;
  } else if (p.mask_kind == AF_MASK_CAUSAL) {
    hi = min(hi, r_end + p.q_offset);
  } else if (p.mask_kind == AF_MASK_WINDOW) {
    lo = max(0, r0 + p.q_offset - p.window + 1);
    hi = min(hi, r_end + p.q_offset + p.window - 1);
  }
  int k0 = lo - TN, k_end = 0, key_base = 0, range_end = hi;
  const uint64_t* tile_bits = nullptr;
  auto advance = [&]() -> bool {
    k0 += TN;
    while (k0 >= range_end) {
      if (++list_at >= list_n) return false;
      const int kb = list[list_at];
      k0 = key_base = kb * p.block_n;
      range_end = min(kb * p.block_n + p.block_n, p.N_kv);
      const int bs = slots ? slots[list_at] : -1;
      tile_bits = bs >= 0 ? p.kv_bits + (int64_t)bs * p.block_m * bit_words : nullptr;
    }
    k_end = min(k0 + TN, range_end);
    return true;
  };

  if (grp == 0) load_tile<T, DMAX, VEC, TM>(sQ, q_base, p.q_stride[2], p.q_stride[3], r0, r_end, p, p.rope != 0, p.q_offset);
  bool more = advance();
  if (G == 2 && grp == 1 && more) more = advance();        // tiles 1, 3, 5, ...
  if (more) load_tile<T, DMAX, VEC, TN>(sK, k_base, p.k_stride[2], p.k_stride[3], k0, k_end, p, p.rope != 0, 0);
  if (VEC) copy_commit();
  if (G == 2) {
    if (VEC) copy_wait<0>();
    __syncthreads();                     // Q for the other group
  }

  const float slope = (p.bias_kind == AF_BIAS_ALIBI) ? load_slope<T>(p.slopes, h) : 0.f;
  float m_i[4], l_i[4];
  uint64_t acc[4][NCH * 2];              // pairs of output columns
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_i[i] = -INFINITY;
    l_i[i] = 0.f;
#pragma unroll
    for (int c = 0; c < NCH * 2; ++c) acc[i][c] = 0ull;
  }

  while (more) {
    // V of this tile flies under the scores, K of the next one under P.V
    load_tile<T, DMAX, VEC, TN>(sV, v_base, p.v_stride[2], p.v_stride[3], k0, k_end, p, false, 0);
    if (VEC) { copy_commit(); copy_wait<1>(); }
    group_sync(grp);

    float s[4][4];
    uint64_t s2[4][4];                   // sums over even and over odd d
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {     // columns D .. of a last group of 4 are zero
      ulonglong2 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(sQ + (ty * 4 + i) * LD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const ulonglong2*>(sK + (tx + 16 * j) * LD + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[i][j] = f32x2_fma(qv[i].x, kv[j].x, s2[i][j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[i][j] = f32x2_fma(qv[i].y, kv[j].y, s2[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float even, odd;
        f32x2_unpack(s2[i][j], even, odd);
        s[i][j] = even + odd;
      }

    // Tile-level decision: only edge tiles pay for element masking.
    bool need_mask = k0 + TN > k_end || tile_bits != nullptr;
    if (p.mask_kind == AF_MASK_CAUSAL) need_mask = need_mask || (k0 + TN - 1 > r0 + p.q_offset);
    if (p.mask_kind == AF_MASK_WINDOW) need_mask = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = r0 + ty * 4 + i;
      const int pos = row + p.q_offset;          // the row's position on the key axis
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + tx + 16 * j;
        float x = s[i][j] * p.sm_scale;
        if (p.bias_kind == AF_BIAS_ALIBI) {
          x += -slope * (float)abs(pos - key);
        } else if (p.bias_kind == AF_BIAS_ADDITIVE) {
          if (row < p.N_q && key < p.N_kv)
            x += ld_elem<T>(p.bias, (int64_t)b * p.bias_stride[0] + (int64_t)h * p.bias_stride[1] +
                                        (int64_t)row * p.bias_stride[2] + (int64_t)key * p.bias_stride[3]);
        }
        if (need_mask) {
          bool keep = key < k_end;
          if (tile_bits != nullptr && keep && row < r_end)
            keep = (tile_bits[(int64_t)(row - qb * p.block_m) * bit_words + ((key - key_base) >> 6)] >> ((key - key_base) & 63)) & 1ull;
          if (p.mask_kind == AF_MASK_CAUSAL) keep = keep && (pos >= key);
          if (p.mask_kind == AF_MASK_WINDOW) keep = keep && (abs(pos - key) < p.window);
          x = keep ? x : -INFINITY;
        }
        s[i][j] = x;
        mx = fmaxf(mx, x);
      }
      if (p.norm_kind == AF_NORM_SOFTMAX) {
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m_i[i], mx);
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        const float alpha = expf(m_i[i] - m_use);  // exp(-inf) = 0 on the first tile
        float rs = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e = expf(s[i][j] - m_use);
          s[i][j] = e;
          rs += e;
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
        l_i[i] = alpha * l_i[i] + rs;
        m_i[i] = m_new;
#pragma unroll
        for (int c = 0; c < NCH * 2; ++c) acc[i][c] = f32x2_mul(acc[i][c], f32x2_pack(alpha, alpha));
      } else {
        float rs = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e = fmaxf(s[i][j], 0.f);
          s[i][j] = e;
          rs += e;
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
        l_i[i] += rs;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(sP + (ty * 4 + i) * LDP + 2 * (tx + 16 * j)) = make_float2(s[i][j], s[i][j]);
    }
    if (VEC) copy_wait<0>();
    group_sync(grp);           // P and V are there, everybody has read K

    more = advance();
    if (G == 2 && more) more = advance();
    if (more) load_tile<T, DMAX, VEC, TN>(sK, k_base, p.k_stride[2], p.k_stride[3], k0, k_end, p, p.rope != 0, 0);
    if (VEC) copy_commit();

#pragma unroll 4
    for (int n = 0; n < TN; n += 2) {
      ulonglong2 pv[4];                  // (p_n, p_n), (p_n+1, p_n+1)
#pragma unroll
      for (int i = 0; i < 4; ++i) pv[i] = *reinterpret_cast<const ulonglong2*>(sP + (ty * 4 + i) * LDP + 2 * n);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(sV + (n + u) * LD + c * 64 + tx * 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t w = u == 0 ? pv[i].x : pv[i].y;
            acc[i][c * 2] = f32x2_fma(w, vv.x, acc[i][c * 2]);
            acc[i][c * 2 + 1] = f32x2_fma(w, vv.y, acc[i][c * 2 + 1]);
          }
        }
      }
    }
    group_sync(grp);           // V and P may be overwritten
  }
  if (VEC) copy_wait<0>();     // a CTA without key tiles still has its Q copies in flight

  if (G == 2) {
    // Merge: group 1 leaves (m, l, accumulators) in its own buffers, group 0 takes them in.  ReLU has no
    // maximum: both weights are 1.
    float* xm = smem + TM * LD + GROUP_FLOATS;             // [TM] m, [TM] l, then [TM][DMAX]
    float* xo = xm + 2 * TM;
    if (grp == 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (tx == 0) { xm[r] = m_i[i]; xm[TM + r] = l_i[i]; }
#pragma unroll
        for (int c = 0; c < NCH; ++c)
          *reinterpret_cast<ulonglong2*>(xo + r * DMAX + c * 64 + tx * 4) = make_ulonglong2(acc[i][c * 2], acc[i][c * 2 + 1]);
      }
    }
    __syncthreads();
    if (grp == 1) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty * 4 + i;
      const float m_o = xm[r], l_o = xm[TM + r];
      float w = 1.f, w_o = 1.f;
      if (p.norm_kind == AF_NORM_SOFTMAX) {
        const float m_new = fmaxf(m_i[i], m_o), m_use = (m_new == -INFINITY) ? 0.f : m_new;
        w = expf(m_i[i] - m_use);
        w_o = expf(m_o - m_use);
        m_i[i] = m_new;
      }
      l_i[i] = l_i[i] * w + l_o * w_o;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const ulonglong2 o = *reinterpret_cast<const ulonglong2*>(xo + r * DMAX + c * 64 + tx * 4);
        acc[i][c * 2] = f32x2_fma(o.x, f32x2_pack(w_o, w_o), f32x2_mul(acc[i][c * 2], f32x2_pack(w, w)));
        acc[i][c * 2 + 1] = f32x2_fma(o.y, f32x2_pack(w_o, w_o), f32x2_mul(acc[i][c * 2 + 1], f32x2_pack(w, w)));
      }
    }
  }

  const int64_t o_off = (int64_t)b * a.o_stride[0] + (int64_t)h * a.o_stride[1];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = r0 + ty * 4 + i;
    if (row >= r_end) continue;
    const float safe_l = (l_i[i] == 0.f) ? 1.f : l_i[i];
    const float inv = 1.f / safe_l;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int d0 = c * 64 + tx * 4;
      float ov[4];
      f32x2_unpack(acc[i][c * 2], ov[0], ov[1]);
      f32x2_unpack(acc[i][c * 2 + 1], ov[2], ov[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) ov[e] *= inv;
      if (VEC) {
        if (d0 < D)
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.o) + o_off + (int64_t)row * a.o_stride[2] + d0) =
              make_float4(ov[0], ov[1], ov[2], ov[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (d0 + e < D)
            reinterpret_cast<T*>(a.o)[o_off + (int64_t)row * a.o_stride[2] + (int64_t)(d0 + e) * a.o_stride[3]] =
                Elem<T>::from_f32(ov[e]);
      }
    }
    if (a.lse != nullptr && tx == 0)
      a.lse[(int64_t)b * a.lse_stride[0] + (int64_t)h * a.lse_stride[1] + (int64_t)row * a.lse_stride[2]] =
          m_i[i] + logf(safe_l);
  }
}

// 16-byte accesses: fp32, unit inner strides, every row of Q, K, V and O on a 16-byte boundary; a
// rotated tile also takes the halves of a row and the table rows 16 bytes at a time.
bool vec_rows(const AfFwdParams& a) {
  const AfProblem& p = a.p;
  if (p.dtype != AF_F32 || p.D % 4 != 0) return false;
  auto ok = [](const void* ptr, const int64_t* st) {
    return ((uintptr_t)ptr & 15) == 0 && st[3] == 1 && st[2] % 4 == 0 && st[1] % 4 == 0 && st[0] % 4 == 0;
  };
  if (!ok(p.q, p.q_stride) || !ok(p.k, p.k_stride) || !ok(p.v, p.v_stride) || !ok(a.o, a.o_stride)) return false;
  if (p.rope && (p.D % 8 != 0 || p.rope_stride_n % 4 != 0 || ((uintptr_t)p.cos & 15) != 0 || ((uintptr_t)p.sin & 15) != 0))
    return false;
  return true;
}

template <typename T, int DMAX, bool VEC>
int launch_one(const AfFwdParams& a, cudaStream_t st) {
  const AfProblem& p = a.p;
  constexpr int G = Groups<DMAX>::value;
  const size_t smem = sizeof(float) * ((size_t)TM * (DMAX + PAD) + (size_t)G * (2 * TN * (DMAX + PAD) + TM * LDP));
  auto kern = fwd_ffma_kernel<T, DMAX, VEC>;
  AF_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int subs = 1, row_tiles;
  if (p.mask_kind == AF_MASK_BLOCKS) {
    subs = (p.block_m + TM - 1) / TM;
    row_tiles = ((p.N_q + p.block_m - 1) / p.block_m) * subs;
  } else {
    row_tiles = (p.N_q + TM - 1) / TM;
  }
  const int64_t ctas = (int64_t)row_tiles * p.B * p.H_q;
  AF_REQUIRE(ctas <= 0x7fffffff, "too many tiles for one launch");
  const dim3 grid((unsigned)ctas);
  kern<<<grid, NT * G, smem, st>>>(a, subs);
  count_launch();
  return check_cuda(cudaGetLastError(), "fwd_ffma launch");
}

template <typename T, bool VEC>
int launch_dtype(const AfFwdParams& a, cudaStream_t st) {
  if (a.p.D <= 64) return launch_one<T, 64, VEC>(a, st);
  if (a.p.D <= 128) return launch_one<T, 128, VEC>(a, st);
  return launch_one<T, 256, VEC>(a, st);
}

}  // namespace

int launch_fwd_ffma(const AfFwdParams& a, cudaStream_t st) {
  if (a.p.N_q == 0 || a.p.B == 0 || a.p.H_q == 0) return AF_OK;
  switch (a.p.dtype) {
    case AF_F16: return launch_dtype<__half, false>(a, st);
    case AF_BF16: return launch_dtype<__nv_bfloat16, false>(a, st);
    case AF_F32: return vec_rows(a) ? launch_dtype<float, true>(a, st) : launch_dtype<float, false>(a, st);
  }
  return fail(AF_ERR_INVALID, "unknown dtype %d", a.p.dtype);
}

}  // namespace af
