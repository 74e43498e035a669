// Chunk-local stage of the chunkwise forward, SIMT (CUDA-core) family: any DK <= 128 (multiple
// of 8), any DV (multiple of 4), fp32 arithmetic throughout. One 256-thread block per
// (chunk, batch*head).
//
// The two intra-chunk matrices are sums over channels of x_r * k_s * exp2(l_{s+1} + .. + l_r), r >= s, l = g * log2(e)
// (exponents <= 0 for decays), evaluated in 4 x 4 tiles of (r, s). On a tile of the diagonal every pair has its own
// exponential (the form the reference uses for its diagonal sub-blocks, intra_diag_kernel, gdn2/forward.py:220-235 of the
// reference project). Below it the exponent is split at the tile's first row, 7 exponentials per channel for the tile's 16.
//
// An exponent is never the difference of two rounded prefix sums: a strong gate (-100, or -inf) would swallow the ones
// after it, and a token-by-token evaluation knows no such loss. The decays stay one by one in shared memory; a span is the
// sum of the up to three at each end and of the four-token groups in between, whose prefix sums are kept as unevaluated
// pairs (high, low), so their difference is right to its own size. Gates are read as max(g, kMinGate), whose exponential is
// zero already: sums stay finite. With one gate of -1e6 in 40 tokens, D = 64, the outputs are off by 1.3e-7 of their norm;
// differences of prefix sums over the chunk gave 4e-2, and NaN for -inf.
//
// The inverse (I + Tm)^-1 is built by 16 x 16 blocks (solve_kernel, gdn2/forward.py:424-434, substitutes column by column),
// then W = Ai E, U = Ai (w*v), KG and Qg follow wy_kernel (gdn2/forward.py:512-533) and the query scaling of
// prefill_scan_kernel (gdn2/inference.py:461).
//
// What bounds it: a call of this family has few chunk-heads (hundreds), so a block's own chain of phases sets the
// time. Hence eight lanes per tile and register tiles of 4 x 4 in every product; one pair per warp and a
// substitution over all 64 rows by one thread per column set the
// pace before. Measured with the scan (scan_simt.cu), B = 2, S = 1000, 8 heads of 64, float32: the call took 501 us,
// now 79 (75.5 with differences of prefix sums).
//
// This family also serves as the exact path for chunks the tensor-core family flags as decaying
// too fast for its factorised diagonal blocks (`only_flagged`).
#include <type_traits>

#include "common.cuh"

namespace gdn2 {

namespace {

constexpr int LT = kChunk + 4;        // floats per row of the transposed 64 x 64 matrices
__host__ __device__ inline int row_stride(int DK) { return DK + 4; }   // floats per token row: 16-byte aligned, rows 4 banks apart

constexpr float kMinGate = -110.f;    // exp(-104) is already below half of float32's smallest number
constexpr int kGroups = kChunk / 4;   // groups of four tokens

// 2^x to the instruction's documented error, a relative 2^-22; zero far below float32's range
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gate_log2(float g) { return (g < kMinGate ? kMinGate : g) * kLog2e; }   // (a NaN stays one)
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                     __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ float4 load4(const __half* p) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> struct alignas(4 * sizeof(T)) Pack4 { T x[4]; };
template <typename T> __device__ __forceinline__ void store4(T* p, T a, T b, T c, T d) {
  *reinterpret_cast<Pack4<T>*>(p) = Pack4<T>{{a, b, c, d}};
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }

// acc[i][j] += a_i * b_j
__device__ __forceinline__ void outer4(float (&acc)[4][4], float4 a, float4 b) {
  const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
  }
}

// The whole chunk-local stage for chunk n of (batch, KEY head) bk, by one 256-thread block: everything that depends
// on q, k, b, g once, then U = Ai (w*v) for each of the H / HK value heads that share the key head. `S` tokens per
// batch entry, NC = ceil(S / 64): the rows past the end count as tokens with k = q = v = 0 and no decay, which leave
// the state alone.
// With packed sequences n counts the chunks of all of them (B = 1) and every sequence has ceil(length / 64), or only its
// whole ones when the tensor-core family made the table.
template <typename TIn, typename TW, typename Seqs>
__device__ __forceinline__ void prep_simt_chunk(const TIn* __restrict__ q, const TIn* __restrict__ k,
                                                const TIn* __restrict__ v, const float* __restrict__ g,
                                                const TIn* __restrict__ b, const TIn* __restrict__ w,
                                                const WsLayout& L, const WsPtrs& P, int S, int H, int HK, int64_t in_bs,
                                                float scale, int n, int bk, const Seqs& seqs) {
  constexpr int BS = kChunk;
  using WT = WsTraits<TW>;
  using TV = typename WT::TV;
  constexpr int E = WT::E;
  const int DK = L.DK, DV = L.DV, LD = row_stride(L.DK);
  int NC, row_tok, rows;               // chunks per row of records; first token and number of tokens of this chunk
  if constexpr (std::is_same<Seqs, PackedSeqs>::value) {
    const int i = packed_find(seqs.n, n, [&](int y) { return seqs.chunk[y]; }), local = (n - seqs.chunk[i]) * BS;
    NC = seqs.chunk[seqs.n];
    row_tok = seqs.tok[i] + local;
    rows = min(BS, seqs.tok[i + 1] - row_tok);
  } else {
    NC = (S + BS - 1) / BS;
    row_tok = n * BS;
    rows = min(BS, S - row_tok);
  }
  const int ib = bk / HK, ihk = bk % HK;
  const int64_t ch = (int64_t)bk * NC + n;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;

  extern __shared__ __align__(16) float sm[];
  float* Ls = sm;                    // [BS][LD] log2 decay of every token
  float* ks = Ls + BS * LD;          // [BS][LD] k
  float* es = ks + BS * LD;          // [BS][LD] b*k, later E = b*k*gamma
  float* qs = es + BS * LD;          // [BS][LD] q, later the w*v tiles
  float* TT = qs + BS * LD;          // [BS][LT] Tm transposed (row s, column r; strictly s < r), later N
  float* AT = TT + BS * LT;          // [BS][LT] (I + Tm)^-1 transposed
  float* Ch = AT + BS * LT;          // [17][LD] decay of the four-token groups before group x: high part ...
  float* Cl = Ch + (kGroups + 1) * LD;   // ... and what its rounding lost

  TW* wq = reinterpret_cast<TW*>(P.wq + (size_t)ch * L.wq_bytes);
  TV* aqk = reinterpret_cast<TV*>(P.aqk + (size_t)ch * L.aqk_bytes);
  TV* kgt = reinterpret_cast<TV*>(P.kgt + (size_t)ch * L.kgt_bytes);

  const size_t tok0 = ((size_t)ib * in_bs + row_tok) * HK + ihk;   // token index of row 0 (stride HK per row)
  const int nq = DK / 4;                                                  // channel quads
#pragma unroll 4
  for (int idx = tid; idx < BS * nq; idx += 256) {
    const int t = idx / nq, c = 4 * (idx % nq);
    const size_t gi = (tok0 + (size_t)t * HK) * DK + c;
    float4 kk = make_float4(0.f, 0.f, 0.f, 0.f), qq = kk, bb = kk, gg = kk;
    if (t < rows) { kk = load4(k + gi); qq = load4(q + gi); bb = load4(b + gi); gg = load4(g + gi); }
    *reinterpret_cast<float4*>(&ks[t * LD + c]) = kk;
    *reinterpret_cast<float4*>(&qs[t * LD + c]) = qq;
    *reinterpret_cast<float4*>(&es[t * LD + c]) = mul4(bb, kk);
    *reinterpret_cast<float4*>(&Ls[t * LD + c]) = make_float4(gate_log2(gg.x), gate_log2(gg.y), gate_log2(gg.z), gate_log2(gg.w));
  }
  __syncthreads();
  // totals of the groups, then their prefix sums as (high, low) pairs: the rounding error of every addition is collected
  // (Knuth's two-sum)
  for (int it = tid; it < kGroups * DK; it += 256) {
    const int c = it % DK, x = it / DK;
    const float* l = &Ls[4 * x * LD + c];
    Ch[(x + 1) * LD + c] = (l[0] + l[LD]) + (l[2 * LD] + l[3 * LD]);
  }
  __syncthreads();
  for (int c = tid; c < DK; c += 256) {
    float hi = 0.f, lo = 0.f;
    Ch[c] = 0.f; Cl[c] = 0.f;
#pragma unroll
    for (int x = 1; x <= kGroups; ++x) {
      const float t = Ch[x * LD + c], sum = hi + t, part = sum - hi;
      lo += (hi - (sum - part)) + (t - part);
      hi = sum;
      Ch[x * LD + c] = hi; Cl[x * LD + c] = lo;
    }
  }
  // the part of the Aqk image above the diagonal tiles
  for (int idx = tid; idx < BS * (BS / 4); idx += 256) {
    const int r = idx % BS, sq = idx / BS;
    if (sq > r / 4) store4(aqk + kc_index<E>(r, 4 * sq, BS), WT::kg_store(0.f), WT::kg_store(0.f), WT::kg_store(0.f), WT::kg_store(0.f));
  }
  __syncthreads();

  // exponent of gamma_t: the groups before t's, then its own group up to t
  auto gamma_log2 = [&](int t, int c) {
    float4 a = *reinterpret_cast<const float4*>(&Ls[(t & ~3) * LD + c]);
#pragma unroll
    for (int x = 1; x < 4; ++x)
      if (x <= (t & 3)) a = add4(a, *reinterpret_cast<const float4*>(&Ls[((t & ~3) + x) * LD + c]));
    return add4(*reinterpret_cast<const float4*>(&Ch[(t >> 2) * LD + c]), add4(*reinterpret_cast<const float4*>(&Cl[(t >> 2) * LD + c]), a));
  };

  // The two matrices: 120 tiles below the diagonal, then the 16 on it; eight lanes per tile share its channels. The loops are a
  // chain of shared-memory loads and exponentials: two turns at a time 36.8 us against 37.8 for one and 37.1 for four (the
  // kernel, float32, B = 2, S = 1000, 8 heads of 64).
  const int l8 = lane & 7;
  for (int grp = wid; grp < 34; grp += 8) {
    const int p = 4 * grp + (lane >> 3);
    float val[32];                                        // [0, 16): q side, [16, 32): erase side; 4 * (r - r0) + (s - s0)
#pragma unroll
    for (int x = 0; x < 32; ++x) val[x] = 0.f;
    int rt, st;
    if (grp < 30) {
      rt = (int)((1.f + sqrtf(8.f * p + 1.f)) * 0.5f);    // largest rt with rt (rt - 1) / 2 <= p
      if (rt * (rt - 1) / 2 > p) --rt;
      if ((rt + 1) * rt / 2 <= p) ++rt;
      st = p - rt * (rt - 1) / 2;
#pragma unroll 2
      for (int u = l8; u < DK / 2; u += 8) {
        const int o_r = 4 * rt * LD + 2 * u, o_s = 4 * st * LD + 2 * u;
        auto at2 = [&](const float* m, int off) { return *reinterpret_cast<const float2*>(m + off); };
        // from the last source token to the tile's first row: the groups in between and that row's own decay
        const float2 h1 = at2(Ch, rt * LD + 2 * u), h0 = at2(Ch, (st + 1) * LD + 2 * u);
        const float2 w1 = at2(Cl, rt * LD + 2 * u), w0 = at2(Cl, (st + 1) * LD + 2 * u), lr = at2(Ls, o_r);
        float2 e = make_float2(((h1.x - h0.x) + (w1.x - w0.x)) + lr.x, ((h1.y - h0.y) + (w1.y - w0.y)) + lr.y);
        float2 kf[4], tail = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          const float2 kj = at2(ks, o_s + j * LD);
          kf[j] = make_float2(kj.x * ex2(e.x + tail.x), kj.y * ex2(e.y + tail.y));
          if (j > 0) tail = add2(tail, at2(Ls, o_s + j * LD));
        }
        float2 head = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 qi = at2(qs, o_r + i * LD), ei = at2(es, o_r + i * LD);
          if (i > 0) {
            head = add2(head, at2(Ls, o_r + i * LD));
            const float ax = ex2(head.x), ay = ex2(head.y);
            qi.x *= ax; qi.y *= ay; ei.x *= ax; ei.y *= ay;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            val[4 * i + j] = fmaf(qi.x, kf[j].x, fmaf(qi.y, kf[j].y, val[4 * i + j]));
            val[16 + 4 * i + j] = fmaf(ei.x, kf[j].x, fmaf(ei.y, kf[j].y, val[16 + 4 * i + j]));
          }
        }
      }
    } else {
      rt = st = p - 120;
#pragma unroll 2
      for (int u = l8; u < DK / 2; u += 8) {
        const int o_r = 4 * rt * LD + 2 * u;
        float2 kk[4];                                      // k_j with the decay up to row i
#pragma unroll
        for (int i = 0; i < 4; ++i) kk[i] = *reinterpret_cast<const float2*>(&ks[o_r + i * LD]);
        float2 span[3];                                    // exponents from rows 0, 1, 2 to row i
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 li = *reinterpret_cast<const float2*>(&Ls[o_r + i * LD]);
#pragma unroll
          for (int j = 0; j < i; ++j) span[j] = j == i - 1 ? li : add2(span[j], li);
          const float2 qi = *reinterpret_cast<const float2*>(&qs[o_r + i * LD]), ei = *reinterpret_cast<const float2*>(&es[o_r + i * LD]);
#pragma unroll
          for (int j = 0; j <= i; ++j) {
            float2 kd = kk[j];
            if (j < i) { kd.x *= ex2(span[j].x); kd.y *= ex2(span[j].y); }
            val[4 * i + j] = fmaf(qi.x, kd.x, fmaf(qi.y, kd.y, val[4 * i + j]));
            if (j < i) val[16 + 4 * i + j] = fmaf(ei.x, kd.x, fmaf(ei.y, kd.y, val[16 + 4 * i + j]));
          }
        }
      }
    }
    // sum over the eight lanes; each step halves what a lane keeps: bit 2 chooses the matrix, bits 1 and 0 the row
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const int half = 16 >> m, bit = 4 >> m;
      const bool up = (lane & bit) != 0;
#pragma unroll
      for (int x = 0; x < half; ++x) {
        const float send = up ? val[x] : val[x + half], keep = up ? val[x + half] : val[x];
        val[x] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
      }
    }
    const int r = 4 * rt + (lane & 3), s0 = 4 * st;
    if (lane & 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) TT[(s0 + j) * LT + r] = val[j];
    } else {
      store4(aqk + kc_index<E>(r, s0, BS), WT::kg_store(val[0] * scale), WT::kg_store(val[1] * scale),
             WT::kg_store(val[2] * scale), WT::kg_store(val[3] * scale));
    }
  }
  __syncthreads();

  // (I + Tm)^-1 by 16 x 16 blocks, everything transposed (a row of AT is a column of the inverse):
  //   X_ii = D_i = (I + T_ii)^-1;   N_ik = D_i T_ik;   X_ij = - sum_{k=j}^{i-1} N_ik X_kj
  if (tid < BS) {
    const int i = tid >> 4, j = tid & 15;
    const float* tb = TT + 16 * i * LT + 16 * i;          // T_ii[r][s] = tb[s * LT + r]
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = r == j ? 1.f : 0.f;
#pragma unroll
    for (int s_ = 0; s_ < 15; ++s_) {
#pragma unroll
      for (int r4 = (s_ + 1) / 4; r4 < 4; ++r4) {
        const float4 t4 = *reinterpret_cast<const float4*>(&tb[s_ * LT + 4 * r4]);
        const float tv[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
        for (int y = 0; y < 4; ++y)
          if (4 * r4 + y > s_) x[4 * r4 + y] = fmaf(-tv[y], x[s_], x[4 * r4 + y]);
      }
    }
#pragma unroll
    for (int r4 = 0; r4 < 4; ++r4)
      *reinterpret_cast<float4*>(&AT[tid * LT + 16 * i + 4 * r4]) = make_float4(x[4 * r4], x[4 * r4 + 1], x[4 * r4 + 2], x[4 * r4 + 3]);
  } else {
    // meanwhile the other six warps: gamma_last, the query rows Qg and KG^T, which need the decays, q and k only
    const int z = tid - BS, nz = 256 - BS;
    for (int idx = z; idx < BS * nq; idx += nz) {          // tokens fastest: 16-byte pieces in a row
      const int t = idx % BS, c = 4 * (idx / BS);
      const float4 G = gamma_log2(t, c), qq = *reinterpret_cast<const float4*>(&qs[t * LD + c]);
      store4(wq + kc_index<E>(BS + t, c, 2 * BS), from_f32<TW>(scale * qq.x * ex2(G.x)), from_f32<TW>(scale * qq.y * ex2(G.y)),
             from_f32<TW>(scale * qq.z * ex2(G.z)), from_f32<TW>(scale * qq.w * ex2(G.w)));
    }
    for (int idx = z; idx < (BS / 4) * DK; idx += nz) {
      const int c = idx % DK, t = 4 * (idx / DK);
      // from t + 3 to the chunk's last token: the groups after this one
      const int x = t / 4 + 1;
      float e = (Ch[kGroups * LD + c] - Ch[x * LD + c]) + (Cl[kGroups * LD + c] - Cl[x * LD + c]), tail = 0.f;
      float kg[4];
#pragma unroll
      for (int y = 3; y >= 0; --y) {
        kg[y] = ks[(t + y) * LD + c] * ex2(e + tail);
        if (y > 0) tail += Ls[(t + y) * LD + c];
      }
      store4(kgt + kc_index<E>(c, t, DK), WT::kg_store(kg[0]), WT::kg_store(kg[1]), WT::kg_store(kg[2]), WT::kg_store(kg[3]));
    }
    float* gl = P.gl + (size_t)ch * DK;
    for (int c = z; c < DK; c += nz) gl[c] = ex2(Ch[kGroups * LD + c] + Cl[kGroups * LD + c]);
  }
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass) {                   // N^T in place over T^T: 6 blocks x 16 rows t x 4 row quads
    const int it = tid + 256 * pass;
    if (it < 384) {                                        // whole warps
      const int blk = it >> 6, t = (it >> 2) & 15, r4 = 4 * (it & 3);
      const int bi = blk < 1 ? 1 : blk < 3 ? 2 : 3, bkk = blk < 1 ? 0 : blk < 3 ? blk - 1 : blk - 3;
      float* trow = TT + (16 * bkk + t) * LT + 16 * bi;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const float4 d = *reinterpret_cast<const float4*>(&AT[(16 * bi + u) * LT + 16 * bi + r4]);
        const float tv = trow[u];
        a.x = fmaf(d.x, tv, a.x); a.y = fmaf(d.y, tv, a.y); a.z = fmaf(d.z, tv, a.z); a.w = fmaf(d.w, tv, a.w);
      }
      __syncwarp();                                        // the four lanes of a row have read it
      *reinterpret_cast<float4*>(&trow[r4]) = a;
    }
  }
  // E = b k gamma in place (needed from here on)
  for (int idx = tid; idx < BS * nq; idx += 256) {
    const int t = idx / nq, c = 4 * (idx % nq);
    const float4 G = gamma_log2(t, c);
    float4* ep = reinterpret_cast<float4*>(&es[t * LD + c]);
    *ep = mul4(*ep, make_float4(ex2(G.x), ex2(G.y), ex2(G.z), ex2(G.w)));
  }
  __syncthreads();
  for (int d = 1; d < 4; ++d) {
    if (tid < 64 * (4 - d)) {
      const int bj = tid >> 6, c = (tid >> 2) & 15, r4 = 4 * (tid & 3), bi = bj + d;
      float* xcol = AT + (16 * bj + c) * LT;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 16
      for (int t = 16 * bj; t < 16 * bi; ++t) {
        const float4 nn = *reinterpret_cast<const float4*>(&TT[t * LT + 16 * bi + r4]);
        const float xv = xcol[t];
        a.x = fmaf(-nn.x, xv, a.x); a.y = fmaf(-nn.y, xv, a.y); a.z = fmaf(-nn.z, xv, a.z); a.w = fmaf(-nn.w, xv, a.w);
      }
      *reinterpret_cast<float4*>(&xcol[16 * bi + r4]) = a;
    }
    __syncthreads();
  }

  // W = Ai E: one thread per 4 tokens x 4 channels; row quad rq needs the source tokens up to its own only
  for (int idx = tid; idx < 16 * nq; idx += 256) {
    const int rq = idx / nq, c = 4 * (idx % nq);
    float acc[4][4] = {};
#pragma unroll 4
    for (int s_ = 0; s_ < 4 * rq + 4; ++s_)
      outer4(acc, *reinterpret_cast<const float4*>(&AT[s_ * LT + 4 * rq]), *reinterpret_cast<const float4*>(&es[s_ * LD + c]));
#pragma unroll
    for (int i = 0; i < 4; ++i)
      store4(wq + kc_index<E>(4 * rq + i, c, 2 * BS), from_f32<TW>(acc[i][0]), from_f32<TW>(acc[i][1]), from_f32<TW>(acc[i][2]),
             from_f32<TW>(acc[i][3]));
  }
  // U = Ai (w*v) for every value head of this key head, value columns in tiles of DK
  const int rep = H / HK;
  for (int hr = 0; hr < rep; ++hr) {
    const int ih = ihk * rep + hr;
    const size_t tok0v = ((size_t)ib * in_bs + row_tok) * H + ih;
    TV* ut = reinterpret_cast<TV*>(P.ut + (size_t)(((int64_t)ib * H + ih) * NC + n) * L.ut_bytes);
    for (int c0 = 0; c0 < DV; c0 += DK) {
      const int cwq = min(DK, DV - c0) / 4;
      if (hr + c0 > 0) __syncthreads();                    // the previous tile has been read (the query rows long since)
#pragma unroll 4
      for (int idx = tid; idx < BS * cwq; idx += 256) {
        const int t = idx / cwq, c = 4 * (idx % cwq);
        const size_t gi = (tok0v + (size_t)t * H) * DV + c0 + c;
        *reinterpret_cast<float4*>(&qs[t * LD + c]) = t < rows ? mul4(load4(w + gi), load4(v + gi)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
      for (int idx = tid; idx < 16 * cwq; idx += 256) {
        const int rq = idx / cwq, c = 4 * (idx % cwq);
        float acc[4][4] = {};
#pragma unroll 4
        for (int s_ = 0; s_ < 4 * rq + 4; ++s_)
          outer4(acc, *reinterpret_cast<const float4*>(&AT[s_ * LT + 4 * rq]), *reinterpret_cast<const float4*>(&qs[s_ * LD + c]));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          store4(ut + kc_index<E>(c0 + c + j, 4 * rq, DV), WT::u_store(acc[0][j]), WT::u_store(acc[1][j]), WT::u_store(acc[2][j]),
                 WT::u_store(acc[3][j]));
      }
    }
  }
}

template <typename TIn, typename TW, typename Seqs>
__global__ void __launch_bounds__(256, 2)
prep_simt_kernel(const TIn* __restrict__ q, const TIn* __restrict__ k, const TIn* __restrict__ v,
                 const float* __restrict__ g, const TIn* __restrict__ b, const TIn* __restrict__ w,
                 WsLayout L, WsPtrs P, int S, int H, int HK, int64_t in_bs, float scale, const __grid_constant__ Seqs seqs) {
  grid_wait();
  prep_simt_chunk<TIn, TW>(q, k, v, g, b, w, L, P, S, H, HK, in_bs, scale, blockIdx.x, blockIdx.y, seqs);
}

// Exact redo of the chunks the tensor-core kernel flagged: a fixed small grid looks through the flags, every block at its
// own share of them (chunk-heads blockIdx.x + i * gridDim.x, so that neighbours that are flagged together spread over the
// blocks). A list of the flagged chunks needed its length cleared before every call, one more operation in the stream;
// the call's time is the same either way (prompt segment of 1037 tokens, 63 us).
template <typename TIn, typename TW, typename Seqs>
__global__ void __launch_bounds__(256, 1)
prep_simt_flagged_kernel(const TIn* __restrict__ q, const TIn* __restrict__ k, const TIn* __restrict__ v,
                         const float* __restrict__ g, const TIn* __restrict__ b, const TIn* __restrict__ w,
                         WsLayout L, WsPtrs P, int S, int H, int HK, int64_t in_bs, float scale, const __grid_constant__ Seqs seqs) {
  const int NC = S / kChunk;                           // chunks per row of records, packed or not
  __shared__ int todo[256], count;
  for (int64_t base = blockIdx.x; base < L.nch; base += (int64_t)256 * gridDim.x) {
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    const int64_t mine = base + (int64_t)threadIdx.x * gridDim.x;
    if (mine < L.nch && P.flags[mine]) todo[atomicAdd(&count, 1)] = (int)mine;
    __syncthreads();
    const int n = count;
    for (int i = 0; i < n; ++i) {
      prep_simt_chunk<TIn, TW>(q, k, v, g, b, w, L, P, S, H, HK, in_bs, scale, todo[i] % NC, todo[i] / NC, seqs);
      __syncthreads();                                 // shared memory is reused by the next chunk
    }
    __syncthreads();                                   // every thread has its count
  }
}

template <typename TIn, typename TW, typename Seqs>
int launch_typed(const void* q, const void* k, const void* v, const float* g, const void* b, const void* w,
                 const WsLayout& L, const WsPtrs& P, int B, int S, int H, int HK, int64_t in_bs, float scale,
                 bool only_flagged, const Seqs& seqs, cudaStream_t st) {
  const size_t smem = ((size_t)(4 * kChunk + 2 * (kGroups + 1)) * row_stride(L.DK) + 2 * kChunk * LT) * sizeof(float);
  const TIn* tq = static_cast<const TIn*>(q); const TIn* tk = static_cast<const TIn*>(k);
  const TIn* tv = static_cast<const TIn*>(v); const TIn* tb = static_cast<const TIn*>(b);
  const TIn* tw = static_cast<const TIn*>(w);
  if (only_flagged) {
    auto kern = prep_simt_flagged_kernel<TIn, TW, Seqs>;
    GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
    const int nch = (int)L.nch;
    kern<<<nch < 296 ? nch : 296, 256, smem, st>>>(tq, tk, tv, g, tb, tw, L, P, S, H, HK, in_bs, scale, seqs);
  } else {
    auto kern = prep_simt_kernel<TIn, TW, Seqs>;
    GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
    dim3 grid((S + kChunk - 1) / kChunk, B * HK);
    GDN2_CUDA_TRY(launch_chained(true, kern, grid, 256, smem, st, tq, tk, tv, g, tb, tw, L, P, S, H, HK, in_bs, scale, seqs));
  }
  GDN2_CUDA_TRY(cudaGetLastError());
  return GDN2_OK;
}

template <typename Seqs>
int launch_any(const void* q, const void* k, const void* v, const float* g, const void* b, const void* w,
               const WsLayout& L, const WsPtrs& P, int B, int S, int H, int HK, int64_t in_bs, float scale, int dtype,
               bool only_flagged, const Seqs& seqs, cudaStream_t st) {
  using bf16 = __nv_bfloat16;
  if (L.esz == 4) {
    switch (dtype) {
      case GDN2_F32: return launch_typed<float, float>(q, k, v, g, b, w, L, P, B, S, H, HK, in_bs, scale, only_flagged, seqs, st);
      case GDN2_BF16: return launch_typed<bf16, float>(q, k, v, g, b, w, L, P, B, S, H, HK, in_bs, scale, only_flagged, seqs, st);
      case GDN2_F16: return launch_typed<__half, float>(q, k, v, g, b, w, L, P, B, S, H, HK, in_bs, scale, only_flagged, seqs, st);
      default: return GDN2_ERR_BAD_DTYPE;
    }
  }
  if (dtype != GDN2_BF16) return GDN2_ERR_UNSUPPORTED;
  return launch_typed<bf16, bf16>(q, k, v, g, b, w, L, P, B, S, H, HK, in_bs, scale, only_flagged, seqs, st);
}

}  // namespace

int launch_prep_simt(const void* q, const void* k, const void* v, const float* g, const void* b, const void* w,
                     const WsLayout& L, const WsPtrs& P, int B, int S, int H, int HK, int64_t in_bs, float scale,
                     int dtype, bool only_flagged, cudaStream_t st) {
  return launch_any(q, k, v, g, b, w, L, P, B, S, H, HK, in_bs, scale, dtype, only_flagged, OneLength{}, st);
}

int launch_prep_simt_packed(const void* q, const void* k, const void* v, const float* g, const void* b, const void* w,
                            const WsLayout& L, const WsPtrs& P, const PackedSeqs& seqs, int H, int HK, float scale,
                            int dtype, bool only_flagged, cudaStream_t st) {
  return launch_any(q, k, v, g, b, w, L, P, 1, seqs.chunk[seqs.n] * kChunk, H, HK, 0, scale, dtype, only_flagged, seqs, st);
}

}  // namespace gdn2
