// Recurrent decode of several tokens for few (batch, head) tiles, DK = DV = 128: a tile spread over blocks by value columns.
//
// The columns of the state evolve independently of one another. Every warp holds 2 * CPT of them in registers for all n tokens and
// evaluates the recurrence token by token,
//     read = S^T (a*b*k);  u = w*v - read;  S <- a*S + k u^T;  o = scale * S^T q        (a = exp g)
// Lane (rl = lane & 15, cl = lane >> 4) has the row pairs rl, rl + 16, .. (four of the 64) of the CPT columns CPT * cl ..
// The sweep that forms o of a token also forms the read of the next: 2 CPT sums per lane, which four exchange steps reduce
// over the sixteen lanes to one per lane (even lanes a read, odd ones an output), and CPT shuffles bring u back to all.
//
// What bounds it is the chain of a token, some 0.3 us; decode_blocked.cu takes a whole tile per SM through a step of 8 tokens
// in 2.7 us and needs a third fewer FMAs, so it is the better one as soon as the tiles are many. Measured (bf16, us, blocked
// against this with CPT 2 / 4): 16 tiles, 16 tokens 11.1 and 7.2 / 8.5, 37 tokens 22.0 and 13.7 / 16.7, 63 tokens 32.9 and
// 21.1 / 26.4; 32 tiles, 37 tokens 22.0 and 17.4 / 16.7; 64 tiles, 37 tokens 22.4 and 26.6 / 21.1; up to 8 tokens no difference.
#include <type_traits>

#include "common.cuh"

namespace gdn2 {

namespace {

constexpr int D = 128;
constexpr int NB = 8;                       // tokens whose tables are in shared memory at a time (two such batches)
constexpr int kColThreads = 128;            // thread = key channel while tables are built

__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return d;
}

template <typename T, typename Seqs, int CPT>
__global__ void __launch_bounds__(kColThreads)
decode_cols_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const float* __restrict__ g,
                   const T* __restrict__ b, const T* __restrict__ w, float* __restrict__ state, T* __restrict__ o, int n,
                   int H, int HK, int64_t in_bs, int64_t o_bs, float scale, const __grid_constant__ Seqs seqs) {
  constexpr int kCols = 8 * CPT, kSlices = D / kCols;
  // per row pair (both rows of each): of token t scale*q, and a*b*k of token t + 1; k and a of token t. Slot NB of the first
  // table holds the a*b*k of the batch's first token.
  __shared__ float4 tab1[2][NB + 1][D / 2];
  __shared__ float4 tab2[2][NB][D / 2];
  __shared__ float wv[2][NB][kCols];        // w * v

  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x / kSlices, col_base = (blockIdx.x % kSlices) * kCols;
  const int ib = tile / H, ih = tile % H, ihk = ih / (H / HK);
  size_t row_in, row_o;                     // first input and output row, in tokens
  if constexpr (std::is_same<Seqs, PackedSeqs>::value) {   // the last len % 64 tokens of a packed sequence, perhaps none
    n = (seqs.tok[ib + 1] - seqs.tok[ib]) % kChunk;
    row_in = row_o = (size_t)(seqs.tok[ib + 1] - n);
    if (n == 0) return;
  } else {
    row_in = (size_t)ib * in_bs;
    row_o = (size_t)ib * o_bs;
  }

  grid_wait();
  grid_launch_dependents();

  using Row = typename std::conditional<CPT == 4, float4, float2>::type;
  const int rl = lane & 15, cl = lane >> 4;
  const int col = 2 * CPT * wid + CPT * cl;                 // first of this thread's columns within the slice
  float2 S[4][CPT];                                           // (row 2p, row 2p + 1) of each column, p = rl + 16 i
  float* gS = state + (size_t)tile * D * D + col_base + col;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t r = (size_t)2 * (rl + 16 * i) * D;
    float lo[CPT], hi[CPT];
    *reinterpret_cast<Row*>(lo) = *reinterpret_cast<const Row*>(gS + r);
    *reinterpret_cast<Row*>(hi) = *reinterpret_cast<const Row*>(gS + r + D);
#pragma unroll
    for (int c = 0; c < CPT; ++c) S[i][c] = make_float2(lo[c], hi[c]);
  }

  // token vectors of one batch: thread = key channel for g, k, q, b; (token, CPT / 2 columns) for v, w
  float rg[NB];
  constexpr int VC = CPT / 2;
  T rk[NB], rq[NB], rb[NB], rv[VC], rw[VC];
  const int vt = tid >> 4, vc = VC * (tid & 15);
  auto fetch = [&](int t0) {
    const int nb = n - t0;
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      if (t < nb) {
        const size_t e = ((row_in + t0 + t) * HK + ihk) * D + tid;
        rg[t] = __ldg(g + e); rk[t] = k[e]; rq[t] = q[e]; rb[t] = b[e];
      }
    }
    if (vt < nb) {
      const size_t e = ((row_in + t0 + vt) * H + ih) * D + col_base + vc;
      
#pragma unroll
      for (int x = 0; x < VC; ++x) { rv[x] = v[e + x]; rw[x] = w[e + x]; }
    }
  };
  auto store_tables = [&](int buf, int nb) {
    const int p = tid >> 1, s = tid & 1;
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      if (t < nb) {
        const float a = exp2f(rg[t] * kLog2e), kk = to_f32(rk[t]);
        reinterpret_cast<float*>(&tab1[buf][t][p])[s] = to_f32(rq[t]) * scale;
        reinterpret_cast<float*>(&tab1[buf][t ? t - 1 : NB][p])[2 + s] = a * (to_f32(rb[t]) * kk);
        reinterpret_cast<float*>(&tab2[buf][t][p])[s] = kk;
        reinterpret_cast<float*>(&tab2[buf][t][p])[2 + s] = a;
      }
    }
#pragma unroll
    for (int x = 0; x < VC; ++x)
      if (vt < nb) wv[buf][vt][vc + x] = to_f32(rw[x]) * to_f32(rv[x]);
  };

  // Sum of val[0 .. 2 CPT) over the sixteen lanes of a half warp. Lane bit 0 picks the lower or the upper CPT of them, the
  // next bits one of those; the lanes that differ in the bits left over get the same.
  constexpr int kPick = CPT == 4 ? 3 : 2;                   // exchange steps that halve what a lane keeps
  auto reduce = [&](float (&val)[2 * CPT]) {
#pragma unroll
    for (int m = 0; m < kPick; ++m) {
      const int half = CPT >> m;
      const bool up = (lane >> m) & 1;
#pragma unroll
      for (int x = 0; x < half; ++x) {
        const float send = up ? val[x] : val[x + half];
        const float keep = up ? val[x + half] : val[x];
        val[x] = keep + __shfl_xor_sync(0xffffffffu, send, 1 << m);
      }
    }
#pragma unroll
    for (int m = kPick; m < 4; ++m) val[0] += __shfl_xor_sync(0xffffffffu, val[0], 1 << m);
    return val[0];
  };
  // the column whose sum is left here, and the lane (of the lower half warp) that has the read of column c
  const int mycol = col + (CPT == 4 ? 2 * ((lane >> 1) & 1) + ((lane >> 2) & 1) : (lane >> 1) & 1);
  auto lane_of = [](int c) { return CPT == 4 ? 2 * ((c >> 1) & 1) + 4 * (c & 1) : 2 * c; };

  fetch(0);
  store_tables(0, n);
  __syncthreads();
  for (int t0 = 0, buf = 0; t0 < n; t0 += NB, buf ^= 1) {
    const int nb = n - t0 < NB ? n - t0 : NB;
    if (t0 + NB < n) fetch(t0 + NB);
    T* po = o + ((row_o + t0) * H + ih) * D + col_base + mycol;
    float sum;                                              // even lanes: the read of the token to come; odd: o of the last
    {
      float2 rd[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) rd[c] = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 P = tab1[buf][NB][rl + 16 * i];
#pragma unroll
        for (int c = 0; c < CPT; ++c) rd[c] = ffma2(S[i][c], make_float2(P.z, P.w), rd[c]);
      }
      float val[2 * CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) { val[c] = rd[c].x + rd[c].y; val[CPT + c] = 0.f; }
      sum = reduce(val);
    }
    for (int t = 0; t < nb; ++t) {
      const float mine = wv[buf][t][mycol] - sum;           // u of column mycol on the even lanes
      float2 u[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const float x = __shfl_sync(0xffffffffu, mine, (lane & 16) + lane_of(c));
        u[c] = make_float2(x, x);
      }
      float2 rd[CPT], ov[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) rd[c] = ov[c] = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 Q = tab2[buf][t][rl + 16 * i], P = tab1[buf][t][rl + 16 * i];
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          S[i][c] = ffma2(make_float2(Q.x, Q.y), u[c], fmul2(make_float2(Q.z, Q.w), S[i][c]));
          rd[c] = ffma2(S[i][c], make_float2(P.z, P.w), rd[c]);
          ov[c] = ffma2(S[i][c], make_float2(P.x, P.y), ov[c]);
        }
      }
      float val[2 * CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) { val[c] = rd[c].x + rd[c].y; val[CPT + c] = ov[c].x + ov[c].y; }
      sum = reduce(val);                                   // the batch's last read is not used (its table is stale)
      if ((lane & (CPT == 4 ? 9 : 13)) == 1) po[(size_t)t * H * D] = from_f32<T>(sum);
    }
    if (t0 + NB < n) {
      store_tables(buf ^ 1, n - t0 - NB);                   // read one batch ago, before the barrier below
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t r = (size_t)2 * (rl + 16 * i) * D;
    float lo[CPT], hi[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) { lo[c] = S[i][c].x; hi[c] = S[i][c].y; }
    *reinterpret_cast<Row*>(gS + r) = *reinterpret_cast<const Row*>(lo);
    *reinterpret_cast<Row*>(gS + r + D) = *reinterpret_cast<const Row*>(hi);
  }
}

}  // namespace

// Whether this form is taken for n tokens of ntiles tiles: with more than one step of the blocked form, and no more blocks than
// SMs (see above). A prompt's ragged tail, or those of a packed batch, take it by the number of tiles alone: how long the other
// tails of a launch are does not change the bits of one.
bool decode_cols_wins(int64_t ntiles, int n, bool tail) { return (tail || n > 8) && ntiles * 4 <= device_sm_count(); }

// ntiles (batch or packed sequence, head) tiles
template <typename T, typename Seqs>
int launch_decode_cols(const T* q, const T* k, const T* v, const float* g, const T* b, const T* w, float* state, T* o,
                       int ntiles, int n, int H, int HK, int64_t in_bs, int64_t o_bs, float scale, const Seqs& seqs, bool chained,
                       cudaStream_t st) {
  auto launch = [&](auto kern, int slices) {
    return launch_chained(chained, kern, dim3(ntiles * slices), kColThreads, 0, st, q, k, v, g, b, w, state, o, n, H, HK, in_bs, o_bs, scale, seqs);
  };
  // eight blocks per tile while they all run at once, then four (decode_cols_wins keeps those within one round)
  if (ntiles * 8 <= device_sm_count()) GDN2_CUDA_TRY(launch(decode_cols_kernel<T, Seqs, 2>, 8));
  else GDN2_CUDA_TRY(launch(decode_cols_kernel<T, Seqs, 4>, 4));
  return GDN2_OK;
}

#define GDN2_INSTANTIATE(T, SEQS)                                                                                          \
  template int launch_decode_cols<T, SEQS>(const T*, const T*, const T*, const float*, const T*, const T*, float*, T*, int, \
                                           int, int, int, int64_t, int64_t, float, const SEQS&, bool, cudaStream_t)
GDN2_INSTANTIATE(float, OneLength);
GDN2_INSTANTIATE(__half, OneLength);
GDN2_INSTANTIATE(__nv_bfloat16, OneLength);
GDN2_INSTANTIATE(__nv_bfloat16, PackedSeqs);
#undef GDN2_INSTANTIATE

}  // namespace gdn2
