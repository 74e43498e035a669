// One token per sequence through the whole GatedDeltaNet2 layer in three kernels, 16-bit storage, DK = DV = 128, four taps,
// at most kMaxRows sequences:
//   front  the seven input projections, a skinny product that reads W_cat once, with everything element-wise that follows
//          them (convolution, SiLU, L2 norm, gates, the new convolution cache) as its epilogue: a block owns the 128 columns
//          of one head of one kind, so a norm needs nothing from another block;
//   core   the recurrence of one token (decode.cu's arithmetic) with the gated RMSNorm as its epilogue, a block per (sequence,
//          head);
//   out    the output projection, a block per 16 columns.
// Against two library products and three kernels this saves two launches, eight allocations and the round trips of the
// projections through memory: hidden 2048, 16 heads, 2 sequences, 61.8 -> 24 us a call (the host), replayed from a graph
// 29.0 -> 20.5; 16 sequences replayed 31.5 -> 27.1. front takes 13.8 us of it, core 5.5, out 5.1 (ncu, cold caches). From 24
// sequences on the legacy tensor path and the library products were level (replayed 33.3 there, 37.6 here), hence kMaxRows.
//
// Every product takes its 16 weight rows as the 16-row operand of mma.sync m16n8k16 and the tokens as the 8-column one: the work is
// reading the weights once (42 + 8 MB at hidden 2048, 16 heads), which the tensor cores only have to keep up with. A lane reads
// 16 bytes of a weight row at a time, eight reduction steps that the two products of a 32-step group take as (words 0, 1) and
// (words 2, 3): any order of the reduction is as good as another as long as both operands use the same.
//
// The kernels are chained (launch_chained). `out` holds its share of the weights in registers before it waits for `core`,
// `core` its state before it waits for `front`: both are complete by then, see there.
#include <cooperative_groups.h>

#include "common.cuh"
#include "layer_math.cuh"

namespace gdn2 {

namespace {

constexpr int D = 128;
constexpr int kMaxRows = 16;        // two groups of eight tokens
constexpr int kFrontThreads = 256, kCoreThreads = 512, kOutThreads = 256;
constexpr int kRedStride = D + 4;

template <typename T> __device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma16816<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// weights: read once, not kept in L1
__device__ __forceinline__ uint4 ld_weight(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

// bytes of a token row in shared memory: 64 bytes more than the row, so that two rows fill the banks
__host__ __device__ constexpr int row_bytes(int K) { return K * 2 + 64; }

// K elements of rows m < M of x (stride apart) to shared memory, zeros up to `rows`; every copy in flight at once
template <typename T>
__device__ __forceinline__ void stage_rows(unsigned char* xs, const T* x, int M, int rows, int K, int stride, int tid, int threads) {
  const int per_row = K / 8;
  for (int i = tid; i < rows * per_row; i += threads) {
    const int m = i / per_row, c = i % per_row;
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(xs + (size_t)m * row_bytes(K) + c * 16));
    const T* src = x + (size_t)(m < M ? m : 0) * stride + c * 8;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(m < M ? 16 : 0) : "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// 64 reduction steps of 16 weight rows: [32-step group][rows g | rows g + 8]
struct Weights64 { uint4 w[2][2]; };
template <typename T>
__device__ __forceinline__ void load64(Weights64& r, const T* row_g, size_t eight_rows, int k0) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    r.w[s][0] = ld_weight(row_g + k0 + 32 * s);
    r.w[s][1] = ld_weight(row_g + eight_rows + k0 + 32 * s);
  }
}
// the same 64 steps of all tokens: xk addresses this lane's token row (lane >> 2) and 16-byte piece (lane & 3) at step k0
template <typename T, int NT>
__device__ __forceinline__ void mma64(float (&acc)[NT][4], const Weights64& r, const unsigned char* xk, int K) {
  uint4 xv[2][NT];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) xv[s][nt] = *reinterpret_cast<const uint4*>(xk + (size_t)nt * 8 * row_bytes(K) + 64 * s);
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      mma16816<T>(acc[nt], r.w[s][0].x, r.w[s][1].x, r.w[s][0].y, r.w[s][1].y, xv[s][nt].x, xv[s][nt].y);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      mma16816<T>(acc[nt], r.w[s][0].z, r.w[s][1].z, r.w[s][0].w, r.w[s][1].w, xv[s][nt].z, xv[s][nt].w);
  }
}

// buffers between the three kernels
struct StepBuffers {
  char *q, *k, *b, *v, *w, *gate, *normed;
  float* g;
};

// ---------------------------------------------------------------- front

// A cluster of two blocks = one head-wide slot (q, k, v, b, w, f or gate of one head), each block half of the reduction. Warp:
// 16 of the 128 columns, kAhead groups of 64 steps in flight. The halves meet in distributed shared memory and the two
// blocks share the tokens of the epilogue: one block per slot would leave 68 of the 148 SMs idle at hidden 2048 and 16 heads (hidden
// 1024 with 4 heads, two sequences, replayed: 14.4 us so, 12.3 with clusters).
template <typename T, int NT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFrontThreads)
layer_step_front_kernel(gdn2_layer_step_args a, StepBuffers buf) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kAhead = 4, kWarps = kFrontThreads / 32;
  grid_wait();
  grid_launch_dependents();
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int M = (int)a.B, hid = (int)a.hidden, H = (int)a.H, HK = (int)a.HK;

  enum { kQ, kK, kV, kB, kW, kF, kGate };
  int kind = kGate, head = blockIdx.x >> 1;
  int64_t off = a.off_gate;
  auto slots = [&](int which, int n, int64_t at) {                     // the first clusters are q heads, then k heads, ..
    if (kind == kGate && head < n) { kind = which; off = at; }
    else if (kind == kGate) head -= n;
  };
  slots(kQ, HK, a.off_q); slots(kK, HK, a.off_k); slots(kV, H, a.off_v);
  slots(kB, HK, a.off_b); slots(kW, H, a.off_w); slots(kF, HK, a.off_f);

  const int groups_all = hid / 64;                                     // of 64 reduction steps
  const int first = groups_all * rank / 2, groups = groups_all * (rank + 1) / 2 - first;
  const int Kh = 64 * groups, Kmost = 64 * ((groups_all + 1) / 2);
  unsigned char* xs = smem;                                            // [NT * 8][row_bytes(Kh)]
  float* red = reinterpret_cast<float*>(smem + (size_t)NT * 8 * row_bytes(Kmost));   // [NT * 8][kRedStride]
  const int g8 = lane >> 2, t4 = lane & 3;
  const T* row_g = static_cast<const T*>(a.w_cat) + (size_t)(off + head * D + 16 * wid + g8) * hid + 64 * first + 8 * t4;
  const size_t eight = (size_t)8 * hid;

  Weights64 w[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i)
    if (i < groups) load64(w[i], row_g, eight, 64 * i);
  stage_rows(xs, static_cast<const T*>(a.x) + 64 * first, M, NT * 8, Kh, hid, tid, kFrontThreads);
  __syncthreads();
  float acc[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  const unsigned char* xl = xs + (size_t)g8 * row_bytes(Kh) + 16 * t4;
  for (int p0 = 0; p0 < groups; p0 += kAhead) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int p = p0 + i;
      if (p < groups) mma64<T, NT>(acc, w[i], xl + 128 * p, Kh);
      if (p + kAhead < groups) load64(w[i], row_g, eight, 64 * (p + kAhead));
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int e = 0; e < 4; ++e) red[(8 * nt + 2 * t4 + (e & 1)) * kRedStride + 16 * wid + g8 + 8 * (e >> 1)] = acc[nt][e];
  }

  // epilogue: warp = token, lane = four adjacent channels
  const int c = 4 * lane, CC = 2 * HK * D + H * D;
  const bool conv = kind == kQ || kind == kK || kind == kV;
  const int cch = (kind == kQ ? 0 : kind == kK ? HK * D : 2 * HK * D) + head * D + c;
  float wt[4][4], bias[4] = {0.f, 0.f, 0.f, 0.f}, old[12];             // old: [channel][last three columns], contiguous
  static_assert(kMaxRows <= 2 * kWarps, "a token for every warp of the two blocks");
  const int m = rank + 2 * wid;
  if (conv && m < M) {                                                 // in flight across the meeting of the two halves
#pragma unroll
    for (int i = 0; i < 4; ++i) load4(static_cast<const T*>(a.conv_weight) + (size_t)(cch + i) * 4, wt[i]);
    if (a.conv_bias) load4(static_cast<const T*>(a.conv_bias) + cch, bias);
    const T* cs = static_cast<const T*>(a.conv_state) + ((size_t)m * CC + cch) * 3;
#pragma unroll
    for (int i = 0; i < 3; ++i) load4(cs + 4 * i, *reinterpret_cast<float(*)[4]>(&old[4 * i]));
  }
  cluster.sync();
  const float* half0 = cluster.map_shared_rank(red, 0);
  const float* half1 = cluster.map_shared_rank(red, 1);
  if (m < M) {
    float p[4];                                                        // rounded to T as a product of its own would be
    {
      const float4 x0 = *reinterpret_cast<const float4*>(half0 + m * kRedStride + c);
      const float4 x1 = *reinterpret_cast<const float4*>(half1 + m * kRedStride + c);
      p[0] = x0.x + x1.x; p[1] = x0.y + x1.y; p[2] = x0.z + x1.z; p[3] = x0.w + x1.w;
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = to_f32(from_f32<T>(p[i]));
    }
    const size_t rk = ((size_t)m * HK + head) * D + c, rv = ((size_t)m * H + head) * D + c;   // of a key / value head's row
    if (conv) {
      float y[4], nw[12];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        y[i] = fmaf(wt[i][0], old[3 * i], bias[i]);
        y[i] = fmaf(wt[i][1], old[3 * i + 1], y[i]);
        y[i] = fmaf(wt[i][2], old[3 * i + 2], y[i]);
        y[i] = silu(fmaf(wt[i][3], p[i], y[i]));
        nw[3 * i] = old[3 * i + 1]; nw[3 * i + 1] = old[3 * i + 2]; nw[3 * i + 2] = p[i];
      }
      // the cache may be updated in place: these channels are read and written by this thread alone
      T* tail = static_cast<T*>(a.new_conv_state) + ((size_t)m * CC + cch) * 3;
#pragma unroll
      for (int i = 0; i < 3; ++i) store4(tail + 4 * i, *reinterpret_cast<float(*)[4]>(&nw[4 * i]));
      if (kind == kV) {
        store4(reinterpret_cast<T*>(buf.v) + rv, y);
      } else {
        const float inv = inv_norm(warp_sum(y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3]));
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] *= inv;
        store4(reinterpret_cast<T*>(kind == kQ ? buf.q : buf.k) + rk, y);
      }
    } else if (kind == kF) {
      float db[4];
      load4(static_cast<const T*>(a.dt_bias) + head * D + c, db);
      const float nega = -__expf(to_f32(static_cast<const T*>(a.A_log)[head]));
      *reinterpret_cast<float4*>(buf.g + rk) = make_float4(nega * softplusf_(p[0] + db[0]), nega * softplusf_(p[1] + db[1]),
                                                           nega * softplusf_(p[2] + db[2]), nega * softplusf_(p[3] + db[3]));
    } else if (kind == kGate) {
      store4(reinterpret_cast<T*>(buf.gate) + rv, p);
    } else {
      float y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        y[i] = sigmoidf_(p[i]);
        if (kind == kB) y[i] = to_f32(from_f32<T>(y[i])) * a.erase_scale;
      }
      store4(kind == kB ? reinterpret_cast<T*>(buf.b) + rk : reinterpret_cast<T*>(buf.w) + rv, y);
    }
  }
  cluster.sync();                                                      // the other half has read this block's sums
}

// ---------------------------------------------------------------- core

// Block = (sequence, value head). Warp w: columns 32 (w & 3) .. + 31, key rows 32 (w >> 2) .. + 31; a lane four columns of
// eight rows, so the 64 KiB of the state are in flight at once, eight 16-byte loads per thread.
template <typename T>
__global__ void __launch_bounds__(kCoreThreads, 2)
layer_step_core_kernel(StepBuffers buf, const T* __restrict__ norm_weight, float* __restrict__ state, int H, int HK, float scale,
                       float eps) {
  __shared__ float s_abk[D], s_qa[D], s_k[D], s_a[D];
  __shared__ float s_red[4][2][D];                     // per row quarter: the read and the decayed state's output
  __shared__ float s_qk[4], s_ss[4];
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, ib = bh / H, ih = bh % H, ihk = ih / (H / HK);
  const int cg = wid & 3, rq = wid >> 2, rg = lane >> 3, cq = lane & 7;
  const int col0 = 32 * cg + 4 * cq, row0 = 32 * rq + 8 * rg;
  // The state is complete before `front` began (it waited for everything before it), and this kernel is launched by a front
  // whose blocks have all passed that wait: its loads may fly before this kernel's own wait, which is for q, k, v, g, b, w.
  float4 S[8];
  float4* gS = reinterpret_cast<float4*>(state + ((size_t)bh * D + row0) * D + col0);
#pragma unroll
  for (int i = 0; i < 8; ++i) S[i] = __ldcg(gS + i * (D / 4));       // (not through L1)
  grid_wait();
  grid_launch_dependents();
  const size_t rk = ((size_t)ib * HK + ihk) * D, rv = (size_t)bh * D;
  if (tid < D) {
    const float av = exp2f(buf.g[rk + tid] * kLog2e);
    const float kk = to_f32(reinterpret_cast<const T*>(buf.k)[rk + tid]);
    const float qs = to_f32(reinterpret_cast<const T*>(buf.q)[rk + tid]) * scale;
    s_abk[tid] = av * to_f32(reinterpret_cast<const T*>(buf.b)[rk + tid]) * kk;
    s_qa[tid] = qs * av; s_k[tid] = kk; s_a[tid] = av;
    const float qk = warp_sum(qs * kk);
    if (lane == 0) s_qk[wid] = qk;
  }
  float wv[4];
  {
    float vv[4];
    load4(reinterpret_cast<const T*>(buf.w) + rv + col0, wv);
    load4(reinterpret_cast<const T*>(buf.v) + rv + col0, vv);
#pragma unroll
    for (int c = 0; c < 4; ++c) wv[c] *= vv[c];
  }
  __syncthreads();
  float rd[4] = {0.f, 0.f, 0.f, 0.f}, oa[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = s_abk[row0 + i], y = s_qa[row0 + i];
    const float sv[4] = {S[i].x, S[i].y, S[i].z, S[i].w};
#pragma unroll
    for (int c = 0; c < 4; ++c) { rd[c] = fmaf(sv[c], x, rd[c]); oa[c] = fmaf(sv[c], y, oa[c]); }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int off = 8; off <= 16; off <<= 1) {
      rd[c] += __shfl_xor_sync(0xffffffffu, rd[c], off);
      oa[c] += __shfl_xor_sync(0xffffffffu, oa[c], off);
    }
  }
  if (rg == 0) {
    *reinterpret_cast<float4*>(&s_red[rq][0][col0]) = make_float4(rd[0], rd[1], rd[2], rd[3]);
    *reinterpret_cast<float4*>(&s_red[rq][1][col0]) = make_float4(oa[0], oa[1], oa[2], oa[3]);
  }
  __syncthreads();
  float u[4];
  {
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 p = *reinterpret_cast<const float4*>(&s_red[x][0][col0]);
      r[0] += p.x; r[1] += p.y; r[2] += p.z; r[3] += p.w;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) u[c] = wv[c] - r[c];
  }
  float y[4];
  if (rq == 0) {                                       // the output row: rounded to T, as a decode of its own leaves it
    const float qk = s_qk[0] + s_qk[1] + s_qk[2] + s_qk[3];
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 p = *reinterpret_cast<const float4*>(&s_red[x][1][col0]);
      r[0] += p.x; r[1] += p.y; r[2] += p.z; r[3] += p.w;
    }
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) { y[c] = to_f32(from_f32<T>(fmaf(qk, u[c], r[c]))); ss = fmaf(y[c], y[c], ss); }
#pragma unroll
    for (int off = 1; off <= 4; off <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (lane == 0) s_ss[cg] = ss;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float kk = s_k[row0 + i], av = s_a[row0 + i];
    __stcs(gS + i * (D / 4), make_float4(fmaf(av, S[i].x, kk * u[0]), fmaf(av, S[i].y, kk * u[1]), fmaf(av, S[i].z, kk * u[2]),
                                         fmaf(av, S[i].w, kk * u[3])));
  }
  __syncthreads();
  if (rq == 0 && rg == 0) {
    const float r = rsqrtf((s_ss[0] + s_ss[1] + s_ss[2] + s_ss[3]) / (float)D + eps);
    float nw[4], gt[4];
    load4(norm_weight + col0, nw);
    load4(reinterpret_cast<const T*>(buf.gate) + rv + col0, gt);
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c] = y[c] * r * nw[c] * silu(gt[c]);
    store4(reinterpret_cast<T*>(buf.normed) + rv + col0, y);
  }
}

// ---------------------------------------------------------------- out

// Block = 16 output columns; the eight warps take every eighth group of 64 reduction steps. A warp keeps up to kHeld groups,
// all of its weights up to 16 heads of 128, in registers while it waits for the normalised rows.
template <typename T, int NT>
__global__ void __launch_bounds__(kOutThreads)
layer_step_out_kernel(const T* __restrict__ x, const T* __restrict__ weight, T* __restrict__ out, int M, int K, int hid) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kHeld = 4, kWarps = kOutThreads / 32;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, g8 = lane >> 2, t4 = lane & 3;
  unsigned char* xs = smem;                                            // [NT * 8][row_bytes(K)]
  float* red = reinterpret_cast<float*>(smem + (size_t)NT * 8 * row_bytes(K));   // [warps][NT * 8][17]
  const T* row_g = weight + (size_t)(16 * blockIdx.x + g8) * K + 8 * t4;
  const size_t eight = (size_t)8 * K;
  const int groups = K / 64;
  // (the weights are not written by `core` or `front`; everything before those had completed when `front` passed its wait)
  Weights64 w[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (wid + kWarps * i < groups) load64(w[i], row_g, eight, 64 * (wid + kWarps * i));
  grid_wait();
  grid_launch_dependents();
  stage_rows(xs, x, M, NT * 8, K, K, tid, kOutThreads);
  __syncthreads();
  float acc[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  const unsigned char* xl = xs + (size_t)g8 * row_bytes(K) + 16 * t4;
  for (int p0 = wid; p0 < groups; p0 += kWarps * kHeld) {
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
      const int p = p0 + kWarps * i;
      if (p < groups) mma64<T, NT>(acc, w[i], xl + 128 * p, K);
      if (p + kWarps * kHeld < groups) load64(w[i], row_g, eight, 64 * (p + kWarps * kHeld));
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      red[((size_t)wid * NT * 8 + 8 * nt + 2 * t4 + (e & 1)) * 17 + g8 + 8 * (e >> 1)] = acc[nt][e];
  }
  __syncthreads();
  for (int i = tid; i < M * 16; i += kOutThreads) {
    const int m = i >> 4, col = i & 15;
    float y = 0.f;
#pragma unroll
    for (int x8 = 0; x8 < kWarps; ++x8) y += red[((size_t)x8 * NT * 8 + m) * 17 + col];
    out[(size_t)m * hid + 16 * blockIdx.x + col] = from_f32<T>(y);
  }
}

// shared memory of the two products for M sequences
size_t front_smem(int64_t rows, int64_t hidden) { return (size_t)rows * row_bytes((int)((hidden / 64 + 1) / 2 * 64)) + (size_t)rows * kRedStride * 4; }
size_t out_smem(int64_t rows, int64_t K) { return (size_t)rows * row_bytes((int)K) + (size_t)kOutThreads / 32 * rows * 17 * 4; }
int64_t padded_rows(int64_t B) { return B <= 8 ? 8 : 16; }

template <typename T, int NT>
int launch_step(const gdn2_layer_step_args& a, const StepBuffers& buf, cudaStream_t st) {
  const size_t fs = front_smem(NT * 8, a.hidden), os = out_smem(NT * 8, a.H * D);
  GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(layer_step_front_kernel<T, NT>), fs));
  GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(layer_step_out_kernel<T, NT>), os));
  GDN2_CUDA_TRY(launch_chained(true, layer_step_front_kernel<T, NT>, dim3((unsigned)(2 * (4 * a.HK + 3 * a.H))), kFrontThreads, fs, st, a, buf));
  GDN2_CUDA_TRY(launch_chained(true, layer_step_core_kernel<T>, dim3((unsigned)(a.B * a.H)), kCoreThreads, 0, st, buf,
                               static_cast<const T*>(a.norm_weight), a.state, (int)a.H, (int)a.HK, a.scale, a.eps));
  GDN2_CUDA_TRY(launch_chained(true, layer_step_out_kernel<T, NT>, dim3((unsigned)(a.hidden / 16)), kOutThreads, os, st,
                               reinterpret_cast<const T*>(buf.normed), static_cast<const T*>(a.o_weight), static_cast<T*>(a.out), (int)a.B,
                               (int)(a.H * D), (int)a.hidden));
  return GDN2_OK;
}
template <typename T>
int launch_step_rows(const gdn2_layer_step_args& a, const StepBuffers& buf, cudaStream_t st) {
  return a.B <= 8 ? launch_step<T, 1>(a, buf, st) : launch_step<T, 2>(a, buf, st);
}

size_t step_bytes(int64_t B, int64_t H, int64_t HK) { return (size_t)B * D * (HK * (3 * 2 + 4) + H * 4 * 2); }

}  // namespace

}  // namespace gdn2

extern "C" {

size_t gdn2_layer_step_workspace_bytes(int64_t B, int64_t hidden, int64_t H, int64_t HK, int64_t DK, int64_t DV, int64_t K, int dtype) {
  using namespace gdn2;
  if (dtype != GDN2_BF16 && dtype != GDN2_F16) return 0;
  if (B < 1 || B > kMaxRows || DK != D || DV != D || K != 4 || H < 1 || HK < 1 || H % HK != 0 || H > 1024 || hidden < 64 || hidden > (1 << 20) ||
      hidden % 64 != 0)
    return 0;
  constexpr size_t kMost = 220 * 1024;                   // shared memory of a block
  if (front_smem(padded_rows(B), hidden) > kMost || out_smem(padded_rows(B), H * D) > kMost) return 0;
  return step_bytes(B, H, HK);
}

int gdn2_layer_step(const gdn2_layer_step_args* args, int dtype, void* stream) {
  using namespace gdn2;
  if (!args) return GDN2_ERR_NULL_POINTER;
  const gdn2_layer_step_args& a = *args;
  if (!a.x || !a.w_cat || !a.conv_state || !a.conv_weight || !a.A_log || !a.dt_bias || !a.norm_weight || !a.o_weight || !a.state ||
      !a.new_conv_state || !a.out || !a.workspace)
    return GDN2_ERR_NULL_POINTER;
  if (dtype != GDN2_F32 && dtype != GDN2_BF16 && dtype != GDN2_F16) return GDN2_ERR_BAD_DTYPE;
  const size_t need = gdn2_layer_step_workspace_bytes(a.B, a.hidden, a.H, a.HK, a.DK, a.DV, a.K, dtype);
  if (need == 0) return GDN2_ERR_UNSUPPORTED;
  if (a.workspace_bytes < need) return GDN2_ERR_WORKSPACE;
  const void* const ptrs[] = {a.x, a.w_cat, a.conv_state, a.conv_weight, a.conv_bias, a.dt_bias, a.norm_weight, a.o_weight, a.state,
                              a.new_conv_state, a.out, a.workspace};
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15u) return GDN2_ERR_MISALIGNED;
  StepBuffers buf;
  char* p = static_cast<char*>(a.workspace);
  const size_t key = (size_t)a.B * a.HK * D * 2, value = (size_t)a.B * a.H * D * 2;
  buf.g = reinterpret_cast<float*>(p); p += 2 * key;
  buf.q = p; p += key;
  buf.k = p; p += key;
  buf.b = p; p += key;
  buf.v = p; p += value;
  buf.w = p; p += value;
  buf.gate = p; p += value;
  buf.normed = p;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return dtype == GDN2_BF16 ? launch_step_rows<__nv_bfloat16>(a, buf, st) : launch_step_rows<__half>(a, buf, st);
}

}  // extern "C"
