// Sequential state scan fused with the output, SIMT (CUDA-core) family, and the chunk-parallel
// output from stored chunk states. fp32 arithmetic; any DK <= 128, any DV.
//
// Scan: one 256-thread block per (value tile, batch*head), sequential over chunks. Per chunk
// (prefill_scan_kernel, gdn2/inference.py:446-475 of the reference project):
//     Un = U - W S ;  o = Qg S + tril(Aqk) Un ;  S <- diag(gamma_C) S + KG^T Un
// Optionally the state entering each chunk is stored (state_kernel, gdn2/forward.py:617-620).
// What bounds it: the chunk-to-chunk chain, since a call of this family has few (batch, head) pairs. The value
// columns never meet, so a head is spread over tiles of 8 of them while SMs are free (16 and 32 beyond that: the
// records are read once per tile). The records arrive by bulk copies in the layout they are stored in, each one
// refilled for the next chunk as soon as its last reader is through, and the two halves of the block form the output
// rows and the new state at the same time: two barriers per chunk.
// Inside a chunk the pace is set by what shared memory can return, 128 bytes a cycle whether lanes share an address or not. A
// thread therefore forms 4 rows x 4 columns over a quarter of the reduction (8 loads of 16 bytes per 64 FMAs, where one row by
// four columns took 5 for 16), and the four quarters, neighbours in a warp, meet in 12 shuffles. Two buffers per record, so that a
// copy has a whole chunk to land, gained nothing (79 -> 84 us); reading U from global memory a chunk ahead, four values a lane, in
// place of sixteen small copies a chunk did (75.6 -> 71.5). Measured
// with the chunk-local stage (prep_simt.cu), B = 2, S = 1000, 8 heads of 64, float32: 71.5 us a call, 78.9 before.
//
// Output: one block per (value tile, chunk, batch*head) doing the first two lines from a stored
// chunk state (output_kernel, gdn2/forward.py:710-725).
#include <type_traits>

#include "common.cuh"
#include "tc_utils.cuh"

namespace gdn2 {

namespace {

constexpr int NV = 32;   // value columns per block of the output kernel

// Shared memory of the output kernel.
struct OutputSmem {
  float *Ws, *Qs, *As, *Us, *Un, *St;
  __device__ OutputSmem(float* base, int DK) {
    Ws = base;                    // [64][DK]
    Qs = Ws + kChunk * DK;        // [64][DK]
    As = Qs + kChunk * DK;        // [64][64]
    Us = As + kChunk * kChunk;    // [64][NV]
    Un = Us + kChunk * NV;        // [64][NV]
    St = Un + kChunk * NV;        // [DK][NV]
  }
  static size_t bytes(int DK) {
    return ((size_t)2 * kChunk * DK + kChunk * kChunk + 2 * kChunk * NV + (size_t)DK * NV) * sizeof(float);
  }
};

template <typename TW>
__device__ __forceinline__ void load_chunk_operands(const WsLayout& L, const WsPtrs& P, int64_t ch, int64_t chv, int lo,
                                                    OutputSmem& s) {
  using WT = WsTraits<TW>;
  using TV = typename WT::TV;
  constexpr int E = WT::E;
  const int DK = L.DK, DV = L.DV, tid = threadIdx.x;
  const TW* wq = reinterpret_cast<const TW*>(P.wq + (size_t)ch * L.wq_bytes);
  const TV* aqk = reinterpret_cast<const TV*>(P.aqk + (size_t)ch * L.aqk_bytes);
  const TV* ut = reinterpret_cast<const TV*>(P.ut + (size_t)chv * L.ut_bytes);   // per value head; the rest per key head
  for (int idx = tid; idx < kChunk * DK; idx += 256) {
    const int t = idx / DK, c = idx % DK;
    s.Ws[idx] = to_f32(wq[kc_index<E>(t, c, 2 * kChunk)]);
    s.Qs[idx] = to_f32(wq[kc_index<E>(kChunk + t, c, 2 * kChunk)]);
  }
  for (int idx = tid; idx < kChunk * kChunk; idx += 256)
    s.As[idx] = WT::kg_load(aqk[kc_index<E>(idx / kChunk, idx % kChunk, kChunk)]);
  for (int idx = tid; idx < kChunk * NV; idx += 256) {
    const int t = idx / NV, c = lo + idx % NV;
    s.Us[idx] = c < DV ? WT::u_load(ut[kc_index<E>(c, t, DV)]) : 0.f;
  }
}

// Un = U - W S and o = Qg S + tril(Aqk) Un for the 8 tokens [wid*8, wid*8+8) and column `lane`.
template <typename TOut>
__device__ __forceinline__ void un_and_output(OutputSmem& s, int DK, int DV, int lo, TOut* __restrict__ o_rows,
                                              size_t o_row_stride) {
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int c = 0; c < DK; ++c) {
    const float sv = s.St[c * NV + lane];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = fmaf(s.Ws[(wid * 8 + i) * DK + c], sv, acc[i]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s.Un[(wid * 8 + i) * NV + lane] = s.Us[(wid * 8 + i) * NV + lane] - acc[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int c = 0; c < DK; ++c) {
    const float sv = s.St[c * NV + lane];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = fmaf(s.Qs[(wid * 8 + i) * DK + c], sv, acc[i]);
  }
  for (int t = 0; t < wid * 8 + 8; ++t) {
    const float un = s.Un[t * NV + lane];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (t <= wid * 8 + i) acc[i] = fmaf(s.As[(wid * 8 + i) * kChunk + t], un, acc[i]);
  }
  if (lo + lane < DV) {
#pragma unroll
    for (int i = 0; i < 8; ++i) o_rows[(size_t)(wid * 8 + i) * o_row_stride + lo + lane] = from_f32<TOut>(acc[i]);
  }
}

enum : uint32_t { kWaitSimtWq = 0x200000u, kWaitSimtAqk = 0x800000u, kWaitSimtKgt = 0x1000000u };

// Shared memory of the scan: the chunk's records as stored (fp32 images), the state tile and Un, value columns outside.
template <int NVT> struct ScanTile {
  float *wq, *aqk, *kgt, *gl, *St, *Un;
  __device__ ScanTile(float* base, int DK) {
    wq = base;                          // [DK/4][128 rows][4]
    kgt = wq + 2 * kChunk * DK;         // [64/4][DK][4]
    aqk = kgt + kChunk * DK;            // [64/4][64 r][4]
    gl = aqk + kChunk * kChunk;         // [DK]
    St = gl + DK;                       // [NVT][DK]: the state transposed
    Un = St + DK * NVT;                 // [NVT][64]
  }
  static size_t bytes(int DK) {
    return ((size_t)3 * kChunk * DK + kChunk * kChunk + kChunk * NVT + DK + (size_t)DK * NVT) * sizeof(float);
  }
};

// acc[i][c] += sum over groups x4 = first, first + 4, .. < end of four reduction steps of row i (rows 8 apart in an image
// [steps/4][stride][4], `rows` its row 0 of this thread) and column c (cols: [column][ld])
template <int NC>
__device__ __forceinline__ void tile_product(float2 (&acc)[4][NC], const float* rows, int stride, const float* cols, int ld, int first, int end) {
#pragma unroll 1
  for (int x4 = first; x4 < end; x4 += 4) {
    float4 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const float4*>(rows + ((size_t)x4 * stride + 8 * i) * 4);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float4 v = *reinterpret_cast<const float4*>(cols + c * ld + 4 * x4);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        acc[i][c] = ffma2(make_float2(r[i].z, r[i].w), make_float2(v.z, v.w), ffma2(make_float2(r[i].x, r[i].y), make_float2(v.x, v.y), acc[i][c]));
    }
  }
}
// The sums of four columns over the four quarters of a warp (lane bits 3 and 4): a lane keeps row 2 * bit 3 + bit 4.
template <int NC>
__device__ __forceinline__ void tile_reduce(const float2 (&acc)[4][NC], int c0, int lane, float (&out)[4]) {
  float v[4][4], h[2][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int c = 0; c < 4; ++c) v[i][c] = acc[i][c0 + c].x + acc[i][c0 + c].y;
  }
  const bool b3 = lane & 8, b4 = lane & 16;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int c = 0; c < 4; ++c) h[i][c] = (b3 ? v[2 + i][c] : v[i][c]) + __shfl_xor_sync(0xffffffffu, b3 ? v[i][c] : v[2 + i][c], 8);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) out[c] = (b4 ? h[1][c] : h[0][c]) + __shfl_xor_sync(0xffffffffu, b4 ? h[0][c] : h[1][c], 16);
}

// S tokens per batch entry, ceil(S / 64) chunks: the rows past the end are not written (the chunk-local stage has made
// them neutral). Warp: rows 32 (wid & 3) .. + 31 of the W | Qg image, half of the tile's columns (wid >> 2) in groups of four. The
// W rows' warps go on to the state update (32 or, when DK > 64, 64 key channels each), the Qg rows' warps to the output.
template <typename TOut, int NVT, typename Seqs>
__global__ void __launch_bounds__(256, 2)
scan_simt_kernel(WsLayout L, WsPtrs P, const float* __restrict__ s0, TOut* __restrict__ o,
                 float* __restrict__ sT, float* __restrict__ hs, int S, int H, int64_t o_bs, uint32_t* status,
                 const __grid_constant__ Seqs seqs) {
  constexpr int kQuads = NVT / 8, kG = kQuads < 2 ? kQuads : 2;   // groups of four columns per warp, and at a time
  const int DK = L.DK, DV = L.DV;
  const int bh = blockIdx.x, ib = bh / H, ih = bh % H;
  const int lo = blockIdx.y * NVT, nv = min(NVT, DV - lo);
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int part = lane >> 3, rl = lane & 7;              // quarter of the reduction; row of eight
  const int rb = wid & 3, quad0 = (wid >> 2) * kQuads;
  const bool is_q = rb >= 2;
  const int mine = rl + 8 * (2 * (part & 1) + (part >> 1));   // row of 32 whose sums this lane keeps (tile_reduce)
  extern __shared__ __align__(128) float sm[];
  ScanTile<NVT> s(sm, DK);
  __shared__ uint64_t bar_wq, bar_aqk, bar_kgt;
  __shared__ int abort_flag;

  // this block's run of chunks: how many, its records (those of its key head, and U of its value head), its first
  // output row and its number of tokens. With packed sequences `ib` is the sequence and there is one row of records.
  int NC, len;
  int64_t ch0, chv0, o_row0;
  if constexpr (std::is_same<Seqs, PackedSeqs>::value) {
    NC = seqs.chunk[ib + 1] - seqs.chunk[ib];
    len = seqs.tok[ib + 1] - seqs.tok[ib];
    ch0 = (int64_t)(ih / L.rep) * seqs.chunk[seqs.n] + seqs.chunk[ib];
    chv0 = (int64_t)ih * seqs.chunk[seqs.n] + seqs.chunk[ib];
    o_row0 = seqs.tok[ib];
  } else {
    NC = (S + kChunk - 1) / kChunk;
    len = S;
    ch0 = ((int64_t)ib * (H / L.rep) + ih / L.rep) * NC;
    chv0 = (int64_t)bh * NC;
    o_row0 = (int64_t)ib * o_bs;
  }
  const char* g_wq = P.wq + (size_t)ch0 * L.wq_bytes;
  const char* g_aqk = P.aqk + (size_t)ch0 * L.aqk_bytes;
  const char* g_kgt = P.kgt + (size_t)ch0 * L.kgt_bytes;
  const float* g_ut = reinterpret_cast<const float*>(P.ut + (size_t)chv0 * L.ut_bytes) + (size_t)lo * 4;
  const float* g_gl = P.gl + (size_t)ch0 * DK;

  // copies of chunk n, issued by one thread
  auto load_wq = [&](int n) {
    if (lane == 0) {
      tc::mbar_expect_tx(&bar_wq, (uint32_t)L.wq_bytes);
      tc::bulk_g2s(s.wq, g_wq + (size_t)n * L.wq_bytes, (uint32_t)L.wq_bytes, &bar_wq);
    }
  };
  auto load_aqk_kgt = [&](int n) {
    if (lane == 0) {
      tc::mbar_expect_tx(&bar_kgt, (uint32_t)L.kgt_bytes + (uint32_t)L.gl_bytes);
      tc::bulk_g2s(s.kgt, g_kgt + (size_t)n * L.kgt_bytes, (uint32_t)L.kgt_bytes, &bar_kgt);
      tc::bulk_g2s(s.gl, g_gl + (size_t)n * DK, (uint32_t)L.gl_bytes, &bar_kgt);
      tc::mbar_expect_tx(&bar_aqk, (uint32_t)L.aqk_bytes);
      tc::bulk_g2s(s.aqk, g_aqk + (size_t)n * L.aqk_bytes, (uint32_t)L.aqk_bytes, &bar_aqk);
    }
  };

  if (tid == 0) {
    tc::mbar_init(&bar_wq, 1); tc::mbar_init(&bar_aqk, 1); tc::mbar_init(&bar_kgt, 1);
    abort_flag = 0;
    tc::mbar_init_fence();
  }
  grid_wait();
  for (int idx = tid; idx < DK * NVT; idx += 256) {
    const int c = idx / NVT, d = idx % NVT;
    s.St[d * DK + c] = (s0 != nullptr && d < nv) ? s0[((size_t)bh * DK + c) * DV + lo + d] : 0.f;
  }
  tc::fence_async_smem();
  __syncthreads();
  if (wid == 0 && NC > 0) { load_wq(0); load_aqk_kgt(0); }

  // After a wait that ran out a warp computes on what is there (the status word says that the results are void) and keeps the
  // block's barriers; the copying warp issues nothing more. Leaving together takes a barrier that carries the result, twice
  // per chunk: 80.1 us for the call above in place of 78.9.
  auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t code) {
    return tc::mbar_wait_warp(bar, parity, &abort_flag, status, code);
  };
  float qs[kQuads][4];                                     // Qg rows: this lane's row of Qg S; W rows: its row of U, a chunk ahead
  auto load_u = [&](int n) {
    const int row = 32 * rb + mine;
    const float* u = g_ut + (size_t)n * (L.ut_bytes / sizeof(float)) + (size_t)(row >> 2) * DV * 4 + (row & 3);
#pragma unroll
    for (int j = 0; j < kQuads; ++j) {
      const int col0 = 4 * (quad0 + j);
#pragma unroll
      for (int c = 0; c < 4; ++c) qs[j][c] = col0 < nv ? __ldg(u + (col0 + c) * 4) : 0.f;      // nv is a multiple of 4
    }
  };
  if (!is_q && NC > 0) load_u(0);
  int wq_ahead = 0, kgt_ahead = 0;                         // last chunk whose copies were issued
  bool ok = true;
  for (int n = 0; n < NC; ++n) {
    const uint32_t ph = n & 1;
    if (hs != nullptr) {
      float* hp = hs + (((size_t)ib * NC + n) * H + ih) * DK * DV + lo;
      for (int idx = tid; idx < DK * NVT; idx += 256) {
        const int c = idx / NVT, d = idx % NVT;
        if (d < nv) hp[(size_t)c * DV + d] = s.St[d * DK + c];
      }
    }
    // ---- rows of W S or Qg S
    ok = ok && wait_all(&bar_wq, ph, kWaitSimtWq);
#pragma unroll
    for (int j0 = 0; j0 < kQuads; j0 += kG) {
      float2 acc[4][4 * kG];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int c = 0; c < 4 * kG; ++c) acc[i][c] = make_float2(0.f, 0.f);
      }
      tile_product(acc, s.wq + (32 * rb + rl) * 4, 2 * kChunk, s.St + 4 * (quad0 + j0) * DK, DK, part, DK / 4);
#pragma unroll
      for (int j = 0; j < kG; ++j) {
        float v[4];
        tile_reduce(acc, 4 * j, lane, v);
        const int col0 = 4 * (quad0 + j0 + j), row = 32 * rb + mine;
        if (is_q) {
#pragma unroll
          for (int c = 0; c < 4; ++c) qs[j0 + j][c] = v[c];
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) s.Un[(col0 + c) * kChunk + row] = qs[j0 + j][c] - v[c];
        }
      }
    }
    if (!is_q && n + 1 < NC) load_u(n + 1);
    __syncthreads();                                       // Un complete; the state and W | Qg have been read
    if (wid == 0 && ok && n + 1 < NC) {
      load_wq(n + 1);
      wq_ahead = n + 1;
    }

    if (is_q) {
      // ---- o = Qg S + tril(Aqk) Un: source tokens up to the warp's last row (Aqk is zero above the diagonal)
      ok = ok && wait_all(&bar_aqk, ph, kWaitSimtAqk);
      const int r = 32 * (rb - 2) + mine, t = n * kChunk + r;
#pragma unroll
      for (int j0 = 0; j0 < kQuads; j0 += kG) {
        float2 acc[4][4 * kG];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
          for (int c = 0; c < 4 * kG; ++c) acc[i][c] = make_float2(0.f, 0.f);
        }
        tile_product(acc, s.aqk + (32 * (rb - 2) + rl) * 4, kChunk, s.Un + 4 * (quad0 + j0) * kChunk, kChunk, part, 8 * (rb - 1));
#pragma unroll
        for (int j = 0; j < kG; ++j) {
          float v[4];
          tile_reduce(acc, 4 * j, lane, v);
          const int col0 = 4 * (quad0 + j0 + j);
          if (t < len && col0 < nv) {                      // nv is a multiple of 4
            TOut* op = o + ((size_t)(o_row0 + t) * H + ih) * DV + lo + col0;
#pragma unroll
            for (int c = 0; c < 4; ++c) op[c] = from_f32<TOut>(qs[j0 + j][c] + v[c]);
          }
        }
      }
    } else {
      // ---- S <- gamma_C S + KG^T Un, 32 channels at a time; rows past DK are formed from the record behind and dropped
      ok = ok && wait_all(&bar_kgt, ph, kWaitSimtKgt);
      for (int c0 = 32 * rb; c0 < DK; c0 += 64) {
        const int ch = c0 + mine;
        const float gm = ch < DK ? s.gl[ch] : 0.f;
#pragma unroll
        for (int j0 = 0; j0 < kQuads; j0 += kG) {
          float2 acc[4][4 * kG];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int c = 0; c < 4 * kG; ++c) acc[i][c] = make_float2(0.f, 0.f);
          }
          tile_product(acc, s.kgt + (c0 + rl) * 4, DK, s.Un + 4 * (quad0 + j0) * kChunk, kChunk, part, kChunk / 4);
#pragma unroll
          for (int j = 0; j < kG; ++j) {
            float v[4];
            tile_reduce(acc, 4 * j, lane, v);
            float* st = s.St + 4 * (quad0 + j0 + j) * DK + ch;
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (ch < DK) st[c * DK] = fmaf(gm, st[c * DK], v[c]);
          }
        }
      }
    }
    __syncthreads();                                       // the new state is complete; Un, Aqk and KG have been read
    if (wid == 0 && ok && n + 1 < NC) {
      load_aqk_kgt(n + 1);
      kgt_ahead = n + 1;
    }
  }
  if (wid == 0 && NC > 0) {                                // copies that no one waited for must land before the block ends
    tc::mbar_drain(&bar_wq, wq_ahead & 1);
    tc::mbar_drain(&bar_kgt, kgt_ahead & 1); tc::mbar_drain(&bar_aqk, kgt_ahead & 1);
  }
  if (sT != nullptr) {
    for (int idx = tid; idx < DK * NVT; idx += 256) {
      const int c = idx / NVT, d = idx % NVT;
      if (d < nv) sT[((size_t)bh * DK + c) * DV + lo + d] = s.St[d * DK + c];
    }
  }
}

template <typename TOut, typename TW>
__global__ void __launch_bounds__(256)
output_simt_kernel(WsLayout L, WsPtrs P, const float* __restrict__ hs, TOut* __restrict__ o, int S, int H, int64_t o_bs) {
  const int DK = L.DK, DV = L.DV, NC = S / kChunk;
  const int n = blockIdx.y, bh = blockIdx.z, ib = bh / H, ih = bh % H;
  const int lo = blockIdx.x * NV;
  const int tid = threadIdx.x;
  extern __shared__ float sm[];
  OutputSmem s(sm, DK);
  const int64_t ch = ((int64_t)ib * (H / L.rep) + ih / L.rep) * NC + n;
  const float* hp = hs + (((size_t)ib * NC + n) * H + ih) * DK * DV;
  for (int idx = tid; idx < DK * NV; idx += 256) {
    const int c = idx / NV, d = lo + idx % NV;
    s.St[idx] = d < DV ? hp[(size_t)c * DV + d] : 0.f;
  }
  load_chunk_operands<TW>(L, P, ch, (int64_t)bh * NC + n, lo, s);
  __syncthreads();
  TOut* o_rows = o + (((size_t)ib * o_bs + (size_t)n * kChunk) * H + ih) * DV;
  un_and_output<TOut>(s, DK, DV, lo, o_rows, (size_t)H * DV);
}

template <typename TOut, typename Seqs>
int launch_scan_typed(const WsLayout& L, const WsPtrs& P, const float* s0, void* o, float* sT, float* hs,
                      int B, int S, int H, int64_t o_bs, const Seqs& seqs, cudaStream_t st) {
  const int BH = B * H, sms = device_sm_count();
  auto launch = [&](auto kern, int nvt, size_t smem) -> int {
    GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
    GDN2_CUDA_TRY(launch_chained(true, kern, dim3(BH, (L.DV + nvt - 1) / nvt), 256, smem, st, L, P, s0, static_cast<TOut*>(o), sT, hs, S, H,
                                 o_bs, device_status_word(), seqs));
    return GDN2_OK;
  };
  // the narrowest tile whose blocks all run at once (two per SM while the records of DK <= 64 leave room)
  const int64_t room = L.DK <= 64 ? 2 * sms : sms;
  if ((int64_t)BH * ((L.DV + 7) / 8) <= room) return launch(scan_simt_kernel<TOut, 8, Seqs>, 8, ScanTile<8>::bytes(L.DK));
  if ((int64_t)BH * ((L.DV + 15) / 16) <= room) return launch(scan_simt_kernel<TOut, 16, Seqs>, 16, ScanTile<16>::bytes(L.DK));
  return launch(scan_simt_kernel<TOut, 32, Seqs>, 32, ScanTile<32>::bytes(L.DK));
}

template <typename TOut, typename TW>
int launch_output_typed(const WsLayout& L, const WsPtrs& P, const float* hs, void* o, int B, int S, int H,
                        int64_t o_bs, cudaStream_t st) {
  const size_t smem = OutputSmem::bytes(L.DK);
  auto kern = output_simt_kernel<TOut, TW>;
  GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
  dim3 grid((L.DV + NV - 1) / NV, S / kChunk, B * H);
  kern<<<grid, 256, smem, st>>>(L, P, hs, static_cast<TOut*>(o), S, H, o_bs);
  GDN2_CUDA_TRY(cudaGetLastError());
  return GDN2_OK;
}

template <typename Seqs>
int launch_scan_any(const WsLayout& L, const WsPtrs& P, const float* s0, void* o, float* sT, float* hs,
                    int B, int S, int H, int64_t o_bs, int dtype, const Seqs& seqs, cudaStream_t st) {
  if (L.esz != 4) return GDN2_ERR_UNSUPPORTED;   // 16-bit records belong to the tensor-core family's kernels
  switch (dtype) {
    case GDN2_F32: return launch_scan_typed<float>(L, P, s0, o, sT, hs, B, S, H, o_bs, seqs, st);
    case GDN2_BF16: return launch_scan_typed<__nv_bfloat16>(L, P, s0, o, sT, hs, B, S, H, o_bs, seqs, st);
    case GDN2_F16: return launch_scan_typed<__half>(L, P, s0, o, sT, hs, B, S, H, o_bs, seqs, st);
    default: return GDN2_ERR_BAD_DTYPE;
  }
}

}  // namespace

int launch_scan_simt(const WsLayout& L, const WsPtrs& P, const float* s0, void* o, float* sT, float* hs,
                     int B, int S, int H, int64_t o_bs, int dtype, cudaStream_t st) {
  return launch_scan_any(L, P, s0, o, sT, hs, B, S, H, o_bs, dtype, OneLength{}, st);
}

int launch_scan_simt_packed(const WsLayout& L, const WsPtrs& P, const PackedSeqs& seqs, const float* s0, void* o,
                            float* sT, int H, int dtype, cudaStream_t st) {
  return launch_scan_any(L, P, s0, o, sT, nullptr, seqs.n, 0, H, 0, dtype, seqs, st);
}

int launch_output_simt(const WsLayout& L, const WsPtrs& P, const float* hs, void* o, int B, int S, int H,
                       int64_t o_bs, int dtype, cudaStream_t st) {
  if (L.esz != 4) return GDN2_ERR_UNSUPPORTED;
  switch (dtype) {
    case GDN2_F32: return launch_output_typed<float, float>(L, P, hs, o, B, S, H, o_bs, st);
    case GDN2_BF16: return launch_output_typed<__nv_bfloat16, float>(L, P, hs, o, B, S, H, o_bs, st);
    case GDN2_F16: return launch_output_typed<__half, float>(L, P, hs, o, B, S, H, o_bs, st);
    default: return GDN2_ERR_BAD_DTYPE;
  }
}

}  // namespace gdn2
