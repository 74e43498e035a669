// Recurrent decode of several tokens at once, DK = DV = 128: the n-token recurrence of
// decode_multi_kernel (gdn2/inference.py:199-303 of the reference project) evaluated in blocks of NB = 4, 6 or
// 8 tokens without a per-token dependent sweep over the state.
//
// With A_t = exp(g_1 + .. + g_t) per key channel (A_t / A_s <= 1 for s <= t, so nothing can overflow):
//     u_t = w_t*v_t - (b_t*k_t*A_t)^T S_0 - sum_{s<t} Akk[t,s] u_s      Akk[t,s] = sum_c b_t k_t k_s A_t/A_s
//     o_t = (scale*q_t*A_t)^T S_0 + sum_{s<=t} Aqk[t,s] u_s              Aqk[t,s] = scale * sum_c q_t k_s A_t/A_s
//     S_NB = diag(A_NB) S_0 + sum_s (k_s * A_NB/A_s) u_s^T
// (the exponent of every A_t / A_s is the sum of the gates s+1 .. t, not a difference of prefix sums, in which one strong gate
// would swallow the ordinary ones after it; gates are read as max(g, kMinGate), whose exponential is zero already)
// which is the token-by-token recurrence S <- diag(exp g) S; u = w*v - S^T(b*k); S <- S + k u^T;
// o = scale S^T q with the sums regrouped: two sweeps over the state tile with 64 and 36 (NB = 8) independent
// accumulation chains per thread instead of 2 n sweeps that each wait for a cross-thread reduction.
//
// Persistent blocks, one per SM, walk over the (batch, head) tiles with four kinds of warps:
//   * one copy thread brings a tile's 64 KiB of fp32 state into shared memory by bulk copies (TMA) two
//     tiles ahead and sends the updated tile back the same way: HBM traffic is the state once in, once
//     out, and no compute thread ever waits on a global load of it;
//   * one output thread sends each step's output rows, staged in shared memory by the sweep warps, as one
//     bulk copy per token row;
//   * four table warps (thread = channel) fetch the token vectors a step ahead as 16-byte pieces, pass them
//     through a staging buffer to read their own channel, and build the step's coefficient tables and the
//     NB x NB pair matrices while the current step is swept;
//   * eight sweep warps do the two sweeps in place: warp w owns value columns 16w .. 16w+15, lane
//     (rgl = lane >> 2, cq = lane & 3) columns 16w + 4cq .. +3 of key rows 16 rgl .. 16 rgl + 15.
// Hand-offs are mbarriers with bounded waits.
// Per-row coefficients sit in shared memory once; the packed f32x2 FMAs pair them over products (sweep 1)
// or tokens (sweep 2), so no duplicated copies are stored or fetched.
#include <type_traits>

#include "common.cuh"
#include "tc_utils.cuh"

namespace gdn2 {

namespace {

constexpr int D = 128;
constexpr float kMinGate = -110.f;          // exp(-104) is already below half of float32's smallest number
constexpr int kGroupFloats = 16 * D + 16;   // 16 state rows + 64 bytes: adjacent row groups land 64 B apart mod 128
constexpr int kTileFloats = 8 * kGroupFloats;
constexpr uint32_t kGroupBytes = 16 * D * 4;
constexpr int kCoefRows = 136;              // 128 rows + one slot per 16-row group
__device__ __forceinline__ int crow(int r) { return r + (r >> 4); }

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int NB>
struct Tables {
  // per key row the 2 NB products, four per chunk: b*k*A_t for t < NB, then scale*q*A_t
  float4 c1[NB / 2][kCoefRows];
  // per key row: k * A_NB/A_s, four per chunk; A_NB itself
  float4 c2[(NB + 3) / 4][kCoefRows];
  float gam[kCoefRows];
  float wv[NB][D];                    // w * v
  float akk[NB][8];                   // strictly lower
  float aqk[NB][8];                   // lower incl. diagonal, scale folded in
};

template <int NB>
struct alignas(128) BlockedSmem {
  float tile[2][kTileFloats];         // the state of two (batch, head) tiles
  Tables<NB> tab[2];                      // coefficient tables of two consecutive steps
  float part[4][64];                  // per 32-channel group: partial sums of the 64 pair entries
  // one step's token vectors as they lie in memory: q, k, b, v, w rows of D elements (up to 4 bytes each), then g
  alignas(16) unsigned char stage[6 * NB * D * 4];
  uint64_t tile_full[2], tile_done[2];   // copy thread -> sweep warps (bytes landed); sweep warps -> copy thread
  uint64_t tab_full[2], tab_empty[2];    // table warps -> sweep warps; sweep warps -> table warps
  uint64_t o_full[2];                    // sweep warps -> output thread (a step's rows are staged)
  int abort_flag;
  alignas(16) unsigned char ostage[2][NB * D * 4];   // a step's output rows [token][value channel] on their way out
};

constexpr int kSweepThreads = 256;    // warps 0..7
constexpr int kTableThreads = 128;    // warps 8..11
constexpr int kAllThreads = kSweepThreads + kTableThreads + 64;   // + warp 12: one thread drives the state copies; warp 13: one thread sends the outputs

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
// one arrival per warp: the lanes' writes are ordered before lane 0's arrival by the warp barrier
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
__device__ __forceinline__ void table_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
// the same barrier fused with an OR over one predicate per thread: every table thread gets the same answer
__device__ __forceinline__ bool table_sync_or(bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}"
      : "=r"(r)
      : "r"((uint32_t)pred)
      : "memory");
  return r != 0;
}

// Bounded wait for hand-offs that have thousands of cycles of slack: the polling thread sleeps between probes
// instead of competing with the sweep warps for issue slots.
[[nodiscard]] __device__ __forceinline__ bool mbar_wait_relaxed(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  uint32_t* status_word, uint32_t code) {
  if (tc::mbar_try_wait(bar, parity)) return true;
  const long long t_begin = clock64();
  while (true) {
    __nanosleep(128);
    if (tc::mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t_begin > tc::kWaitCycles) {
      *abort_flag = 1;
      atomicOr(status_word, code);
      return false;
    }
  }
}

enum : uint32_t { kWaitTile = 0x10000u, kWaitTab = 0x20000u, kWaitEmpty = 0x40000u, kWaitDone = 0x80000u, kWaitOut = 0x100000u };

template <typename T, typename Seqs, int NB>
__global__ void __launch_bounds__(kAllThreads, 1)
decode_blocked_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                      const float* __restrict__ g, const T* __restrict__ b, const T* __restrict__ w,
                      float* __restrict__ state, T* __restrict__ o, int ntiles, int n, int H, int HK, int64_t in_bs,
                      int64_t o_bs, float scale, uint32_t* status, const __grid_constant__ Seqs seqs) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  static_assert(NB % 2 == 0 && NB >= 4 && NB <= 8, "products are paired, pair matrices have eight columns");
  using Smem = BlockedSmem<NB>;
  Smem& s = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;

  // tokens of a tile, and its first input and output row (in tokens). Packed sequences: the last len % 64 tokens of
  // the tile's sequence, which may be none; such a tile is passed over by every role.
  auto tile_tokens = [&](int tile, size_t* row_in, size_t* row_o) -> int {
    const int ib = tile / H;
    if constexpr (std::is_same<Seqs, PackedSeqs>::value) {
      const int m = (seqs.tok[ib + 1] - seqs.tok[ib]) % kChunk;
      if (row_in) *row_in = seqs.tok[ib + 1] - m;
      if (row_o) *row_o = seqs.tok[ib + 1] - m;
      return m;
    } else {
      if (row_in) *row_in = (size_t)ib * in_bs;
      if (row_o) *row_o = (size_t)ib * o_bs;
      return n;
    }
  };
  // the next tile of this block that has tokens, from `tile` on (>= ntiles: none)
  auto from_tile = [&](int tile) -> int {
    if constexpr (std::is_same<Seqs, PackedSeqs>::value)
      while (tile < ntiles && tile_tokens(tile, nullptr, nullptr) == 0) tile += gridDim.x;
    return tile;
  };

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&s.tile_full[i], 1);
      tc::mbar_init(&s.tile_done[i], kSweepThreads / 32);     // one arrival per warp
      tc::mbar_init(&s.tab_full[i], kTableThreads / 32);
      // a table buffer is free when the eight sweep warps have finished its step AND the output thread has sent
      // the step's rows: the tables of step k + 2 are then built after the staging rows of step k were read, and
      // the sweep warps (which wait for those tables) may overwrite the rows without a hand-off of their own
      tc::mbar_init(&s.tab_empty[i], kSweepThreads / 32 + 1);
      tc::mbar_init(&s.o_full[i], kSweepThreads / 32);
    }
    s.abort_flag = 0;
    tc::mbar_init_fence();
  }
  __syncthreads();

  grid_wait();
  grid_launch_dependents();

  if (wid == 13) {
    // =============================== output thread: a step's rows leave as bulk copies ==========
    // (256-byte rows for 16-bit outputs: eight scattered 2-byte stores per lane of the sweep warps otherwise)
    if (lane == 0) {
      bool ok = true;
      for (int tile = from_tile(blockIdx.x), step = 0; ok && tile < ntiles; tile = from_tile(tile + gridDim.x)) {
        const int ih = tile % H;
        size_t row_o;
        const int nt = tile_tokens(tile, nullptr, &row_o);
        for (int t0 = 0; t0 < nt; t0 += NB, ++step) {
          const int nb = min(NB, nt - t0);
          ok = mbar_wait_relaxed(&s.o_full[step & 1], (step >> 1) & 1, &s.abort_flag, status, kWaitOut);
          if (!ok) break;
          const T* src = reinterpret_cast<const T*>(s.ostage[step & 1]);
          for (int t = 0; t < nb; ++t) tc::bulk_s2g(o + ((row_o + t0 + t) * H + ih) * D, src + t * D, D * sizeof(T));
          tc::bulk_commit();
          tc::bulk_wait_read_all();                      // the staging rows may be overwritten
          mbar_arrive(&s.tab_empty[step & 1]);
        }
      }
      tc::bulk_wait_all();
    }
  } else if (wid == 12) {
    // =============================== copy thread: tiles in, tiles out ==========================
    if (lane == 0) {
      auto load_tile = [&](int tile, int buf) {          // 8 bulk copies of 16 rows each
        tc::mbar_expect_tx(&s.tile_full[buf], 8 * kGroupBytes);
        const float* src = state + (size_t)tile * D * D;
#pragma unroll
        for (int gidx = 0; gidx < 8; ++gidx)
          tc::bulk_g2s(&s.tile[buf][gidx * kGroupFloats], src + gidx * 16 * D, kGroupBytes, &s.tile_full[buf]);
      };
      const int stride = gridDim.x;
      int tile = from_tile(blockIdx.x);
      int next = tile < ntiles ? from_tile(tile + stride) : ntiles;
      int loaded = 0;                                    // tiles whose copies were issued
      if (tile < ntiles) { load_tile(tile, 0); ++loaded; }
      if (next < ntiles) { load_tile(next, 1); ++loaded; }
      for (int it = 0; tile < ntiles; ++it) {
        const int buf = it & 1;
        if (!mbar_wait_relaxed(&s.tile_done[buf], (it >> 1) & 1, &s.abort_flag, status, kWaitDone)) break;
        float* dst = state + (size_t)tile * D * D;
#pragma unroll
        for (int gidx = 0; gidx < 8; ++gidx)
          tc::bulk_s2g(dst + gidx * 16 * D, &s.tile[buf][gidx * kGroupFloats], kGroupBytes);
        tc::bulk_commit();
        const int after = next < ntiles ? from_tile(next + stride) : ntiles;
        if (after < ntiles) {
          tc::bulk_wait_read_all();                      // the buffer may be overwritten once the store has read it
          load_tile(after, buf);
          ++loaded;
        }
        tile = next;
        next = after;
      }
      tc::bulk_wait_all();
      // a block that gave up leaves copies behind: they must land before it gives its shared memory back
      for (int x = loaded > 1 ? loaded - 2 : 0; x < loaded; ++x) tc::mbar_drain(&s.tile_full[x & 1], (x >> 1) & 1);
    }
  } else if (wid >= 8) {
    // =============================== table warps: thread = key / value channel =================
    const int c = tid - kSweepThreads;
    const int pw_ = wid - 8;                             // 32-channel group
    // A step's token vectors are NB rows of D elements per tensor, contiguous per row: the 128 threads fetch them
    // as 16-byte pieces (CH pieces per thread and tensor, CG for g), ONE STEP AHEAD, into registers; at the
    // top of a step the pieces go to the staging buffer and every thread reads its own channel from there.
    constexpr int kRowPieces = D * (int)sizeof(T) / 16;  // 16-byte pieces per row
    constexpr int CH = (NB * kRowPieces + kTableThreads - 1) / kTableThreads;   // ... per thread and tensor, the last ones perhaps past NB rows
    constexpr int CG = (NB * (D / 4) + kTableThreads - 1) / kTableThreads;
    uint4 ldT[5][CH], ldG[CG];
    auto issue_loads = [&](int ptile, int pt0) {
      const int pih = ptile % H, pihk = pih / (H / HK);
      size_t prow;
      const int pnb = min(NB, tile_tokens(ptile, &prow, nullptr) - pt0);
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int e = c + kTableThreads * j, tokr = e / kRowPieces, within = e % kRowPieces;
        const int tt = pt0 + (tokr < pnb ? tokr : pnb - 1);                 // padding tokens re-read the last real one
        const size_t rowk = ((prow + tt) * HK + pihk) * D, rowv = ((prow + tt) * H + pih) * D;
        ldT[0][j] = __ldg(reinterpret_cast<const uint4*>(q + rowk) + within);
        ldT[1][j] = __ldg(reinterpret_cast<const uint4*>(k + rowk) + within);
        ldT[2][j] = __ldg(reinterpret_cast<const uint4*>(b + rowk) + within);
        ldT[3][j] = __ldg(reinterpret_cast<const uint4*>(v + rowv) + within);
        ldT[4][j] = __ldg(reinterpret_cast<const uint4*>(w + rowv) + within);
      }
#pragma unroll
      for (int j = 0; j < CG; ++j) {
        const int e = c + kTableThreads * j, tokr = e / (D / 4), within = e % (D / 4);
        const int tt = pt0 + (tokr < pnb ? tokr : pnb - 1);
        ldG[j] = __ldg(reinterpret_cast<const uint4*>(g + ((prow + tt) * HK + pihk) * D) + within);
      }
    };
    T* stT = reinterpret_cast<T*>(s.stage);                                // [5][NB][D]
    float* stG = reinterpret_cast<float*>(s.stage + 5 * NB * D * sizeof(T));   // [NB][D]
    int tile = from_tile(blockIdx.x), t0 = 0;
    if (tile < ntiles) issue_loads(tile, t0);
    for (int step = 0; tile < ntiles; ++step) {
      {
        const int nt = tile_tokens(tile, nullptr, nullptr), nb = min(NB, nt - t0);
        t0 += NB;                                        // the step after this one
        if (t0 >= nt) { t0 = 0; tile = from_tile(tile + gridDim.x); }
        Tables<NB>& tb = s.tab[step & 1];
        // every thread has read the previous step's staging buffer (two table barriers lie in between)
#pragma unroll
        for (int j = 0; j < CH; ++j) {
#pragma unroll
          for (int x = 0; x < 5; ++x)
            if (c + kTableThreads * j < NB * kRowPieces) reinterpret_cast<uint4*>(stT + (size_t)x * NB * D)[c + kTableThreads * j] = ldT[x][j];
        }
#pragma unroll
        for (int j = 0; j < CG; ++j)
          if (c + kTableThreads * j < NB * (D / 4)) reinterpret_cast<uint4*>(stG)[c + kTableThreads * j] = ldG[j];
        if (tile < ntiles) issue_loads(tile, t0);
        table_sync();
        float graw[NB];
        T kraw[NB], braw[NB], qraw[NB], wraw[NB], vraw[NB];
#pragma unroll
        for (int t = 0; t < NB; ++t) {
          graw[t] = stG[t * D + c];
          qraw[t] = stT[(0 * NB + t) * D + c]; kraw[t] = stT[(1 * NB + t) * D + c]; braw[t] = stT[(2 * NB + t) * D + c];
          vraw[t] = stT[(3 * NB + t) * D + c]; wraw[t] = stT[(4 * NB + t) * D + c];
        }
        float l[NB], kk[NB], bk[NB], qs[NB], wvv[NB];
#pragma unroll
        for (int t = 0; t < NB; ++t) {
          const bool real = t < nb;                      // padding token: no decay, no write, no read
          l[t] = real ? (graw[t] < kMinGate ? kMinGate : graw[t]) * kLog2e : 0.f;   // (a NaN stays one)
          kk[t] = real ? to_f32(kraw[t]) : 0.f;
          bk[t] = real ? to_f32(braw[t]) * kk[t] : 0.f;
          qs[t] = real ? to_f32(qraw[t]) * scale : 0.f;
          wvv[t] = real ? to_f32(wraw[t]) * to_f32(vraw[t]) : 0.f;
        }
        // the sweep warps have finished with this table buffer (two steps ago)
        // (one warp polls, with pauses; the other three sleep at the barrier below)
        bool okw = true;
        if (wid == 8) okw = mbar_wait_relaxed(&s.tab_empty[step & 1], ((step >> 1) & 1) ^ 1, &s.abort_flag, status, kWaitEmpty);
        // uniform over the table warps; it also orders this step after the reads of the previous step's partial sums
        if (table_sync_or(!okw)) break;
        {
          const int pr = crow(c);
          float c1v[2 * NB], c2v[4 * ((NB + 3) / 4)], An = 1.f;
          float run = 0.f, rest = 0.f;                   // log2 of A_t and of A_NB / A_t
#pragma unroll
          for (int t = 0; t < NB; ++t) {
            run += l[t];
            An = ex2(run);
            c1v[t] = bk[t] * An;
            c1v[NB + t] = qs[t] * An;
            tb.wv[t][c] = wvv[t];
          }
#pragma unroll
          for (int t = NB - 1; t >= 0; --t) {
            c2v[t] = kk[t] * ex2(rest);
            rest += l[t];
          }
#pragma unroll
          for (int t = NB; t < 4 * ((NB + 3) / 4); ++t) c2v[t] = 0.f;
#pragma unroll
          for (int j = 0; j < NB / 2; ++j) tb.c1[j][pr] = make_float4(c1v[4 * j], c1v[4 * j + 1], c1v[4 * j + 2], c1v[4 * j + 3]);
#pragma unroll
          for (int j = 0; j < (NB + 3) / 4; ++j) tb.c2[j][pr] = make_float4(c2v[4 * j], c2v[4 * j + 1], c2v[4 * j + 2], c2v[4 * j + 3]);
          tb.gam[pr] = An;
        }
        // Slot (t, sx) holds the Akk[t, sx] term for sx < t and the Aqk[sx, t] term for sx >= t (the upper
        // triangle is free). Summing over the warp's 32 channels: each step halves what a lane keeps.
        float span[NB];                                  // span[sx] = l[sx + 1] + .. + l[t], log2 of A_t / A_sx
#pragma unroll
        for (int hb = 0; hb < (NB + 3) / 4; ++hb) {
          float term[32];
#pragma unroll
          for (int tt = 0; tt < 4; ++tt) {
            const int t = 4 * hb + tt;
            float ahead = 0.f;
#pragma unroll
            for (int sx = 0; sx < 8; ++sx) {
              float val = 0.f;
              if (t >= NB || sx >= NB) {                                      // (slots of no token)
              } else if (sx < t) {                                                   // Akk[t, sx], A_t / A_s <= 1
                span[sx] = sx == t - 1 ? l[t] : span[sx] + l[t];
                val = bk[t] * kk[sx] * ex2(span[sx]);
              } else if (sx == t) {                                           // Aqk[t, t]
                val = qs[t] * kk[t];
              } else {                                                        // Aqk[sx, t]
                ahead = sx == t + 1 ? l[sx] : ahead + l[sx];
                val = qs[sx] * kk[t] * ex2(ahead);
              }
              term[tt * 8 + sx] = val;
            }
          }
#pragma unroll
          for (int m = 0; m < 5; ++m) {
            const int half = 16 >> m;                    // values kept after this step
            const int bit = 16 >> m;
            const bool up = (lane & bit) != 0;
#pragma unroll
            for (int x = 0; x < half; ++x) {
              const float send = up ? term[x] : term[x + half];
              const float keep = up ? term[x + half] : term[x];
              term[x] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
            }
          }
          int idx = 0;                                   // the lane bit tested at step m chose the upper half of 16 >> m entries
#pragma unroll
          for (int m = 0; m < 5; ++m) idx += ((lane >> (4 - m)) & 1) * (16 >> m);
          s.part[pw_][32 * hb + idx] = term[0];
        }
        table_sync();
        if (c < 64) {
          const float sum = s.part[0][c] + s.part[1][c] + s.part[2][c] + s.part[3][c];
          const int t = c >> 3, sx = c & 7;
          if (t >= NB || sx >= NB) {}
          else if (sx < t) tb.akk[t][sx] = sum;          // Akk[t, sx]
          else tb.aqk[sx][t] = sum;                      // slot (t, sx) with sx >= t holds Aqk[sx, t]
        }
        warp_arrive(&s.tab_full[step & 1], lane);
      }
      // (a block that gave up is left at the next step's table_sync_or, by all four warps together)
    }
  } else {
    // =============================== sweep warps ================================================
    const int rgl = lane >> 2, cq = lane & 3;
    const int col0 = 16 * wid + 4 * cq;
    int it = 0, step = 0;
    for (int tile = from_tile(blockIdx.x); tile < ntiles; tile = from_tile(tile + gridDim.x), ++it) {
      const int nt = tile_tokens(tile, nullptr, nullptr);
      const int buf = it & 1;
      float* S = s.tile[buf];
      bool ok = true;
      for (int t0 = 0; t0 < nt; t0 += NB, ++step) {
        const Tables<NB>& tb = s.tab[step & 1];
        ok = tc::mbar_wait(&s.tab_full[step & 1], (step >> 1) & 1, &s.abort_flag, status, kWaitTab);
        if (ok && t0 == 0) ok = tc::mbar_wait(&s.tile_full[buf], (it >> 1) & 1, &s.abort_flag, status, kWaitTile);
        ok = __all_sync(0xffffffffu, ok);                // the warp leaves together: what follows uses full-warp shuffles
        if (!ok) break;

        // ---- sweep 1: the 2 NB products (NB erase rows, NB query rows) of S_0 for this thread's rows and columns
        //      packed over PAIRS OF PRODUCTS: acc[pp][col] = (product 2pp, product 2pp+1) of column col, so the
        //      coefficients are used as stored (no duplicated copies in shared memory) and the state value is
        //      the operand that is duplicated, in registers
        float2 acc[NB][4];
#pragma unroll
        for (int p = 0; p < NB; ++p) {
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) acc[p][cc] = make_float2(0.f, 0.f);
        }
        const float* Srow = S + rgl * kGroupFloats + col0;
        const int cr0 = 17 * rgl;
#pragma unroll                             // all 16 rows: the loads of later rows are scheduled under the FMAs of earlier ones
        for (int i = 0; i < 16; ++i) {
          const float4 sv = *reinterpret_cast<const float4*>(Srow + i * D);
          const float2 sd[4] = {make_float2(sv.x, sv.x), make_float2(sv.y, sv.y), make_float2(sv.z, sv.z),
                                make_float2(sv.w, sv.w)};
#pragma unroll
          for (int j = 0; j < NB / 2; ++j) {
            const float4 cf = tb.c1[j][cr0 + i];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
              acc[2 * j][cc] = ffma2(sd[cc], make_float2(cf.x, cf.y), acc[2 * j][cc]);
              acc[2 * j + 1][cc] = ffma2(sd[cc], make_float2(cf.z, cf.w), acc[2 * j + 1][cc]);
            }
          }
        }
        // reduce over the 8 row groups. Index = (half * 4 + column) * NB + t (half 0: erase products, 1: query
        // products); lane (rgl) ends with the NB values of half rgl >> 2, column rgl & 3.
        float pv[NB];
        {
          float val[8 * NB];
#pragma unroll
          for (int pp = 0; pp < NB; ++pp) {
            const int half = pp / (NB / 2), base = half * 4 * NB + 2 * pp - half * NB;       // products 2pp, 2pp + 1
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) { val[base + cc * NB] = acc[pp][cc].x; val[base + cc * NB + 1] = acc[pp][cc].y; }
          }
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int half = (4 * NB) >> m;
            const int bit = 16 >> m;                     // lane bits 4, 3, 2 = rgl bits 2, 1, 0
            const bool up = (lane & bit) != 0;
#pragma unroll
            for (int x = 0; x < half; ++x) {
              const float send = up ? val[x] : val[x + half];
              const float keep = up ? val[x + half] : val[x];
              val[x] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
            }
          }
#pragma unroll
          for (int t = 0; t < NB; ++t) pv[t] = val[t];
        }
        // ---- forward substitution for u on the lanes that hold the erase products; the lanes that hold
        //      the query products of the same column take u from them and form the outputs
        const bool has_q = (rgl & 4) != 0;
        const int mycol = col0 + (rgl & 3);
        float u[NB];
        {
          float4 ak[NB][2];                              // rows of Akk, fetched ahead of the dependent chain
#pragma unroll
          for (int t = 1; t < NB; ++t) {
            ak[t][0] = *reinterpret_cast<const float4*>(&tb.akk[t][0]);
            if (t > 4) ak[t][1] = *reinterpret_cast<const float4*>(&tb.akk[t][4]);
          }
          float wvt[NB];
#pragma unroll
          for (int t = 0; t < NB; ++t) wvt[t] = tb.wv[t][mycol];
#pragma unroll
          for (int t = 0; t < NB; ++t) {
            float x = wvt[t] - pv[t];
            const float arow[8] = {ak[t][0].x, ak[t][0].y, ak[t][0].z, ak[t][0].w, ak[t][1].x, ak[t][1].y, ak[t][1].z, ak[t][1].w};
#pragma unroll
            for (int sx = 0; sx < t; ++sx) x = fmaf(-arow[sx], u[sx], x);
            u[t] = x;                                    // meaningful on the erase lanes only
          }
#pragma unroll
          for (int t = 0; t < NB; ++t) {
            const float other = __shfl_xor_sync(0xffffffffu, u[t], 16);
            if (has_q) u[t] = other;
          }
        }
        if (has_q) {
#pragma unroll
          for (int t = 0; t < NB; ++t) {
            const float4 a0 = *reinterpret_cast<const float4*>(&tb.aqk[t][0]);
            const float4 a1 = *reinterpret_cast<const float4*>(&tb.aqk[t][4]);
            const float arow[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            float ov = pv[t];
#pragma unroll
            for (int sx = 0; sx <= t; ++sx) ov = fmaf(arow[sx], u[sx], ov);
            reinterpret_cast<T*>(s.ostage[step & 1])[t * D + mycol] = from_f32<T>(ov);
          }
        }
        tc::fence_async_smem();                          // the staged rows are read by the bulk store
        warp_arrive(&s.o_full[step & 1], lane);
        // gather u of the thread's four columns from the lanes that share cq (rgl bits 0 and 1 = lane bits 2, 3)
        //      and pair them over tokens: up[tp][c] = (u_{2tp}, u_{2tp+1}) of column col0 + c
        float2 up[NB / 2][4];
#pragma unroll
        for (int t = 0; t < NB; ++t) {
          const float o4 = __shfl_xor_sync(0xffffffffu, u[t], 4);      // column (rgl & 3) ^ 1
          const float e = (rgl & 1) ? o4 : u[t];                       // even column of my pair
          const float od = (rgl & 1) ? u[t] : o4;                      // odd column of my pair
          const float e2 = __shfl_xor_sync(0xffffffffu, e, 8);         // the other pair
          const float od2 = __shfl_xor_sync(0xffffffffu, od, 8);
          const float uc[4] = {(rgl & 2) ? e2 : e, (rgl & 2) ? od2 : od, (rgl & 2) ? e : e2, (rgl & 2) ? od : od2};
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            if (t & 1) up[t >> 1][cc].y = uc[cc];
            else up[t >> 1][cc].x = uc[cc];
          }
        }
        // ---- sweep 2: S <- A_NB * S + sum_s (k_s A_NB/A_s) u_s^T, in place
        {
          float* Sw = S + rgl * kGroupFloats + col0;
#pragma unroll 4
          for (int i = 0; i < 16; ++i) {
            // per column a dot product over the NB tokens, packed over token pairs (coefficients as stored)
            const float4 sv = *reinterpret_cast<const float4*>(Sw + i * D);
            float2 kp[NB / 2];
#pragma unroll
            for (int j = 0; j < (NB + 3) / 4; ++j) {
              const float4 kq = tb.c2[j][cr0 + i];
              kp[2 * j] = make_float2(kq.x, kq.y);
              if (2 * j + 1 < NB / 2) kp[2 * j + 1] = make_float2(kq.z, kq.w);
            }
            const float ga = tb.gam[cr0 + i];
            const float svv[4] = {sv.x, sv.y, sv.z, sv.w};
            float nn[4];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
              float2 d = fmul2(kp[NB / 2 - 1], up[NB / 2 - 1][cc]);
#pragma unroll
              for (int j = NB / 2 - 2; j >= 0; --j) d = ffma2(kp[j], up[j][cc], d);
              nn[cc] = fmaf(ga, svv[cc], d.x + d.y);
            }
            *reinterpret_cast<float4*>(Sw + i * D) = make_float4(nn[0], nn[1], nn[2], nn[3]);
          }
        }
        warp_arrive(&s.tab_empty[step & 1], lane);       // this step's tables may be overwritten
      }
      if (!ok) break;
      tc::fence_async_smem();                            // the tile's new values are visible to the bulk store
      warp_arrive(&s.tile_done[buf], lane);
    }
  }
}

}  // namespace

template <typename T>
int launch_decode_blocked(const T* q, const T* k, const T* v, const float* g, const T* b, const T* w, float* state,
                          T* o, int B, int n, int H, int HK, int64_t in_bs, int64_t o_bs, float scale, bool chained,
                          cudaStream_t st) {
  const int ntiles = B * H;
  const int sms = device_sm_count();
  const int grid = ntiles < sms ? ntiles : sms;
  auto launch = [&](auto kern, size_t smem) -> int {
    GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
    GDN2_CUDA_TRY(launch_chained(chained, kern, dim3(grid), kAllThreads, smem, st, q, k, v, g, b, w, state, o, ntiles, n, H, HK, in_bs, o_bs,
                                 scale, device_status_word(), OneLength{}));
    return GDN2_OK;
  };
  // Tokens per step: padding tokens cost what real ones do, so the fewest that n needs; in several steps 6 or 8, whichever takes
  // less, a step of 6 being about four fifths of one of 8. bf16, 16 heads, 256 / 24 conversations, us (steps of 8 before): n = 4
  // 113 -> 91 / 18.6 -> 14.3, n = 5 114 -> 97 / 18.9 -> 16.6, n = 12 213 -> 171 / 30.1 -> 25.4; steps of 6 for n = 16 would take 251 / 34.3
  // in place of 214 / 30.3.
  // A prompt's ragged tail of four or more tokens (not chained) takes steps of 8 whatever its length, as the packed launch does for
  // the tails of all lengths: a sequence has the same bits there and alone. (Tails of one to three tokens are swept token by token when
  // alone, by this kernel when packed.)
  if (!chained) return launch(decode_blocked_kernel<T, OneLength, 8>, sizeof(BlockedSmem<8>) + 128);
  if (n <= 4) return launch(decode_blocked_kernel<T, OneLength, 4>, sizeof(BlockedSmem<4>) + 128);
  if ((n + 5) / 6 * 4 < (n + 7) / 8 * 5) return launch(decode_blocked_kernel<T, OneLength, 6>, sizeof(BlockedSmem<6>) + 128);
  return launch(decode_blocked_kernel<T, OneLength, 8>, sizeof(BlockedSmem<8>) + 128);
}

int launch_decode_packed_tails(const void* q, const void* k, const void* v, const float* g, const void* b, const void* w,
                               float* state, void* o, const PackedSeqs& seqs, int H, int HK, float scale, cudaStream_t st) {
  using T = __nv_bfloat16;
  const size_t smem = sizeof(BlockedSmem<8>) + 128;
  auto kern = decode_blocked_kernel<T, PackedSeqs, 8>;
  GDN2_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
  const int ntiles = seqs.n * H, sms = device_sm_count();
  GDN2_CUDA_TRY(launch_chained(false, kern, dim3(ntiles < sms ? ntiles : sms), kAllThreads, smem, st, static_cast<const T*>(q),
                               static_cast<const T*>(k), static_cast<const T*>(v), g, static_cast<const T*>(b), static_cast<const T*>(w),
                               state, static_cast<T*>(o), ntiles, 0, H, HK, 0, 0, scale, device_status_word(), seqs));
  return GDN2_OK;
}

template int launch_decode_blocked<float>(const float*, const float*, const float*, const float*, const float*,
                                          const float*, float*, float*, int, int, int, int, int64_t, int64_t, float, bool, cudaStream_t);
template int launch_decode_blocked<__nv_bfloat16>(const __nv_bfloat16*, const __nv_bfloat16*, const __nv_bfloat16*,
                                                  const float*, const __nv_bfloat16*, const __nv_bfloat16*, float*,
                                                  __nv_bfloat16*, int, int, int, int, int64_t, int64_t, float, bool, cudaStream_t);
template int launch_decode_blocked<__half>(const __half*, const __half*, const __half*, const float*, const __half*,
                                           const __half*, float*, __half*, int, int, int, int, int64_t, int64_t, float, bool, cudaStream_t);

}  // namespace gdn2
