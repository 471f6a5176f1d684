// Decode path (T <= B200MOE_DECODE_MAX_T tokens): two kernels, weights streamed from HBM once per expert that has a token.
//
// With a handful of tokens every expert sees one or a few rows: a 128-row tile is padding, and the sort, the gather and
// the tile pipeline of the larger paths cost more than the weights' journey from HBM.  Both kernels run one persistent
// CTA per SM and keep the next pieces of weights in flight in registers (~110 KB per SM; HBM needs ~55).
//
//   k_gemv1_swiglu  (route, selection bits,) GEMM1 + SwiGLU.  Every CTA routes the whole batch by itself, a warp per token,
//                   after the activations were put into shared memory as f16: no launch and no hand-over between routing
//                   and the weight stream.  A task is eight intermediate columns of one expert as one
//                     mma.sync m16n8k16, f16 x f16 -> f32 (e4m3 -> f16 is exact)
//                   M rows 0..7 = W1 rows n.., M rows 8..15 = W3 rows 2048 + n.., N = the expert's tokens, so one thread
//                   holds up and gate of the same (column, token).  K is permuted the same way on both sides: the 16
//                   bytes a lane loads of a row are its A fragments, without a trip through shared memory.  Seven warps
//                   take every seventh of the 56 K blocks of a task (a team reads 896 contiguous bytes per row at a time)
//                   and add their sums through shared memory.
//                   The instruction costs the same for one token and for eight, which is what it is for: packed half FMAs
//                   take 61 us instead of 26 for eight tokens on five hot experts (37 instead of 43 where every expert has
//                   one token).  e4m3 mma.sync (m16n8k32) was slower: 40 us per call at T = 1 against 27.
//   k_gemv2_reduce  GEMM2 and the weighted sum over experts with the same instruction.  A warp task is four output columns
//                   for the whole batch: 8 KB of W2 per expert in registers, requested at once, the intermediate rows in
//                   shared memory as f16 scaled per 128 columns (11-bit rounding of each element, the only one below 32
//                   bits).  M = four columns x four quarters of K and N = the quarters of two tokens, or two columns x eight
//                   eighths and the eighths of one token (half the shared-memory reads: 15 experts with a token each
//                   122.5 us per call, 120.9 with it): a warp needs no other warp's sums.
//                   With packed half FMAs and one scale per row instead, the un-rounded sums were 4.9e-4 off 64 bits, now 1.7e-4
//                   (one 128-column block 1e6 times larger than the others: 1.3e-2, now 1.7e-4).  us per call, those / now:
//                   T = 1 / 32 experts 22.5 / 22.7, T = 7 54.5 / 54.7, T = 8 hot experts 55.5 / 49.3, T = 8 / 256 experts 358 / 366,
//                   hot 200 / 188, T = 2 / 256 118.7 / 120.9.  Refilling the registers for the next expert piece by piece took
//                   7 % longer (the requests of a warp's 8 KB no longer go out together).
// Measured: see the dispatch rule in api.cu.
// Reference counterpart: the T = 1 path, solution/python/pure_triton_impl.py:2025-2123 (_kernel_t1) with
// _t1_fused_gemm2_reduce_kernel (:1676-1750); oracle math solution/cuda/binding.py:157-182.
#include <cuda_fp16.h>
#include "common.cuh"
#include "gemm_common.cuh"
#include "route_token.cuh"

namespace b200moe {

constexpr int DEC_T = B200MOE_DECODE_MAX_T;
constexpr int DEC_PAIRS = DEC_T * TOP_K;
constexpr int DEC_N = 8;                                // tokens of one list = N of the instruction
static_assert(DEC_T <= DEC_N, "an expert's tokens are one N tile, and one lane each in GEMV2's sums");

// streaming 16-byte load (see ld_dep): weights are read once, keep them out of L1
__device__ __forceinline__ uint4 ld_stream(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t half2_bits(const __half2& h) { return *reinterpret_cast<const uint32_t*>(&h); }
// Four e4m3 values -> f16, exactly.
__device__ __forceinline__ uint2 cvt4_h2(uint32_t w) {
  const __half2_raw a = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w & 0xffffu), __NV_E4M3);
  const __half2_raw b = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w >> 16), __NV_E4M3);
  return make_uint2(half2_bits(__half2(a)), half2_bits(__half2(b)));
}
// c += 16 K columns: a0 / a1 = the lane's four of M rows g and g + 8, b0 b1 = the same four of N column g.
__device__ __forceinline__ void mma_k16(float (&c)[4], const uint2& a0, const uint2& a1, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0.x), "r"(a1.x), "r"(a0.y), "r"(a1.y), "r"(b0), "r"(b1));
}
// c += 64 K columns of 16 weight rows x 8 tokens.  lo / hi: the lane's 16 weights of M rows g and g + 8; b: the same 16 K
// columns of token g (f16).  Four MMAs, each taking four of the lane's columns.
__device__ __forceinline__ void mma_k64(float (&c)[4], const uint4& lo, const uint4& hi, const uint8_t* b) {
  const uint4 b0 = reinterpret_cast<const uint4*>(b)[0], b1 = reinterpret_cast<const uint4*>(b)[1];
  mma_k16(c, cvt4_h2(lo.x), cvt4_h2(hi.x), b0.x, b0.y);
  mma_k16(c, cvt4_h2(lo.y), cvt4_h2(hi.y), b0.z, b0.w);
  mma_k16(c, cvt4_h2(lo.z), cvt4_h2(hi.z), b1.x, b1.y);
  mma_k16(c, cvt4_h2(lo.w), cvt4_h2(hi.w), b1.z, b1.w);
}
// Ask for bytes [p, p + bytes) to be brought into L2 (16-byte aligned, a multiple of 16; no completion to wait for).
__device__ __forceinline__ void l2_prefetch_bulk(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// The batch seen expert by expert: lists of the tokens of each active local expert, experts ascending, tokens ascending.
// Pair r of this order is row r of the intermediate.
struct ExpertLists {
  int n;                           // active experts
  int warp_sum[E_GLOBAL / 32];
  uint32_t mask[E_GLOBAL];         // bit t: token t selected the local expert
  int e[DEC_PAIRS];
  int first[DEC_PAIRS + 1];        // first pair of list u
  uint8_t token[DEC_PAIRS];
};

// L.mask is complete (visible to the CTA).  Ends with a barrier.  The CTA has at least E_GLOBAL threads.
__device__ __forceinline__ void build_lists(ExpertLists& L, int E_local) {
  const int e = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t mask = 0;
  int incl = 0;
  if (warp < E_GLOBAL / 32) {
    mask = e < E_local ? L.mask[e] : 0u;
    incl = (__popc(mask) << 16) | (mask != 0u);   // pairs and active experts in one scan
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) L.warp_sum[warp] = incl;
  }
  __syncthreads();
  if (warp < E_GLOBAL / 32) {
    for (int w = 0; w < warp; ++w) incl += L.warp_sum[w];
    if (mask) {
      const int u = (incl & 0xffff) - 1;
      int at = (incl >> 16) - __popc(mask);
      L.e[u] = e;
      L.first[u] = at;
      for (uint32_t m = mask; m; m &= m - 1) L.token[at++] = static_cast<uint8_t>(__ffs(m) - 1);
    }
    if (threadIdx.x == E_GLOBAL - 1) {
      L.n = incl & 0xffff;
      L.first[incl & 0xffff] = incl >> 16;
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------------------------
// GEMM1 + SwiGLU
// ---------------------------------------------------------------------------------------------------------
constexpr int G1_TEAM_WARPS = 7;                          // 56 K blocks, eight per warp
constexpr int G1_TEAMS = 2;
constexpr int G1_THREADS = G1_TEAMS * G1_TEAM_WARPS * 32; // 448: four warps on a quarter of the SM, 128 registers per thread
constexpr int G1_COLS = 8;
constexpr int G1_ROW = 2 * H + 16;        // pitch of an activation row: tokens 16 bytes apart modulo 128, B loads without conflicts
constexpr int G1_SCALES = H_BLOCKS + 1;
constexpr int PART_PITCH = 20;        // floats per token of a partial sum: 16 rows + 4 (conflict-free stores)
static_assert(G1_TEAM_WARPS * 8 == H_BLOCKS && G1_THREADS >= E_GLOBAL, "K split, list building");
constexpr uint32_t W2_PREFETCH_BYTES = 32u << 20;         // about what HBM delivers while GEMV2 starts

struct Gemv1Shared {
  ExpertLists L;
  float part[G1_TEAMS][G1_TEAM_WARPS][DEC_N * PART_PITCH];
  float scale[DEC_T * G1_SCALES];     // activation scales, [token][K block]
};
static size_t gemv1_smem(int T) { return sizeof(Gemv1Shared) + 16 + static_cast<size_t>(T) * G1_ROW; }

template <bool ROUTE>
__global__ void __launch_bounds__(G1_THREADS, 1)
k_gemv1_swiglu(const float* logits, const uint16_t* bias, float scale_factor,
               int* topk_idx, float* topk_w, uint32_t* chunk_bits,
               const uint8_t* hidden, const float* hidden_scale, int T, int local_offset,
               int E_local, const uint8_t* w13, const float* w13_scale,
               const uint8_t* w2, float* inter) {
  extern __shared__ __align__(16) uint8_t dyn[];
  uint8_t* rows = dyn;                                        // [T][G1_ROW]
  Gemv1Shared& S = *reinterpret_cast<Gemv1Shared*>(dyn + static_cast<size_t>(T) * G1_ROW);
  ExpertLists& L = S.L;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < E_GLOBAL) L.mask[threadIdx.x] = 0;
  pdl_wait();
  pdl_launch_dependents();
  for (int c = threadIdx.x; c < T * (H / 16); c += G1_THREADS) {
    const int t = c / (H / 16), u = c - t * (H / 16);
    const uint4 h = ld_dep(reinterpret_cast<const uint4*>(hidden + static_cast<size_t>(t) * H) + u);
    const uint2 h0 = cvt4_h2(h.x), h1 = cvt4_h2(h.y), h2 = cvt4_h2(h.z), h3 = cvt4_h2(h.w);
    uint4* dst = reinterpret_cast<uint4*>(rows + t * G1_ROW + u * 32);
    dst[0] = make_uint4(h0.x, h0.y, h1.x, h1.y);
    dst[1] = make_uint4(h2.x, h2.y, h3.x, h3.y);
  }
  for (int c = threadIdx.x; c < T * H_BLOCKS; c += G1_THREADS) {
    const int kb = c / T, t = c - kb * T;
    S.scale[t * G1_SCALES + kb] = ld_dep(hidden_scale + c);
  }
  __syncthreads();   // masks are zero
  for (int t = warp; t < T; t += G1_TEAMS * G1_TEAM_WARPS) {
    int idx = 0;
    if (ROUTE) {
      float w;
      route_token(logits + static_cast<size_t>(t) * E_GLOBAL, bias, scale_factor, lane, idx, w);
      if (blockIdx.x == 0 && lane < TOP_K) {
        topk_idx[t * TOP_K + lane] = idx;
        topk_w[t * TOP_K + lane] = w;
      }
    } else if (lane < TOP_K) {
      idx = ld_dep(topk_idx + t * TOP_K + lane);
    }
    const int le = idx - local_offset;
    if (lane < TOP_K && le >= 0 && le < E_local) atomicOr(&L.mask[le], 1u << t);
  }
  __syncthreads();
  if (ROUTE && blockIdx.x == 0 && threadIdx.x < E_local) chunk_bits[threadIdx.x] = L.mask[threadIdx.x];   // T <= 32: one chunk
  build_lists(L, E_local);

  const int team = warp / G1_TEAM_WARPS, wt = warp - team * G1_TEAM_WARPS;
  const int tid_team = threadIdx.x - team * (G1_TEAM_WARPS * 32);
  const int g = lane >> 2, q = lane & 3;
  constexpr int TASKS_PER_LIST = I / G1_COLS;
  const int n_teams = static_cast<int>(gridDim.x) * G1_TEAMS, my_team = blockIdx.x * G1_TEAMS + team;
  const int tasks = L.n * TASKS_PER_LIST;
  const int task_begin = tasks * my_team / n_teams, task_end = tasks * (my_team + 1) / n_teams;

  // this lane's share of block kb of a task: 16 bytes at q * 16 and 64 + q * 16 of W1 row n + g and of W3 row n + g
  auto task_ptr = [&](int task) {
    const int u = task / TASKS_PER_LIST, n0 = (task - u * TASKS_PER_LIST) * G1_COLS;
    return w13 + (static_cast<size_t>(L.e[u]) * 2 * I + n0 + g) * H + wt * 128 + q * 16;
  };
  // lanes 0..7: scales of W1 for the warp's eight blocks, lanes 8..15: of W3
  auto task_scale = [&](int task) {
    const int u = task / TASKS_PER_LIST, n0 = (task - u * TASKS_PER_LIST) * G1_COLS;
    return ld_dep(w13_scale + (static_cast<size_t>(L.e[u]) * 32 + (lane & 8) * 2 + (n0 >> 7)) * H_BLOCKS + (lane & 7) * G1_TEAM_WARPS + wt);
  };
  uint4 ring[4][4];
  auto load = [&](uint4 (&s)[4], const uint8_t* p) {
    s[0] = ld_stream(p);
    s[1] = ld_stream(p + 64);
    s[2] = ld_stream(p + static_cast<size_t>(I) * H);
    s[3] = ld_stream(p + static_cast<size_t>(I) * H + 64);
  };
  const uint8_t* ptr = nullptr;
  float wsc = 0.f;
  if (task_begin < task_end) {
    ptr = task_ptr(task_begin);
#pragma unroll
    for (int i = 0; i < 4; ++i) load(ring[i], ptr + i * (G1_TEAM_WARPS * 128));
    wsc = task_scale(task_begin);
  }
#pragma unroll 1
  for (int task = task_begin; task < task_end; ++task) {
    const int u = task / TASKS_PER_LIST, n0 = (task - u * TASKS_PER_LIST) * G1_COLS;
    const int first = L.first[u], m = L.first[u + 1] - first;
    const bool more = task + 1 < task_end;
    const uint8_t* next = more ? task_ptr(task + 1) : ptr;
    const float wsc_next = more ? task_scale(task + 1) : 0.f;
    // columns past the list's last token repeat it; their sums are not used
    const uint8_t* b_row = rows + L.token[first + min(g, m - 1)] * G1_ROW + wt * 256 + q * 32;
    const float* x0 = S.scale + L.token[first + min(2 * q, m - 1)] * G1_SCALES + wt;
    const float* x1 = S.scale + L.token[first + min(2 * q + 1, m - 1)] * G1_SCALES + wt;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint4 (&s)[4] = ring[i & 3];
      const float w1 = __shfl_sync(0xffffffffu, wsc, i), w3 = __shfl_sync(0xffffffffu, wsc, 8 + i);
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      mma_k64(c, s[0], s[2], b_row + i * (G1_TEAM_WARPS * 256));
      mma_k64(c, s[1], s[3], b_row + i * (G1_TEAM_WARPS * 256) + 128);
      acc[0] = fmaf(c[0], x0[i * G1_TEAM_WARPS] * w1, acc[0]);
      acc[1] = fmaf(c[1], x1[i * G1_TEAM_WARPS] * w1, acc[1]);
      acc[2] = fmaf(c[2], x0[i * G1_TEAM_WARPS] * w3, acc[2]);
      acc[3] = fmaf(c[3], x1[i * G1_TEAM_WARPS] * w3, acc[3]);
      if (i < 4) load(s, ptr + (i + 4) * (G1_TEAM_WARPS * 128));
      else if (more) load(s, next + (i - 4) * (G1_TEAM_WARPS * 128));
    }
    float* a = S.part[team][wt] + 2 * q * PART_PITCH + g;
    a[0] = acc[0];
    a[PART_PITCH] = acc[1];
    a[8] = acc[2];
    a[PART_PITCH + 8] = acc[3];
    asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(G1_TEAM_WARPS * 32) : "memory");
    if (tid_team < m * G1_COLS) {
      const float* p = S.part[team][0] + (tid_team >> 3) * PART_PITCH + (tid_team & 7);
      float up = 0.f, gate = 0.f;
#pragma unroll
      for (int w = 0; w < G1_TEAM_WARPS; ++w) {
        up += p[w * (DEC_N * PART_PITCH)];
        gate += p[w * (DEC_N * PART_PITCH) + 8];
      }
      inter[static_cast<size_t>(first + (tid_team >> 3)) * I + n0 + (tid_team & 7)] = gate / (1.0f + expf(-gate)) * up;
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(G1_TEAM_WARPS * 32) : "memory");
    ptr = next;
    wsc = wsc_next;
  }
  // GEMV2 reads W2 of the same experts: have its first rows on their way into L2 while the last columns finish here and
  // the next kernel starts.
  if (lane == 0 && L.n > 0 && w2) {
    constexpr uint32_t PIECE = 8192, PER_EXPERT = static_cast<uint32_t>(H) * I / PIECE;
    uint32_t per = W2_PREFETCH_BYTES / PIECE / static_cast<uint32_t>(L.n);
    per = per < PER_EXPERT ? per : PER_EXPERT;
    for (uint32_t i = blockIdx.x + gridDim.x * warp; i < per * L.n; i += gridDim.x * (G1_TEAMS * G1_TEAM_WARPS)) {
      const uint32_t u = i / per;
      l2_prefetch_bulk(w2 + static_cast<size_t>(L.e[u]) * H * I + static_cast<size_t>(i - u * per) * PIECE, PIECE);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// GEMM2 + weighted sum over experts
// ---------------------------------------------------------------------------------------------------------
// Hides from the compiler that `w` is the same in every round of a loop.  Without it the f16 form of all weights a thread
// holds is computed once before the loop over an expert's tokens (usually one): twice the registers, spilled.
__device__ __forceinline__ void keep_packed(uint4& w) {
  asm volatile("" : "+r"(w.x), "+r"(w.y), "+r"(w.z), "+r"(w.w));
}

constexpr int G2_WARPS = 16;
constexpr int G2_THREADS = G2_WARPS * 32;
constexpr int GEMV2_BATCH = 24;   // intermediate rows staged at a time (4 KB each)
constexpr int GEMV2_COLS = 4;     // output columns per warp task
constexpr int GEMV2_STEPS = I / 256;   // a lane's 16-byte pieces of a weight row
constexpr int G2_ROW = 2 * I + 16;   // pitch of a staged row: the rows of a token pair 16 bytes apart modulo 128

struct Gemv2Shared {
  uint8_t row[GEMV2_BATCH + 1][G2_ROW];          // f16, scaled to |x| <= 256 per 128 columns
  float scale[I_BLOCKS][GEMV2_BATCH + 1];        // what undoes it, times the routing weight
  ExpertLists L;
};

// P pairs of tokens (list entries r .., rows r - p0 .. of the staged batch; `n` of the 2 P are real) of one expert against
// four rows of W2.  M rows 4 c + j and 8 + 4 c + j: quarter j of the K columns of columns c and 2 + c; N column 2 j + t: the
// same quarter of token t of the pair.  Quarter 2 a + b is half b (64 columns) of each of the 128-column blocks 8 a .. 8 a + 7:
// the eight lanes of a (column, a) read whole lines.  Only equal quarters belong together, so lane 16 c + 5 j holds four
// sums and the others nothing of use; that costs the tensor core three quarters of its work, of which it has plenty, and
// keeps each warp's weights, sums and columns to itself.  Lane 8 c + t adds column c of token t to `tot`.
template <int P>
__device__ __forceinline__ void gemv2_rows(const Gemv2Shared& S, int r, int p0, int n, int lane,
                                           uint4 (&w)[GEMV2_STEPS][2], float w_scale, float& tot) {
  const int g = lane >> 2, q = lane & 3;
  // Slots past the last token take whatever the next row holds (the arrays have a row more for that): an N column's sums come
  // from its own values alone, and those of such a slot are not used.
  const uint8_t* b = S.row[r - p0 + (g & 1)] + (g >> 2) * (GEMV2_STEPS * 256) + (g >> 1 & 1) * 128 + q * 32;
  const int swap = (g >> 1 & 1) * 16;
  const float* x = &S.scale[(q >> 1) * GEMV2_STEPS][r - p0];
  float acc[P][4];
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[p][j] = 0.f;
#pragma unroll
  for (int i = 0; i < GEMV2_STEPS; ++i) {
    keep_packed(w[i][0]);
    keep_packed(w[i][1]);
    const uint32_t lo[4] = {w[i][0].x, w[i][0].y, w[i][0].z, w[i][0].w}, hi[4] = {w[i][1].x, w[i][1].y, w[i][1].z, w[i][1].w};
    float c[P][4];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int j = 0; j < 4; ++j) c[p][j] = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint4 bv[P];
#pragma unroll
      for (int p = 0; p < P; ++p) bv[p] = *reinterpret_cast<const uint4*>(b + p * (2 * G2_ROW) + i * 256 + (h * 16 ^ swap));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint2 a0 = cvt4_h2(lo[2 * h + k]), a1 = cvt4_h2(hi[2 * h + k]);
#pragma unroll
        for (int p = 0; p < P; ++p) mma_k16(c[p], a0, a1, k ? bv[p].z : bv[p].x, k ? bv[p].w : bv[p].y);
      }
    }
    const float f = __shfl_sync(0xffffffffu, w_scale, (g >> 1 & 1) * GEMV2_STEPS + i);
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const float f0 = x[i * (GEMV2_BATCH + 1) + 2 * p] * f, f1 = x[i * (GEMV2_BATCH + 1) + 2 * p + 1] * f;
      acc[p][0] = fmaf(c[p][0], f0, acc[p][0]);
      acc[p][1] = fmaf(c[p][1], f1, acc[p][1]);
      acc[p][2] = fmaf(c[p][2], f0, acc[p][2]);
      acc[p][3] = fmaf(c[p][3], f1, acc[p][3]);
    }
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    // add the four quarters (lanes 16 c + 5 j); afterwards lane 16 c + 5 (k + 2 t) holds column c + 2 k of token t
    const bool hi = (lane & 1) != 0, odd = (lane & 2) != 0;
    float y0 = hi ? acc[p][2] : acc[p][0], y1 = hi ? acc[p][3] : acc[p][1];
    y0 += __shfl_xor_sync(0xffffffffu, hi ? acc[p][0] : acc[p][2], 5);
    y1 += __shfl_xor_sync(0xffffffffu, hi ? acc[p][1] : acc[p][3], 5);
    float z = odd ? y1 : y0;
    z += __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 10);
    const int src = (lane & 8) * 2 + (lane >> 4) * 5;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float v = __shfl_sync(0xffffffffu, z, src + 10 * t);
      if (2 * p + t < n && (lane & 7) == S.L.token[r + 2 * p + t]) tot += v;
    }
  }
}

// The same for an expert with one token (`row` of the staged batch): M rows j and 8 + j: eighth j of the K columns of two of the
// four columns, N column j: the same eighth of the token.  Eighth 2 a + b is half b of the blocks 4 a .. 4 a + 3.
__device__ __forceinline__ void gemv2_row(const Gemv2Shared& S, int row, int token, int lane, const uint4 (&w)[4][4], float w_scale,
                                          float& tot) {
  const int g = lane >> 2, q = lane & 3;
  const uint8_t* b = S.row[row] + (lane >> 3) * 1024 + (g & 1) * 128 + q * 32;
  const int swap = (g & 1) * 16;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float c[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) c[0][j] = c[1][j] = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 bv = *reinterpret_cast<const uint4*>(b + i * 256 + (h * 16 ^ swap));
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const uint4 &lo = w[2 * p][i], &hi = w[2 * p + 1][i];
          mma_k16(c[p], cvt4_h2(h ? (k ? lo.w : lo.z) : (k ? lo.y : lo.x)), cvt4_h2(h ? (k ? hi.w : hi.z) : (k ? hi.y : hi.x)),
                  k ? bv.z : bv.x, k ? bv.w : bv.y);
        }
    }
    const float f = __shfl_sync(0xffffffffu, w_scale, (lane >> 3) * 4 + i) * S.scale[q * 4 + i][row];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = fmaf(g & 1 ? c[j >> 1][(j & 1) * 2 + 1] : c[j >> 1][(j & 1) * 2], f, acc[j]);
  }
  // add the eight eighths (lanes 4 j + j / 2); afterwards lane 4 k + 9 l holds column 2 k + l
  const bool hi = (lane & 4) != 0, odd = (lane & 8) != 0;
  float y0 = hi ? acc[2] : acc[0], y1 = hi ? acc[3] : acc[1];
  y0 += __shfl_xor_sync(0xffffffffu, hi ? acc[0] : acc[2], 4);
  y1 += __shfl_xor_sync(0xffffffffu, hi ? acc[1] : acc[3], 4);
  float z = odd ? y1 : y0;
  z += __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 9);
  z += __shfl_xor_sync(0xffffffffu, z, 18);
  const float v = __shfl_sync(0xffffffffu, z, (lane >> 4) * 4 + (lane >> 3 & 1) * 9);
  if ((lane & 7) == token) tot += v;
}

// out[t, n] = sum over the token's local experts of weight * (inter[p] . W2[e][n]).
__global__ void __launch_bounds__(G2_THREADS, 1)
k_gemv2_reduce(const float* inter, const int* topk_idx, const float* topk_w,
               int T, int local_offset, int E_local, const uint8_t* w2, const float* w2_scale,
               uint16_t* out, float* out_f32) {
  extern __shared__ __align__(16) uint8_t dyn[];
  Gemv2Shared& S = *reinterpret_cast<Gemv2Shared*>(dyn);
  ExpertLists& L = S.L;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = gridDim.x;
  if (threadIdx.x < E_GLOBAL) L.mask[threadIdx.x] = 0;
  pdl_launch_dependents();
  pdl_wait();
  __syncthreads();
  if (threadIdx.x < T * TOP_K) {
    const int le = ld_dep(topk_idx + threadIdx.x) - local_offset;
    if (le >= 0 && le < E_local) atomicOr(&L.mask[le], 1u << (threadIdx.x / TOP_K));
  }
  __syncthreads();
  build_lists(L, E_local);
  const int n_lists = L.n, n_pairs = L.first[L.n];

  // Column groups of this CTA, one per warp and round.  A round keeps its sums while the batch's intermediate rows pass
  // through shared memory GEMV2_BATCH at a time (one pass unless the batch has more pairs than that).
  constexpr int GROUPS = H / GEMV2_COLS;
  const int g_begin = GROUPS * blockIdx.x / G, g_end = GROUPS * (blockIdx.x + 1) / G;
  const bool vec_store = ((reinterpret_cast<uintptr_t>(out) & 7u) | (reinterpret_cast<uintptr_t>(out_f32) & 15u)) == 0;
  int staged = -1;   // first pair of the rows in shared memory
  for (int g0 = g_begin; g0 < g_end; g0 += G2_WARPS) {
    const int g = g0 + warp;
    const int n0 = g * GEMV2_COLS;
    float tot = 0.f;   // lane 8 c + t: column n0 + c of token t
    int u = 0;
    for (int p0 = 0; p0 < n_pairs; p0 += GEMV2_BATCH) {
      const int p1 = p0 + GEMV2_BATCH < n_pairs ? p0 + GEMV2_BATCH : n_pairs;
      if (staged != p0) {
        if (staged >= 0) __syncthreads();   // everybody has finished with the rows that are replaced
        // a warp per 512 columns of a row: f16 scaled to |x| <= 256 by the largest magnitude of each 128 (eight lanes' share)
#pragma unroll 1
        for (int h = warp; h < 4 * (p1 - p0); h += G2_WARPS) {
          const int r = h >> 2, c = (h & 3) * 32 + lane;   // this lane's 16 columns
          const float4* x = reinterpret_cast<const float4*>(inter + static_cast<size_t>(p0 + r) * I) + c * 4;
          float4 v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) v[q] = ld_dep(x + q);
          // the routing weight: the slot in which the pair's token holds the pair's expert
          int u_r = 0;
          while (L.first[u_r + 1] <= p0 + r) ++u_r;
          const int at = L.token[p0 + r] * TOP_K + (lane & (TOP_K - 1));
          const float wk = ld_dep(topk_w + at);
          const uint32_t hit = __ballot_sync(0xffffffffu, ld_dep(topk_idx + at) == L.e[u_r] + local_offset);
          const float weight = __shfl_sync(0xffffffffu, wk, __ffs(hit) - 1);
          float m = 1e-36f;   // 256 / m stays finite
#pragma unroll
          for (int q = 0; q < 4; ++q)
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v[q].x), fabsf(v[q].y)), fmaxf(fabsf(v[q].z), fabsf(v[q].w))));
#pragma unroll
          for (int d = 4; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
          const float k = 256.0f / m;
          uint4* dst = reinterpret_cast<uint4*>(S.row[r] + c * 32);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float4 &a = v[2 * q], &b = v[2 * q + 1];
            // the halves of every second 64 columns are swapped: gemv2_row reads two such pieces at a time
            dst[q ^ (c >> 2 & 1)] =
                make_uint4(half2_bits(__floats2half2_rn(a.x * k, a.y * k)), half2_bits(__floats2half2_rn(a.z * k, a.w * k)),
                           half2_bits(__floats2half2_rn(b.x * k, b.y * k)), half2_bits(__floats2half2_rn(b.z * k, b.w * k)));
          }
          if ((lane & 7) == 0) S.scale[c >> 3][r] = weight * (m * (1.0f / 256.0f));
        }
        staged = p0;
        __syncthreads();
      }
      if (g >= g_end) continue;
      while (u < n_lists && L.first[u] < p1) {
        const int e = L.e[u];
        // lanes 0..15: the scales of the 16 K blocks
        const float w_scale =
            ld_dep(w2_scale + (static_cast<size_t>(e) * H_BLOCKS + (n0 >> 7)) * I_BLOCKS + (lane & (I_BLOCKS - 1)));
        const uint8_t* w_cols = w2 + (static_cast<size_t>(e) * H + n0) * I + (lane & 7) * 16;
        const int first = L.first[u], last = L.first[u + 1];
        const int r1 = last < p1 ? last : p1;
        int r = first > p0 ? first : p0;
        if (r1 - r == 1) {
          uint4 w[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) w[j][i] = ld_stream(w_cols + (lane >> 3) * 512 + j * I + i * 128);
          gemv2_row(S, r - p0, L.token[r], lane, w, w_scale, tot);
        } else {
          // this lane's 64-column halves of the blocks 8 a + i of columns n0 + c and n0 + 2 + c (lane = 16 c + 8 a + 4 b + q)
          w_cols += (lane >> 4) * I + (lane >> 3 & 1) * (GEMV2_STEPS * 128);
          uint4 w[GEMV2_STEPS][2];
#pragma unroll
          for (int i = 0; i < GEMV2_STEPS; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) w[i][j] = ld_stream(w_cols + j * (2 * I) + i * 128);
#pragma unroll 1
          for (; r + 2 < r1; r += 4) gemv2_rows<2>(S, r, p0, min(r1 - r, 4), lane, w, w_scale, tot);
          if (r < r1) gemv2_rows<1>(S, r, p0, r1 - r, lane, w, w_scale, tot);
        }
        if (last > p1) break;   // the rest of this expert's tokens are in the next batch of rows
        ++u;
      }
    }
    const float c1 = __shfl_down_sync(0xffffffffu, tot, 8), c2 = __shfl_down_sync(0xffffffffu, tot, 16),
                c3 = __shfl_down_sync(0xffffffffu, tot, 24);
    if (g < g_end && lane < T) {
      const float v[GEMV2_COLS] = {tot, c1, c2, c3};
      const size_t at = static_cast<size_t>(lane) * H + n0;
      if (out) {
        uint16_t b[GEMV2_COLS];
#pragma unroll
        for (int j = 0; j < GEMV2_COLS; ++j) {
          const __nv_bfloat16 x = __float2bfloat16_rn(v[j]);
          b[j] = *reinterpret_cast<const uint16_t*>(&x);
        }
        if (vec_store) {
          *reinterpret_cast<uint2*>(out + at) = make_uint2(b[0] | (static_cast<uint32_t>(b[1]) << 16),
                                                           b[2] | (static_cast<uint32_t>(b[3]) << 16));
        } else {
#pragma unroll
          for (int j = 0; j < GEMV2_COLS; ++j) out[at + j] = b[j];
        }
      }
      if (out_f32) {
        if (vec_store) {
          *reinterpret_cast<float4*>(out_f32 + at) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int j = 0; j < GEMV2_COLS; ++j) out_f32[at + j] = v[j];
        }
      }
    }
  }
}

// `inter` lives in the workspace's expert_out array (unused by this path): one row of 2048 floats per local pair.
template <bool ROUTE>
static int launch_gemv1_as(const b200moe_problem* p, const b200moe_workspace* ws, int num_sms, cudaStream_t st) {
  if (p->T == 0) return B200MOE_OK;
  static bool attr_set[64] = {};
  int dev = 0;
  B200MOE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && !attr_set[dev]) {
    B200MOE_CUDA_TRY(cudaFuncSetAttribute(k_gemv1_swiglu<ROUTE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(gemv1_smem(DEC_T))));
    attr_set[dev] = true;
  }
  B200MOE_CUDA_TRY(launch_pdl(k_gemv1_swiglu<ROUTE>, dim3(num_sms), dim3(G1_THREADS), gemv1_smem(p->T), st,
                              p->routing_logits, p->routing_bias, p->routed_scaling_factor, ws->topk_idx, ws->topk_w,
                              ws->chunk_bits, p->hidden_states, p->hidden_states_scale, p->T, p->local_expert_offset,
                              p->E_local, p->gemm1_weights, p->gemm1_weights_scale,
                              ROUTE ? p->gemm2_weights : nullptr, ws->expert_out));   // the stage call leaves W2 alone
  return B200MOE_OK;
}
int launch_gemv1(const b200moe_problem* p, const b200moe_workspace* ws, int num_sms, cudaStream_t st) {
  return launch_gemv1_as<false>(p, ws, num_sms, st);
}
// routing, selection bits and GEMV1 in one launch
int launch_route_gemv1(const b200moe_problem* p, const b200moe_workspace* ws, int num_sms, cudaStream_t st) {
  return launch_gemv1_as<true>(p, ws, num_sms, st);
}

int launch_gemv2(const b200moe_problem* p, const b200moe_workspace* ws, int num_sms, cudaStream_t st) {
  if (p->T == 0) return B200MOE_OK;
  static bool attr_set[64] = {};
  int dev = 0;
  constexpr int SMEM = sizeof(Gemv2Shared);
  B200MOE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && !attr_set[dev]) {
    B200MOE_CUDA_TRY(cudaFuncSetAttribute(k_gemv2_reduce, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          SMEM));
    attr_set[dev] = true;
  }
  B200MOE_CUDA_TRY(launch_pdl(k_gemv2_reduce, dim3(num_sms), dim3(G2_THREADS), SMEM, st, ws->expert_out,
                              ws->topk_idx, ws->topk_w, p->T, p->local_expert_offset, p->E_local, p->gemm2_weights,
                              p->gemm2_weights_scale, p->output, p->output_f32));
  return B200MOE_OK;
}

}  // namespace b200moe
