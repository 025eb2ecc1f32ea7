// The reference's CPU operators (the cbm_mkl_cpp module,
// cbm/cbm_extensions.cpp:351-919) as stateless GPU products on the reference's
// own layout.
//
// The reference binds eight products over a CSR matrix given by begin/end row
// pointers (MKL's four-array CSR) and, for the CBM forms, the compression tree
// as branch offsets plus (parent, child) edges in BFS order per branch.  They
// keep no state between calls, so neither do these: every call reads the
// caller's arrays directly (no plan, no re-layout, no upload).  The only
// memory they need beyond their operands is a caller-owned workspace of
// 256 + 8 N bytes: a status word and claim counters, and per node a
// "has a parent" stamp and a "row is final" stamp.  Stamps are compared with a
// per-call value from a process-wide counter, so the workspace is never
// cleared between calls (it must be zero-filled once, before its first use).
//
// Kernels (all on the caller's stream, none synchronises):
//   direct_mark    every tree edge: stamp its child; check indices, that no
//                  node has two parents and that the branch offsets are a
//                  prefix sum ending at the edge count; zero the claim counters.
//   direct_spmm    Y[i] = sum_k val_k X[col_k] over row i's entries in order
//                  (one FMA per entry, the order of the oracle's restatement;
//                  MKL's own summation order may differ in the last bits):
//                  long rows by column slices through cp.async rings, a team
//                  of lanes for each other row, 16-byte gathers of X rows;
//                  optionally + (1 + eps) X[i] fused into the store.
//   direct_update  tree edges claimed in their listed order (parents precede
//                  children in BFS order, so the earliest unfinished edge
//                  never waits): wait (bounded) until the parent row is final
//                  when the parent has a parent itself, then
//                  Y[v] = Y[v] + Y[u]                     (update)
//                  Y[v] = fma(Y[u], m[v] / m[u], Y[v])    (fused update, the
//                  rounding of cbm/cbm_extensions.cpp:660-697), and mark v final.
//   direct_spmm_t  Y = A^T X: each row's X row scattered into the rows of its
//                  columns with vector atomic adds (order not deterministic).
//   direct_axpy    Y += (1 + eps) X element-wise (the reference's cblas_saxpy),
//                  after the update of the GIN form.

#include "cbm_b200.h"
#include "launch.cuh"

#include <atomic>

namespace cbm {
namespace {

constexpr int kDirectThreads = 256;
constexpr int64_t kDirectHeader = 256;  // QueueState, padded

struct DirectArgs {
  const int32_t* rp_b;
  const int32_t* rp_e;
  const int32_t* col;
  const float* val;  // NULL: every entry 1
  int64_t n_rows, n_cols, nnz;
  const float* x;  // [n_x_rows, c]
  float* y;        // [n_rows (n_cols for the transpose), c]
  int64_t c;
  float self_scale;
  int32_t claim_runs;  // the SpMM's runs of rows are claimed (next_chunk, zeroed by direct_mark)
  int32_t self_term;  // y = fma(self_scale, x[i], (A x)[i]) in the SpMM store
  const int32_t* branches;
  int64_t n_branch_offsets;
  const int32_t* src;
  const int32_t* dst;
  int64_t n_edges;
  const float* mult;  // NULL: plain update
  QueueState* qs;     // workspace header
  unsigned* has_parent;
  unsigned* ready;
  unsigned epoch;
  long long timeout_ns;
};

__device__ __forceinline__ void record(QueueState* qs, int code, long long info) {
  if (atomicCAS(&qs->error, 0, code) == 0) qs->error_info = info;
}

__global__ void __launch_bounds__(kDirectThreads) direct_mark(const DirectArgs a) {
  if (blockIdx.x == 0 && threadIdx.x == 0) a.qs->next_row = a.qs->next_chunk = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < a.n_edges; e += stride) {
    const int32_t u = a.src[e], v = a.dst[e];
    if (u < 0 || u >= a.n_rows || v < 0 || v >= a.n_rows || u == v) {
      record(a.qs, CBM_ERR_INDEX, e);
      continue;
    }
    if (atomicExch(a.has_parent + v, a.epoch) == a.epoch) record(a.qs, CBM_ERR_STRUCTURE, e);  // two parents
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n_branch_offsets; i += stride) {
    const int32_t b = a.branches[i];
    const bool bad = b < 0 || b > a.n_edges || (i == 0 && b != 0) ||
                     (i == a.n_branch_offsets - 1 && b != a.n_edges) || (i > 0 && a.branches[i - 1] > b);
    if (bad) record(a.qs, CBM_ERR_STRUCTURE, i);
  }
}

// ---- direct_spmm ------------------------------------------------------------------
// A row's sum is one chain of FMAs in entry order, so a long row cannot be
// split by entries; it is split by columns instead, and its gathers run far
// ahead of its FMAs.  A block takes a run of rows, lists the long ones, and its
// warps draw tasks: first every (giant row, slice of 32 columns), then every
// (long row, slice of 128), then the other rows, a team of TL lanes each.
// Narrow slices put a giant's chain on more warps; wide ones cost a third of
// the instructions per byte.
//
// Bound: the X-row gathers (L2, and DRAM where X is larger), with the longest
// rows' chains behind them.  Fused-update products on B200, every row by one
// team with four gathers in flight -> as here (us, bit-identical): 250,000-node
// power-law graph of mean degree 20, 256 columns 1933 -> 840, a million nodes
// 6330 -> 3380; 100,000 nodes of mean degree 14, 128 / 40 columns 692 / 546 ->
// 311 / 229; 20,000 nodes, one column 146 -> 87.
//
// Long: more than 16 entries (256 columns: 840 us, 876 from 32 and 927 from
// 64), 64 where a row fills no slice of 32 columns (4 columns: 123 us against
// 152).  Giant: more than 512 entries, 256 up to 128 columns, which have one
// wide slice only (7 columns: 175 us against 187).
__device__ __forceinline__ int long_len(int64_t c) { return c >= 32 ? 16 : 64; }
__device__ __forceinline__ int giant_len(int64_t c) { return c > 128 ? 512 : 256; }
// Ring of a slice task: a giant's holds 6 groups of 8 entries x 128 bytes of X
// rows and their weights (40 entries in flight while 8 are summed), a long
// row's 3 groups of 4 entries x 512 bytes.
constexpr int kRingGroups = 6;
constexpr int kRingEntries = 8 * kRingGroups;
constexpr int kRingFloats = kRingEntries * 33;  // 32 columns and a weight each
constexpr int kWideGroups = 3;
static_assert(kWideGroups * 4 * 128 <= kRingFloats, "one ring serves both");
constexpr int kDirectWarps = kDirectThreads / 32;

// One entry of a slice task: its column (-1 past the end, or out of range and
// recorded) and its weight.
__device__ __forceinline__ void slice_entry(const DirectArgs& a, int b, int n, int64_t c0, int k, int32_t& c,
                                            float& w) {
  c = -1;
  w = 0.f;
  if (k < n) {
    c = __ldg(a.col + b + k);
    w = a.val ? __ldg(a.val + b + k) : 1.f;
    if (c < 0 || c >= a.n_cols) {
      if (c0 == 0) record(a.qs, CBM_ERR_INDEX, b + k);
      c = -1;
      w = 0.f;
    }
  }
}

template <int V>
__device__ __forceinline__ void cp_async_piece(float* smem, const float* gmem, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (V == 4) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gmem), "r"(valid ? 16u : 0u) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(gmem), "r"(valid ? 4u : 0u) : "memory");
  }
}

// Giant rows: columns [c0, c0 + 32) of row `row`, entries [b, b + n), by one warp: X-row
// pieces come through the warp's ring by cp.async, each lane then sums one
// column.  An entry whose column is out of range (recorded) copies nothing and
// weighs 0: its zero-filled slot leaves the sum as it is.
template <int V>
__device__ __forceinline__ void hub_slice(const DirectArgs& a, int64_t row, int b, int n, int64_t c0, float* ring) {
  constexpr int kPieces = 32 / V;     // lanes that copy one entry's 32 columns
  constexpr int kAtOnce = 32 / kPieces;  // entries per copy instruction
  const int lane = threadIdx.x & 31;
  const int piece = lane % kPieces, sub = lane / kPieces;
  const bool in = c0 + piece * V < a.c;
  float* weights = ring + kRingEntries * 32;
  const float* x0 = a.x + c0 + (in ? piece * V : 0);
  // entries come in batches of 32, one per lane, the next batch loaded ahead
  int32_t col = 0, col_n = 0;
  float w = 0.f, w_n = 0.f;
  slice_entry(a, b, n, c0, lane, col, w);
  slice_entry(a, b, n, c0, 32 + lane, col_n, w_n);
  const int groups = (n + 7) / 8;
  int made = 0;  // groups issued
  auto produce = [&]() {
    if (made < groups) {
      if (made > 0 && (made & 3) == 0) {  // a new batch of 32 entries
        col = col_n;
        w = w_n;
        slice_entry(a, b, n, c0, (made + 4) * 8 + lane, col_n, w_n);
      }
      const int slot = made % kRingGroups * 8, e0 = (made & 3) * 8;
      const float we = __shfl_sync(0xffffffffu, w, e0 + (lane & 7));
      if (lane < 8) weights[slot + lane] = we;
#pragma unroll
      for (int u = 0; u < 8; u += kAtOnce) {
        const int32_t c = __shfl_sync(0xffffffffu, col, e0 + u + sub);
        cp_async_piece<V>(ring + (slot + u + sub) * 32 + piece * V, x0 + (int64_t)(c < 0 ? 0 : c) * a.c,
                          in && c >= 0);
      }
    }
    cp_async_commit();
    ++made;
  };
#pragma unroll 1
  for (int g = 0; g < kRingGroups - 1; ++g) produce();
  float acc = 0.f;
#pragma unroll 1
  for (int g = 0; g < groups; ++g) {
    produce();  // into the slot that the previous step summed
    cp_async_wait<kRingGroups - 1>();
    __syncwarp();
    const float* slot = ring + g % kRingGroups * 8 * 32;
    const float* ws = weights + g % kRingGroups * 8;
#pragma unroll
    for (int u = 0; u < 8; ++u) acc = fmaf(ws[u], slot[u * 32 + lane], acc);
    __syncwarp();
  }
  cp_async_wait<0>();
  __syncwarp();
  if (c0 + lane < a.c) {
    const int64_t at = row * a.c + c0 + lane;
    a.y[at] = a.self_term ? fmaf(a.self_scale, __ldg(a.x + at), acc) : acc;
  }
}

// Long rows: columns [c0, c0 + 128), four per lane (one vector, or every 32nd
// scalar).  A lane copies and sums only its own pieces, so its own cp.async
// groups are all it waits for.
template <int V>
__device__ __forceinline__ void wide_slice(const DirectArgs& a, int64_t row, int b, int n, int64_t c0, float* ring) {
  constexpr int P = 4 / V;  // pieces per lane
  const int lane = threadIdx.x & 31;
  int32_t col = 0, col_n = 0;
  float w = 0.f, w_n = 0.f, w_p = 0.f;  // weights of the producer's batch of 32, the next and the previous one
  slice_entry(a, b, n, c0, lane, col, w);
  slice_entry(a, b, n, c0, 32 + lane, col_n, w_n);
  const float* x0 = a.x + c0 + (c0 + lane * V < a.c ? lane * V : 0);
  bool in[P];
#pragma unroll
  for (int q = 0; q < P; ++q) in[q] = c0 + (q * 32 + lane) * V < a.c;
  const int groups = (n + 3) / 4;
  int made = 0;  // groups issued
  auto produce = [&](int slot) {
    if (made < groups) {
      if (made > 0 && (made & 7) == 0) {
        w_p = w;
        col = col_n;
        w = w_n;
        slice_entry(a, b, n, c0, (made + 8) * 4 + lane, col_n, w_n);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int32_t c = __shfl_sync(0xffffffffu, col, (made & 7) * 4 + u);
        const float* xr = x0 + (int64_t)(c < 0 ? 0 : c) * a.c;
#pragma unroll
        for (int q = 0; q < P; ++q)
          cp_async_piece<V>(ring + (slot * 4 + u) * 128 + (q * 32 + lane) * V, xr + (in[q] ? q * 32 : 0),
                            in[q] && c >= 0);
      }
    }
    cp_async_commit();
    ++made;
  };
#pragma unroll
  for (int g = 0; g < kWideGroups - 1; ++g) produce(g);
  float acc[P][V];
#pragma unroll
  for (int q = 0; q < P; ++q)
#pragma unroll
    for (int j = 0; j < V; ++j) acc[q][j] = 0.f;
  int slot = 0;
#pragma unroll 1
  for (int g = 0; g < groups; ++g) {
    produce(slot == 0 ? kWideGroups - 1 : slot - 1);  // into the slot that the previous step summed
    cp_async_wait<kWideGroups - 1>();
    // the producer, at most 3 groups ahead, may be one batch of 8 groups on
    const int last = (made < groups ? made : groups) - 1;
    const float ws = last / 8 == g / 8 ? w : w_p;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float wu = __shfl_sync(0xffffffffu, ws, (g & 7) * 4 + u);
#pragma unroll
      for (int q = 0; q < P; ++q) {
        const float* xs = ring + (slot * 4 + u) * 128 + (q * 32 + lane) * V;
        if constexpr (V == 4) {
          const float4 t = *reinterpret_cast<const float4*>(xs);
          acc[q][0] = fmaf(wu, t.x, acc[q][0]);
          acc[q][1] = fmaf(wu, t.y, acc[q][1]);
          acc[q][2] = fmaf(wu, t.z, acc[q][2]);
          acc[q][3] = fmaf(wu, t.w, acc[q][3]);
        } else {
          acc[q][0] = fmaf(wu, xs[0], acc[q][0]);
        }
      }
    }
    slot = slot + 1 == kWideGroups ? 0 : slot + 1;
  }
  cp_async_wait<0>();
#pragma unroll
  for (int q = 0; q < P; ++q) {
    if (!in[q]) continue;
    const int64_t at = row * a.c + c0 + (q * 32 + lane) * V;
    if (a.self_term) {
      float xs[V];
      Vec<float, V>::load(a.x + at, xs);
#pragma unroll
      for (int j = 0; j < V; ++j) acc[q][j] = fmaf(a.self_scale, xs[j], acc[q][j]);
    }
    store_vec<float, V>(a.y + at, acc[q]);
  }
}

// One row by a team of TL lanes; a lane owns VPL vectors of V floats per pass
// of TL * VPL * V columns.
template <int TL, int VPL, int V>
__device__ __forceinline__ void team_row(const DirectArgs& a, int64_t row, int64_t b, int64_t e, int tl) {
  constexpr int U = (VPL * V >= 8) ? 4 : 8;  // entries whose gathers are in flight together
  constexpr int64_t kPass = (int64_t)TL * VPL * V;
  for (int64_t c0 = 0; c0 < a.c; c0 += kPass) {
    float acc[VPL][V];
#pragma unroll
    for (int q = 0; q < VPL; ++q)
#pragma unroll
      for (int j = 0; j < V; ++j) acc[q][j] = 0.f;
    // wide rows (groups of 4): the next group's columns and values are
    // loaded while the current group's X rows are gathered; narrow rows
    // (groups of 8) load each group's own at its start, which keeps their
    // registers within four blocks per SM
    constexpr bool kPrefetch = U == 4;
    int32_t pc[U];
    float pw[U];
    auto fetch = [&](int64_t k) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = k + u < e;
        pc[u] = in ? __ldg(a.col + k + u) : 0;
        pw[u] = (in && a.val) ? __ldg(a.val + k + u) : 1.f;
      }
    };
    if (kPrefetch && b < e) fetch(b);
    for (int64_t k0 = b; k0 < e; k0 += U) {
      const int n = (int)((e - k0) < U ? (e - k0) : U);
      int64_t off[U];
      float w[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        off[u] = -1;
        w[u] = 0.f;
        if (u < n) {
          const int32_t cj = kPrefetch ? pc[u] : __ldg(a.col + k0 + u);
          if (cj < 0 || cj >= a.n_cols) {
            if (tl == 0) record(a.qs, CBM_ERR_INDEX, k0 + u);
          } else {
            off[u] = (int64_t)cj * a.c;
            w[u] = kPrefetch ? pw[u] : (a.val ? __ldg(a.val + k0 + u) : 1.f);
          }
        }
      }
      if (kPrefetch && k0 + U < e) fetch(k0 + U);
      float xv[U][VPL][V];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < VPL; ++q) {
          const int64_t cc = c0 + ((int64_t)q * TL + tl) * V;
          if (off[u] >= 0 && cc < a.c) {
            Vec<float, V>::load(a.x + off[u] + cc, xv[u][q]);
          } else {
#pragma unroll
            for (int j = 0; j < V; ++j) xv[u][q][j] = 0.f;
          }
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (off[u] >= 0)
#pragma unroll
          for (int q = 0; q < VPL; ++q)
#pragma unroll
            for (int j = 0; j < V; ++j) acc[q][j] = fmaf(w[u], xv[u][q][j], acc[q][j]);
    }
#pragma unroll
    for (int q = 0; q < VPL; ++q) {
      const int64_t cc = c0 + ((int64_t)q * TL + tl) * V;
      if (cc >= a.c) continue;
      if (a.self_term) {
        float xs[V];
        Vec<float, V>::load(a.x + row * a.c + cc, xs);
#pragma unroll
        for (int j = 0; j < V; ++j) acc[q][j] = fmaf(a.self_scale, xs[j], acc[q][j]);
      }
      store_vec<float, V>(a.y + row * a.c + cc, acc[q]);
    }
  }
}

template <int TL, int VPL, int V>
__global__ void __launch_bounds__(kDirectThreads, 4) direct_spmm(const DirectArgs a) {
  extern __shared__ __align__(16) float rings[];
  // a run's rows; giants listed from the front of s_long, long rows from its end
  __shared__ int s_beg[kDirectThreads], s_len[kDirectThreads], s_long[kDirectThreads];
  __shared__ int s_giants, s_longs, s_task;
  __shared__ unsigned s_run;
  constexpr int kTeams = kDirectThreads / TL;
  constexpr int kPerWarp = 32 / TL;  // rows of one row task
  // rows per run: one per team, up to four where every block then still gets
  // several runs, fewer (whole warps' shares) where the rows would else leave
  // blocks without one (2,215 rows, 8 columns: 65 us with a block's full run of 128
  // rows, 38 with 16).  Runs are claimed in turn in the forms with a tree, whose
  // calls own the workspace (direct_mark zeroed the counter); the others may
  // share it with products on other streams and deal their runs out instead.
  const int64_t per_team = a.n_rows / ((int64_t)gridDim.x * kTeams * 4);
  const int64_t shares = (a.n_rows + (int64_t)gridDim.x * kPerWarp - 1) / ((int64_t)gridDim.x * kPerWarp);
  const int run = shares < kTeams / kPerWarp
                      ? kPerWarp * (int)shares
                      : kTeams * (int)(TL < 4 || per_team < 1 ? 1 : per_team < 4 ? per_team : 4);
  const int lane = threadIdx.x & 31;
  const int tl = lane % TL;
  float* ring = rings + (threadIdx.x >> 5) * kRingFloats;
  const int long_row = long_len(a.c), giant = giant_len(a.c);
  const int narrow = (int)((a.c + 31) / 32), wide = (int)((a.c + 127) / 128);
  for (unsigned turn = blockIdx.x;; turn += gridDim.x) {
    __syncthreads();  // the previous run's lists are no longer read
    if (threadIdx.x == 0) {
      s_giants = s_longs = s_task = 0;
      s_run = a.claim_runs ? atomicAdd(&a.qs->next_chunk, 1u) : turn;
    }
    __syncthreads();
    const int64_t r0 = (int64_t)s_run * run;
    if (r0 >= a.n_rows) break;
    if ((int)threadIdx.x < run) {
      const int64_t row = r0 + threadIdx.x;
      int64_t b = 0, e = 0;
      const bool have = row < a.n_rows;
      if (have) {
        b = a.rp_b[row], e = a.rp_e[row];
        if (b < 0 || e < b || e > a.nnz) {
          record(a.qs, CBM_ERR_INDEX, row);
          b = e = 0;
        }
      }
      s_beg[threadIdx.x] = (int)b;
      s_len[threadIdx.x] = have ? (int)(e - b) : -1;
      if (e - b > giant)
        s_long[atomicAdd(&s_giants, 1)] = threadIdx.x;
      else if (e - b > long_row)
        s_long[kDirectThreads - 1 - atomicAdd(&s_longs, 1)] = threadIdx.x;
    }
    __syncthreads();
    const int64_t giant_tasks = (int64_t)s_giants * narrow, long_tasks = giant_tasks + (int64_t)s_longs * wide;
    const int64_t tasks = long_tasks + run / kPerWarp;
    for (;;) {
      int task = 0;
      if (lane == 0) task = atomicAdd(&s_task, 1);
      task = __shfl_sync(0xffffffffu, task, 0);
      if (task >= tasks) break;
      if (task < giant_tasks) {
        const int i = s_long[task / narrow];
        hub_slice<V>(a, r0 + i, s_beg[i], s_len[i], (int64_t)(task % narrow) * 32, ring);
      } else if (task < long_tasks) {
        const int k = task - (int)giant_tasks;
        const int i = s_long[kDirectThreads - 1 - k / wide];
        wide_slice<V>(a, r0 + i, s_beg[i], s_len[i], (int64_t)(k % wide) * 128, ring);
      } else {
        const int i = (task - (int)long_tasks) * kPerWarp + lane / TL;
        if (s_len[i] >= 0 && s_len[i] <= long_row)
          team_row<TL, VPL, V>(a, r0 + i, s_beg[i], (int64_t)s_beg[i] + s_len[i], tl);
        __syncwarp();
      }
    }
  }
}

template <int TL, int VPL, int V>
__global__ void __launch_bounds__(kDirectThreads) direct_update(const DirectArgs a) {
  constexpr int64_t kPass = (int64_t)TL * VPL * V;
  const int tl = threadIdx.x % TL;
  const int lane = threadIdx.x & 31;
  const unsigned tmask = TL == 32 ? 0xffffffffu : (((1u << TL) - 1u) << (lane / TL * TL));
  for (;;) {
    unsigned base = 0;
    if (tl == 0) base = atomicAdd(&a.qs->next_row, 1u);
    base = __shfl_sync(tmask, base, 0, TL);
    if ((int64_t)base >= a.n_edges) break;
    const int64_t e = base;
    const int32_t u = a.src[e], v = a.dst[e];
    if (u < 0 || u >= a.n_rows || v < 0 || v >= a.n_rows || u == v) continue;  // recorded by direct_mark
    bool ok = true;
    if (a.has_parent[u] == a.epoch) ok = wait_flag(a.ready + u, a.epoch, a.qs, a.timeout_ns, e);
    if (ok) {
      const float r = a.mult ? __fdiv_rn(a.mult[v], a.mult[u]) : 1.f;
      const float* yu = a.y + (int64_t)u * a.c;
      float* yv = a.y + (int64_t)v * a.c;
      for (int64_t c0 = 0; c0 < a.c; c0 += kPass) {
#pragma unroll
        for (int q = 0; q < VPL; ++q) {
          const int64_t cc = c0 + ((int64_t)q * TL + tl) * V;
          if (cc >= a.c) continue;
          float pu[V], pv[V];
          load_f32_cg<V>(yu + cc, pu);
          load_f32_cg<V>(yv + cc, pv);
#pragma unroll
          for (int j = 0; j < V; ++j) pv[j] = a.mult ? fmaf(pu[j], r, pv[j]) : __fadd_rn(pv[j], pu[j]);
          store_f32<V>(yv + cc, pv);
        }
      }
    }
    // v is marked final even after a failed wait, so that no wait on it hangs
    __threadfence();
    __syncwarp(tmask);
    if (tl == 0) st_release(a.ready + v, a.epoch);
  }
}

template <int TL, int VPL, int V>
__global__ void __launch_bounds__(kDirectThreads) direct_spmm_t(const DirectArgs a) {
  constexpr int kTeams = kDirectThreads / TL;
  constexpr int64_t kPass = (int64_t)TL * VPL * V;
  const int tl = threadIdx.x % TL;
  const int64_t n_teams = (int64_t)gridDim.x * kTeams;
  for (int64_t row = (int64_t)blockIdx.x * kTeams + threadIdx.x / TL; row < a.n_rows; row += n_teams) {
    int64_t b = a.rp_b[row], e = a.rp_e[row];
    if (b < 0 || e < b || e > a.nnz) {
      if (tl == 0) record(a.qs, CBM_ERR_INDEX, row);
      continue;
    }
    if (b == e) continue;
    for (int64_t c0 = 0; c0 < a.c; c0 += kPass) {
      float xr[VPL][V];
#pragma unroll
      for (int q = 0; q < VPL; ++q) {
        const int64_t cc = c0 + ((int64_t)q * TL + tl) * V;
        if (cc < a.c) {
          Vec<float, V>::load(a.x + row * a.c + cc, xr[q]);
        } else {
#pragma unroll
          for (int j = 0; j < V; ++j) xr[q][j] = 0.f;
        }
      }
      for (int64_t k = b; k < e; ++k) {
        const int32_t cj = __ldg(a.col + k);
        if (cj < 0 || cj >= a.n_cols) {
          if (tl == 0 && c0 == 0) record(a.qs, CBM_ERR_INDEX, k);
          continue;
        }
        const float w = a.val ? __ldg(a.val + k) : 1.f;
        float* yr = a.y + (int64_t)cj * a.c;
#pragma unroll
        for (int q = 0; q < VPL; ++q) {
          const int64_t cc = c0 + ((int64_t)q * TL + tl) * V;
          if (cc >= a.c) continue;
          if constexpr (V == 4) {
            atomicAdd(reinterpret_cast<float4*>(yr + cc),
                      make_float4(w * xr[q][0], w * xr[q][1], w * xr[q][2], w * xr[q][3]));
          } else {
            atomicAdd(yr + cc, w * xr[q][0]);
          }
        }
      }
    }
  }
}

template <int V>
__global__ void __launch_bounds__(kDirectThreads) direct_axpy(const DirectArgs a) {
  const int64_t n = a.n_rows * a.c / V;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float xs[V], ys[V];
    Vec<float, V>::load(a.x + i * V, xs);
    load_f32_cg<V>(a.y + i * V, ys);
#pragma unroll
    for (int j = 0; j < V; ++j) ys[j] = fmaf(a.self_scale, xs[j], ys[j]);
    store_f32<V>(a.y + i * V, ys);
  }
}

int current_device() {
  int d = 0;
  return cudaGetDevice(&d) == cudaSuccess ? d : -1;
}

template <typename K>
int launch_direct(GridCache& cache, K kern, const DirectArgs& a, cudaStream_t st, int smem = 0) {
  const int grid = cached_grid(cache, kern, current_device(), kDirectThreads, smem);
  if (grid <= 0) return CBM_ERR_CUDA;
  kern<<<grid, kDirectThreads, smem, st>>>(a);
  return cuda_status(cudaGetLastError());
}

enum DirectKernel { K_SPMM = 0, K_UPDATE = 1, K_SPMM_T = 2 };

template <int TL, int VPL, int V>
int launch_shape(int which, const DirectArgs& a, cudaStream_t st) {
  static GridCache c_spmm, c_update, c_spmm_t;
  switch (which) {
    case K_SPMM:
      return launch_direct(c_spmm, direct_spmm<TL, VPL, V>, a, st, kDirectWarps * kRingFloats * (int)sizeof(float));
    case K_UPDATE: return launch_direct(c_update, direct_update<TL, VPL, V>, a, st);
    default: return launch_direct(c_spmm_t, direct_spmm_t<TL, VPL, V>, a, st);
  }
}

// Lanes per row and vectors per lane for c columns: 16-byte vectors when the
// operands allow them, a full warp per row from 32 vectors on, two vectors
// per lane from 64 on (passes of 256 columns), else the smallest power-of-two
// team that covers the row.
int launch_kernel(int which, const DirectArgs& a, bool vec, cudaStream_t st) {
  if (!vec) return launch_shape<32, 1, 1>(which, a, st);
  const int64_t nvec = a.c / 4;
  if (nvec >= 64) return launch_shape<32, 2, 4>(which, a, st);
  if (nvec > 16) return launch_shape<32, 1, 4>(which, a, st);
  if (nvec > 8) return launch_shape<16, 1, 4>(which, a, st);
  if (nvec > 4) return launch_shape<8, 1, 4>(which, a, st);
  if (nvec > 2) return launch_shape<4, 1, 4>(which, a, st);
  if (nvec > 1) return launch_shape<2, 1, 4>(which, a, st);
  return launch_shape<1, 1, 4>(which, a, st);
}

std::atomic<unsigned> g_call_epoch{0};

unsigned next_epoch() {
  unsigned e = g_call_epoch.fetch_add(1u) + 1u;
  if (e == 0) e = g_call_epoch.fetch_add(1u) + 1u;  // 0 is the zero-filled workspace's value
  return e;
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// One call: optional SpMM (or its transpose), optional tree update, optional
// trailing (1 + eps) X term.
struct DirectCall {
  bool spmm = false, transpose = false, update = false, axpy = false;
  const int32_t* rp_b = nullptr;
  const int32_t* rp_e = nullptr;
  const int32_t* col = nullptr;
  const float* val = nullptr;
  int64_t n_rows = 0, n_cols = 0, nnz = 0;
  const float* x = nullptr;
  int64_t c = 0;
  float self_scale = 1.f;
  const int32_t* branches = nullptr;
  int64_t n_branch_offsets = 0;
  const int32_t* src = nullptr;
  const int32_t* dst = nullptr;
  int64_t n_edges = 0;
  const float* mult = nullptr;
  float* y = nullptr;
  int64_t n_y_rows = 0;
  void* ws = nullptr;
  int64_t ws_bytes = 0;
  void* stream = nullptr;
};

int run(const DirectCall& k) {
  CbmRange range("cbm direct product");
  if (k.n_rows < 0 || k.n_cols < 0 || k.nnz < 0 || k.c < 0 || k.n_edges < 0 || k.n_branch_offsets < 0 ||
      k.n_y_rows < 0)
    return CBM_ERR_INVALID;
  if (!k.ws || k.ws_bytes < cbm_direct_workspace_bytes(k.n_y_rows) || !aligned16(k.ws)) return CBM_ERR_WORKSPACE;
  if (k.spmm && k.n_rows > 0 && (!k.rp_b || !k.rp_e || (k.nnz > 0 && !k.col))) return CBM_ERR_INVALID;
  if (k.update && k.n_edges > 0 && (!k.src || !k.dst)) return CBM_ERR_INVALID;
  if (k.update && k.n_branch_offsets > 0 && !k.branches) return CBM_ERR_INVALID;
  if (k.n_rows >= INT32_MAX || k.n_cols >= INT32_MAX || k.nnz >= INT32_MAX) return CBM_ERR_TOO_LARGE;
  if (k.c == 0 || k.n_y_rows == 0) return CBM_OK;
  if (!k.y || ((k.spmm || k.axpy) && !k.x)) return CBM_ERR_INVALID;
  // x and y must not overlap (the update reads and writes y in place)
  if (k.x) {
    const int64_t x_rows = k.transpose ? k.n_rows : (k.spmm ? k.n_cols : k.n_y_rows);
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(k.x), y0 = reinterpret_cast<uintptr_t>(k.y);
    const uintptr_t xb = (uintptr_t)(x_rows * k.c * 4), yb = (uintptr_t)(k.n_y_rows * k.c * 4);
    if (x0 < y0 + yb && y0 < x0 + xb) return CBM_ERR_SHAPE;
  }
  cudaStream_t st = static_cast<cudaStream_t>(k.stream);
  DirectArgs a;
  memset(&a, 0, sizeof(a));
  a.rp_b = k.rp_b;
  a.rp_e = k.rp_e;
  a.col = k.col;
  a.val = k.val;
  a.n_rows = k.spmm ? k.n_rows : k.n_y_rows;
  a.n_cols = k.n_cols;
  a.nnz = k.nnz;
  a.x = k.x;
  a.y = k.y;
  a.c = k.c;
  a.self_scale = k.self_scale;
  a.branches = k.branches;
  a.n_branch_offsets = k.n_branch_offsets;
  a.src = k.src;
  a.dst = k.dst;
  a.n_edges = k.n_edges;
  a.mult = k.mult;
  a.qs = static_cast<QueueState*>(k.ws);
  a.has_parent = reinterpret_cast<unsigned*>(static_cast<char*>(k.ws) + kDirectHeader);
  a.ready = a.has_parent + k.n_y_rows;
  a.epoch = next_epoch();
  a.timeout_ns = 1000000000ll;
  const bool vec = k.c % 4 == 0 && aligned16(k.y) && (!k.x || aligned16(k.x));
  int rc;
  const bool tree = k.update && (k.n_edges > 0 || k.n_branch_offsets > 0);
  if (tree) {
    // the tree's nodes are the output rows
    a.n_rows = k.n_y_rows;
    direct_mark<<<sm_count(current_device()) * 4, kDirectThreads, 0, st>>>(a);
    if ((rc = cuda_status(cudaGetLastError()))) return rc;
    a.n_rows = k.spmm ? k.n_rows : k.n_y_rows;
    a.claim_runs = 1;
  }
  if (k.spmm && k.transpose) {
    if (cudaMemsetAsync(k.y, 0, (size_t)(k.n_y_rows * k.c * 4), st) != cudaSuccess) return CBM_ERR_CUDA;
    if ((rc = launch_kernel(K_SPMM_T, a, vec, st))) return rc;
  } else if (k.spmm) {
    // GIN without a tree: (1 + eps) X fused into the SpMM's store
    a.self_term = k.axpy && !tree;
    if ((rc = launch_kernel(K_SPMM, a, vec, st))) return rc;
    a.self_term = 0;
  }
  if (tree && k.n_edges > 0) {
    a.n_rows = k.n_y_rows;
    if ((rc = launch_kernel(K_UPDATE, a, vec, st))) return rc;
  }
  if (k.axpy && (tree || !k.spmm)) {
    a.n_rows = k.n_y_rows;
    static GridCache c4, c1;
    rc = vec ? launch_direct(c4, direct_axpy<4>, a, st) : launch_direct(c1, direct_axpy<1>, a, st);
    if (rc) return rc;
  }
  return CBM_OK;
}

}  // namespace
}  // namespace cbm

using cbm::DirectCall;

extern "C" {

int64_t cbm_direct_workspace_bytes(int64_t n_rows) {
  if (n_rows < 0) return -1;
  return (cbm::kDirectHeader + 8 * n_rows + 255) / 256 * 256;
}

int cbm_direct_status(void* workspace, void* stream, int32_t* device_status, int64_t* info) {
  if (!workspace || !device_status) return CBM_ERR_INVALID;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cbm::QueueState qs;
  if (cudaMemcpyAsync(&qs, workspace, sizeof(qs), cudaMemcpyDeviceToHost, st) != cudaSuccess) return CBM_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return CBM_ERR_CUDA;
  *device_status = qs.error;
  if (info) *info = qs.error_info;
  if (qs.error != 0) {
    // clear the status (error and error_info) for the next calls
    if (cudaMemsetAsync(&static_cast<cbm::QueueState*>(workspace)->error, 0, 16, st) != cudaSuccess)
      return CBM_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return CBM_ERR_CUDA;
  }
  return CBM_OK;
}

int cbm_s_spmm_csr_int32(const int32_t* rp_b, const int32_t* rp_e, const int32_t* col, const float* val,
                         int64_t n_rows, int64_t n_cols, int64_t nnz, const float* rhs, int64_t n_rhs_cols,
                         float* out, void* workspace, int64_t workspace_bytes, void* stream) {
  DirectCall k;
  k.spmm = true;
  k.rp_b = rp_b, k.rp_e = rp_e, k.col = col, k.val = val, k.n_rows = n_rows, k.n_cols = n_cols, k.nnz = nnz;
  k.x = rhs, k.c = n_rhs_cols, k.y = out, k.n_y_rows = n_rows;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_spmm_csr_t_int32(const int32_t* rp_b, const int32_t* rp_e, const int32_t* col, const float* val,
                           int64_t n_rows, int64_t n_cols, int64_t nnz, const float* rhs, int64_t n_rhs_cols,
                           float* out, void* workspace, int64_t workspace_bytes, void* stream) {
  DirectCall k;
  k.spmm = true;
  k.transpose = true;
  k.rp_b = rp_b, k.rp_e = rp_e, k.col = col, k.val = val, k.n_rows = n_rows, k.n_cols = n_cols, k.nnz = nnz;
  k.x = rhs, k.c = n_rhs_cols, k.y = out, k.n_y_rows = n_cols;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_spmm_add_csr_int32(const int32_t* rp_b, const int32_t* rp_e, const int32_t* col, const float* val,
                             int64_t n_rows, int64_t n_cols, int64_t nnz, const float* rhs, int64_t n_rhs_cols,
                             float epsilon, float* out, void* workspace, int64_t workspace_bytes, void* stream) {
  if (n_rows != n_cols) return CBM_ERR_SHAPE;  // X[i] must exist for every row i
  DirectCall k;
  k.spmm = true;
  k.axpy = true;
  k.self_scale = 1.0f + epsilon;
  k.rp_b = rp_b, k.rp_e = rp_e, k.col = col, k.val = val, k.n_rows = n_rows, k.n_cols = n_cols, k.nnz = nnz;
  k.x = rhs, k.c = n_rhs_cols, k.y = out, k.n_y_rows = n_rows;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_spmm_update_csr_int32(const int32_t* rp_b, const int32_t* rp_e, const int32_t* col, const float* val,
                                int64_t n_rows, int64_t n_cols, int64_t nnz, const float* rhs, int64_t n_rhs_cols,
                                const int32_t* branches, int64_t n_branch_offsets, const int32_t* src,
                                const int32_t* dst, int64_t n_edges, float* out, void* workspace,
                                int64_t workspace_bytes, void* stream) {
  DirectCall k;
  k.spmm = true;
  k.update = true;
  k.rp_b = rp_b, k.rp_e = rp_e, k.col = col, k.val = val, k.n_rows = n_rows, k.n_cols = n_cols, k.nnz = nnz;
  k.x = rhs, k.c = n_rhs_cols, k.y = out, k.n_y_rows = n_rows;
  k.branches = branches, k.n_branch_offsets = n_branch_offsets, k.src = src, k.dst = dst, k.n_edges = n_edges;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_spmm_fused_update_csr_int32(const int32_t* rp_b, const int32_t* rp_e, const int32_t* col,
                                      const float* val, int64_t n_rows, int64_t n_cols, int64_t nnz,
                                      const float* rhs, int64_t n_rhs_cols, const int32_t* branches,
                                      int64_t n_branch_offsets, const int32_t* src, const int32_t* dst,
                                      int64_t n_edges, const float* multiplier, float* out, void* workspace,
                                      int64_t workspace_bytes, void* stream) {
  if (!multiplier && n_edges > 0) return CBM_ERR_INVALID;
  DirectCall k;
  k.spmm = true;
  k.update = true;
  k.mult = multiplier;
  k.rp_b = rp_b, k.rp_e = rp_e, k.col = col, k.val = val, k.n_rows = n_rows, k.n_cols = n_cols, k.nnz = nnz;
  k.x = rhs, k.c = n_rhs_cols, k.y = out, k.n_y_rows = n_rows;
  k.branches = branches, k.n_branch_offsets = n_branch_offsets, k.src = src, k.dst = dst, k.n_edges = n_edges;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_spmm_update_add_csr_int32(const int32_t* rp_b, const int32_t* rp_e, const int32_t* col,
                                    const float* val, int64_t n_rows, int64_t n_cols, int64_t nnz,
                                    const float* rhs, int64_t n_rhs_cols, float epsilon, const int32_t* branches,
                                    int64_t n_branch_offsets, const int32_t* src, const int32_t* dst,
                                    int64_t n_edges, float* out, void* workspace, int64_t workspace_bytes,
                                    void* stream) {
  if (n_rows != n_cols) return CBM_ERR_SHAPE;
  DirectCall k;
  k.spmm = true;
  k.update = true;
  k.axpy = true;
  k.self_scale = 1.0f + epsilon;
  k.rp_b = rp_b, k.rp_e = rp_e, k.col = col, k.val = val, k.n_rows = n_rows, k.n_cols = n_cols, k.nnz = nnz;
  k.x = rhs, k.c = n_rhs_cols, k.y = out, k.n_y_rows = n_rows;
  k.branches = branches, k.n_branch_offsets = n_branch_offsets, k.src = src, k.dst = dst, k.n_edges = n_edges;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_update_csr_int32(const int32_t* branches, int64_t n_branch_offsets, const int32_t* src,
                           const int32_t* dst, int64_t n_edges, float* out, int64_t n_out_rows,
                           int64_t n_out_cols, void* workspace, int64_t workspace_bytes, void* stream) {
  DirectCall k;
  k.update = true;
  k.y = out, k.n_y_rows = n_out_rows, k.c = n_out_cols;
  k.branches = branches, k.n_branch_offsets = n_branch_offsets, k.src = src, k.dst = dst, k.n_edges = n_edges;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

int cbm_s_fused_update_csr_int32(const int32_t* branches, int64_t n_branch_offsets, const int32_t* src,
                                 const int32_t* dst, int64_t n_edges, const float* multiplier, float* out,
                                 int64_t n_out_rows, int64_t n_out_cols, void* workspace, int64_t workspace_bytes,
                                 void* stream) {
  if (!multiplier && n_edges > 0) return CBM_ERR_INVALID;
  DirectCall k;
  k.update = true;
  k.mult = multiplier;
  k.y = out, k.n_y_rows = n_out_rows, k.c = n_out_cols;
  k.branches = branches, k.n_branch_offsets = n_branch_offsets, k.src = src, k.dst = dst, k.n_edges = n_edges;
  k.ws = workspace, k.ws_bytes = workspace_bytes, k.stream = stream;
  return cbm::run(k);
}

}  // extern "C"
