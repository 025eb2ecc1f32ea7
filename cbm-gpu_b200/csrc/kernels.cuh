// Device code of the CBM product: one persistent kernel per product.
//
//   Y[v] = sum_k s_k * X[col_k]   (the delta row of v)          cbm/cbm.cu:184-189
//        + Y[parent(v)]            (tree propagation)            cbm/cbm.cu:25-57
//        or + Y[parent(v)] * m[v] / m[parent(v)]                 cbm/cbm.cu:59-91
//
// The reference runs a cuSPARSE SpMM over all rows, then walks each tree branch
// serially in one thread block.  Here a single kernel does both in one pass:
// rows are taken from a device work queue in tree-level order, a team of lanes
// gathers the row's X rows with 16-byte loads, adds the parent's finished row
// (waiting on the parent's ready flag, a bounded wait), and writes Y[v] once.
// Rows longer than the chunk size are summed in chunks by other teams first
// (chunk items precede row items in the queue) and combined in a fixed order.
//
// Progress: items are claimed in queue order by running warps, every item
// depends only on earlier items, and each team finishes its items in claim
// order, so the earliest unfinished item never waits: no deadlock for any grid
// size.  Every wait is still bounded (globaltimer), recording CBM_ERR_TIMEOUT.
#pragma once

#include <cuda.h>  // CUtensorMap (the TMA descriptor type)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <climits>

namespace cbm {

constexpr int kThreads = 256;
// Forward entry word: column in bits 0-29, bit 30 set for the columns gathered
// most often (L2 keeps their X rows), bit 31 the sign.
constexpr uint32_t kColMask = 0x3fffffffu;
constexpr uint32_t kHotBit = 0x40000000u;

// Element offset of row r with leading dimension ld (below 2^31, which the
// host checks): one widening 32 x 32 -> 64-bit multiply per gathered row
// instead of a 64-bit one.
__device__ __forceinline__ uint64_t row_off(uint32_t r, int64_t ld) { return (uint64_t)r * (uint32_t)ld; }

enum ScaleMode : int {
  SCALE_SIGN = 0,       // s
  SCALE_DCOL = 1,       // s * m[col]
  SCALE_DCOL_DROW = 2,  // (s * m[col]) * m[row]
  SCALE_VALUES = 3      // stored value
};
enum PropMode : int { PROP_ADD = 0, PROP_RATIO = 1 };

struct QueueState {
  unsigned int next_chunk;
  unsigned int next_row;
  unsigned int done_blocks;
  unsigned int epoch;
  int error;
  int pad;
  long long error_info;
};

struct FwdArgs {
  // rows in level order
  int32_t n_items;
  // register kernel: one record per item (layout at the kernel) and the items'
  // slots, in record order (level by level, as the items)
  const int4* meta;
  const int32_t* rec_self_slot;
  const int32_t* rec_par_slot;
  const int32_t* node;       // node id per item; bit 31 set: node has children
  const int64_t* ptr;        // [n_items + 1]
  const uint32_t* ent;       // column | sign << 31
  const float* val;          // values (SCALE_VALUES) or null
  const float* sval;         // s * m[col] per entry of ent (SCALE_DCOL*), or null: formed from mult
  const float* csval;        // the same per entry of cent
  const int32_t* par;        // parent node id, -1 for children of the virtual root
  const int32_t* par_item;   // queue position of the parent's item, -1
  const int32_t* self_slot;  // internal-node slot of the item's node, -1 if leaf
  const int32_t* par_slot;   // internal-node slot of the parent, -1
  const int32_t* chunk0;     // first chunk of a split row, -1
  // chunks of long rows (entries in cent / cval)
  const uint32_t* cent;
  const float* cval;
  int32_t n_chunks;
  const int32_t* chunk_item;
  const int64_t* chunk_beg;
  const int64_t* chunk_end;
  // state
  const float* mult;
  unsigned int* node_flag;   // [n_rows], ready epoch of internal nodes
  unsigned int* chunk_flag;  // [n_chunks], then one per presummed row
  QueueState* qs;
  // register kernel: presummed rows (item, node, first entry, entries), longest
  // first, and its kClaimQueues row counters, kClaimStride apart
  int32_t n_pre;
  const int4* pre;
  unsigned int* claims;
  // operands
  const void* x;
  int64_t ldx;
  void* y;
  int64_t ldy;
  int32_t nvec;        // vectors per row (columns / V)
  int32_t ldp;         // floats per row of partial / parent-state scratch
  float* partial;      // [n_chunks, ldp]
  float* pre_rows;     // [n_pre, ldp] sums of presummed rows, or null: kept in Y (FP32)
  float* pstate;       // [n_internal, ldp] fp32 parent rows when Y is bf16
  int32_t scale_mode;
  int32_t prop_mode;
  int32_t team;        // lanes per row: 1, 2, 4, 8, 16 or 32
  int32_t rows_per_claim;       // staged kernel: level-0 rows a team takes per claim
  int32_t rows_per_claim_deep;  // staged kernel: rows below level 0 a team takes per claim
  int32_t n_root;               // items [0, n_root) are level 0 (no parent)
  // staged kernel with several teams per warp: claims of one unit per team,
  // unit u = items [unit[u], unit[u + 1]) (at most 8), level-0 units balanced
  // by entries (null, or full-warp teams: claims of rows_per_claim /
  // rows_per_claim_deep items)
  const int32_t* unit;
  int32_t n_units;
  int32_t hints;       // L2 cache policies on (staged kernel)
  // compensated propagation (register kernel, COMP = true): items from
  // comp_item0 on (tree depth >= the plan's threshold) add their parent term
  // with an error-free sum and carry the rounding residual; items from
  // comp_read0 on (depth >= threshold + 1) read their parent's residual row
  int32_t comp_item0;
  int32_t comp_read0;
  float* pcomp;        // [n_internal, ldp] residual rows of internal nodes
  int32_t tma_rb;      // TMA variant: bytes of one gathered row (nvec * 16)
  // GIN form (register kernel only): Y[v] = (A X)[v] + gin_scale * X[v]
  // (gin_scale = 1 + epsilon), the self term added in the final store only;
  // internal nodes then keep their (A X) rows in pstate for their children,
  // as with BF16 Y
  int32_t gin;
  float gin_scale;
  // first pass of a two-pass product (FP32 Y): rows store their delta sums
  // only (no parent term, no ready flags); prop_kernel adds the parents
  int32_t skip_parent;
  int32_t publish_epoch;  // the last block publishes the launch epoch (0: a pass that another follows)
  long long timeout_ns;
};

// ---- memory-model helpers ----------------------------------------------------
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr long long kMaxSpins = 1ll << 22;

// Bounded wait until *flag == target.  Records the first failure in qs.
// Once any wait of the launch has failed, later waits give up at once, so a
// launch ends within about one timeout whatever goes wrong.
static __device__ __noinline__ bool wait_flag(const unsigned int* flag, unsigned int target, QueueState* qs,
                                              long long timeout_ns, long long info) {
  if (ld_acquire(flag) == target) return true;
  if (*(volatile int*)&qs->error != 0) return false;
  const unsigned long long t0 = global_ns();
  unsigned int ns = 32;
  for (long long it = 0; it < kMaxSpins; ++it) {
    __nanosleep(ns);
    if (ns < 1024) ns <<= 1;
    if (ld_acquire(flag) == target) return true;
    if ((long long)(global_ns() - t0) > timeout_ns) break;
    if ((it & 63) == 63 && *(volatile int*)&qs->error != 0) return false;
  }
  if (atomicCAS(&qs->error, 0, 8 /* CBM_ERR_TIMEOUT */) == 0) qs->error_info = info;
  return false;
}

// One round of a wait that polls several flags: sleeps, and says whether the
// time is over (or an earlier wait of the launch has failed).  t0: 0 at first.
static __device__ __noinline__ bool poll_over(unsigned long long& t0, QueueState* qs, long long timeout_ns) {
  if (t0 == 0) t0 = global_ns();
  __nanosleep(64);
  return *(volatile int*)&qs->error != 0 || (long long)(global_ns() - t0) > timeout_ns;
}

// ---- vector loads / stores ---------------------------------------------------
template <typename T, int V>
struct Vec;

template <>
struct Vec<float, 4> {
  static __device__ __forceinline__ void load(const float* p, float (&o)[4]) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
  }
};
template <>
struct Vec<float, 1> {
  static __device__ __forceinline__ void load(const float* p, float (&o)[1]) { o[0] = __ldg(p); }
};
template <>
struct Vec<__nv_bfloat16, 4> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&o)[4]) {
    const uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
    o[0] = __uint_as_float(t.x << 16);
    o[1] = __uint_as_float(t.x & 0xffff0000u);
    o[2] = __uint_as_float(t.y << 16);
    o[3] = __uint_as_float(t.y & 0xffff0000u);
  }
};
template <>
struct Vec<__nv_bfloat16, 8> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&o)[8]) {
    const uint4 t = __ldg(reinterpret_cast<const uint4*>(p));
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <>
struct Vec<__nv_bfloat16, 1> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&o)[1]) {
    const unsigned short b = __ldg(reinterpret_cast<const unsigned short*>(p));
    o[0] = __uint_as_float(((uint32_t)b) << 16);
  }
};

// store V floats as T
template <typename T, int V>
__device__ __forceinline__ void store_vec(T* p, const float (&v)[V]);

template <>
__device__ __forceinline__ void store_vec<float, 4>(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void store_vec<float, 8>(float* p, const float (&v)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
template <>
__device__ __forceinline__ void store_vec<float, 1>(float* p, const float (&v)[1]) {
  *p = v[0];
}
template <>
__device__ __forceinline__ void store_vec<__nv_bfloat16, 8>(__nv_bfloat16* p, const float (&v)[8]) {
  __nv_bfloat162 h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(h);
}
template <>
__device__ __forceinline__ void store_vec<__nv_bfloat16, 4>(__nv_bfloat16* p, const float (&v)[4]) {
  __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
}
template <>
__device__ __forceinline__ void store_vec<__nv_bfloat16, 1>(__nv_bfloat16* p, const float (&v)[1]) {
  *p = __float2bfloat16_rn(v[0]);
}

// evict-first (streaming) stores of V floats as T
template <typename T, int V>
__device__ __forceinline__ void store_vec_cs(T* p, const float (&v)[V]) {
  if constexpr (sizeof(T) == 4 && V % 4 == 0) {
#pragma unroll
    for (int i = 0; i < V / 4; ++i)
      __stcs(reinterpret_cast<float4*>(p) + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
  } else if constexpr (sizeof(T) == 2 && V == 8) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    __stcs(reinterpret_cast<uint4*>(p), *reinterpret_cast<const uint4*>(h));
  } else {
    store_vec<T, V>(p, v);
  }
}

// fp32 scratch rows (partials, parent state): L2-coherent loads after an acquire
template <int V>
__device__ __forceinline__ void load_f32_cg(const float* p, float (&o)[V]) {
  if constexpr (V % 4 == 0) {
#pragma unroll
    for (int i = 0; i < V / 4; ++i) {
      const float4 t = __ldcg(reinterpret_cast<const float4*>(p) + i);
      o[4 * i] = t.x; o[4 * i + 1] = t.y; o[4 * i + 2] = t.z; o[4 * i + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) o[i] = __ldcg(p + i);
  }
}
template <int V>
__device__ __forceinline__ void store_f32(float* p, const float (&v)[V]) {
  if constexpr (V % 4 == 0) {
#pragma unroll
    for (int i = 0; i < V / 4; ++i)
      reinterpret_cast<float4*>(p)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = v[i];
  }
}
// parent row stored as T (Y itself): L2-coherent load
template <typename T, int V>
__device__ __forceinline__ void load_y_cg(const T* p, float (&o)[V]) {
  if constexpr (sizeof(T) == 4) {
    load_f32_cg<V>(reinterpret_cast<const float*>(p), o);
  } else {
    // bf16 parent rows are never read: the fp32 parent state is used instead
#pragma unroll
    for (int i = 0; i < V; ++i) o[i] = 0.f;
  }
}

template <int VPL, int V>
__host__ __device__ constexpr int unroll_for() {
  return (32 / (VPL * V)) < 1 ? 1 : ((32 / (VPL * V)) > 8 ? 8 : (32 / (VPL * V)));
}

// ---- register kernel: gathers ---------------------------------------------------
// V elements of T as loaded (16 bytes or one element), widened when consumed, so
// a gather in flight costs no more registers than its bytes.
template <typename T, int V>
struct Raw;
template <>
struct Raw<float, 4> {
  using type = float4;
  static constexpr int regs = 4;
  static __device__ __forceinline__ type zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  static __device__ __forceinline__ type load(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
  static __device__ __forceinline__ void widen(const type& r, float (&o)[4]) {
    o[0] = r.x; o[1] = r.y; o[2] = r.z; o[3] = r.w;
  }
};
template <>
struct Raw<float, 1> {
  using type = float;
  static constexpr int regs = 1;
  static __device__ __forceinline__ type zero() { return 0.f; }
  static __device__ __forceinline__ type load(const float* p) { return __ldg(p); }
  static __device__ __forceinline__ void widen(const type& r, float (&o)[1]) { o[0] = r; }
};
template <>
struct Raw<__nv_bfloat16, 8> {
  using type = uint4;
  static constexpr int regs = 4;
  static __device__ __forceinline__ type zero() { return make_uint4(0u, 0u, 0u, 0u); }
  static __device__ __forceinline__ type load(const __nv_bfloat16* p) {
    return __ldg(reinterpret_cast<const uint4*>(p));
  }
  static __device__ __forceinline__ void widen(const type& r, float (&o)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <>
struct Raw<__nv_bfloat16, 1> {
  using type = unsigned short;
  static constexpr int regs = 1;
  static __device__ __forceinline__ type zero() { return 0; }
  static __device__ __forceinline__ type load(const __nv_bfloat16* p) {
    return __ldg(reinterpret_cast<const unsigned short*>(p));
  }
  static __device__ __forceinline__ void widen(const type& r, float (&o)[1]) {
    o[0] = __uint_as_float(((uint32_t)r) << 16);
  }
};

// How the register kernel claims and gathers (CLAIMS).  With two groups claimed
// ahead, the first third of the resident warps takes all the rows of a plan that has
// one group of them per warp, longest rows first, and works through them with the
// rest of the chip idle; and on such a plan the time is the chain of gathers of the
// longest rows, so more of them in flight count for more than occupancy.  Small
// plans (the rule is at the launch) therefore claim one group at a time; teams of 8
// lanes and more also keep twice the gathers in flight (narrower ones gather no
// faster so: 8,000 nodes, 24 BF16 columns 65 -> 72 us).  Measured on B200, two groups
// ahead -> as here (us, bit-identical): 8,000 nodes of mean degree 30, shallow tree, 128
// FP32 / 256 BF16 columns 66 / 87 -> 38 / 42; 2,000 nodes, GIN with 128 / 256 columns 60 /
// 74 -> 27 / 40; GCN graph of 20,000 nodes, 128 / 256 columns 56 / 65 -> 44 / 48; 4,096
// nodes, 64 columns 14.6 -> 11.9.  Twice the gathers on large plans cost a resident
// block and were slower (170,000-node GCN graph, 128 BF16 columns: 152 -> 174).
enum RowClaims : int {
  CLAIMS_AHEAD = 0,  // the next two groups claimed while one is worked on
  CLAIMS_LONE = 1,   // one group at a time
  CLAIMS_FEW = 2     // one group at a time, twice the gathers in flight
};

// Gathers in flight per lane: 16 registers' worth (32 from four pieces per lane
// on and with CLAIMS_FEW), at most 8.
template <typename XT, int VPL, int V, int CLAIMS>
__host__ __device__ constexpr int reg_in_flight() {
  const int u = (VPL >= 4 || CLAIMS == CLAIMS_FEW ? 32 : 16) / (VPL * Raw<XT, V>::regs);
  return u < 1 ? 1 : (u > 8 ? 8 : u);
}

// Entry idx's scale before the row factor: s, the stored value, or s * m[col]
// (from the plan's array when it has one).
__device__ __forceinline__ float reg_scale(uint32_t e, const float* __restrict__ vals, int idx, int scale_mode,
                                           const float* __restrict__ mult) {
  const float sgn = (e >> 31) ? -1.f : 1.f;
  if (scale_mode == SCALE_SIGN) return sgn;
  if (vals) return __ldg(vals + idx);
  return sgn * __ldg(mult + (e & kColMask));
}

// A lane's place in the rows of X: its first piece's address and, for each of
// its VPL pieces, the byte offset from there (0 for a piece past the row's end:
// the lane then reads its first piece again into sums no store reads; a lane
// with no piece at all reads the row's first).  ldb: bytes between rows; WIDE
// allows 2^32 of them and more.
template <typename XT, int VPL, int V, bool WIDE>
struct Lane {
  const char* x;
  uint32_t off[VPL];
  uint32_t ldb, ldb_hi;
  __device__ __forceinline__ Lane(const void* xv, int64_t ldx, int nvec, int tl, int TL) {
    constexpr int piece = V * (int)sizeof(XT);
    x = static_cast<const char*>(xv) + (tl < nvec ? tl * piece : 0);
#pragma unroll
    for (int v = 0; v < VPL; ++v) off[v] = tl + v * TL < nvec ? (uint32_t)(v * TL * piece) : 0u;
    const uint64_t ld = (uint64_t)ldx * sizeof(XT);
    ldb = (uint32_t)ld;
    ldb_hi = (uint32_t)(ld >> 32);
  }
  __device__ __forceinline__ const char* row(uint32_t c) const {
    const char* r = x + (uint64_t)c * ldb;
    return WIDE ? r + ((uint64_t)(c * ldb_hi) << 32) : r;
  }
};

// Lanes per team as a template parameter (TLC): 32, or one of these.
constexpr int kTeamAny = 0;   // run-time team size; entries come by shuffles
// run-time team size of one or two lanes: a batch of one entry per lane would
// be less than a group, so every lane reads its team's entries itself (100,000
// nodes, one FP32 column: 268 -> 172 us, 8 BF16 columns 231 -> 160; with four
// lanes shuffles are faster, 16 FP32 columns 96 against 119)
constexpr int kTeamNarrow = 1;

// acc += sum of scale_k * X[col_k] over the `len` entries of ent, in order, one
// FMA each.  Every lane of the warp calls it: the trip counts come from wlen,
// the largest len of the warp's teams, so teams that share a warp step through
// one instruction stream (a shuffle with per-team masks would split it), and a
// team past its end is predicated off.  e / s: the lane's entry of the first
// TL (loaded ahead by the caller); later batches of TL are loaded one batch
// ahead.  `between` runs once, after the first group's gathers are issued and
// before anything waits for them: the place for loads the next row needs, and
// for an acquire, whose latency then hides under the gathers'.
template <typename XT, int VPL, int V, int TLC, int U, bool WIDE, typename Between>
__device__ __forceinline__ void gather_row(float (&acc)[VPL][V], const Lane<XT, VPL, V, WIDE>& ln,
                                           const uint32_t* __restrict__ ent, const float* __restrict__ vals, int len,
                                           int wlen, uint32_t e, float s, float dv, int scale_mode,
                                           const float* __restrict__ mult, int tl, int team_lanes, Between between) {
  using R = Raw<XT, V>;
  const int TL = TLC == 32 ? 32 : team_lanes;
  if (wlen <= 0) {
    between();
    return;
  }
  if constexpr (TLC == kTeamNarrow) {
    // one address per team; the next group's entries load a group ahead
    uint32_t eg[U];
    float sg[U];
    auto fetch = [&](int j) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        eg[u] = 0;
        sg[u] = 0.f;
        if (j + u < len) {
          eg[u] = __ldg(ent + j + u);
          if (vals) sg[u] = __ldg(vals + j + u);
        }
      }
    };
    fetch(0);
#pragma unroll 1
    for (int j = 0; j < wlen; j += U) {
      typename R::type raw[U][VPL];
      float sc[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const char* row = ln.row(eg[u] & kColMask);
        if (j + u < len) {
#pragma unroll
          for (int v = 0; v < VPL; ++v) raw[u][v] = R::load(reinterpret_cast<const XT*>(row + ln.off[v]));
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        sc[u] = vals ? sg[u] : j + u < len ? reg_scale(eg[u], nullptr, 0, scale_mode, mult) : 0.f;
      if (j == 0) between();
      if (j + U < wlen) fetch(j + U);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j + u < len) {
          const float su = __fmul_rn(sc[u], dv);
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            float t[V];
            R::widen(raw[u][v], t);
#pragma unroll
            for (int k = 0; k < V; ++k) acc[v][k] = fmaf(su, t[k], acc[v][k]);
          }
        }
      }
    }
  } else {
    for (int b = 0; b < wlen; b += TL) {
      const int in = b + TL + tl;
      uint32_t en = 0;
      float sn = 0.f;
      if (in < len) {
        en = __ldg(ent + in);
        if (vals) sn = __ldg(vals + in);
      }
      const uint32_t c = e & kColMask;
      const int cnt = len - b < TL ? len - b : TL;   // this team's entries in the batch (<= 0: none)
      const int wc = wlen - b < TL ? wlen - b : TL;  // the warp's
      typename R::type raw[U][VPL];
      auto load = [&](int j, int u) {
        const char* row = ln.row(__shfl_sync(0xffffffffu, c, j + u, TL));
#pragma unroll
        for (int v = 0; v < VPL; ++v) raw[u][v] = R::load(reinterpret_cast<const XT*>(row + ln.off[v]));
      };
      auto add = [&](float su, int u) {
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          float t[V];
          R::widen(raw[u][v], t);
#pragma unroll
          for (int k = 0; k < V; ++k) acc[v][k] = fmaf(su, t[k], acc[v][k]);
        }
      };
      auto after_loads = [&](int j) {
        if (b + j == 0) {
          between();
          s = __fmul_rn(s, dv);
        }
      };
      int j = 0;
      if (TLC == 32) {
        // whole groups without predicates
#pragma unroll 1
        for (; j + U <= cnt; j += U) {
#pragma unroll
          for (int u = 0; u < U; ++u) load(j, u);
          after_loads(j);
#pragma unroll
          for (int u = 0; u < U; ++u) add(__shfl_sync(0xffffffffu, s, j + u, TL), u);
        }
      }
#pragma unroll 1
      for (; j < wc; j += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const char* row = ln.row(__shfl_sync(0xffffffffu, c, j + u, TL));
          if (j + u < cnt) {
#pragma unroll
            for (int v = 0; v < VPL; ++v) raw[u][v] = R::load(reinterpret_cast<const XT*>(row + ln.off[v]));
          }
        }
        after_loads(j);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float su = __shfl_sync(0xffffffffu, s, j + u, TL);
          if (j + u < cnt) add(su, u);
        }
      }
      e = en;
      if (!vals) sn = in < len ? reg_scale(en, vals, in, scale_mode, mult) : 0.f;
      s = __fmul_rn(sn, dv);
    }
  }
}

// Resident blocks per SM of the register kernel (registers per thread are
// capped to fit them): four for full-warp rows of one vector per lane
// (200,000-node power-law graph, 128 FP32 columns: 348 us with three, 295
// with four), three where teams share a warp (40 BF16 columns on the GCN
// graph: 103 against 121) and for two vectors per lane (47 scalar columns: 103
// against 137 with two).
template <typename XT, typename YT, int VPL, int FORM, int TLC, int CLAIMS>
__host__ __device__ constexpr int fwd_min_blocks() {
  return FORM == 2 || VPL > 4 ? 1 : CLAIMS == CLAIMS_FEW || VPL == 4 ? 2 : VPL == 1 && TLC == 32 ? 4 : 3;
}

// s + e == a + b exactly (Knuth's TwoSum; explicit roundings, no contraction)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// The register kernel hands out rows from kClaimQueues counters, one per warp
// of a block: warp w of every block takes every kClaimQueues-th group.  Atomics
// on one address complete one after another, about 0.9 ns apart on B200, which
// alone cost 150 us of a 170,000-row product with one-row claims.  Each counter
// is handed out in queue order and every block serves all of them, so the
// progress argument of one queue holds.
constexpr int kClaimQueues = kThreads / 32;
constexpr int kClaimStride = 256;  // unsigned, 1 KiB: counters in separate L2 lines

// The last block to finish resets the queue counters and, unless another pass
// of the same product follows, publishes the launch epoch.
__device__ __forceinline__ void finish_block(QueueState* qs, unsigned epoch, bool publish = true,
                                             unsigned* claims = nullptr) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(&qs->done_blocks, 1u);
    if (prev == gridDim.x - 1) {
      qs->next_chunk = 0;
      qs->next_row = 0;
      qs->done_blocks = 0;
      for (int q = 0; claims && q < kClaimQueues; ++q) claims[q * kClaimStride] = 0;
      __threadfence();
      if (publish) atomicExch(&qs->epoch, epoch);
    }
  }
}

// ---- register kernel ------------------------------------------------------------
// Short rows on an operand that L2 holds are bound by latency: a row is a chain
// of dependent loads (claim, record, entries, gathers, parent's flag, parent's
// row).  Each warp therefore runs its rows as a pipeline: while the gathers of
// row i are in flight, row i + 1's entries load and its parent's flag is
// acquired, and the claim and the record of the row after that are made; the
// parent's row of row i + 1 is then fetched together with its gathers.
//
// Teams that share a warp (rows narrower than 32 vectors) step together.  A
// wait then holds up the whole warp, which is safe as long as what it waits
// for is not the warp's own: an item whose parent lies fewer than 32 queue
// positions before it carries kNearBit, and a group of items with one runs its
// row ends team by team, in queue order; with one group claimed at a time (small
// plans, whose levels may be narrower than a warp) all teams at once whose parents
// are ready, polled without blocking (2,145 nodes, 16 BF16 columns: 39 us one by one).
//
// Progress: a warp finishes its groups in the order it claimed them, also with
// the next claim already made, and an item depends on earlier items only.
// Record of an item: x = node | kNearBit | internal << 31, y = parent node or
// -1, z = first entry and w = entries of the row; a split row has its first
// chunk and minus the number of chunks there, a presummed row its place among
// the presummed rows and kPreMark.
//
// Measured on B200 against one row per claim and warp with every load in turn
// (bit-identical): 170,000-node GCN graph, 128 FP32 columns 259 -> 160 us, 128
// BF16 208 -> 145, 40 BF16 174 -> 102-115; 100,000 nodes, 47 FP32 columns (no
// 16-byte vectors) 272 -> 103, GIN with 64 columns 120 -> 77.  What is left is
// instruction issue and the exposed round trip per row, not bandwidth: no
// gather at all leaves 66 us of the first (timed by leaving parts out).
constexpr int kNearBit = 0x40000000;
constexpr int kNodeMask = 0x3fffffff;
// null records past the last item: a group there starts at item n at most
constexpr int kMetaPad = 32;
// entry count of a presummed row's record
constexpr int kPreMark = INT_MIN;
// One past the last chunk of a record (z, w); z itself where the row is not split.
__host__ __device__ constexpr int chunk_stop(int z, int w) { return w < 0 && w != kPreMark ? z - w : z; }
static_assert(chunk_stop(INT_MAX, kPreMark) == INT_MAX && chunk_stop(5, 12) == 5 && chunk_stop(5, -3) == 8,
              "a presummed row's record, whose mark has no negative, walks no chunks");

// What a register-kernel instantiation leaves out: FORM_PLAIN has no GIN term
// and no compensation.
enum RowForm : int { FORM_PLAIN = 0, FORM_GIN = 1, FORM_COMP = 2 };

template <typename XT, typename YT, int VPL, int V, int FORM, int TLC, int CLAIMS>
__global__ void __launch_bounds__(kThreads, (fwd_min_blocks<XT, YT, VPL, FORM, TLC, CLAIMS>()))
    fwd_kernel(const FwdArgs a) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr bool COMP = FORM == FORM_COMP;
  constexpr bool kPlain = FORM == FORM_PLAIN;
  constexpr bool AHEAD = CLAIMS == CLAIMS_AHEAD;
  constexpr int U = reg_in_flight<XT, VPL, V, CLAIMS>();
  // parents' rows come from the FP32 state rows
  const bool state = sizeof(YT) != 4 || FORM == FORM_GIN || (COMP && a.gin);
  const int lane = threadIdx.x & 31;
  const int TL = TLC == 32 ? 32 : a.team;
  const int tl = lane & (TL - 1);
  const int team = lane / TL;
  const unsigned teams = 32 / TL;
  const unsigned epoch = *(volatile unsigned*)&a.qs->epoch + 1u;
  const Lane<XT, VPL, V, TLC != 32> ln(a.x, a.ldx, a.nvec, tl, TL);
  const bool drow = a.scale_mode == SCALE_DCOL_DROW;
  const bool ratio = a.prop_mode == PROP_RATIO;
  const float* vals = a.scale_mode == SCALE_SIGN ? nullptr : a.scale_mode == SCALE_VALUES ? a.val : a.sval;
  const unsigned n = (unsigned)a.n_items;

  // ---- sums that wait on nothing: chunks of split rows, then the presummed
  // rows; one per team and claim, the next claim made ahead
  const unsigned n_split = (unsigned)a.n_chunks;
  const unsigned n_sums = n_split + (unsigned)a.n_pre;
  if (n_sums > 0) {
    const float* cvals = a.scale_mode == SCALE_SIGN ? nullptr : a.scale_mode == SCALE_VALUES ? a.cval : a.csval;
    unsigned pend = 0;
    if (lane == 0) pend = atomicAdd(&a.qs->next_chunk, teams);
    for (;;) {
      const unsigned base = __shfl_sync(kAll, pend, 0);
      if (base >= n_sums) break;
      if (lane == 0) pend = atomicAdd(&a.qs->next_chunk, teams);
      const unsigned k = base + team;
      const bool have = k < n_sums;
      const bool split = k < n_split;
      const uint32_t* ent = a.ent;
      const float* cv = vals;
      float* out = nullptr;
      int len = 0, node = 0;
      if (have) {
        if (split) {
          const int64_t cb = a.chunk_beg[k];
          len = (int)(a.chunk_end[k] - cb);
          node = a.node[a.chunk_item[k]] & 0x7fffffff;
          ent = a.cent + cb;
          cv = cvals ? cvals + cb : nullptr;
          out = a.partial + (int64_t)k * a.ldp;
        } else {
          const int4 r = __ldg(a.pre + (k - n_split));
          len = r.w;
          node = r.y;
          ent = a.ent + (uint32_t)r.z;
          if (vals) cv = vals + (uint32_t)r.z;
          out = a.pre_rows ? a.pre_rows + (int64_t)(k - n_split) * a.ldp
                           : static_cast<float*>(a.y) + row_off(node, a.ldy);
        }
      }
      uint32_t e = 0;
      float s = 0.f;
      if (tl < len) {
        e = __ldg(ent + tl);
        s = reg_scale(e, cv, tl, a.scale_mode, a.mult);
      }
      const float dv = drow ? __ldg(a.mult + node) : 1.f;
      float acc[VPL][V];
#pragma unroll
      for (int v = 0; v < VPL; ++v)
#pragma unroll
        for (int q = 0; q < V; ++q) acc[v][q] = 0.f;
      gather_row<XT, VPL, V, TLC, U>(acc, ln, ent, cv, len, TLC == 32 ? len : __reduce_max_sync(kAll, len), e, s, dv,
                                  a.scale_mode, a.mult, tl, TL, [] {});
      if (have) {
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) store_f32<V>(out + vi * V, acc[v]);
        }
      }
      // the barrier orders the team's stores before its first lane's release,
      // which carries them (cumulativity)
      __syncwarp();
      if (have && tl == 0) st_release(a.chunk_flag + k, epoch);
    }
  }

  // ---- rows: one group of `teams` items per claim from the warp's queue, the
  // next claim made ahead if AHEAD
  const unsigned wq = threadIdx.x >> 5;
  unsigned pend = 0;
  auto claim = [&] {
    if (lane == 0) pend = atomicAdd(a.claims + wq * kClaimStride, 1u);
  };
  // first item of the warp's next group; n when the queue is exhausted
  auto next_group = [&]() -> unsigned {
    const unsigned g = (__shfl_sync(kAll, pend, 0) * kClaimQueues + wq) * teams;
    if (g >= n) return n;  // the claim stays pending: every later call ends here too
    if (AHEAD) claim();
    return g;
  };
  unsigned g0, g1 = n, f0;
  int4 m0, m1;
  uint32_t e0;
  float s0;
  // the next group, with nothing of it claimed or loaded yet
  auto begin = [&] {
    claim();
    g0 = next_group();
    if (g0 >= n) return;
    m0 = __ldg(a.meta + g0 + team);
    e0 = 0;
    s0 = 0.f;
    f0 = 0;
    if (tl < m0.w) {
      e0 = __ldg(a.ent + (uint32_t)m0.z + tl);
      s0 = reg_scale(e0, vals ? vals + (uint32_t)m0.z : nullptr, tl, a.scale_mode, a.mult);
    }
    if (AHEAD) g1 = next_group();
    m1 = __ldg(a.meta + g1 + team);
    if (a.skip_parent) m0.y = -1, m1.y = -1;
    if (m0.y >= 0) f0 = ld_acquire(a.node_flag + m0.y);
  };
  begin();
  while (g0 < n) {
    const unsigned item = g0 + team;
    const bool have = TLC == 32 || item < n;
    const int node = m0.x & kNodeMask;
    const int p = m0.y;
    const float dv = drow || ratio ? __ldg(a.mult + node) : 1.f;
    // the parent's row, if that is final already
    const bool ready = p >= 0 && f0 == epoch;
    float yp[VPL][V];
    float dp = 1.f;
    auto load_parent = [&]() {
      const float* src;
      if (state) {
        src = a.pstate + (int64_t)__ldg(a.rec_par_slot + item) * a.ldp;
      } else {
        src = static_cast<const float*>(a.y) + row_off(p, a.ldy);
      }
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = tl + v * TL;
        if (vi < a.nvec) load_f32_cg<V>(src + (int64_t)vi * V, yp[v]);
      }
    };
    if (ready) load_parent();
    typename Raw<XT, V>::type xself[VPL];  // GIN: the row's own X, for its store
    auto load_self = [&]() {
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        xself[v] = Raw<XT, V>::zero();
        if (a.gin && have) xself[v] = Raw<XT, V>::load(reinterpret_cast<const XT*>(ln.row(node) + ln.off[v]));
      }
    };
    // ahead of the gathers, but for one piece per lane, where those registers
    // are worth more as occupancy (100,000-node GIN, 256 FP32 columns: 198 ->
    // 178 us; 200,000 nodes, 128 columns: 376 -> 353 us the other way)
    if (!kPlain && VPL > 1) load_self();
    if (ratio && p >= 0) dp = __ldg(a.mult + p);
    float acc[VPL][V];
#pragma unroll
    for (int v = 0; v < VPL; ++v)
#pragma unroll
      for (int q = 0; q < V; ++q) acc[v][q] = 0.f;
    const int len = m0.w > 0 ? m0.w : 0;
    uint32_t e1 = 0;
    float s1 = 0.f;
    unsigned f1 = 0;
    gather_row<XT, VPL, V, TLC, U>(acc, ln, a.ent + (uint32_t)m0.z, vals ? vals + (uint32_t)m0.z : nullptr, len,
                                TLC == 32 ? len : __reduce_max_sync(kAll, len), e0, s0, drow ? dv : 1.f,
                                a.scale_mode, a.mult, tl, TL, [&] {
                                  if (tl < m1.w) {
                                    e1 = __ldg(a.ent + (uint32_t)m1.z + tl);
                                    if (vals) s1 = __ldg(vals + (uint32_t)m1.z + tl);
                                  }
                                  if (m1.y >= 0) f1 = ld_acquire(a.node_flag + m1.y);
                                });

    if (!kPlain && VPL == 1) load_self();

    // ---- the row's end: chunk partials, parent, store, ready flag
    const bool near_any = TLC != 32 && __any_sync(kAll, have && (m0.x & kNearBit) != 0);
    const int turns = AHEAD && !near_any ? 1 : AHEAD ? (int)teams : INT_MAX;
    bool todo = have;
    unsigned long long t0 = 0;
    for (int turn = 0; turn < turns; ++turn) {
      bool go = todo;
      if constexpr (AHEAD) {
        // a group that may hold an item and its parent: team by team, in queue order
        go = have && (turns == 1 || team == turn);
      } else if (near_any) {
        // here those whose parent is ready
        if (go && p >= 0) go = ld_acquire(a.node_flag + p) == epoch;
        go = __shfl_sync(kAll, go, team * TL);  // the team's first lane's answer
        if (!__any_sync(kAll, go)) go = todo && poll_over(t0, a.qs, a.timeout_ns);
        go = __shfl_sync(kAll, go, team * TL);
      }
      if (go) {
        todo = false;
        if (m0.w == kPreMark) {
          // summed ahead: record z is its place among the presummed rows
          if (wait_flag(a.chunk_flag + n_split + m0.z, epoch, a.qs, a.timeout_ns, (long long)m0.z)) {
            const float* prow = a.pre_rows ? a.pre_rows + (int64_t)m0.z * a.ldp
                                           : static_cast<const float*>(a.y) + row_off(node, a.ldy);
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
              const int vi = tl + v * TL;
              if (vi < a.nvec) load_f32_cg<V>(prow + vi * V, acc[v]);
            }
          }
        }
        for (int k = m0.z, ke = chunk_stop(m0.z, m0.w); k < ke; ++k) {
          if (!wait_flag(a.chunk_flag + k, epoch, a.qs, a.timeout_ns, (long long)k)) continue;
          const float* prow = a.partial + (int64_t)k * a.ldp;
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            const int vi = tl + v * TL;
            if (vi < a.nvec) {
              float part[V];
              load_f32_cg<V>(prow + vi * V, part);
#pragma unroll
              for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], part[q]);
            }
          }
        }
        // compensated arithmetic for this row, a residual to read from the parent
        const bool cmode = COMP && (int)item >= a.comp_item0;
        const bool cread = COMP && (int)item >= a.comp_read0;
        float cres[VPL][V];  // unused (and removed by the compiler) without COMP
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
          for (int q = 0; q < V; ++q) cres[v][q] = 0.f;
        // after a failed (timed-out) wait the parent is left out; the error is recorded
        bool add = ready;
        if (p >= 0 && !ready && wait_flag(a.node_flag + p, epoch, a.qs, a.timeout_ns, (long long)node)) {
          load_parent();
          add = true;
        }
        if (add) {
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            const int vi = tl + v * TL;
            if (vi < a.nvec) {
              if (COMP && cmode) {
                // parent value = yp + rp (rp: its residual); add with TwoSum and keep
                // the rounding errors (of the ratio's product and quotient too)
                float rp[V];
                if (cread) {
                  load_f32_cg<V>(a.pcomp + (int64_t)__ldg(a.rec_par_slot + item) * a.ldp + vi * V, rp);
                } else {
#pragma unroll
                  for (int q = 0; q < V; ++q) rp[q] = 0.f;
                }
#pragma unroll
                for (int q = 0; q < V; ++q) {
                  float y = yp[v][q], r = rp[q];
                  if (ratio) {
                    const float prod = __fmul_rn(yp[v][q], dv);
                    const float pe = fmaf(yp[v][q], dv, -prod);  // prod + pe == yp * dv
                    y = __fdiv_rn(prod, dp);
                    const float qe = __fdiv_rn(fmaf(-y, dp, prod), dp);  // y + qe ~ prod / dp
                    r = __fadd_rn(__fdiv_rn(fmaf(r, dv, pe), dp), qe);
                  }
                  float s_, e_;
                  two_sum(acc[v][q], y, s_, e_);
                  acc[v][q] = s_;
                  cres[v][q] = __fadd_rn(r, e_);
                }
              } else if (ratio) {
#pragma unroll
                for (int q = 0; q < V; ++q)
                  acc[v][q] = __fadd_rn(acc[v][q], __fdiv_rn(__fmul_rn(yp[v][q], dv), dp));
              } else {
#pragma unroll
                for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], yp[v][q]);
              }
            }
          }
        }
        const bool keep = m0.x < 0 && !a.skip_parent;  // children read this row
        const int ss = keep && (state || COMP) ? __ldg(a.rec_self_slot + item) : 0;
        if (COMP && cmode) {
          // the row's value is acc + cres, rounded once; its residual is kept for
          // the children of an internal node
#pragma unroll
          for (int v = 0; v < VPL; ++v)
#pragma unroll
            for (int q = 0; q < V; ++q) {
              float s_, e_;
              two_sum(acc[v][q], cres[v][q], s_, e_);
              acc[v][q] = s_;
              cres[v][q] = e_;
            }
          if (keep) {
            float* crow = a.pcomp + (int64_t)ss * a.ldp;
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
              const int vi = tl + v * TL;
              if (vi < a.nvec) store_f32<V>(crow + vi * V, cres[v]);
            }
          }
        }
        YT* yrow = static_cast<YT*>(a.y) + row_off(node, a.ldy);
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) {
            if constexpr (kPlain) {
              store_vec<YT, V>(yrow + (int64_t)vi * V, acc[v]);
            } else {
              float xs[V], out[V];
              Raw<XT, V>::widen(xself[v], xs);
#pragma unroll
              for (int q = 0; q < V; ++q) out[q] = a.gin ? fmaf(a.gin_scale, xs[q], acc[v][q]) : acc[v][q];
              store_vec<YT, V>(yrow + (int64_t)vi * V, out);
            }
          }
        }
        if (keep) {
          if (state) {
            float* srow = a.pstate + (int64_t)ss * a.ldp;
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
              const int vi = tl + v * TL;
              if (vi < a.nvec) store_f32<V>(srow + vi * V, acc[v]);
            }
          }
          // as for the chunks: the team's stores before its first lane's release
          __syncwarp(TLC == 32 || TL == 32 ? kAll : (((1u << TL) - 1u) << (team * TL)));
          if (tl == 0) st_release(a.node_flag + node, epoch);
        }
      }
      __syncwarp();
      if (!AHEAD && !(near_any && __any_sync(kAll, todo))) break;
    }
    // ---- on to the next row: its entries are here, the record behind it loads
    if constexpr (!AHEAD) {
      begin();
      continue;
    }
    g0 = g1;
    m0 = m1;
    e0 = e1;
    s0 = vals ? s1 : tl < m0.w ? reg_scale(e0, nullptr, 0, a.scale_mode, a.mult) : 0.f;
    f0 = f1;
    g1 = next_group();
    m1 = __ldg(a.meta + g1 + team);
    if (a.skip_parent) m1.y = -1;
  }
  finish_block(a.qs, epoch, a.publish_epoch != 0, a.claims);
}

// ============================================================================
// Second pass of a two-pass product (FP32 Y): the first pass (fwd_kernel or
// fwd_stream_kernel with skip_parent) left every row's delta sum in Y; this
// pass adds the parent term to the rows below tree level 0, in level order
// (items [n_root, n_items)): wait (bounded) until the parent is final when it
// is itself below level 0, then
//   Y[v] = Y[v] + Y[u]                 (PROP_ADD)
//   Y[v] = Y[v] + (Y[u] m[v]) / m[u]   (PROP_RATIO, cbm/cbm.cu:88)
// the same additions, in the same order, as the one-pass kernels, so results
// are bit-identical.  A deep tree's rows then gather X without waiting on
// their parents, and the waits left here are short (no gathers behind them).
// ============================================================================
struct PropArgs {
  int32_t n_items;
  int32_t n_root;
  const int32_t* node;
  const int32_t* par;
  const int32_t* par_item;
  float* y;
  int64_t ldy;
  int32_t nvec;
  const float* mult;
  int32_t prop_mode;
  unsigned int* node_flag;
  QueueState* qs;
  int32_t team;
  long long timeout_ns;
};

template <int VPL, int V>
__global__ void __launch_bounds__(kThreads) prop_kernel(const PropArgs a) {
  const int lane = threadIdx.x & 31;
  const int TL = a.team;
  const int team = lane / TL;
  const int tl = lane & (TL - 1);
  const int teams = 32 / TL;
  const unsigned tmask = (TL == 32) ? 0xffffffffu : (((1u << TL) - 1u) << (team * TL));
  const unsigned epoch = *(volatile unsigned*)&a.qs->epoch + 1u;
  const unsigned n_deep = (unsigned)(a.n_items - a.n_root);
  for (;;) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&a.qs->next_row, (unsigned)teams);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n_deep) break;
    const unsigned k = base + team;
    if (k < n_deep) {
      const int item = a.n_root + (int)k;
      const int nodew = a.node[item];
      const int node = nodew & 0x7fffffff;
      const int p = a.par[item];
      bool ok = p >= 0;
      if (ok && a.par_item[item] >= a.n_root)
        ok = wait_flag(a.node_flag + p, epoch, a.qs, a.timeout_ns, (long long)node);
      if (ok) {
        const bool ratio = a.prop_mode == PROP_RATIO;
        const float dv = ratio ? __ldg(a.mult + node) : 1.f;
        const float dp = ratio ? __ldg(a.mult + p) : 1.f;
        const float* yp_row = a.y + (int64_t)p * a.ldy;
        float* yv_row = a.y + (int64_t)node * a.ldy;
        // passes of TL * VPL vectors cover rows of any width
        for (int vb = 0; vb < a.nvec; vb += TL * VPL) {
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = vb + tl + v * TL;
          if (vi < a.nvec) {
            float yp[V], yv[V];
            load_f32_cg<V>(yp_row + vi * V, yp);
            load_f32_cg<V>(yv_row + vi * V, yv);
            if (ratio) {
#pragma unroll
              for (int q = 0; q < V; ++q) yv[q] = __fadd_rn(yv[q], __fdiv_rn(__fmul_rn(yp[q], dv), dp));
            } else {
#pragma unroll
              for (int q = 0; q < V; ++q) yv[q] = __fadd_rn(yv[q], yp[q]);
            }
            store_f32<V>(yv_row + vi * V, yv);
          }
        }
        }
      }
      if (nodew < 0) {
        // marked final even after a failed wait, so that no wait on it hangs
        __threadfence();
        __syncwarp(tmask);
        if (tl == 0) st_release(a.node_flag + node, epoch);
      }
    }
    __syncwarp();
  }
  finish_block(a.qs, epoch);
}

// ============================================================================
// Staged variant of the forward kernel (16-byte vector path, teams of >= 8
// lanes).  The work a team claims is a run of consecutive items, and the
// stream layout stores their entries contiguously, so the team walks one flat
// entry range.  X rows are fetched with cp.async into a per-thread ring of S
// slots in shared memory, S entries ahead of the consumer, independent of row
// boundaries: S gathers stay in flight without holding registers.  Each lane
// copies and later reads only its own 16-byte pieces, so the only waits are
// the lane's own cp.async groups.  Column indices come in batches of TL (one
// coalesced load per batch), three batches in flight; the items' metadata for
// a claim is held one item per lane.  Rows are finished (chunk partials,
// parent, store, ready flag) when the consumer crosses their end.
// ============================================================================
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16_hint(void* smem, const void* gmem, uint64_t policy) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "l"(policy)
               : "memory");
}
// copies `bytes` (16 or 0) and zero-fills the rest: a copy that may be empty
// without a branch (the address must still point into the operand)
__device__ __forceinline__ void cp_async16_hint_n(void* smem, const void* gmem, unsigned bytes, uint64_t policy) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(s), "l"(gmem), "r"(bytes),
               "l"(policy)
               : "memory");
}
// the same without an L2 policy
__device__ __forceinline__ void cp_async16_n(void* smem, const void* gmem, unsigned bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- TMA (tile::gather4) and mbarrier helpers ------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// makes initialised barriers visible to the TMA unit (the async proxy)
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// orders this thread's earlier generic-proxy shared-memory accesses before
// later async-proxy (TMA) writes
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// four rows r0..r3 of a 2-D tensor (box: all columns from col0, one row high)
// into dst, one after another; completion counted on bar
__device__ __forceinline__ void tma_gather4(void* dst, const CUtensorMap* map, int col0, int r0, int r1, int r2, int r3,
                                            uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7], %8;" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(col0), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(smem_u32(bar)),
      "l"(policy)
      : "memory");
}
// Bounded wait for a barrier phase: try_wait (which itself suspends for a
// while) until the phase completes or timeout_ns pass.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, long long timeout_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (long long it = 0; it < kMaxSpins; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((long long)(global_ns() - t0) > timeout_ns) break;
  }
  return false;
}

template <typename XT, int V>
__device__ __forceinline__ void unpack16(const uint4& r, float (&o)[V]) {
  if constexpr (sizeof(XT) == 4) {
    o[0] = __uint_as_float(r.x);
    o[1] = __uint_as_float(r.y);
    o[2] = __uint_as_float(r.z);
    o[3] = __uint_as_float(r.w);
  } else {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
}

// Scale of one entry before the row factor: s, s * m[col] (both for
// SCALE_DCOL and SCALE_DCOL_DROW, whose consumer then multiplies by m[row]) or
// the stored value.
__device__ __forceinline__ float entry_scale(uint32_t e, int64_t idx, bool valid, int scale_mode, const float* mult,
                                             const float* val) {
  if (!valid) return 0.f;
  const float sgn = (e >> 31) ? -1.f : 1.f;
  if (scale_mode == SCALE_SIGN) return sgn;
  if (scale_mode == SCALE_VALUES) return __ldg(val + idx);
  return sgn * __ldg(mult + (e & kColMask));
}

// One team's pipelined pass over the `len` entries ent[k0, k0 + len).  With
// lockstep every lane of the warp calls it (a team with nothing to do passes
// len = 0).
// Positions are 32-bit and relative to k0; batches of TL entries start at
// multiples of TL.  next_end() gives the relative position where the
// current item ends (INT_MAX when none is left); on_end(acc) finishes it,
// resets acc and advances, updating row_dv (the row factor: m[row] under
// SCALE_DCOL_DROW, exactly 1 otherwise).
template <typename XT, int TL, int VPL, int V, int S, int BLOCK, bool OFF32, bool HINTS, typename NextEnd,
          typename OnEnd>
__device__ __forceinline__ void stream_pass(const XT* __restrict__ x, int64_t ldx, int nvec,
                                            const uint32_t* __restrict__ ent, const float* __restrict__ val,
                                            int64_t k0, int len, int scale_mode, const float* __restrict__ mult,
                                            uint4* __restrict__ ring, int tl, unsigned tmask, NextEnd next_end,
                                            OnEnd on_end, const float& row_dv, bool hints, bool lockstep) {
  static_assert(S <= TL && TL % S == 0, "ring depth must divide the team size");
  uint64_t pol_keep, pol_stream;
  if (hints) {
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_keep));
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_stream));
  } else {
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol_keep));
    pol_stream = pol_keep;
  }
  const uint32_t* ent0 = ent + k0;
  const float* val0 = val ? val + k0 : nullptr;
  const XT* xl = x + (int64_t)tl * V;  // this lane's first element of any row
  uint4* my = ring + threadIdx.x;      // this thread's ring: slot s, piece v at my[(s * VPL + v) * BLOCK]
  bool piece_ok[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) piece_ok[v] = tl + v * TL < nvec;

  // three batches of TL entries: A (holds the consumer position), B, C
  int bA = 0;
  uint32_t eA = 0, eB = 0, eC = 0;
  float sA = 0.f, sB = 0.f;
  {
    const int ia = tl, ib = TL + tl, ic = 2 * TL + tl;
    if (ia < len) eA = __ldcs(ent0 + ia);
    if (ib < len) eB = __ldcs(ent0 + ib);
    if (ic < len) eC = __ldcs(ent0 + ic);
    sA = entry_scale(eA, ia, ia < len, scale_mode, mult, val0);
    sB = entry_scale(eB, ib, ib < len, scale_mode, mult, val0);
  }
  // X row of entry word e from a lane's base: with OFF32 (X holds fewer than
  // 2^32 elements) a 32-bit element offset and one scaled add, else 64-bit
  auto row_at = [&](const XT* base, uint32_t e) -> const XT* {
    if constexpr (OFF32) {
      return base + (uint32_t)((e & kColMask) * (uint32_t)ldx);
    } else {
      return base + row_off(e & kColMask, ldx);
    }
  };
  // entry p's pieces into ring slot sp (no commit).  One piece per lane
  // (narrow rows): branch-free.  An entry past the stream's end (its word is
  // 0, so the address is X's first row) copies 0 bytes and zero-fills the
  // slot.  A lane without a piece (a row narrower than the team) copies the
  // first 16 bytes of the row, a valid address, into a slot whose sums no
  // store reads (every store is limited to the row's pieces); so the
  // per-entry code tests only the stream's end, with a constant size.
  // Several pieces per lane: pieces outside the row and entries past the end
  // are skipped (the slots keep old data, never read).
  const XT* xp = piece_ok[0] ? xl : x;
  auto produce = [&](int p, uint4* sp) {
    // HINTS: the entry's hot bit picks its L2 policy; without (a plan with
    // no hot set) the copies carry no policy and need no per-entry choice
    if constexpr (VPL == 1) {
      const bool inA = p < bA + TL;
      const uint32_t e = __shfl_sync(tmask, inA ? eA : eB, p & (TL - 1), TL);
      const XT* row = row_at(xp, e);
      if constexpr (HINTS) {
        const uint64_t pol = (e & kHotBit) ? pol_keep : pol_stream;
        cp_async16_hint_n(sp, row, p < len ? 16u : 0u, pol);
      } else {
        cp_async16_n(sp, row, p < len ? 16u : 0u);
      }
    } else if (p < len) {
      const bool inA = p < bA + TL;
      const uint32_t e = __shfl_sync(tmask, inA ? eA : eB, p & (TL - 1), TL);
      const XT* row = row_at(xl, e);
      const uint64_t pol = (e & kHotBit) ? pol_keep : pol_stream;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        if (piece_ok[v]) {
          if constexpr (HINTS) {
            cp_async16_hint(sp + v * BLOCK, row + v * TL * V, pol);
          } else {
            cp_async16(sp + v * BLOCK, row + v * TL * V);
          }
        }
      }
    }
  };
  // Entries move in groups of U (one cp.async group each, S / U groups in
  // flight); a group without a row end inside is consumed by straight-line
  // code (all U scales, then all U pieces, then the FMAs), one with a row end
  // (or past the stream's end) entry by entry.
  constexpr int U = S >= 8 ? 4 : 2;
  constexpr int G = S / U;
  static_assert(S % U == 0 && TL % U == 0, "groups must tile the ring and the batches");
#pragma unroll
  for (int j = 0; j < S; ++j) {
    produce(j, my + j * (VPL * BLOCK));
    if (j % U == U - 1) cp_async_commit();
  }

  float acc[VPL][V];
#pragma unroll
  for (int v = 0; v < VPL; ++v)
#pragma unroll
    for (int q = 0; q < V; ++q) acc[v][q] = 0.f;
  int end_at = next_end();
  int slot = 0;  // ring slot of entry k (a multiple of U)
  // With lockstep, all teams of the warp step together (to the warp's longest
  // stream) so that one instruction serves every team, finished teams idling.
  // Only when no team waits on a row another team of the warp produces in the
  // same pass (the caller checks): a wait would then block the producer at
  // the per-step warp barrier.
  // (a full-warp team is alone in its warp: no lockstep, every step active)
  const bool ls = TL < 32 && lockstep;
  const int wlen = ls ? __reduce_max_sync(0xffffffffu, len) : len;
  auto consume = [&](int kk, uint4* sp, bool active) {
    float sc = __fmul_rn(__shfl_sync(tmask, sA, kk & (TL - 1), TL), row_dv);
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      if (piece_ok[v] && active) {
        float t[V];
        unpack16<XT, V>(sp[v * BLOCK], t);
#pragma unroll
        for (int q = 0; q < V; ++q) acc[v][q] = fmaf(sc, t[q], acc[v][q]);
      }
    }
  };
  for (int k = 0; k < wlen; k += U) {
    if (k == bA + TL) {
      // rotate: A <- B (scales ready), B <- C (scales now), load a new C
      bA += TL;
      eA = eB;
      sA = sB;
      eB = eC;
      const int ib = bA + TL + tl, ic = bA + 2 * TL + tl;
      sB = entry_scale(eB, ib, ib < len, scale_mode, mult, val0);
      eC = ic < len ? __ldcs(ent0 + ic) : 0u;
    }
    cp_async_wait<G - 1>();
    uint4* sp = my + slot * (VPL * BLOCK);
    if (k + U <= len && end_at >= k + U) {
      // row_dv is m[row] under SCALE_DCOL_DROW and exactly 1 otherwise
      if constexpr (VPL == 1) {
        // all U scales, then all U pieces, then the FMAs (lanes outside the
        // row add their placeholder pieces to accumulators no store reads)
        float sc[U];
        uint4 raw[U];
#pragma unroll
        for (int u = 0; u < U; ++u) sc[u] = __fmul_rn(__shfl_sync(tmask, sA, (k + u) & (TL - 1), TL), row_dv);
#pragma unroll
        for (int u = 0; u < U; ++u) raw[u] = sp[u * BLOCK];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float t[V];
          unpack16<XT, V>(raw[u], t);
#pragma unroll
          for (int q = 0; q < V; ++q) acc[0][q] = fmaf(sc[u], t[q], acc[0][q]);
        }
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u) consume(k + u, sp + u * (VPL * BLOCK), true);
      }
    } else {
      for (int u = 0; u < U; ++u) {
        const int kk = k + u;
        const bool active = kk < len;
        if (active) {
          while (kk == end_at) {
            on_end(acc);
            end_at = next_end();
          }
        }
        consume(kk, sp + u * (VPL * BLOCK), active);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) produce(k + S + u, sp + u * (VPL * BLOCK));
    cp_async_commit();
    slot = (slot + U == S) ? 0 : slot + U;
    if (ls) __syncwarp();
  }
  cp_async_wait<0>();
  while (end_at <= len) {
    on_end(acc);
    end_at = next_end();
  }
  if (ls) __syncwarp();
}

// TMA variant of stream_pass: the team's rows come in groups of four by one
// tile::gather4 copy (issued by the team's first lane) into the team's ring of
// G slots of four rows, completion counted on one mbarrier per slot.
// Every lane owns every piece of a row here (nvec == TL * VPL, rows of 16-byte
// multiples, 128-byte multiples per row), so a lane reads pieces tl + v * TL of
// each gathered row.  The summation order is stream_pass's (sequential FMAs
// per row).  A wait that runs out records CBM_ERR_TIMEOUT and stops further
// copies; the copies already issued are waited for (bounded) before return.
template <typename XT, int TL, int VPL, int V, int G, typename NextEnd, typename OnEnd>
__device__ __forceinline__ void stream_pass_tma(const CUtensorMap* tmap, int rb, const uint32_t* __restrict__ ent,
                                                const float* __restrict__ val, int64_t k0, int len, int scale_mode,
                                                const float* __restrict__ mult, uint8_t* tring, uint64_t* tbar,
                                                unsigned& phase, int tl, unsigned tmask, NextEnd next_end,
                                                OnEnd on_end, const float& row_dv, bool hints, bool lockstep,
                                                QueueState* qs, long long timeout_ns) {
  static_assert(G >= 2 && (G & (G - 1)) == 0 && 4 * G <= TL, "G slots of four rows, 4G entries within two batches");
  uint64_t pol_keep, pol_stream;
  if (hints) {
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_keep));
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_stream));
  } else {
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol_keep));
    pol_stream = pol_keep;
  }
  const uint32_t* ent0 = ent + k0;
  const float* val0 = val ? val + k0 : nullptr;
  // a failure earlier in this launch: no more copies (the results are void)
  bool broken = *(volatile int*)&qs->error != 0;

  int bA = 0;
  uint32_t eA = 0, eB = 0, eC = 0;
  float sA = 0.f, sB = 0.f;
  {
    const int ia = tl, ib = TL + tl, ic = 2 * TL + tl;
    if (ia < len) eA = __ldcs(ent0 + ia);
    if (ib < len) eB = __ldcs(ent0 + ib);
    if (ic < len) eC = __ldcs(ent0 + ic);
    sA = entry_scale(eA, ia, ia < len, scale_mode, mult, val0);
    sB = entry_scale(eB, ib, ib < len, scale_mode, mult, val0);
  }
  int issued = 0;  // groups issued so far (group g: entries 4g .. 4g + 3)
  // entries of group g lie in batches A and B: the consumer is at 4g - 4G or
  // later, and 4G <= TL
  auto issue = [&](int g) {
    const int p0 = 4 * g;
    if (p0 >= len || broken) return;
    uint32_t e4[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = p0 + u < len ? p0 + u : len - 1;  // padding repeats the last row
      e4[u] = __shfl_sync(tmask, p < bA + TL ? eA : eB, p & (TL - 1), TL);
    }
    if (tl == 0) {
      const int sl = g & (G - 1);
      const uint64_t pol = ((e4[0] | e4[1] | e4[2] | e4[3]) & kHotBit) ? pol_keep : pol_stream;
      fence_proxy_async();
      mbar_expect_tx(tbar + sl, 4u * (unsigned)rb);
      tma_gather4(tring + (size_t)sl * 4 * rb, tmap, 0, (int)(e4[0] & kColMask), (int)(e4[1] & kColMask),
                  (int)(e4[2] & kColMask), (int)(e4[3] & kColMask), tbar + sl, pol);
    }
    issued = g + 1;
  };
#pragma unroll
  for (int g = 0; g < G; ++g) issue(g);

  float acc[VPL][V];
#pragma unroll
  for (int v = 0; v < VPL; ++v)
#pragma unroll
    for (int q = 0; q < V; ++q) acc[v][q] = 0.f;
  int end_at = next_end();
  const bool ls = TL < 32 && lockstep;
  const int wlen = ls ? __reduce_max_sync(0xffffffffu, len) : len;
  int waited = 0;  // groups waited for
  auto consume = [&](int kk, const uint8_t* rowp, bool active) {
    const float sc = __fmul_rn(__shfl_sync(tmask, sA, kk & (TL - 1), TL), row_dv);
    if (active) {
      const uint4* pr = reinterpret_cast<const uint4*>(rowp) + tl;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        float t[V];
        unpack16<XT, V>(pr[v * TL], t);
#pragma unroll
        for (int q = 0; q < V; ++q) acc[v][q] = fmaf(sc, t[q], acc[v][q]);
      }
    }
  };
  for (int k = 0; k < wlen; k += 4) {
    if (k == bA + TL) {
      bA += TL;
      eA = eB;
      sA = sB;
      eB = eC;
      const int ib = bA + TL + tl, ic = bA + 2 * TL + tl;
      sB = entry_scale(eB, ib, ib < len, scale_mode, mult, val0);
      eC = ic < len ? __ldcs(ent0 + ic) : 0u;
    }
    const int g = k >> 2;
    const int sl = g & (G - 1);
    if (k < len && g < issued) {
      if (mbar_wait_bounded(tbar + sl, (phase >> sl) & 1u, timeout_ns)) {
        phase ^= 1u << sl;
      } else if (!broken) {
        broken = true;
        if (tl == 0 && atomicCAS(&qs->error, 0, 8 /* CBM_ERR_TIMEOUT */) == 0) qs->error_info = -1 - (long long)g;
      }
      waited = g + 1;
    }
    const uint8_t* slot = tring + (size_t)sl * 4 * rb;
    if (k + 4 <= len && end_at >= k + 4) {
      float sc[4];
      uint4 raw[4][VPL];
#pragma unroll
      for (int u = 0; u < 4; ++u) sc[u] = __fmul_rn(__shfl_sync(tmask, sA, (k + u) & (TL - 1), TL), row_dv);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < VPL; ++v) raw[u][v] = reinterpret_cast<const uint4*>(slot + u * rb)[tl + v * TL];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          float t[V];
          unpack16<XT, V>(raw[u][v], t);
#pragma unroll
          for (int q = 0; q < V; ++q) acc[v][q] = fmaf(sc[u], t[q], acc[v][q]);
        }
    } else {
      for (int u = 0; u < 4; ++u) {
        const int kk = k + u;
        const bool active = kk < len;
        if (active) {
          while (kk == end_at) {
            on_end(acc);
            end_at = next_end();
          }
        }
        consume(kk, slot + u * rb, active);
      }
    }
    // every lane of the team is done with the slot before it is refilled
    __syncwarp(tmask);
    issue(g + G);
    if (ls) __syncwarp();
  }
  // after a failure: wait (bounded) for the copies still in flight
  for (int g = waited; g < issued; ++g) {
    const int sl = g & (G - 1);
    if (mbar_wait_bounded(tbar + sl, (phase >> sl) & 1u, timeout_ns)) phase ^= 1u << sl;
  }
  while (end_at <= len) {
    on_end(acc);
    end_at = next_end();
  }
  if (ls) __syncwarp();
}

// TMA = true: rows arrive by tile::gather4 copies into per-team rings (the
// dynamic shared memory then holds BLOCK / TL teams x S / 4 slots of four
// rows of tma_rb bytes, followed by one mbarrier per slot: S entries in flight
// per team, as in the cp.async ring); `tmap` describes
// X (columns [0, nvec * V), every row, one-row box).  TMA = false: the
// per-thread cp.async ring of stream_pass (tmap unused).
template <typename XT, typename YT, int TL, int VPL, int V, int S, int BLOCK, bool TMA = false, bool OFF32 = false,
          bool HINTS = true>
__global__ void __launch_bounds__(BLOCK) fwd_stream_kernel(const FwdArgs a, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(128) uint4 ring[];
  const int lane = threadIdx.x & 31;
  const int team = lane / TL;
  const int tl = lane & (TL - 1);
  constexpr int teams = 32 / TL;
  const unsigned tmask = (TL == 32) ? 0xffffffffu : (((1u << TL) - 1u) << (team * TL));
  const unsigned epoch = *(volatile unsigned*)&a.qs->epoch + 1u;
  const XT* x = static_cast<const XT*>(a.x);
  const bool hints = a.hints != 0;
  float ch_dv = 1.f;
  // TMA rings and barriers of this thread's team
  uint8_t* tring = nullptr;
  uint64_t* tbar = nullptr;
  unsigned tphase = 0;
  constexpr int G = S / 4;
  if constexpr (TMA) {
    constexpr int n_teams = BLOCK / TL;
    const int bt = threadIdx.x / TL;
    uint8_t* base = reinterpret_cast<uint8_t*>(ring);
    tring = base + (size_t)bt * G * 4 * a.tma_rb;
    tbar = reinterpret_cast<uint64_t*>(base + (size_t)n_teams * G * 4 * a.tma_rb) + bt * G;
    if (tl == 0) {
#pragma unroll
      for (int g = 0; g < G; ++g) mbar_init(tbar + g, 1);
      mbar_init_fence();
    }
    __syncwarp(tmask);
  }

  // ---- chunks of long rows: one chunk per team per claim ----
  if (a.n_chunks > 0) {
    for (;;) {
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(&a.qs->next_chunk, (unsigned)teams);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= (unsigned)a.n_chunks) break;
      const unsigned k = base + team;
      const bool have = k < (unsigned)a.n_chunks;
      int64_t cb = 0;
      int clen = 0;
      if (have) {
        const int item = a.chunk_item[k];
        const int node = a.node[item] & 0x7fffffff;
        ch_dv = (a.scale_mode == SCALE_DCOL_DROW) ? __ldg(a.mult + node) : 1.f;
        cb = a.chunk_beg[k];
        clen = (int)(a.chunk_end[k] - cb);
      }
      bool done = !have;
      auto next_end = [&]() -> int { return done ? INT_MAX : clen; };
      auto on_end = [&](float (&acc)[VPL][V]) {
        float* prow = a.partial + (int64_t)k * a.ldp;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) store_f32<V>(prow + vi * V, acc[v]);
        }
        __threadfence();
        __syncwarp(tmask);
        if (tl == 0) st_release(a.chunk_flag + k, epoch);
        done = true;
      };
      // chunks depend on nothing: always in lockstep
      if constexpr (TMA) {
        stream_pass_tma<XT, TL, VPL, V, G>(&tmap, a.tma_rb, a.cent, a.cval, cb, clen, a.scale_mode, a.mult, tring, tbar,
                                        tphase, tl, tmask, next_end, on_end, ch_dv, hints, true, a.qs, a.timeout_ns);
      } else {
        stream_pass<XT, TL, VPL, V, S, BLOCK, OFF32, HINTS>(x, a.ldx, a.nvec, a.cent, a.cval, cb, clen, a.scale_mode, a.mult,
                                              ring, tl, tmask, next_end, on_end, ch_dv, hints, true);
      }
    }
  }

  // ---- rows: a team takes R consecutive items per claim: rows_per_claim while
  // the queue is in level 0, rows_per_claim_deep below it (sized by where the
  // warp's last claim fell)
  const bool need_dv = (a.scale_mode == SCALE_DCOL_DROW) || (a.prop_mode == PROP_RATIO);
  const int64_t hi = a.n_items;
  unsigned last = 0;
  for (;;) {
    // this team's items [i0, i1); base: the first item of the warp's claim
    int64_t i0, i1;
    unsigned base;
    // units pay off where teams share a warp (they step together); a full-warp
    // team keeps the plain claims (one dependent load fewer per claim)
    if (TL < 32 && a.unit) {
      unsigned claimed = 0;
      if (lane == 0) claimed = atomicAdd(&a.qs->next_row, (unsigned)teams);
      const unsigned ub = __shfl_sync(0xffffffffu, claimed, 0);
      if (ub >= (unsigned)a.n_units) break;
      const unsigned u = ub + team;
      base = (unsigned)a.unit[ub];
      i0 = u < (unsigned)a.n_units ? a.unit[u] : hi;
      i1 = u < (unsigned)a.n_units ? a.unit[u + 1] : hi;
    } else {
      const int Rp = last < (unsigned)a.n_root ? a.rows_per_claim : a.rows_per_claim_deep;
      const int R = Rp < TL ? Rp : TL;
      unsigned claimed = 0;
      if (lane == 0) claimed = atomicAdd(&a.qs->next_row, (unsigned)(teams * R));
      base = __shfl_sync(0xffffffffu, claimed, 0);
      if ((int64_t)base >= hi) break;
      last = base;
      i0 = (int64_t)base + (int64_t)team * R;
      i1 = (i0 + R < hi) ? i0 + R : hi;
    }
    {
      const int nit = i0 < hi ? (int)(i1 - i0) : 0;
      const int64_t k0 = nit > 0 ? a.ptr[i0] : 0;
      // item metadata, one item per lane; ends relative to k0
      int m_node = 0, m_par = -1, m_chunk = -1, m_pslot = -1, m_sslot = -1, m_end = 0;
      float m_dv = 1.f;
      bool dep_in_claim = false;
      if (tl < nit) {
        const int64_t it = i0 + tl;
        m_node = a.node[it];
        m_par = a.skip_parent ? -1 : a.par[it];
        dep_in_claim = m_par >= 0 && a.par_item[it] >= (int)base;
        m_chunk = a.chunk0[it];
        m_pslot = a.par_slot[it];
        m_sslot = a.self_slot[it];
        m_end = (int)(a.ptr[it + 1] - k0);
        if (need_dv) m_dv = __ldg(a.mult + (m_node & 0x7fffffff));
      }
      const int len = nit > 0 ? __shfl_sync(tmask, m_end, nit - 1, TL) : 0;
      int cur = 0;  // item (relative) the consumer is in
      const bool drow = a.scale_mode == SCALE_DCOL_DROW;
      float row_dv = drow ? __shfl_sync(tmask, m_dv, 0, TL) : 1.f;
      auto next_end = [&]() -> int { return cur < nit ? __shfl_sync(tmask, m_end, cur, TL) : INT_MAX; };
      // Parent rows are fetched ahead: the parent's ready flag of item i+1 is
      // acquired when item i starts, and if it was set, item i+1's parent row is
      // loaded into registers when item i+1 starts; the row end then finds it
      // there.  A flag not yet set falls back to the bounded wait at the end.
      bool pf_ok = false;
      float pbuf[VPL][V];
      // claims without any parent skip this bookkeeping
      const bool any_parent = __any_sync(tmask, tl < nit && m_par >= 0);
      auto acquire_for = [&](int it) -> unsigned {
        if (!any_parent || it >= nit) return 0u;
        const int p = __shfl_sync(tmask, m_par, it, TL);
        return p >= 0 ? ld_acquire(a.node_flag + p) : 0u;
      };
      auto prefetch = [&](int it, unsigned fval) {
        pf_ok = false;
        if (!any_parent || it >= nit) return;
        const int p = __shfl_sync(tmask, m_par, it, TL);
        const int ps = __shfl_sync(tmask, m_pslot, it, TL);
        if (p < 0 || fval != epoch) return;
        pf_ok = true;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) {
            if constexpr (sizeof(YT) == 4) {
              load_y_cg<YT, V>(static_cast<const YT*>(a.y) + (int64_t)p * a.ldy + (int64_t)vi * V, pbuf[v]);
            } else {
              load_f32_cg<V>(a.pstate + (int64_t)ps * a.ldp + vi * V, pbuf[v]);
            }
          }
        }
      };
      unsigned flag_next;
      {
        const unsigned f0 = acquire_for(0);
        flag_next = acquire_for(1);
        prefetch(0, f0);
      }
      auto on_end = [&](float (&acc)[VPL][V]) {
        const int nodew = __shfl_sync(tmask, m_node, cur, TL);
        const int node = nodew & 0x7fffffff;
        const int c0 = __shfl_sync(tmask, m_chunk, cur, TL);
        const int p = __shfl_sync(tmask, m_par, cur, TL);
        const int ps = __shfl_sync(tmask, m_pslot, cur, TL);
        const int ss = __shfl_sync(tmask, m_sslot, cur, TL);
        const float dv = __shfl_sync(tmask, m_dv, cur, TL);
        if (c0 >= 0) {
          const int item = (int)(i0 + cur);
          for (int k = c0; k < a.n_chunks && a.chunk_item[k] == item; ++k) {
            if (!wait_flag(a.chunk_flag + k, epoch, a.qs, a.timeout_ns, (long long)k)) continue;
            const float* prow = a.partial + (int64_t)k * a.ldp;
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
              const int vi = tl + v * TL;
              if (vi < a.nvec) {
                float t[V];
                load_f32_cg<V>(prow + vi * V, t);
#pragma unroll
                for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], t[q]);
              }
            }
          }
        }
        if (p >= 0 && (pf_ok || wait_flag(a.node_flag + p, epoch, a.qs, a.timeout_ns, (long long)node))) {
          const float dp = (a.prop_mode == PROP_RATIO) ? __ldg(a.mult + p) : 1.f;
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            const int vi = tl + v * TL;
            if (vi < a.nvec) {
              float yp[V];
              if (pf_ok) {
#pragma unroll
                for (int q = 0; q < V; ++q) yp[q] = pbuf[v][q];
              } else if constexpr (sizeof(YT) == 4) {
                load_y_cg<YT, V>(static_cast<const YT*>(a.y) + (int64_t)p * a.ldy + (int64_t)vi * V, yp);
              } else {
                load_f32_cg<V>(a.pstate + (int64_t)ps * a.ldp + vi * V, yp);
              }
              if (a.prop_mode == PROP_RATIO) {
#pragma unroll
                for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], __fdiv_rn(__fmul_rn(yp[q], dv), dp));
              } else {
#pragma unroll
                for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], yp[q]);
              }
            }
          }
        }
        YT* yrow = static_cast<YT*>(a.y) + (int64_t)node * a.ldy;
        // leaves are not read again by this kernel: stream them past L2 (not
        // in a first pass, whose rows the second pass reads back)
        const bool stream_y = hints && nodew >= 0 && !a.skip_parent;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) {
            if (stream_y)
              store_vec_cs<YT, V>(yrow + (int64_t)vi * V, acc[v]);
            else
              store_vec<YT, V>(yrow + (int64_t)vi * V, acc[v]);
          }
        }
        if (nodew < 0 && !a.skip_parent) {
          if constexpr (sizeof(YT) != 4) {
            float* srow = a.pstate + (int64_t)ss * a.ldp;
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
              const int vi = tl + v * TL;
              if (vi < a.nvec) store_f32<V>(srow + vi * V, acc[v]);
            }
          }
          __threadfence();
          __syncwarp(tmask);
          if (tl == 0) st_release(a.node_flag + node, epoch);
        }
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
          for (int q = 0; q < V; ++q) acc[v][q] = 0.f;
        ++cur;
        const float next_dv = __shfl_sync(tmask, m_dv, cur < nit ? cur : 0, TL);
        row_dv = drow ? next_dv : 1.f;
        const unsigned f_cur = flag_next;
        flag_next = acquire_for(cur + 1);
        prefetch(cur, f_cur);
      };
      // a parent row inside this warp's claim: let the teams run independently
      const bool lockstep = !__any_sync(0xffffffffu, dep_in_claim);
      if constexpr (TMA) {
        stream_pass_tma<XT, TL, VPL, V, G>(&tmap, a.tma_rb, a.ent, a.val, k0, len, a.scale_mode, a.mult, tring, tbar,
                                        tphase, tl, tmask, next_end, on_end, row_dv, hints, lockstep, a.qs,
                                        a.timeout_ns);
      } else {
        stream_pass<XT, TL, VPL, V, S, BLOCK, OFF32, HINTS>(x, a.ldx, a.nvec, a.ent, a.val, k0, len, a.scale_mode, a.mult, ring,
                                              tl, tmask, next_end, on_end, row_dv, hints, lockstep);
      }
    }
  }
  finish_block(a.qs, epoch, a.publish_epoch != 0);
}

// ============================================================================
// Adjoint: dX = Delta^T P^T G' with P the tree-prefix operator (A = P Delta).
//   reverse pass   H[w] = G'[w] + sum over children c of H[c]   (deepest first)
//   transposed     dX[j] = m[j]^(ADX/DADX) * sum over (v, j, s) of s * H[v]
// with G' = m o G for DADX.  Leaves are not materialised: their H is G'.
// ============================================================================
constexpr uint32_t kInternalBit = 0x40000000u;
constexpr uint32_t kIndexMask = 0x3fffffffu;

struct RevArgs {
  // items, deepest level first: for each internal node its chunk items (long
  // children lists), then the node item
  int32_t n_items;
  const int4* meta;      // x = node, -1 for a chunk item; y = internal slot or chunk id;
                         // z = first child and w = children, or first chunk and minus the chunks
  const uint32_t* ent;   // child | internal bit (slot then)
  const float* mult;
  int32_t scale_g;       // G' = m o G
  unsigned int* flag;    // [n_internal]
  unsigned int* chunk_flag;  // [chunks]
  unsigned int* claims;  // kClaimQueues counters
  float* partial;        // [chunks, ldp]
  QueueState* qs;
  const void* g;
  int64_t ldg;
  float* h;              // [n_internal, ldp]
  int32_t ldp;
  int32_t nvec;
  int32_t team;
  long long timeout_ns;
};

// Entries above which a list is split over all teams of a warp.  Measured above 32, 64
// and 0 (the chunks then in a phase of their own), 40 FP32 columns: 10,000-node GCN
// graph 85 us each, 170,000 nodes 169, 168 and 199.
constexpr int kSoloLen = 64;

struct TrArgs {
  int32_t n_items;       // chunks of long lists, then the columns of Delta
  int32_t n_solo;        // of these, the first ones: a warp takes each alone
  const int4* meta;      // per item, columns longest lists first: x = column, z = first
                         // entry and w = entries, or first chunk and minus the chunks;
                         // a chunk's x is ~its number
  const uint32_t* ent;   // row | internal bit (slot then) | sign << 31
  unsigned int* chunk_flag;
  unsigned int* claims;  // kClaimQueues counters
  const float* mult;
  int32_t scale_g;       // leaves read m[v] * G[v]
  int32_t scale_out;     // dX[j] *= m[j]
  QueueState* qs;
  const void* g;
  int64_t ldg;
  const float* h;
  int32_t ldp;
  void* dx;
  int64_t lddx;
  int32_t nvec;
  float* partial;
  int32_t team;
  long long timeout_ns;
};

// acc += sum over the `len` children in ent of (internal ? H[slot] : scale * G[row]),
// each internal child's ready flag awaited first.  e: the lane's child of the
// first TL; later batches of TL load one batch ahead.
template <typename GT, int VPL, int V>
__device__ __forceinline__ void gather_children(float (&acc)[VPL][V], const RevArgs& a, const GT* __restrict__ g,
                                                const uint32_t* __restrict__ ent, int len, uint32_t e, unsigned epoch,
                                                int tl, int TL, unsigned tmask) {
  constexpr int U = unroll_for<VPL, V>();
  for (int base = 0; base < len; base += TL) {
    const int at = base + TL + tl;
    const uint32_t en = at < len ? __ldg(ent + at) : 0u;
    const int cnt = len - base < TL ? len - base : TL;
    float sc = 0.f;
    if (tl < cnt) {
      const uint32_t r = e & kIndexMask;
      if (e & kInternalBit) {
        sc = 1.f;
        // each lane acquires the flag of its own entry; the team barrier below
        // orders every lane's later reads of those rows after these acquires
        wait_flag(a.flag + r, epoch, a.qs, a.timeout_ns, (long long)r);
      } else {
        sc = a.scale_g ? __ldg(a.mult + r) : 1.f;
      }
    }
    __syncwarp(tmask);
    for (int j = 0; j < cnt; j += U) {
      float buf[U][VPL][V];
      float s[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int src = j + u < cnt ? j + u : 0;
        const uint32_t eu = __shfl_sync(tmask, e, src, TL);
        s[u] = __shfl_sync(tmask, sc, src, TL);
        const uint32_t r = eu & kIndexMask;
        const bool in = (eu & kInternalBit) != 0;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (j + u < cnt && vi < a.nvec) {
            if (in) {
              load_f32_cg<V>(a.h + row_off(r, a.ldp) + vi * V, buf[u][v]);
            } else {
              Vec<GT, V>::load(g + row_off(r, a.ldg) + (int64_t)vi * V, buf[u][v]);
            }
          } else {
#pragma unroll
            for (int k = 0; k < V; ++k) buf[u][v][k] = 0.f;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j + u < cnt) {
#pragma unroll
          for (int v = 0; v < VPL; ++v)
#pragma unroll
            for (int k = 0; k < V; ++k) acc[v][k] = fmaf(s[u], buf[u][v][k], acc[v][k]);
        }
      }
    }
    e = en;
  }
}

template <typename GT, int VPL, int V>
__global__ void __launch_bounds__(kThreads) rev_kernel(const RevArgs a) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int TL = a.team;
  const int team = lane / TL;
  const int tl = lane & (TL - 1);
  const unsigned teams = 32 / TL;
  const unsigned tmask = (TL == 32) ? kAll : (((1u << TL) - 1u) << (team * TL));
  const unsigned epoch = *(volatile unsigned*)&a.qs->epoch + 1u;
  const GT* g = static_cast<const GT*>(a.g);
  const unsigned n = (unsigned)a.n_items;
  const unsigned wq = threadIdx.x >> 5;
  for (;;) {
    // one item per team and claim, and nothing claimed ahead: an item waits on
    // children claimed just before it, and one held back behind another item of
    // its warp holds up its parents (with a claim and a record made ahead, as in
    // the forward kernel, 80 -> 94-112 us on the GCN graph)
    unsigned g0 = 0;
    if (lane == 0) g0 = atomicAdd(a.claims + wq * kClaimStride, 1u);
    g0 = (__shfl_sync(kAll, g0, 0) * kClaimQueues + wq) * teams;
    if (g0 >= n) break;
    const int4 m0 = __ldg(a.meta + g0 + team);
    const uint32_t e0 = tl < m0.w ? __ldg(a.ent + (uint32_t)m0.z + tl) : 0u;
    if (g0 + team < n) {
      const int w = m0.x;
      float acc[VPL][V];
#pragma unroll
      for (int v = 0; v < VPL; ++v)
#pragma unroll
        for (int q = 0; q < V; ++q) acc[v][q] = 0.f;
      if (w >= 0) {
        // node item: its own G' row
        const float sw = a.scale_g ? __ldg(a.mult + w) : 1.f;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) {
            float t[V];
            Vec<GT, V>::load(g + row_off(w, a.ldg) + (int64_t)vi * V, t);
#pragma unroll
            for (int q = 0; q < V; ++q) acc[v][q] = __fmul_rn(sw, t[q]);
          }
        }
        // partial sums of its chunks, in order
        for (int k = m0.z, ke = m0.z - m0.w; k < ke && m0.w < 0; ++k) {
          if (!wait_flag(a.chunk_flag + k, epoch, a.qs, a.timeout_ns, (long long)k)) continue;
          const float* prow = a.partial + (int64_t)k * a.ldp;
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            const int vi = tl + v * TL;
            if (vi < a.nvec) {
              float t[V];
              load_f32_cg<V>(prow + vi * V, t);
#pragma unroll
              for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], t[q]);
            }
          }
        }
      }
      gather_children<GT, VPL, V>(acc, a, g, a.ent + (uint32_t)m0.z, m0.w, e0, epoch, tl, TL, tmask);
      float* orow = (w >= 0 ? a.h : a.partial) + (int64_t)m0.y * a.ldp;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = tl + v * TL;
        if (vi < a.nvec) store_f32<V>(orow + vi * V, acc[v]);
      }
      // the barrier orders the team's stores before its first lane's release,
      // which carries them (cumulativity)
      __syncwarp(tmask);
      if (tl == 0) st_release((w >= 0 ? a.flag : a.chunk_flag) + m0.y, epoch);
    }
    __syncwarp();
  }
  finish_block(a.qs, epoch, true, a.claims);
}

// V elements of a row of G (type GT) or of H (FP32) as loaded.  BF16 rows come in
// vectors of four elements here, as H's do, so that a vector of either takes the
// same registers (170,000 nodes, 128 columns: 361 us with vectors of eight,
// 279 with four).
template <typename GT, int V>
struct Dual;
template <int V>
struct Dual<float, V> {
  using type = typename Raw<float, V>::type;
  static constexpr int regs = Raw<float, V>::regs;
  static __device__ __forceinline__ type load(const char* g, const char* h, bool in) {
    return Raw<float, V>::load(reinterpret_cast<const float*>(in ? h : g));
  }
  static __device__ __forceinline__ void widen(const type& r, bool, float (&o)[V]) { Raw<float, V>::widen(r, o); }
};
template <>
struct Dual<__nv_bfloat16, 4> {
  using type = uint4;
  static constexpr int regs = 4;
  static __device__ __forceinline__ type load(const char* g, const char* h, bool in) {
    if (in) return __ldg(reinterpret_cast<const uint4*>(h));
    const uint2 t = __ldg(reinterpret_cast<const uint2*>(g));
    return make_uint4(t.x, t.y, 0u, 0u);
  }
  static __device__ __forceinline__ void widen(const type& r, bool in, float (&o)[4]) {
    o[0] = __uint_as_float(in ? r.x : r.x << 16);
    o[1] = __uint_as_float(in ? r.y : r.x & 0xffff0000u);
    o[2] = __uint_as_float(in ? r.z : r.y << 16);
    o[3] = __uint_as_float(in ? r.w : r.y & 0xffff0000u);
  }
};
template <>
struct Dual<__nv_bfloat16, 1> {
  using type = uint32_t;
  static constexpr int regs = 1;
  static __device__ __forceinline__ type load(const char* g, const char* h, bool in) {
    return in ? __ldg(reinterpret_cast<const uint32_t*>(h))
              : (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(g)) << 16;
  }
  static __device__ __forceinline__ void widen(const type& r, bool, float (&o)[1]) { o[0] = __uint_as_float(r); }
};

// Gathers in flight per lane: 16 registers' worth, at most 8 (170,000-node GCN
// graph, 40 FP32 columns, the whole adjoint: 160 us, 177 with 32 registers).
template <typename GT, int VPL, int V>
__host__ __device__ constexpr int dual_in_flight() {
  const int u = 16 / (VPL * Dual<GT, V>::regs);
  return u < 1 ? 1 : (u > 8 ? 8 : u);
}

// Scale of one transposed entry: the sign, times m[row] for a leaf of a scaled G.
__device__ __forceinline__ float dual_scale(uint32_t e, bool scale_g, const float* __restrict__ mult) {
  const float sgn = (e >> 31) ? -1.f : 1.f;
  return (!scale_g || (e & kInternalBit)) ? sgn : sgn * __ldg(mult + (e & kIndexMask));
}

// sums += sum of s * (internal ? H[slot] : G[row]) over `len` entries, dealt over
// the S sums in turn: gather_row (above) with a row source per entry.
template <typename GT, int VPL, int V, int TLC, int S, typename Between>
__device__ __forceinline__ void gather_dual_row(float (&acc)[S][VPL][V], const Lane<GT, VPL, V, true>& lg,
                                                const Lane<float, VPL, V, false>& lh,
                                                const uint32_t* __restrict__ ent, int len, int wlen, uint32_t e,
                                                float s, bool scale_g, const float* __restrict__ mult, int tl,
                                                int team_lanes, Between between) {
  constexpr int U = dual_in_flight<GT, VPL, V>();
  static_assert(S == 1 || U % S == 0, "a group's entries are dealt over the sums");
  using D = Dual<GT, V>;
  const int TL = TLC == 32 ? 32 : team_lanes;
  if (wlen <= 0) {
    between();
    return;
  }
  if constexpr (TLC == kTeamNarrow) {
    uint32_t eg[U];
    auto fetch = [&](int j) {
#pragma unroll
      for (int u = 0; u < U; ++u) eg[u] = j + u < len ? __ldg(ent + j + u) : 0u;
    };
    fetch(0);
#pragma unroll 1
    for (int j = 0; j < wlen; j += U) {
      typename D::type raw[U][VPL];
      float sc[U];
      bool in[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t r = eg[u] & kIndexMask;
        in[u] = (eg[u] & kInternalBit) != 0;
        if (j + u < len) {
          const char* g = lg.row(r);
          const char* h = lh.row(r);
#pragma unroll
          for (int v = 0; v < VPL; ++v) raw[u][v] = D::load(g + lg.off[v], h + lh.off[v], in[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) sc[u] = j + u < len ? dual_scale(eg[u], scale_g, mult) : 0.f;
      if (j == 0) between();
      if (j + U < wlen) fetch(j + U);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j + u < len) {
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            float t[V];
            D::widen(raw[u][v], in[u], t);
#pragma unroll
            for (int k = 0; k < V; ++k) acc[u % S][v][k] = fmaf(sc[u], t[k], acc[u % S][v][k]);
          }
        }
      }
    }
  } else {
    for (int b = 0; b < wlen; b += TL) {
      const int at = b + TL + tl;
      const uint32_t en = at < len ? __ldg(ent + at) : 0u;
      const int cnt = len - b < TL ? len - b : TL;
      const int wc = wlen - b < TL ? wlen - b : TL;
#pragma unroll 1
      for (int j = 0; j < wc; j += U) {
        typename D::type raw[U][VPL];
        uint32_t eu[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          eu[u] = __shfl_sync(0xffffffffu, e, j + u, TL);
          const uint32_t r = eu[u] & kIndexMask;
          const bool in = (eu[u] & kInternalBit) != 0;
          if (j + u < cnt) {
            const char* g = lg.row(r);
            const char* h = lh.row(r);
#pragma unroll
            for (int v = 0; v < VPL; ++v) raw[u][v] = D::load(g + lg.off[v], h + lh.off[v], in);
          }
        }
        if (b + j == 0) between();
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float su = __shfl_sync(0xffffffffu, s, j + u, TL);
          if (j + u < cnt) {
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
              float t[V];
              D::widen(raw[u][v], (eu[u] & kInternalBit) != 0, t);
#pragma unroll
              for (int k = 0; k < V; ++k) acc[u % S][v][k] = fmaf(su, t[k], acc[u % S][v][k]);
            }
          }
        }
      }
      e = en;
      s = at < len ? dual_scale(en, scale_g, mult) : 0.f;
    }
  }
}

// Sums a team keeps of its share of a list, the entries dealt over them in turn.
// Four chains of a quarter of the length where teams share a warp: a list is then
// split at least as finely as over every team of a warp (170,000-node GCN graph,
// 40 FP32 columns, error against 64 bits: 8.1e-8 over the warp's two teams, 8.8e-8 by
// one team in one chain, 7.6e-8 by one team in four).
template <int TLC>
__host__ __device__ constexpr int dual_sums() {
  return TLC == 32 ? 1 : 4;
}
template <int VPL, int V, int S>
__device__ __forceinline__ void add_sums(float (&acc)[VPL][V], const float (&sums)[S][VPL][V]) {
#pragma unroll
  for (int v = 0; v < VPL; ++v)
#pragma unroll
    for (int q = 0; q < V; ++q) {
      if constexpr (S == 4)
        acc[v][q] = __fadd_rn(__fadd_rn(sums[0][v][q], sums[1][v][q]), __fadd_rn(sums[2][v][q], sums[3][v][q]));
      else
        acc[v][q] = sums[0][v][q];
    }
}

// The transposed gather, a pipeline like the register forward kernel's: lists
// of like length share a warp (the items are in length order), the next list's
// record, entries and claim load under the current one's gathers, and the rows
// are handed out from eight counters.  A list of more than kSoloLen entries, and a
// chunk of one that is split, has a warp to itself, in equal runs over its teams
// whose sums are added by shuffles (no order is kept here, the adjoint is held
// to FP64).  The others run up to four to a warp, on their share of its teams.
//
// The chunks are the queue's first items.  A phase of their own ahead of the
// lists had some SMs work through several while the longest lists, claimed two
// ahead, waited behind them (10,000 nodes of mean degree 20, 128 FP32 columns: 67 us
// with the phase, 52 as items; 10,000-node GCN graph, 40 columns 95 -> 68; 50,000 nodes
// 113 -> 91).  Progress: every counter hands its chunks out before its lists, and
// only lists wait.
//
// Bound by the chain of gathers of the longest lists on small graphs, by
// instruction issue on large ones.  Measured on B200, the whole adjoint, a column
// per team or warp with every load in turn -> as here (us): GCN graph of
// 170,000 nodes, 40 FP32 columns 222 -> 162, 128 FP32 299 -> 203, 40 / 256 BF16 267 / 501
// -> 217 / 358; of 10,000 nodes, 40 FP32 columns 80 -> 68, 128 86 -> 71; 200,000 nodes on
// a shallow tree, 8 / 40 / 128 columns 158 / 226 / 361 -> 85 / 164 / 260.
template <typename GT, typename DT, int VPL, int V, int TLC>
__global__ void __launch_bounds__(kThreads, (VPL > 2 ? 1 : VPL == 2 ? 2 : 3)) tr_kernel(const TrArgs a) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int S = dual_sums<TLC>();
  const int lane = threadIdx.x & 31;
  const int TL = TLC == 32 ? 32 : a.team;
  const int tl = lane & (TL - 1);
  const int team = lane / TL;
  const unsigned teams = 32 / TL;
  const unsigned epoch = *(volatile unsigned*)&a.qs->epoch + 1u;
  const Lane<GT, VPL, V, true> lg(a.g, a.ldg, a.nvec, tl, TL);
  const Lane<float, VPL, V, false> lh(a.h, a.ldp, a.nvec, tl, TL);
  const bool scale_g = a.scale_g != 0;
  const unsigned n = (unsigned)a.n_items, n_solo = (unsigned)a.n_solo;
  const unsigned lists = teams < 4u ? teams : 4u;  // lists of a group behind the solo ones
  const int ps_solo = __ffs((int)teams) - 1;       // log2 of the teams per list: all of them,
  const int ps_shared = teams > 4u ? __ffs((int)teams) - 3 : 0;  // or the list's share
  const unsigned wq = threadIdx.x >> 5;
  unsigned pend = 0;
  auto claim = [&] {
    if (lane == 0) pend = atomicAdd(a.claims + wq * kClaimStride, 1u);
  };
  // first item of the warp's next group; n when the queue is exhausted
  auto next_group = [&]() -> unsigned {
    unsigned g = __shfl_sync(kAll, pend, 0) * kClaimQueues + wq;
    if (g > n_solo) g = n_solo + (g - n_solo) * lists;
    if (g >= n) return n;  // the claim stays pending: every later call ends here too
    claim();
    return g;
  };
  auto split_of = [&](unsigned g) { return g < n_solo ? ps_solo : ps_shared; };
  // this team's run [from, from + len) of a list of w entries split over 2^ps teams
  auto part_of = [&](int w, int ps, int& from, int& len) {
    w = w > 0 ? w : 0;
    const int part = team & ((1 << ps) - 1);
    const int run = (w + (1 << ps) - 1) >> ps;
    from = part * run < w ? part * run : w;
    len = w - from < run ? w - from : run;
  };
  claim();
  unsigned g0 = next_group();
  if (g0 < n) {
    unsigned g1 = next_group();
    int ps0 = split_of(g0), ps1 = split_of(g1);
    int4 m0 = __ldg(a.meta + g0 + (team >> ps0)), m1 = __ldg(a.meta + g1 + (team >> ps1));
    int from0, len0;
    part_of(m0.w, ps0, from0, len0);
    uint32_t e0 = tl < len0 ? __ldg(a.ent + (uint32_t)m0.z + from0 + tl) : 0u;
    while (g0 < n) {
      const float s0 = tl < len0 ? dual_scale(e0, scale_g, a.mult) : 0.f;
      int from1, len1;
      uint32_t e1 = 0;
      float sums[S][VPL][V] = {};
      gather_dual_row<GT, VPL, V, TLC, S>(sums, lg, lh, a.ent + (uint32_t)m0.z + from0, len0,
                                          __reduce_max_sync(kAll, len0), e0, s0, scale_g, a.mult, tl, TL, [&] {
                                            part_of(m1.w, ps1, from1, len1);
                                            if (tl < len1) e1 = __ldg(a.ent + (uint32_t)m1.z + from1 + tl);
                                          });
      float acc[VPL][V];
      add_sums<VPL, V>(acc, sums);
      for (int off = TL; off < TL << ps0; off <<= 1) {
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
          for (int q = 0; q < V; ++q) acc[v][q] += __shfl_xor_sync(kAll, acc[v][q], off);
      }
      const bool writer = (team & ((1 << ps0) - 1)) == 0 && g0 + (team >> ps0) < n;
      if (m0.x < 0) {
        // a chunk, alone on its warp: its sum, then its ready flag
        float* prow = a.partial + (int64_t)(~m0.x) * a.ldp;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (writer && vi < a.nvec) store_f32<V>(prow + vi * V, acc[v]);
        }
        // the barrier orders the team's stores before lane 0's release, which carries them
        __syncwarp();
        if (lane == 0) st_release(a.chunk_flag + ~m0.x, epoch);
      } else if (writer) {
        for (int k = m0.z, ke = chunk_stop(m0.z, m0.w); k < ke; ++k) {
          if (!wait_flag(a.chunk_flag + k, epoch, a.qs, a.timeout_ns, (long long)k)) continue;
          const float* prow = a.partial + (int64_t)k * a.ldp;
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            const int vi = tl + v * TL;
            if (vi < a.nvec) {
              float t[V];
              load_f32_cg<V>(prow + vi * V, t);
#pragma unroll
              for (int q = 0; q < V; ++q) acc[v][q] = __fadd_rn(acc[v][q], t[q]);
            }
          }
        }
        // an empty column contributes nothing; do not scale it (m may be inf there)
        const bool scaled = a.scale_out && m0.w != 0;
        const float so = scaled ? __ldg(a.mult + m0.x) : 1.f;
        DT* drow = static_cast<DT*>(a.dx) + row_off(m0.x, a.lddx);
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = tl + v * TL;
          if (vi < a.nvec) {
            if (scaled) {
#pragma unroll
              for (int q = 0; q < V; ++q) acc[v][q] = __fmul_rn(acc[v][q], so);
            }
            store_vec<DT, V>(drow + (int64_t)vi * V, acc[v]);
          }
        }
      }
      __syncwarp();
      g0 = g1;
      m0 = m1;
      e0 = e1;
      from0 = from1;
      len0 = len1;
      ps0 = ps1;
      g1 = next_group();
      ps1 = split_of(g1);
      m1 = __ldg(a.meta + g1 + (team >> ps1));
    }
  }
  finish_block(a.qs, epoch, true, a.claims);
}

}  // namespace cbm
