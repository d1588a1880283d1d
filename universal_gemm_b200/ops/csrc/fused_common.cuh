// Device helpers shared by the fused GEMM kernels (one-CTA tiles in fused_gemm.cu, CTA-pair tiles in
// fused_gemm_pair.cu): bounded waits, tile raster, UMMA descriptors, epilogue stores, fetch-warp copy.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "ptx_sm100.cuh"
#include "ugemm_b200.h"

namespace ugfused {

using namespace ugptx;

constexpr int kNumThreads = 448;      // 14 warps: producer, UMMA, 8 epilogue, 4 fetch
constexpr int kProducerWarp = 0;
constexpr int kMmaWarp = 1;
constexpr int kEpiWarp0 = 2;    // warps 2..9 are the epilogue: two per TMEM lane quadrant (warp & 3), the first
constexpr int kNumEpiWarps = 8; // four drain the left part of a tile's columns, the other four the right part
constexpr int kFetchWarp0 = 10; // warps 10..13 fetch

constexpr uint32_t kBChunkBytes = UG_BK * 64 * 2;      // 8 KiB: 64 k rows x 64 n elements
constexpr uint32_t kBBytes = 4 * kBChunkBytes;         // 32 KiB
constexpr uint32_t kEpiWarpBytes = 32 * 128;           // 32 rows of 128 bytes, 16-byte groups XOR-swizzled by row
constexpr uint32_t kEpiBytes = kNumEpiWarps * kEpiWarpBytes;   // one transpose buffer per epilogue warp
constexpr uint32_t kCtlBytes = 512;                    // barriers, flags and the tile queue; the epilogue buffers follow
constexpr uint32_t kTmemCols = 512;                    // 128 lanes x 512 fp32 columns: all of TMEM

struct WaitCtl {
  volatile uint32_t* abort;
  uint32_t* status;
  uint64_t deadline;
  uint32_t peer_abort;   // shared::cluster address of the abort word of the other CTA of a pair (0: no partner)
};

// First error wins the status word; the CTA (and its partner in a CTA pair, which would otherwise only leave when
// its own waits run out) drains and returns.  The partner cannot have exited yet: both CTAs meet at a cluster
// barrier before they leave.
__device__ __forceinline__ void raise_error(const WaitCtl& ctl, uint32_t code) {
  atomicCAS(ctl.status, 0u, code);
  *ctl.abort = 1u;
  if (ctl.peer_abort != 0u) st_shared_cluster_u32(ctl.peer_abort, 1u);
}

// In-kernel check of the work tables (UG_ERR_BAD_TABLE): indices a tile is about to use must lie inside the tables
// the launch declared.  A failed check records the error and the tile is never touched.
__device__ __forceinline__ bool task_in_bounds(const UgFusedParams& P, const UgTask& t) {
  return t.seg_begin >= 0 && t.seg_count >= 0 && t.seg_begin + t.seg_count <= P.num_segs;
}
// K ranges of staged operands: [0, 256), [256, 512), [512, 1024), then 1024 each.
__device__ __forceinline__ int k_range(int k) { return k < 256 ? 0 : k < 512 ? 1 : k < 1024 ? 2 : 2 + (k >> 10); }
__device__ __forceinline__ int k_range_end(int k) { return k < 256 ? 256 : k < 512 ? 512 : ((k >> 10) + 1) << 10; }
// a_chunk: chunk of A the tile needs, b_chunk: the last one of B, cta_chunks: 64-column chunks of B a CTA loads.
__device__ __forceinline__ bool segment_in_bounds(const UgFusedParams& P, const UgSegment& sg, int a_chunk,
                                                  int b_chunk, int cta_chunks) {
  if (sg.k_pos < 0 || sg.k_len <= 0 || sg.a_step < 0 || sg.b_step < 0) return false;
  const int last = k_range(sg.k_pos + sg.k_len - 1);
  const int a_flag_last = sg.a_flag + last * sg.a_step + a_chunk, b_flag_last = sg.b_flag + last * sg.b_step + b_chunk;
  return (sg.b_box <= 1 || sg.b_box == cta_chunks) && sg.a_map >= 0 && sg.a_map < P.num_maps && sg.b_map >= 0 && sg.b_map < P.num_maps && sg.k_len > 0 &&
         (sg.a_flag < 0 || a_flag_last < P.num_flags) && (sg.b_flag < 0 || b_flag_last < P.num_flags);
}

// Optional timeline (UgFusedParams::trace != 0): one 64-byte record per (CTA, tile iteration), written by
// single threads with plain stores; the host reads it after the kernel.  Costs one uniform branch when off.
__device__ __forceinline__ uint64_t* trace_slot(const UgFusedParams& P, int cta, int iter) {
  if (P.trace == 0 || iter > P.trace_slots) return nullptr;
  return reinterpret_cast<uint64_t*>(P.trace) + (static_cast<int64_t>(cta) * (P.trace_slots + 1) + iter) * UG_TR_FIELDS;
}
__device__ __forceinline__ void trace_put(const UgFusedParams& P, int cta, int iter, int field, uint64_t v) {
  if (P.trace == 0 || iter >= P.trace_slots) return;
  trace_slot(P, cta, iter)[field] = v;
}
__device__ __forceinline__ void trace_now(const UgFusedParams& P, int cta, int iter, int field) {
  if (P.trace == 0 || iter >= P.trace_slots) return;
  trace_slot(P, cta, iter)[field] = global_timer_ns();
}
// Summary record of the CTA (index trace_slots).
__device__ __forceinline__ uint64_t* trace_summary(const UgFusedParams& P, int cta) {
  return P.trace == 0 ? nullptr : trace_slot(P, cta, P.trace_slots);
}

// Tile hand-off inside a CTA when tiles are claimed dynamically (UgFusedParams::sched): the TMA producer claims the
// tile of iteration i and publishes (i + 1) << 32 | tile in slot i % 16 with one 64-bit store; the UMMA issuer and
// the epilogue warps read it from there.  No role is ever 16 tiles ahead of another (the operand ring and the two
// accumulator buffers bound the lead), so a slot is not overwritten before everyone has read it.
constexpr int kTileQueueSlots = 16;
struct TileQueue {
  volatile unsigned long long slot[kTileQueueSlots];
};
__device__ __forceinline__ unsigned long long tileq_word(int iter, int tile) {
  return (static_cast<unsigned long long>(iter + 1) << 32) | static_cast<uint32_t>(tile);
}
__device__ __forceinline__ void tileq_publish(TileQueue* q, int iter, int tile) {
  q->slot[iter & (kTileQueueSlots - 1)] = tileq_word(iter, tile);
}
// Bounded wait for the tile of iteration `iter`; -1 after an abort or a timeout.
__device__ __forceinline__ int tileq_get(const TileQueue* q, int iter, const WaitCtl& ctl);

// Bounded mbarrier wait.  Returns false after an abort or a timeout.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const WaitCtl& ctl) {
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0xffu) == 0u) {
      if (*ctl.abort) return false;
      if (global_timer_ns() > ctl.deadline) {
        raise_error(ctl, UG_ERR_TIMEOUT_MBAR);
        return false;
      }
    }
  }
  return true;
}

// The same wait with a pause between polls, for roles that wait a whole main loop (the epilogue warps): fewer
// issue slots and less power spent on polling, at the price of up to `sleep_ns` of wake-up latency.
__device__ __forceinline__ bool mbar_wait_backoff(uint32_t bar, uint32_t parity, const WaitCtl& ctl, uint32_t sleep_ns) {
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (sleep_ns != 0u) __nanosleep(sleep_ns);
    if ((++spins & 0xffu) == 0u) {
      if (*ctl.abort) return false;
      if (global_timer_ns() > ctl.deadline) {
        raise_error(ctl, UG_ERR_TIMEOUT_MBAR);
        return false;
      }
    }
  }
  return true;
}

// Bounded wait until counter >= need (a staged chunk has fully landed).
__device__ __forceinline__ bool flag_wait(const uint32_t* counter, uint32_t need, const WaitCtl& ctl) {
  uint32_t spins = 0;
  while (ld_acquire_gpu(counter) < need) {
    __nanosleep(64);
    if ((++spins & 0x3fu) == 0u) {
      if (*ctl.abort) return false;
      if (global_timer_ns() > ctl.deadline) {
        raise_error(ctl, UG_ERR_TIMEOUT_FLAG);
        return false;
      }
    }
  }
  return true;
}

__device__ __forceinline__ int tileq_get(const TileQueue* q, int iter, const WaitCtl& ctl) {
  const unsigned long long want = static_cast<unsigned long long>(iter + 1);
  uint32_t spins = 0;
  for (;;) {
    const unsigned long long w = q->slot[iter & (kTileQueueSlots - 1)];
    if ((w >> 32) == want) return static_cast<int>(static_cast<uint32_t>(w));
    if ((++spins & 0x3fu) == 0u) {
      if (*ctl.abort) return -1;
      if (global_timer_ns() > ctl.deadline) {
        raise_error(ctl, UG_ERR_TIMEOUT_MBAR);
        return -1;
      }
      __nanosleep(32);
    }
  }
}

// Columns per output tile of a task: UG_BN, or a narrower width stored in the upper half of c_vec
// (used for the last, partly filled wave of tiles); bit 0 of c_vec says whether 16-byte accesses to C are legal.
__device__ __forceinline__ int task_tile_n(const UgTask& t) {
  const int v = t.c_vec >> 16;
  return v > 0 ? v : UG_BN;
}
__device__ __forceinline__ bool task_c_vec(const UgTask& t) { return (t.c_vec & 1) != 0; }
// Bit 1 of c_vec: the row pitch of C is a multiple of 16 bytes (and C is element-aligned), so every row of a region
// has the same alignment phase even when the region starts on an odd column.
__device__ __forceinline__ bool task_c_pitch_vec(const UgTask& t) { return (t.c_vec & 2) != 0; }
// Bit 2 of c_vec: the task's output rows live in several places (a task merged from tasks of different C tiles);
// c_ptr is then the address of a table uint64[m] with the address of every row's first column, and ldc is unused.
// All rows share one 16-byte alignment phase (checked when the table is built).
__device__ __forceinline__ bool task_c_rows_indirect(const UgTask& t) { return (t.c_vec & 4) != 0; }

// Bit 3 of c_vec: a bf16 C that only this task adds to (c_mode 0) may take the reduction instruction where whole aligned
// chunks are added; they round the sum to bf16 before they add it either way.  The ragged end of a row adds in fp32.
__device__ __forceinline__ int task_chunk_mode(const UgTask& t) { return (t.c_vec & 8) != 0 ? 1 : t.c_mode; }

// Where the 32 rows of an epilogue warp go: rows of one region (base + r * ldc) or rows named by a table.
struct CRows {
  const uint64_t* tab;   // entry of the warp's first row, or nullptr
  float* base;           // first row of the warp at the region's first column (direct), unused with a table
  int64_t ldc;
  int col;               // column offset added to a table entry
  __device__ __forceinline__ float* row(int r) const {
    return tab != nullptr ? reinterpret_cast<float*>(tab[r]) + col : base + r * ldc;
  }
};

struct TileCoord {
  int task;
  int mt, nt;
};

__device__ __forceinline__ int find_task(const UgTask* __restrict__ tasks, int num_tasks, int tile) {
  int lo = 0, hi = num_tasks - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (tasks[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Banded raster: inside a band of group_m tile rows, m runs fastest so the A band
// stays in L2 while the CTAs sweep across n.
__device__ __forceinline__ TileCoord locate(const UgTask* __restrict__ tasks, int num_tasks, int tile) {
  TileCoord tc;
  tc.task = find_task(tasks, num_tasks, tile);
  const UgTask& t = tasks[tc.task];
  int idx = tile - t.tile_begin;
  int gm = t.group_m > 0 ? t.group_m : t.m_tiles;
  int band_tiles = gm * t.n_tiles;
  int band = idx / band_tiles;
  int first_m = band * gm;
  int band_m = min(gm, t.m_tiles - first_m);
  int rem = idx - band * band_tiles;
  tc.mt = first_m + rem % band_m;
  tc.nt = rem / band_m;
  return tc;
}

// UMMA shared-memory descriptors (sm_100 format, version 1, 128-byte swizzle).
// A tile: K-major, rows of 128 bytes, 8-row groups 1024 bytes apart (SBO).
__device__ __forceinline__ uint64_t make_desc_a(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3fffu);
  d |= static_cast<uint64_t>(1u) << 16;                  // LBO (unused for swizzled K-major)
  d |= static_cast<uint64_t>(1024u >> 4) << 32;          // SBO
  d |= static_cast<uint64_t>(1u) << 46;                  // descriptor version
  d |= static_cast<uint64_t>(2u) << 61;                  // SWIZZLE_128B
  return d;
}
// B tile: N-major.  One k row = 64 n elements = 128 bytes; 8-k-row groups are 1024
// bytes apart (SBO); the next 64 n elements start kBChunkBytes later (LBO).
__device__ __forceinline__ uint64_t make_desc_b(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3fffu);
  d |= static_cast<uint64_t>(kBChunkBytes >> 4) << 16;   // LBO
  d |= static_cast<uint64_t>(1024u >> 4) << 32;          // SBO
  d |= static_cast<uint64_t>(1u) << 46;
  d |= static_cast<uint64_t>(2u) << 61;
  return d;
}
// Instruction descriptor: D fp32, A/B bf16, A K-major, B MN-major, M = 128, N = n.
__device__ __forceinline__ uint32_t make_idesc(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (0u << 15) | (1u << 16) | ((n >> 3) << 17) |
         ((static_cast<uint32_t>(UG_BM) >> 4) << 24);
}

// ---------------------------------------------------------------- epilogue stores
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Word offset of 16-byte group `group` (0..7) of row `row` in a transpose buffer.  Rows are 128 bytes without
// padding; XOR-ing the group with the row number keeps both phases free of bank conflicts: lanes of a quarter warp
// write the same group of 8 different rows, and read 8 different groups of one row.
__device__ __forceinline__ int epi_off(int row, int group) { return row * 32 + ((group ^ (row & 7)) << 2); }

// Full, 16-byte aligned chunks: the warp's 32 x 32 block of accumulators goes through a
// shared-memory buffer so that each store / reduction instruction covers whole 128-byte row
// segments (4 rows of fp32, 8 rows of bf16) instead of 32 different rows.  This matters most for
// red.add into a peer's memory, where every instruction becomes a few full NVLink packets.
__device__ __forceinline__ void store_chunk_f32(float* sb, const uint32_t (&v)[32], int lane, float* c_base,
                                                int64_t ldc, int rows_valid, int mode) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(sb + epi_off(lane, j)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  const int rsub = lane >> 3, cseg = (lane & 7) * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + rsub;
    if (r < rows_valid) {
      float4 x = *reinterpret_cast<const float4*>(sb + epi_off(r, lane & 7));
      float4* g = reinterpret_cast<float4*>(c_base + r * ldc + cseg);
      if (mode == 1) {
        red_add_v4_f32(g, x.x, x.y, x.z, x.w);
      } else {
        if (mode == 0) {
          const float4 old = *g;
          x.x += old.x; x.y += old.y; x.z += old.z; x.w += old.w;
        }
        *g = x;
      }
    }
  }
  __syncwarp();
}

__device__ __forceinline__ void store_chunk_bf16(float* sbf, const uint32_t (&v)[32], int lane,
                                                 __nv_bfloat16* c_base, int64_t ldc, int rows_valid, int mode) {
  // 64 payload bytes per row, rows 80 bytes apart.
  unsigned char* sb = reinterpret_cast<unsigned char*>(sbf);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4 q;
    q.x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
    q.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
    q.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
    q.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
    *reinterpret_cast<uint4*>(sb + lane * 80 + j * 16) = q;
  }
  __syncwarp();
  const int rsub = lane >> 2, cseg = (lane & 3) * 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * 8 + rsub;
    if (r < rows_valid) {
      uint4 x = *reinterpret_cast<const uint4*>(sb + r * 80 + (lane & 3) * 16);
      uint4* g = reinterpret_cast<uint4*>(c_base + r * ldc + cseg);
      if (mode == 1) {
        red_add_v4_bf16x2(g, x.x, x.y, x.z, x.w);
      } else {
        if (mode == 0) {
          const uint4 old = *g;
          const __nv_bfloat162* o = reinterpret_cast<const __nv_bfloat162*>(&old);
          __nv_bfloat162* n = reinterpret_cast<__nv_bfloat162*>(&x);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 a = __bfloat1622float2(n[e]), b = __bfloat1622float2(o[e]);
            n[e] = __floats2bfloat162_rn(a.x + b.x, a.y + b.y);
          }
        }
        *g = x;
      }
    }
  }
  __syncwarp();
}

// 64 bf16 columns at a time: rows of 128 payload bytes, so that every store / reduction instruction covers
// four full 128-byte row segments (half-line segments made the NVLink pushes of bf16 partial tiles inefficient).
__device__ __forceinline__ void store_chunk_bf16_64(float* sbf, const uint32_t (&v0)[32], const uint32_t (&v1)[32],
                                                    int lane, __nv_bfloat16* c_base, int64_t ldc, int rows_valid,
                                                    int mode) {
  // rows of 128 payload bytes, swizzled like the fp32 rows
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4 q;
    q.x = pack_bf16x2(__uint_as_float(v0[8 * j + 0]), __uint_as_float(v0[8 * j + 1]));
    q.y = pack_bf16x2(__uint_as_float(v0[8 * j + 2]), __uint_as_float(v0[8 * j + 3]));
    q.z = pack_bf16x2(__uint_as_float(v0[8 * j + 4]), __uint_as_float(v0[8 * j + 5]));
    q.w = pack_bf16x2(__uint_as_float(v0[8 * j + 6]), __uint_as_float(v0[8 * j + 7]));
    *reinterpret_cast<uint4*>(sbf + epi_off(lane, j)) = q;
    q.x = pack_bf16x2(__uint_as_float(v1[8 * j + 0]), __uint_as_float(v1[8 * j + 1]));
    q.y = pack_bf16x2(__uint_as_float(v1[8 * j + 2]), __uint_as_float(v1[8 * j + 3]));
    q.z = pack_bf16x2(__uint_as_float(v1[8 * j + 4]), __uint_as_float(v1[8 * j + 5]));
    q.w = pack_bf16x2(__uint_as_float(v1[8 * j + 6]), __uint_as_float(v1[8 * j + 7]));
    *reinterpret_cast<uint4*>(sbf + epi_off(lane, j + 4)) = q;
  }
  __syncwarp();
  const int rsub = lane >> 3, seg = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + rsub;
    if (r < rows_valid) {
      uint4 x = *reinterpret_cast<const uint4*>(sbf + epi_off(r, seg));
      uint4* g = reinterpret_cast<uint4*>(c_base + r * ldc + seg * 8);
      if (mode == 1) {
        red_add_v4_bf16x2(g, x.x, x.y, x.z, x.w);
      } else {
        if (mode == 0) {
          const uint4 old = *g;
          const __nv_bfloat162* o = reinterpret_cast<const __nv_bfloat162*>(&old);
          __nv_bfloat162* n = reinterpret_cast<__nv_bfloat162*>(&x);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 a = __bfloat1622float2(n[e]), b = __bfloat1622float2(o[e]);
            n[e] = __floats2bfloat162_rn(a.x + b.x, a.y + b.y);
          }
        }
        *g = x;
      }
    }
  }
  __syncwarp();
}

// Any alignment, any width: the 32 x 32 block goes through shared memory and every instruction handles 32
// consecutive columns of ONE row (a coalesced, possibly misaligned 128-byte / 64-byte segment).  Used when C
// rows are not 16-byte aligned (odd column offsets of odd-shaped partitions) and for ragged right edges.
__device__ __forceinline__ void store_chunk_scalar(float* sb, const uint32_t (&v)[32], int lane, uint64_t c_ptr,
                                                   int64_t elem_off, int64_t ldc, int rows_valid, int ncols, int mode,
                                                   int dtype) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(sb + epi_off(lane, j)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  if (lane < ncols) {
    for (int r = 0; r < rows_valid; ++r) {
      const float x = sb[epi_off(r, lane >> 2) + (lane & 3)];
      const int64_t off = elem_off + r * ldc + lane;
      if (dtype == 0) {
        float* g = reinterpret_cast<float*>(c_ptr) + off;
        if (mode == 1) red_add_f32(g, x);
        else if (mode == 0) *g += x;
        else *g = x;
      } else {
        __nv_bfloat16* g = reinterpret_cast<__nv_bfloat16*>(c_ptr) + off;
        if (mode == 1) atomicAdd(g, __float2bfloat16_rn(x));
        else if (mode == 0) *g = __float2bfloat16_rn(__bfloat162float(*g) + x);
        else *g = __float2bfloat16_rn(x);
      }
    }
  }
  __syncwarp();
}

// Sum of the accumulator columns [lo, hi) of this lane's row (the checksum a launch can ask for).
__device__ __forceinline__ float sum_columns(const uint32_t (&v)[32], int lo, int hi) {
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (j >= lo && j < hi) s += __uint_as_float(v[j]);
  return s;
}

// The same transpose for a 32-column chunk of which only columns [lo, hi) are to be written (lo a multiple of 4;
// c_base 16-byte aligned): whole 16-byte groups inside the range go out as vectors, the ragged end element by element.
__device__ __forceinline__ void store_chunk_f32_ragged(float* sb, const uint32_t (&v)[32], int lane, const CRows& rows,
                                                       int col, int rows_valid, int mode, int lo, int hi) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(sb + epi_off(lane, j)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  const int rsub = lane >> 3, cseg = (lane & 7) * 4;
  if (cseg >= lo && cseg < hi) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + rsub;
      if (r < rows_valid) {
        float4 x = *reinterpret_cast<const float4*>(sb + epi_off(r, lane & 7));
        float* g = rows.row(r) + col + cseg;
        if (cseg + 4 <= hi) {
          float4* g4 = reinterpret_cast<float4*>(g);
          if (mode == 1) {
            red_add_v4_f32(g4, x.x, x.y, x.z, x.w);
          } else {
            if (mode == 0) {
              const float4 old = *g4;
              x.x += old.x; x.y += old.y; x.z += old.z; x.w += old.w;
            }
            *g4 = x;
          }
        } else {
          const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            if (cseg + e < hi) {
              if (mode == 1) red_add_f32(g + e, xs[e]);
              else if (mode == 0) g[e] += xs[e];
              else g[e] = xs[e];
            }
          }
        }
      }
    }
  }
  __syncwarp();
}

// Sums of the other parts of a tile whose K blocks were cut (UgTask::part_count): `base` is this epilogue warp's block of
// the first part: groups of four columns, in a group 16 bytes per row, so that a warp's access is four whole lines.
struct Partials {
  const float* base;
  int64_t stride;      // to the same block of the next part
  int count;
};
__device__ __forceinline__ void load_partial(float4 (&x)[8], const Partials& pt, int p, int c, int lane) {
  const float4* q = reinterpret_cast<const float4*>(pt.base + p * pt.stride) + (c >> 2) * 32 + lane;
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = __ldcg(q + j * 32);
}
__device__ __forceinline__ void add_partial(uint32_t (&v)[32], const float4 (&x)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[4 * j] = __float_as_uint(__uint_as_float(v[4 * j]) + x[j].x);
    v[4 * j + 1] = __float_as_uint(__uint_as_float(v[4 * j + 1]) + x[j].y);
    v[4 * j + 2] = __float_as_uint(__uint_as_float(v[4 * j + 2]) + x[j].z);
    v[4 * j + 3] = __float_as_uint(__uint_as_float(v[4 * j + 3]) + x[j].w);
  }
}
// Add them to this warp's accumulator columns in place (TMEM), so that the drain that follows is the ordinary one.  Bound
// by the latency of the reads (L2), a block of 4 KiB per warp at a time: a second one in registers would spill.  Cut tiles as
// a whole, 64 x 16383 x 16383 (64 tiles on 148 SMs, two parts each): 104 us per call, 124 with whole pair tiles.
__device__ __forceinline__ void add_partials(uint32_t taddr, int n_rem, const Partials& pt, int lane) {
#pragma unroll 1
  for (int c = 0; c < n_rem; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
#pragma unroll 1
    for (int p = 0; p < pt.count; ++p) {
      float4 x[8];
      load_partial(x, pt, p, c, lane);
      add_partial(v, x);
    }
    tmem_st_32x32(taddr + c, v);
  }
  tmem_st_wait();
}
__device__ __forceinline__ void store_partials(uint32_t taddr, int n_rem, float* base, int lane) {
#pragma unroll 1
  for (int c = 0; c < n_rem; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
    uint4* q = reinterpret_cast<uint4*>(base) + (c >> 2) * 32 + lane;
#pragma unroll
    for (int j = 0; j < 8; ++j) __stcg(q + j * 32, make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
  }
}
// This warp's block of part 0 of a tile.  `slot`: the warp's number among the tile's epilogue warps (and halves), of `slots`.
__device__ __forceinline__ Partials tile_partials(const UgTask& t, int tile, int slot, int slots) {
  const int tiles = t.m_tiles * t.n_tiles;
  const int64_t block = 32 * (task_tile_n(t) / 2);
  Partials pt;
  pt.base = reinterpret_cast<const float*>(t.part_ptr) + (static_cast<int64_t>(tile - t.tile_begin) * slots + slot) * block;
  pt.stride = static_cast<int64_t>(tiles) * slots * block;
  pt.count = t.part_count - 1;
  return pt;
}
// Counter of one epilogue warp of a cut tile.
__device__ __forceinline__ uint32_t* part_counter(const UgFusedParams& P, const UgTask& t, int tile, int warp_slot) {
  return reinterpret_cast<uint32_t*>(P.part_flags) + t.part_flag + (tile - t.tile_begin) * 16 + warp_slot;
}
__device__ __forceinline__ void part_done(uint32_t* counter, int lane) {
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    red_add_gpu(counter, 1u);
  }
}
// Bounded wait of a whole warp for the other parts of a tile.  Lane 0 acquires; the warp barrier orders the reads of the
// other lanes after it (the shuffle alone orders no memory).
__device__ __forceinline__ bool parts_wait(const uint32_t* counter, uint32_t need, int lane, const WaitCtl& ctl) {
  int ok = 1;
  if (lane == 0) ok = flag_wait(counter, need, ctl) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();
  return ok != 0;
}
__device__ __forceinline__ bool part_in_bounds(const UgFusedParams& P, const UgTask& t) {
  return t.part_count <= 1 || (t.part_ptr != 0 && t.part_flag >= 0 && t.part_index >= 0 && t.part_index < t.part_count &&
                               t.part_flag + t.m_tiles * t.n_tiles * 16 <= P.num_part_flags);
}

// fp32 C whose rows are 16 bytes apart in phase but whose region starts on any column (odd-shaped partitions) and has
// any width: up to three head columns go out element by element, then 32-column chunks that start on a 16-byte
// boundary of C.  `avail` TMEM columns can be read from `taddr`; a last chunk that would read past them is moved back
// by a multiple of four columns and writes only what the chunks before it have not written.
__device__ __forceinline__ void epilogue_drain_f32_shifted(uint32_t taddr, const UgTask& t, int row0, int col0,
                                                           int n_rem, int avail, float* epi_buf, int lane, float* acc) {
  const int rows_valid = min(32, t.m - row0);
  if (rows_valid <= 0) return;
  CRows rows;
  if (task_c_rows_indirect(t)) {
    rows.tab = reinterpret_cast<const uint64_t*>(t.c_ptr) + row0;
    rows.base = nullptr;
    rows.ldc = 0;
    rows.col = col0;
  } else {
    rows.tab = nullptr;
    rows.base = reinterpret_cast<float*>(t.c_ptr) + static_cast<int64_t>(row0) * t.ldc + col0;
    rows.ldc = t.ldc;
    rows.col = 0;
  }
  const int phase = static_cast<int>((reinterpret_cast<uint64_t>(rows.row(0)) >> 2) & 3u);
  const int head = min((4 - phase) & 3, n_rem);
  uint32_t v[32];
  if (head > 0) {
    tmem_ld_32x32(taddr, v);
    tmem_ld_wait();
    if (acc != nullptr && lane < rows_valid) *acc += sum_columns(v, 0, head);
    if (lane < rows_valid) {
      float* g = rows.row(lane);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j < head) {
          const float x = __uint_as_float(v[j]);
          if (t.c_mode == 1) red_add_f32(g + j, x);
          else if (t.c_mode == 0) g[j] += x;
          else g[j] = x;
        }
      }
    }
  }
  int c = head;
  for (; c < n_rem && c + 32 <= avail; c += 32) {
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
    if (acc != nullptr && lane < rows_valid) *acc += sum_columns(v, 0, min(32, n_rem - c));
    store_chunk_f32_ragged(epi_buf, v, lane, rows, c, rows_valid, t.c_mode, 0, min(32, n_rem - c));
  }
  if (c < n_rem) {
    // Fewer than 32 columns are left and a chunk on this boundary would read past the readable TMEM columns: move it
    // back by a multiple of four columns (it then skips what is written already); up to three columns can remain
    // beyond its end, they go out element by element from a chunk that ends with the region.
    const int lo = (c + 32 - avail + 3) & ~3;
    const int start = c - lo;
    const int hi = min(32, n_rem - start);
    if (lo < hi) {
      tmem_ld_32x32(taddr + start, v);
      tmem_ld_wait();
      if (acc != nullptr && lane < rows_valid) *acc += sum_columns(v, lo, hi);
      store_chunk_f32_ragged(epi_buf, v, lane, rows, start, rows_valid, t.c_mode, lo, hi);
    }
    const int rem = n_rem - min(start + 32, n_rem);
    if (rem > 0) {
      tmem_ld_32x32(taddr + n_rem - 32, v);
      tmem_ld_wait();
      if (acc != nullptr && lane < rows_valid) *acc += sum_columns(v, 32 - rem, 32);
      if (lane < rows_valid) {
        float* g = rows.row(lane) + n_rem - 32;
#pragma unroll
        for (int j = 29; j < 32; ++j) {
          if (j >= 32 - rem) {
            const float x = __uint_as_float(v[j]);
            if (t.c_mode == 1) red_add_f32(g + j, x);
            else if (t.c_mode == 0) g[j] += x;
            else g[j] = x;
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------- fetch warps
__device__ __forceinline__ float4 ld_stream_f4(const void* p) {
  const uint4 u = ld_stream_v4(p);
  return make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
}
__device__ __forceinline__ uint16_t ld_stream_u16(const void* p) {
  uint16_t v;
  asm volatile("ld.global.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream_f1(const void* p) {
  float v;
  asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
// High and low bf16 parts of two fp32 values: hi = bf16(x), lo = bf16(x - hi), packed as bf16x2.
__device__ __forceinline__ void split_bf16x2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat16 h0 = __float2bfloat16_rn(x0), h1 = __float2bfloat16_rn(x1);
  const __nv_bfloat162 hp = __halves2bfloat162(h0, h1);
  const __nv_bfloat162 lp = __floats2bfloat162_rn(x0 - __bfloat162float(h0), x1 - __bfloat162float(h1));
  hi = *reinterpret_cast<const uint32_t*>(&hp);
  lo = *reinterpret_cast<const uint32_t*>(&lp);
}

// Copy an fp32 piece (possibly from a peer) into two bf16 buffers: the high parts at pc.dst, the low parts
// (pc.mode >> 8) KiB further on.  A 16-byte destination vector holds eight elements, i.e. 32 source bytes.
// `aligned`: source rows start on 16-byte boundaries (two vector loads per destination vector), else 4-byte loads.
// Elements past the end of a row are written as zeros.
__device__ __forceinline__ void copy_piece_split_f32(const UgPiece& pc, int lane, int vec_per_row, uint32_t nvec,
                                                     bool aligned) {
  const char* src = reinterpret_cast<const char*>(pc.src);
  char* dst = reinterpret_cast<char*>(pc.dst);
  const int64_t low = static_cast<int64_t>(static_cast<uint32_t>(pc.mode) >> 8) << 10;
  const uint32_t vpr = static_cast<uint32_t>(vec_per_row);
  const int row_elems = pc.row_bytes >> 1;
  constexpr uint32_t U = 4;                       // destination vectors per lane and batch: 8 x 16 B loads in flight
  for (uint32_t base = 0; base < nvec; base += 32u * U) {
    float f[U][8];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t idx = min(base + u * 32u + static_cast<uint32_t>(lane), nvec - 1u);
      const uint32_t r = idx / vpr, c = idx - r * vpr;
      const char* sp = src + static_cast<int64_t>(r) * pc.src_ld + (static_cast<int64_t>(c) << 5);
      const int valid = row_elems - static_cast<int>(c << 3);          // elements of this vector inside the row
      if (aligned) {
        const float4 a = ld_stream_f4(sp);
        const float4 b = valid > 4 ? ld_stream_f4(sp + 16) : make_float4(0.f, 0.f, 0.f, 0.f);
        f[u][0] = a.x; f[u][1] = a.y; f[u][2] = a.z; f[u][3] = a.w;
        f[u][4] = b.x; f[u][5] = b.y; f[u][6] = b.z; f[u][7] = b.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[u][e] = e < valid ? ld_stream_f1(sp + 4 * e) : 0.f;
      }
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e >= valid) f[u][e] = 0.f;
    }
    asm volatile("" ::: "memory");
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t idx = base + u * 32u + static_cast<uint32_t>(lane);
      if (idx < nvec) {
        const uint32_t r = idx / vpr, c = idx - r * vpr;
        uint4 hi, lo;
        split_bf16x2(f[u][0], f[u][1], hi.x, lo.x);
        split_bf16x2(f[u][2], f[u][3], hi.y, lo.y);
        split_bf16x2(f[u][4], f[u][5], hi.z, lo.z);
        split_bf16x2(f[u][6], f[u][7], hi.w, lo.w);
        char* dp = dst + static_cast<int64_t>(r) * pc.dst_ld + (static_cast<int64_t>(c) << 4);
        *reinterpret_cast<uint4*>(dp) = hi;
        *reinterpret_cast<uint4*>(dp + low) = lo;
      }
    }
  }
}

// Mode 0 (16-byte aligned source): the piece is walked as one flat sequence of 16-byte vectors (row after row); a
// warp takes 32 x U consecutive vectors per batch, whatever the piece's shape (one 24 KiB row or 128 rows of 256
// bytes).  The batch is straight-line code: U unconditional loads (lanes past the end re-read the last vector), a
// compiler barrier, then the predicated stores, so one warp keeps U x 512 bytes on the wire: over NVLink the copy
// rate is (bytes in flight) / (about 2 us of latency), and a copy loop whose loads are issued one at a time reaches
// a quarter of the link rate.  U is chosen per launch (UgFusedParams::fetch_depth): loads in flight share the SM's
// outstanding-request capacity with the TMA operand loads, so a plan that needs its remote data slowly asks for less.
template <uint32_t U>
__device__ __forceinline__ void copy_flat_vec(const UgPiece& pc, int lane, int vec_per_row, uint32_t nvec) {
  const char* src = reinterpret_cast<const char*>(pc.src);
  char* dst = reinterpret_cast<char*>(pc.dst);
  const uint32_t vpr = static_cast<uint32_t>(vec_per_row);
  for (uint32_t base = 0; base < nvec; base += 32u * U) {
    uint4 buf[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t idx = min(base + u * 32u + static_cast<uint32_t>(lane), nvec - 1u);
      const uint32_t r = idx / vpr, c = idx - r * vpr;
      buf[u] = ld_stream_v4(src + static_cast<int64_t>(r) * pc.src_ld + (static_cast<int64_t>(c) << 4));
    }
    asm volatile("" ::: "memory");
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t idx = base + u * 32u + static_cast<uint32_t>(lane);
      if (idx < nvec) {
        const uint32_t r = idx / vpr, c = idx - r * vpr;
        *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(r) * pc.dst_ld + (static_cast<int64_t>(c) << 4)) = buf[u];
      }
    }
  }
}

// Copy one piece with the 32 lanes of a warp.  mode 0: 16-byte vectors, `depth` in flight per lane.  mode 1: the source is
// only 2-byte aligned; every 16-byte destination vector is shifted out of the two aligned source vectors that cover it.
// Modes 2 and 3: fp32 sources, split into two bf16 parts (copy_piece_split_f32), 16-byte aligned or not.
__device__ __forceinline__ void copy_piece(const UgPiece& pc, int lane, int depth) {
  const int vec_per_row = (pc.row_bytes + 15) >> 4;
  if (vec_per_row <= 0) return;
  const int64_t total = static_cast<int64_t>(pc.rows) * vec_per_row;
  const char* src = reinterpret_cast<const char*>(pc.src);
  char* dst = reinterpret_cast<char*>(pc.dst);
  const int mode = pc.mode & 0xff;
  if (mode >= 2) {
    copy_piece_split_f32(pc, lane, vec_per_row, static_cast<uint32_t>(total), mode == 2);
    return;
  }
  if (mode == 0) {
    if (depth <= 4) copy_flat_vec<4>(pc, lane, vec_per_row, static_cast<uint32_t>(total));
    else if (depth <= 8) copy_flat_vec<8>(pc, lane, vec_per_row, static_cast<uint32_t>(total));
    else copy_flat_vec<16>(pc, lane, vec_per_row, static_cast<uint32_t>(total));
  } else {
    // Source only 2-byte aligned (odd column offsets or pitches of odd-shaped partitions).  Every 16-byte destination
    // vector is cut out of the two 16-byte-aligned source vectors that cover it (funnel shifts by the source's byte
    // offset), so the copy still moves whole 16-byte vectors over the link: 2-byte loads from a peer cost a 32-byte
    // sector each.  The second vector is only read when it holds needed bytes, so no read leaves the source row.
    // Eight destination vectors per lane and batch keep up to sixteen loads in flight.
    constexpr uint32_t U = 8;
    const uint32_t vpr = static_cast<uint32_t>(vec_per_row);
    const uint32_t nvec = static_cast<uint32_t>(total);
    for (uint32_t base = 0; base < nvec; base += 32u * U) {
      uint4 lo[U], hi[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
        const uint32_t idx = min(base + u * 32u + static_cast<uint32_t>(lane), nvec - 1u);
        const uint32_t r = idx / vpr, c = idx - r * vpr;
        const uint64_t sp = reinterpret_cast<uint64_t>(src) + static_cast<uint64_t>(r) * pc.src_ld + (static_cast<uint64_t>(c) << 4);
        const int valid_bytes = min(16, pc.row_bytes - static_cast<int>(c << 4));
        const uint32_t shift = static_cast<uint32_t>(sp & 15u);
        const char* ap = reinterpret_cast<const char*>(sp - shift);
        lo[u] = ld_stream_v4(ap);
        hi[u] = (static_cast<int>(shift) + valid_bytes > 16) ? ld_stream_v4(ap + 16) : make_uint4(0u, 0u, 0u, 0u);
      }
      asm volatile("" ::: "memory");
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
        const uint32_t idx = base + u * 32u + static_cast<uint32_t>(lane);
        if (idx < nvec) {
          const uint32_t r = idx / vpr, c = idx - r * vpr;
          const uint32_t shift = static_cast<uint32_t>(reinterpret_cast<uint64_t>(src) + static_cast<uint64_t>(r) * pc.src_ld) & 15u;
          const uint32_t w[9] = {lo[u].x, lo[u].y, lo[u].z, lo[u].w, hi[u].x, hi[u].y, hi[u].z, hi[u].w, 0u};
          const uint32_t q = shift >> 2, bits = (shift & 3u) * 8u;
          uint32_t o[4];
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) {
            uint32_t a = 0u, b = 0u;
#pragma unroll
            for (uint32_t qq = 0; qq < 4; ++qq)
              if (q == qq) { a = w[i + qq]; b = w[i + qq + 1]; }
            o[i] = __funnelshift_r(a, b, bits);
          }
          const int valid = min(8, (pc.row_bytes - static_cast<int>(c << 4)) >> 1);     // elements inside the row
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (2 * i >= valid) o[i] = 0u;
            else if (2 * i + 1 >= valid) o[i] &= 0xffffu;
          }
          *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(r) * pc.dst_ld + (static_cast<int64_t>(c) << 4)) =
              make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
  }
}


// Fetch loop of one warp: claim staged pieces until none is left.  With `until` (the epilogue warps: the barrier of
// their first accumulator) also until that barrier's first phase completes.
//
// Staged data arrives as fast as the loads in flight allow (bytes in flight / latency), and at the start of a launch
// every tile waits for it while the eight epilogue warps have nothing to do: with them an SM has three times the loads
// in flight.  fp32 operands, 4096^3 (128 MiB read, 128 MiB written by the split): the last piece landed after 86 us
// instead of 209, the kernel took 343 us instead of 399; eight emulated ranks of the 2048-token up-projection: 29 us
// instead of 85 for a rank's 44 MB.
__device__ __forceinline__ unsigned long long fetch_pieces(const UgFusedParams& P, const WaitCtl& ctl, int lane, uint32_t until) {
  const UgPiece* __restrict__ pieces = reinterpret_cast<const UgPiece*>(P.pieces);
  uint32_t* counter = reinterpret_cast<uint32_t*>(P.piece_counter);
  uint32_t* wflags = reinterpret_cast<uint32_t*>(P.flags);
  unsigned long long copied = 0;
  const uint32_t count = P.num_pieces > 0 ? static_cast<uint32_t>(P.num_pieces) : 0u;
  auto claim = [&]() -> uint32_t {
    if (count == 0u || *ctl.abort || (until != 0u && mbar_test_wait(until, 0u) != 0u)) return count;
    return atomicAdd(counter, 1u);
  };
  uint32_t next = lane == 0 ? claim() : 0u;
  for (;;) {
    const uint32_t p = __shfl_sync(0xffffffffu, next, 0);
    if (p >= count) break;
    if (lane == 0) next = claim();                    // on its way while this piece is copied
    const UgPiece pc = pieces[p];
    if (pc.flag < 0 || pc.flag >= P.num_flags) {      // warp-uniform: never copy for a counter that does not exist
      if (lane == 0) raise_error(ctl, UG_ERR_BAD_TABLE);
      break;
    }
    copy_piece(pc, lane, P.fetch_depth == 0 ? 16 : P.fetch_depth);
    // One fence by one lane publishes the whole warp's stores (the warp barrier orders them before it): a fence waits
    // for the stores in flight, and with one per lane and one per counter a piece took 6 us on top of its copy.
    __syncwarp();
    if (lane == 0) {
      __threadfence();
      red_add_gpu(wflags + pc.flag, 1u);
      red_add_gpu(counter + 1, 1u);                   // all pieces together: see all_landed
    }
    ++copied;
  }
  return copied;
}

// True once every piece of the launch has landed: a producer that has seen it polls no more chunk counters (a poll is
// a round trip to L2, about as long as the operand ring covers; with seven of them per tile the main loop of tiles
// whose data had long arrived took 82 instead of 75 us).
__device__ __forceinline__ bool all_landed(const UgFusedParams& P) {
  return P.num_pieces > 0 &&
         ld_acquire_gpu(reinterpret_cast<const uint32_t*>(P.piece_counter) + 1) >= static_cast<uint32_t>(P.num_pieces);
}

// Bounded wait until K range `range` of the staged chunks of one tile is in place (a 512-column tile spans two chunks of B).
__device__ __forceinline__ bool range_wait(const UgFusedParams& P, const UgSegment& sg, int range, int a_chunk, int b_chunk,
                                           int b_chunks, const WaitCtl& ctl) {
  const uint32_t* flags = reinterpret_cast<const uint32_t*>(P.flags);
  const int32_t* need = reinterpret_cast<const int32_t*>(P.flag_need);
  bool ok = true;
  if (sg.a_flag >= 0) {
    const int f = sg.a_flag + range * sg.a_step + a_chunk;
    ok = flag_wait(flags + f, static_cast<uint32_t>(need[f]), ctl);
  }
  if (sg.b_flag >= 0) {
    const int f = sg.b_flag + range * sg.b_step + b_chunk;
    for (int i = 0; ok && i < b_chunks; ++i) ok = flag_wait(flags + f + i, static_cast<uint32_t>(need[f + i]), ctl);
  }
  if (ok) fence_proxy_async();
  return ok;
}

__device__ __forceinline__ void trace_fetch(const UgFusedParams& P, int cta, int lane, unsigned long long copied) {
  if (lane == 0 && P.num_pieces > 0) {
    if (uint64_t* ts = trace_summary(P, cta)) {
      atomicMax(reinterpret_cast<unsigned long long*>(ts + UG_TR_S_FETCH_END),
                static_cast<unsigned long long>(global_timer_ns()));
      atomicAdd(reinterpret_cast<unsigned long long*>(ts + UG_TR_S_PIECES), copied);
    }
  }
}

// Called by all threads of a worker's CTA (the leader's, of a pair) once every role of the worker is done: the last
// worker of the launch puts the counters back to zero, so that the next launch needs no clearing pass before it
// (2.3 us and a launch gap per call).  The count of finished workers wraps by itself: should two launches of a program
// overlap after all (replays of one graph on two streams), it and with it every counter is back at zero when both are done.
__device__ __forceinline__ void rearm_counters(const UgFusedParams& P, uint32_t workers, uint32_t* last) {
  if (P.finished == 0) return;
  if (threadIdx.x == 0) {
    __threadfence();
    *last = atomicInc(reinterpret_cast<uint32_t*>(P.finished), workers - 1u) == workers - 1u ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  if (*last == 0u) return;
  uint32_t* flags = reinterpret_cast<uint32_t*>(P.flags);
  if (P.num_pieces > 0)
    for (int i = threadIdx.x; i < P.num_flags + 2; i += blockDim.x) flags[i] = 0u;
  uint32_t* part_flags = reinterpret_cast<uint32_t*>(P.part_flags);
  for (int i = threadIdx.x; i < P.num_part_flags; i += blockDim.x) part_flags[i] = 0u;
  if (threadIdx.x == 0 && P.sched != 0) *reinterpret_cast<uint32_t*>(P.sched) = 0u;
}

// Store a 32 x 32 block of fp32 C and, as bf16, its gelu (an MLP's hidden layer: the activation is the operand of the
// next product, so the epilogue writes it beside C instead of a pass that reads C back).  Bound by the arithmetic of the
// distribution function (about 30 instructions per element on eight warps): 11.0 us per 256 x 256 pair tile instead of
// 3.9, mostly behind the next main loop (32 K blocks: 15.6 instead of 14.1 us).  4096 x 8192 x 2048: 126 us with the
// activation, against 109 for the product, 43 for the activation and 26 for its conversion as separate passes.
__device__ __forceinline__ void store_chunk_f32_gelu(float* sb, const uint32_t (&v)[32], int lane, float* c_base,
                                                     __nv_bfloat16* act_base, int64_t ldc, int rows_valid) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(sb + epi_off(lane, j)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  const int rsub = lane >> 3, cseg = (lane & 7) * 4;
#pragma unroll 4
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + rsub;
    if (r < rows_valid) {
      const float4 x = *reinterpret_cast<const float4*>(sb + epi_off(r, lane & 7));
      // C is not what the next product reads: it should leave L2 before the activation does
      __stcs(reinterpret_cast<float4*>(c_base + r * ldc + cseg), x);
      *reinterpret_cast<uint2*>(act_base + r * ldc + cseg) =
          make_uint2(pack_bf16x2(gelu_erf(x.x), gelu_erf(x.y)), pack_bf16x2(gelu_erf(x.z), gelu_erf(x.w)));
    }
  }
  __syncwarp();
}

// The drain of a task with an activation output; returns the sum of the lane's row (the checksum's share).  Whole aligned
// 32-column chunks go out as vectors, the rest one row at a time.
__device__ __forceinline__ float epilogue_drain_gelu(uint32_t taddr, const UgTask& t, int row0, int col0, int n_rem,
                                                 float* epi_buf, int lane) {
  float sum = 0.f;
  const int rows_valid = min(32, t.m - row0);
  const int64_t off = static_cast<int64_t>(row0) * t.ldc + col0;
  float* c_base = reinterpret_cast<float*>(t.c_ptr) + off;
  __nv_bfloat16* act_base = reinterpret_cast<__nv_bfloat16*>(t.act_ptr) + off;
#pragma unroll 1
  for (int c = 0; c < n_rem; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
    const int ncols = min(32, n_rem - c);
    if (lane < rows_valid) sum += sum_columns(v, 0, ncols);
    if (task_c_vec(t) && (t.act_ptr & 7u) == 0 && ncols == 32) {
      store_chunk_f32_gelu(epi_buf, v, lane, c_base + c, act_base + c, t.ldc, rows_valid);
      continue;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      *reinterpret_cast<uint4*>(epi_buf + epi_off(lane, j)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    __syncwarp();
    if (lane < ncols) {
      for (int r = 0; r < rows_valid; ++r) {
        const float x = epi_buf[epi_off(r, lane >> 2) + (lane & 3)];
        c_base[r * t.ldc + c + lane] = x;
        act_base[r * t.ldc + c + lane] = __float2bfloat16_rn(gelu_erf(x));
      }
    }
    __syncwarp();
  }
  return sum;
}

// Drain this warp's 32 TMEM lanes x n_rem accumulator columns (first column at `taddr`) into rows row0.. and
// columns col0.. of the task's C.  The common case (fp32 C, 16-byte aligned, whole 32-column chunks) is software
// pipelined: the TMEM load of the next chunk is in flight while the current chunk goes through shared memory.
__device__ __forceinline__ void epilogue_drain(uint32_t taddr, const UgTask& t, int row0, int col0, int n_rem,
                                               int avail, float* epi_buf, int lane, float* acc) {
  const int rows_valid = min(32, t.m - row0);               // <= 0 when the warp is past the region
  if (t.c_dtype == 0 && task_c_pitch_vec(t) &&
      (task_c_rows_indirect(t) || !(task_c_vec(t) && (n_rem & 31) == 0 && (col0 & 3) == 0))) {
    epilogue_drain_f32_shifted(taddr, t, row0, col0, n_rem, avail, epi_buf, lane, acc);
    return;
  }
  if (task_c_vec(t) && t.c_dtype == 0 && (n_rem & 31) == 0) {
    float* c_row = reinterpret_cast<float*>(t.c_ptr) + static_cast<int64_t>(row0) * t.ldc + col0;
    uint32_t va[32], vb[32];
    tmem_ld_32x32(taddr, va);
    for (int c = 0; c < n_rem; c += 64) {
      tmem_ld_wait();
      const bool second = c + 32 < n_rem;
      if (second) tmem_ld_32x32(taddr + c + 32, vb);
      if (acc != nullptr && lane < rows_valid) *acc += sum_columns(va, 0, 32);
      store_chunk_f32(epi_buf, va, lane, c_row + c, t.ldc, rows_valid, t.c_mode);
      if (second) {
        tmem_ld_wait();
        if (acc != nullptr && lane < rows_valid) *acc += sum_columns(vb, 0, 32);
        if (c + 64 < n_rem) tmem_ld_32x32(taddr + c + 64, va);
        store_chunk_f32(epi_buf, vb, lane, c_row + c + 32, t.ldc, rows_valid, t.c_mode);
      }
    }
    return;
  }
  for (int c = 0; c < n_rem; c += 32) {
    if (t.c_dtype == 1 && task_c_vec(t) && n_rem - c >= 64) {
      // bf16 output: two 32-column loads make one 128-byte row segment per row
      uint32_t v0[32], v1[32];
      tmem_ld_32x32(taddr + c, v0);
      tmem_ld_32x32(taddr + c + 32, v1);
      tmem_ld_wait();
      if (acc != nullptr && lane < rows_valid) *acc += sum_columns(v0, 0, 32) + sum_columns(v1, 0, 32);
      store_chunk_bf16_64(epi_buf, v0, v1, lane,
                          reinterpret_cast<__nv_bfloat16*>(t.c_ptr) + static_cast<int64_t>(row0) * t.ldc + col0 + c,
                          t.ldc, rows_valid, task_chunk_mode(t));
      c += 32;
      continue;
    }
    uint32_t v[32];
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
    const int ncols = min(32, n_rem - c);
    if (acc != nullptr && lane < rows_valid) *acc += sum_columns(v, 0, ncols);
    const int64_t off0 = static_cast<int64_t>(row0) * t.ldc + col0 + c;
    if (task_c_vec(t) && ncols == 32) {
      if (t.c_dtype == 0)
        store_chunk_f32(epi_buf, v, lane, reinterpret_cast<float*>(t.c_ptr) + off0, t.ldc, rows_valid, t.c_mode);
      else
        store_chunk_bf16(epi_buf, v, lane, reinterpret_cast<__nv_bfloat16*>(t.c_ptr) + off0, t.ldc, rows_valid,
                         task_chunk_mode(t));
    } else {
      store_chunk_scalar(epi_buf, v, lane, t.c_ptr, off0, t.ldc, rows_valid, ncols, t.c_mode, t.c_dtype);
    }
  }
}

// Add an epilogue warp's checksum share of one tile to the launch's checksum (a double in device memory).
__device__ __forceinline__ void checksum_flush(uint64_t checksum_ptr, float acc, int lane) {
  if (checksum_ptr == 0) return;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (lane == 0) atomicAdd(reinterpret_cast<double*>(checksum_ptr), static_cast<double>(acc));
}

}  // namespace ugfused
