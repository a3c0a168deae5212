// Shared helpers of the eppgcn_b200 C-ABI library: status plumbing, launch
// checks and the packed tile descriptor used by the single-pass scans.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/eppgcn_b200.h"

// Entry points are the only symbols the shared library exports.
#define EPP_EXPORT extern "C" __attribute__((visibility("default")))

namespace epp {

void set_error(const char *fmt, ...);

#define EPP_CUDA_TRY(expr)                                                        \
  do {                                                                            \
    cudaError_t _e = (expr);                                                      \
    if (_e != cudaSuccess) {                                                      \
      ::epp::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),    \
                       __FILE__, __LINE__);                                       \
      return EPP_ERR_CUDA;                                                        \
    }                                                                             \
  } while (0)

#define EPP_CHECK_LAUNCH(name)                                                    \
  do {                                                                            \
    cudaError_t _e = cudaPeekAtLastError();                                       \
    if (_e != cudaSuccess) {                                                      \
      ::epp::set_error("launch of %s failed: %s", name, cudaGetErrorString(_e));  \
      (void)cudaGetLastError();                                                   \
      return EPP_ERR_CUDA;                                                        \
    }                                                                             \
  } while (0)

#define EPP_REQUIRE(cond, msg)                                                    \
  do {                                                                            \
    if (!(cond)) {                                                                \
      ::epp::set_error("%s: %s", __func__, msg);                                  \
      return EPP_ERR_BAD_ARG;                                                     \
    }                                                                             \
  } while (0)

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

__host__ __device__ inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }

// Flag words another GPU writes or reads: release / acquire at system scope.
__device__ __forceinline__ void store_release_sys(unsigned *p, unsigned v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned load_acquire_sys(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ---------------------------------------------------------------------------
// Device-side clock of a stream, behind the same print_time keys as the event
// timers of single operators.  Two events per operation and their resolution
// cost a third of a small graph's epoch on the host, and events cannot be part
// of a replayed graph; here the kernels of an operation leave their own times.
// The first kernel of an operation closes what is open (whose kernels have all
// finished: same stream) and opens its slot, every kernel pushes its slot's end
// forward.  Operations that follow each other use different slots, so that no
// block can push the end of the operation that its kernel's first block is about
// to close: slots 0 and 1 for those that come in pairs (also where a graph replays
// them), 2 and 3 in turn for those that may follow themselves.
// ---------------------------------------------------------------------------
constexpr int kClockSlots = 4;
struct StreamClock {
  unsigned long long start[kClockSlots], end[kClockSlots];     // ns of the global timer
  int category[kClockSlots], layer[kClockSlots];
  alignas(16) int open[kClockSlots];
  unsigned long long acc[11];              // closed operations, indexed like the host's accumulators
};
struct ClockMark {
  StreamClock *clock;                      // NULL: nothing is timed
  int slot, category, layer;               // category -1: not the first kernel of the operation
};
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// One thread of the grid, before its work.
__device__ __forceinline__ void clock_begin(const ClockMark &m) {
  if (!m.clock || m.category < 0) return;
  StreamClock *c = m.clock;
  const int4 all = *reinterpret_cast<const int4 *>(c->open);     // at once: the block's work waits for this
  const int open[kClockSlots] = {all.x, all.y, all.z, all.w};
#pragma unroll
  for (int s = 0; s < kClockSlots; ++s) {
    if (!open[s]) continue;
    const unsigned long long ns = c->end[s] > c->start[s] ? c->end[s] - c->start[s] : 0;
    c->acc[c->category[s]] += ns;
    if (c->category[s] == 2 && c->layer[s] >= 1 && c->layer[s] <= 6) c->acc[4 + c->layer[s]] += ns;
    c->open[s] = 0;
  }
  c->start[m.slot] = global_ns();
  c->category[m.slot] = m.category;
  c->layer[m.slot] = m.layer;
  c->open[m.slot] = 1;
}
// One thread of every block, after its work.
__device__ __forceinline__ void clock_end(const ClockMark &m) {
  if (m.clock) atomicMax(&m.clock->end[m.slot], global_ns());
}
// The mark of the calling thread's current operation for its next kernel (see eppgcn_mark_begin).
ClockMark take_mark();

// ---------------------------------------------------------------------------
// Rows that an aggregation adds to with atomics, and rows without an edge, are cleared in front of it.  A kernel of its
// own for that costs its launch, 2 us in a recorded step and 4 - 6 between others, for a few thousand rows: the kernel that
// runs before the aggregation clears them on its way (eppgcn_clear_begin).
// ---------------------------------------------------------------------------
struct ClearList {
  float *out;                              // rows of ld floats, 16-byte aligned
  long long ld;
  const int *rows;
  int count, quads;                        // rows; 16-byte pieces per row
};
__device__ __forceinline__ void clear_rows(const ClearList &c) {
  const long long total = static_cast<long long>(c.count) * c.quads;
  const long long block = blockIdx.x + static_cast<long long>(gridDim.x) * (blockIdx.y + static_cast<long long>(gridDim.y) * blockIdx.z);
  const long long stride = static_cast<long long>(gridDim.x) * gridDim.y * gridDim.z * blockDim.x;
  for (long long i = block * blockDim.x + threadIdx.x; i < total; i += stride)
    *reinterpret_cast<float4 *>(c.out + __ldg(c.rows + i / c.quads) * c.ld + i % c.quads * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
}
// What the calling thread wants cleared, for its next kernel on the stream; and how it says so.
ClearList take_clear(cudaStream_t s);
void want_clear(const ClearList &c, cudaStream_t s);

// ---------------------------------------------------------------------------
// Tile descriptor of the chained (decoupled look-back) scans.
// One 64-bit word per tile: bits 63..62 state, 61..31 field B, 30..0 field A.
// Both fields are partial sums of int32 totals that the host has checked to be
// below 2^31, so they never carry into each other.
// ---------------------------------------------------------------------------
constexpr unsigned long long kTileEmpty = 0ull;
constexpr unsigned long long kTileAggregate = 1ull;   // sum of this tile only
constexpr unsigned long long kTilePrefix = 2ull;      // sum of tiles 0..this

__host__ __device__ inline unsigned long long tile_pack(unsigned long long state, unsigned a, unsigned b) {
  return (state << 62) | (static_cast<unsigned long long>(b) << 31) | static_cast<unsigned long long>(a);
}
__host__ __device__ inline unsigned tile_state(unsigned long long w) { return static_cast<unsigned>(w >> 62); }
__host__ __device__ inline unsigned tile_a(unsigned long long w) { return static_cast<unsigned>(w & 0x7fffffffull); }
__host__ __device__ inline unsigned tile_b(unsigned long long w) { return static_cast<unsigned>((w >> 31) & 0x7fffffffull); }

// Layout of the scratch buffer handed to the scan entry points.
struct ScanHeader {
  unsigned int ticket;      // next tile id to hand out
  int error;                // EPP_OK or EPP_ERR_SCAN_TIMEOUT
  unsigned int pad[62];     // keeps the descriptors 256-byte aligned
};
static_assert(sizeof(ScanHeader) == 256, "ScanHeader must be 256 bytes");

}  // namespace epp
