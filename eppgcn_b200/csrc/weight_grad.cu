// Weight gradient of a layer:  dw[k][c] += sum over rows r of f(x[r][k]) * d[r][c]
// (the X^T * d' product of the backward wrapper, EPPGCN_kernel.cu:615).  A tall
// reduction with a tiny result: at best bound by reading the listed rows of x once.
//
// A warp owns 32 * MI values of k and all columns (at most 8 * NT) and adds up 16
// rows per step on the tensor cores, operands split into three bf16 pieces that
// hold every bit (mma_split.cuh); rows are the contracted index, so that a lane
// packs the same element of neighbouring rows.  Rows of x and d come through a
// ring of shared memory that belongs to the warp (cp.async; no block barrier in
// the loop), their ids one step ahead; steps are dealt round-robin, so that at any
// time the grid reads one contiguous window of the (listed) rows.  Lane t of a
// group takes rows t, t + 4, t + 8, t + 12, and rows of a stage lie 32 bytes modulo
// 128 apart: 8 lanes reading 16 bytes touch all banks.  At the end the warps of a
// block add their tiles in shared memory, and the block issues one vector atomic
// per four elements.
//
// By FMA (a lane with 4 x 16 accumulators, one outer product per row) this took
// about 150 instructions per row of 128 features, mostly staging in pieces whose
// alignment was looked up per piece, and was bound by their issue.
#include "mma_split.cuh"

namespace epp {
namespace {

constexpr int kWgWarps = 8;

struct WeightGradArgs {
  float *dw;
  long long ld_dw;
  const float *x;
  long long ldx;
  const float *d;
  long long ldd;
  const int *rows;                 // row ids, or NULL: rows 0 .. n - 1
  int n, k, dout;
  bool relu_x, x_vec, d_vec, dw_vec;
  ClockMark mark;
};

template <int NT, int MI>
struct WeightGradShape {
  static constexpr int RESIDENT = NT <= 2 || (NT == 3 && MI == 1) ? 2 : 1;             // blocks per SM
  static constexpr int STAGES = RESIDENT == 2 ? 2 : 3;
  static constexpr int XS = 32 * MI + 8;                       // floats between rows of x: 32 bytes modulo 128
  static constexpr int DS = NT == 1 ? 8 : NT <= 3 ? 24 : NT <= 5 ? 40 : NT <= 7 ? 56 : 72;   // of d: 8 or 24 words modulo 32
  static constexpr int STAGE = 16 * (XS + DS);
  static constexpr int RING = STAGES * STAGE;
  static constexpr int SMEM = 4 * kWgWarps * RING;
  static_assert(32 * MI * 8 * NT <= RING, "a warp's tile takes the place of its ring");
  static_assert(SMEM <= (RESIDENT == 2 ? 113 : 227) * 1024, "shared memory of a block");
};

template <int NT, int MI>
__global__ void __launch_bounds__(kWgWarps * 32, (WeightGradShape<NT, MI>::RESIDENT)) weight_grad_kernel(const WeightGradArgs a) {
  using Shape = WeightGradShape<NT, MI>;
  constexpr int S = Shape::STAGES, XS = Shape::XS, DS = Shape::DS, QUADS = 2 * NT;
  extern __shared__ __align__(16) float wg_smem[];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) clock_begin(a.mark);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  float *const ring = wg_smem + warp * Shape::RING;
  const unsigned ring_addr = static_cast<unsigned>(__cvta_generic_to_shared(ring));
  const int k0 = blockIdx.y * 32 * MI;
  const int k_have = min(32 * MI, a.k - k0);
  const int all = static_cast<int>((static_cast<long long>(a.n) + 15) / 16);
  const int stride = static_cast<int>(gridDim.x) * kWgWarps;
  const int first = static_cast<int>(blockIdx.x) * kWgWarps + warp;

  // ids of the 16 rows of a step, in lanes 0 - 15; -1: no row
  auto load_ids = [&](int step) {
    const long long at = static_cast<long long>(step) * 16 + (lane & 15);
    if (step >= all || at >= a.n) return -1;
    return a.rows ? __ldg(a.rows + at) : static_cast<int>(at);
  };
  int s_step = first, s_slot = 0, ids = load_ids(first);
  auto stage = [&]() {
    if (s_step < all) {
      const unsigned xs = ring_addr + s_slot * (Shape::STAGE * 4), ds = xs + 16 * XS * 4;
      if (a.x_vec) {
        constexpr int PER_ROW = 8 * MI, ROWS = 32 / PER_ROW;       // 16-byte pieces of a row, rows per instruction
        const int c = lane % PER_ROW * 4, bytes = max(0, min(4, k_have - c)) * 4;
#pragma unroll
        for (int i = 0; i < 16 / ROWS; ++i) {
          const int r = i * ROWS + lane / PER_ROW, id = __shfl_sync(kFull, ids, r);
          const bool in = id >= 0 && bytes > 0;
          cp16_some(xs + (r * XS + c) * 4, in ? a.x + id * a.ldx + k0 + c : a.x, in ? bytes : 0);
        }
      } else {
#pragma unroll 4
        for (int r = 0; r < 16; ++r) {
          const int id = __shfl_sync(kFull, ids, r);
#pragma unroll
          for (int i = 0; i < MI; ++i) {
            const int c = i * 32 + lane;
            const bool in = id >= 0 && c < k_have;
            cp4_some(xs + (r * XS + c) * 4, in ? a.x + id * a.ldx + k0 + c : a.x, in ? 4 : 0);
          }
        }
      }
      if (a.d_vec) {
#pragma unroll
        for (int i = 0; i < (16 * QUADS + 31) / 32; ++i) {
          const int e = i * 32 + lane, r = e / QUADS, c = e % QUADS * 4, id = __shfl_sync(kFull, ids, r & 15);
          const bool in = id >= 0 && c < a.dout;
          if (16 * QUADS % 32 == 0 || r < 16)
            cp16_some(ds + (r * DS + c) * 4, in ? a.d + id * a.ldd + c : a.d, in ? min(4, a.dout - c) * 4 : 0);
        }
      } else {
#pragma unroll 4
        for (int i = 0; i < 4 * NT; ++i) {
          const int e = i * 32 + lane, r = e / (8 * NT), c = e % (8 * NT), id = __shfl_sync(kFull, ids, r);
          const bool in = id >= 0 && c < a.dout;
          cp4_some(ds + (r * DS + c) * 4, in ? a.d + id * a.ldd + c : a.d, in ? 4 : 0);
        }
      }
      s_slot = s_slot + 1 == S ? 0 : s_slot + 1;
      s_step += stride;
      ids = load_ids(s_step);
    }
    cp_commit();
  };

  float top[NT][MI][2][4], rest[NT][MI][2][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) top[j][i][m][q] = rest[j][i][m][q] = 0.f;
#pragma unroll
  for (int u = 0; u < S - 1; ++u) stage();
  int slot = 0;
  for (int step = first; step < all; step += stride) {
    stage();
    cp_wait<S - 1>();
    __syncwarp();
    const float *xs = ring + slot * Shape::STAGE + t * XS + 4 * g, *ds = ring + slot * Shape::STAGE + 16 * XS + t * DS + g;
    slot = slot + 1 == S ? 0 : slot + 1;
    uint2 w[MI == 1 ? 1 : NT][3];
    auto split_d = [&](int j, uint2 (&f)[3]) {
      split3(ds[8 * j], ds[8 * j + 4 * DS], f[0].x, f[1].x, f[2].x);
      split3(ds[8 * j + 8 * DS], ds[8 * j + 12 * DS], f[0].y, f[1].y, f[2].y);
    };
    if constexpr (MI > 1) {
#pragma unroll
      for (int j = 0; j < NT; ++j) split_d(j, w[j]);
    }
    // two 16 x 16 pieces of x^T at a time: elements 32i + 4g and + 1 of each row, elements + 2 and + 3
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      float4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q] = *reinterpret_cast<const float4 *>(xs + 4 * q * XS + 32 * i);
        if (a.relu_x) v[q] = relu4(v[q]);
      }
      unsigned x[2][3][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {                    // rows t, t + 4, then t + 8, t + 12
        const float4 &u = v[2 * h], &o = v[2 * h + 1];
        split3(u.x, o.x, x[0][0][2 * h], x[0][1][2 * h], x[0][2][2 * h]);
        split3(u.y, o.y, x[0][0][2 * h + 1], x[0][1][2 * h + 1], x[0][2][2 * h + 1]);
        split3(u.z, o.z, x[1][0][2 * h], x[1][1][2 * h], x[1][2][2 * h]);
        split3(u.w, o.w, x[1][0][2 * h + 1], x[1][1][2 * h + 1], x[1][2][2 * h + 1]);
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        uint2 (&f)[3] = w[MI == 1 ? 0 : j];
        if constexpr (MI == 1) split_d(j, f);
        multiply_split(top[j][i], rest[j][i], x, f[0], f[1], f[2]);
      }
    }
    __syncwarp();          // the slot is copied over by the next stage()
  }
  cp_wait<0>();
  __syncthreads();         // every ring is drained: the warps' tiles of dw take their places
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < NT; ++j)
          *reinterpret_cast<float2 *>(ring + (32 * i + 4 * g + 2 * m + h) * (8 * NT) + 8 * j + 2 * t) =
              make_float2(top[j][i][m][2 * h] + rest[j][i][m][2 * h], top[j][i][m][2 * h + 1] + rest[j][i][m][2 * h + 1]);
  __syncthreads();
  constexpr int PIECES = (32 * MI * QUADS + kWgWarps * 32 - 1) / (kWgWarps * 32);      // of four columns, per thread
  float4 v[PIECES];
  bool bad = false;
  // has() of a piece: e = threadIdx.x + i * blockDim.x, element (e / QUADS, e % QUADS * 4) of the block's tile
  auto has = [&](int e, int q) { return e < k_have * QUADS && e % QUADS * 4 + q < a.dout; };
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int e = threadIdx.x + i * kWgWarps * 32;
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!has(e, 0)) continue;
    for (int w = 0; w < kWgWarps; ++w) {
      const float4 o = *reinterpret_cast<const float4 *>(wg_smem + w * Shape::RING + e / QUADS * (8 * NT) + e % QUADS * 4);
      v[i].x += o.x; v[i].y += o.y; v[i].z += o.z; v[i].w += o.w;
    }
    bad |= isnan(v[i].x) || (has(e, 1) && isnan(v[i].y)) || (has(e, 2) && isnan(v[i].z)) || (has(e, 3) && isnan(v[i].w));
  }
  if (__syncthreads_or(bad)) {
    // An infinity or a NaN among the operands: the block's rows once more through the rings, by FMA, until every result that
    // is to be replaced has become NaN here too or the rows end.  2 M x 128 -> 16: 254 us without a NaN, 264 where d' or x
    // is NaN throughout, 690 with one infinity in x, 1030 with one in d' (a thread that walked all rows of its block for
    // every four results: 6.8 to 7.1 ms).
    float4 sum[PIECES];
#pragma unroll
    for (int i = 0; i < PIECES; ++i) sum[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    s_step = first;
    s_slot = 0;
    ids = load_ids(first);
#pragma unroll 1
    for (int u = 0; u < S - 1; ++u) stage();
    const float *at = wg_smem;
    for (int step = static_cast<int>(blockIdx.x) * kWgWarps; step < all; step += stride) {
      stage();
      cp_wait<S - 1>();
      __syncthreads();
      const int warps = min(kWgWarps, all - step);     // that have a step
      bool open = false;
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const int e = threadIdx.x + i * kWgWarps * 32;
        if (!has(e, 0)) continue;
        for (int w = 0; w < warps; ++w) {
          const float *x_at = at + w * Shape::RING + e / QUADS, *d_at = at + w * Shape::RING + 16 * XS + e % QUADS * 4;
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            const float xk = a.relu_x ? max_nan(x_at[r * XS], 0.f) : x_at[r * XS];
            const float4 d4 = *reinterpret_cast<const float4 *>(d_at + r * DS);
            sum[i].x = fmaf(xk, d4.x, sum[i].x);
            sum[i].y = fmaf(xk, d4.y, sum[i].y);
            sum[i].z = fmaf(xk, d4.z, sum[i].z);
            sum[i].w = fmaf(xk, d4.w, sum[i].w);
          }
        }
        open |= (isnan(v[i].x) && !isnan(sum[i].x)) || (has(e, 1) && isnan(v[i].y) && !isnan(sum[i].y)) ||
                (has(e, 2) && isnan(v[i].z) && !isnan(sum[i].z)) || (has(e, 3) && isnan(v[i].w) && !isnan(sum[i].w));
      }
      if (!__syncthreads_or(open)) break;
      at = at == wg_smem + (S - 1) * Shape::STAGE ? wg_smem : at + Shape::STAGE;
    }
    cp_wait<0>();
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
      if (isnan(v[i].x)) v[i].x = sum[i].x;
      if (isnan(v[i].y)) v[i].y = sum[i].y;
      if (isnan(v[i].z)) v[i].z = sum[i].z;
      if (isnan(v[i].w)) v[i].w = sum[i].w;
    }
  }
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int e = threadIdx.x + i * kWgWarps * 32, c = e % QUADS * 4;
    if (!has(e, 0)) continue;
    float *dst = a.dw + (k0 + e / QUADS) * a.ld_dw + c;
    if (a.dw_vec && c + 4 <= a.dout) {
      atomicAdd(reinterpret_cast<float4 *>(dst), v[i]);
    } else {
      const float o[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (c + q < a.dout) atomicAdd(dst + q, o[q]);
    }
  }
  if (threadIdx.x == 0) clock_end(a.mark);
}

template <int NT, int MI>
int launch_weight_grad(const WeightGradArgs &a, int sms, cudaStream_t s) {
  using Shape = WeightGradShape<NT, MI>;
  static SmemOptIn memo;                         // per instantiation; remembers the opt-in per device
  if (const int rc = smem_opt_in(memo, reinterpret_cast<const void *>(weight_grad_kernel<NT, MI>), Shape::SMEM); rc != EPP_OK)
    return rc;
  // one wave: as many blocks per slab of k as the chip holds, no warp without a step
  const long long slabs = ceil_div_ll(a.k, 32 * MI), steps = ceil_div_ll(a.n, 16);
  long long per_slab = static_cast<long long>(sms) * Shape::RESIDENT / slabs;
  if (per_slab > ceil_div_ll(steps, kWgWarps)) per_slab = ceil_div_ll(steps, kWgWarps);
  if (per_slab < 1) per_slab = 1;
  const dim3 grid(static_cast<unsigned>(per_slab), static_cast<unsigned>(slabs));
  weight_grad_kernel<NT, MI><<<grid, kWgWarps * 32, Shape::SMEM, s>>>(a);
  EPP_CHECK_LAUNCH("weight_grad_kernel");
  return EPP_OK;
}

// 64 values of k per warp while their accumulators leave room in the register file, 32 for wide results, short rows and
// 65 .. 96 values, where a second slab of 64 would be half empty (1.13 M x 96 -> 16: 137 us, 120).
template <int NT>
int weight_grad_block(const WeightGradArgs &a, int sms, cudaStream_t s) {
  if constexpr (NT <= 4) {
    if (a.k > 32 && (a.k <= 64 || a.k > 96)) return launch_weight_grad<NT, 2>(a, sms, s);
  }
  return launch_weight_grad<NT, 1>(a, sms, s);
}

}  // namespace
}  // namespace epp

EPP_EXPORT int eppgcn_weight_grad_add(float *dw, const float *x, long long ldx, const float *d, long long ldd,
                                      const int *rows, int num_rows, int k, int dout, int relu_x, void *stream) {
  using namespace epp;
  EPP_REQUIRE(num_rows >= 0 && k >= 1 && dout >= 1, "negative size, k < 1 or dout < 1");
  EPP_REQUIRE(dw, "null pointer");
  if (num_rows == 0) return EPP_OK;
  EPP_REQUIRE(x && d && ldx >= k && ldd >= dout, "null pointer or row stride smaller than the row");
  EPP_REQUIRE(aligned(x, 16) && aligned(d, 16), "x and d must be 16-byte aligned");
  EPP_REQUIRE(k <= 65535 * 32, "more than 2 097 120 columns of x");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int sms = 148;
  if (const int rc = device_sm_count(&sms); rc != EPP_OK) return rc;
  // blocks of at most 64 columns, about equally wide
  const int blocks = (dout + 63) / 64, width = ((dout + blocks - 1) / blocks + 7) / 8 * 8;
  for (int c0 = 0; c0 < dout; c0 += width) {
    WeightGradArgs a{};
    a.dw = dw + c0; a.ld_dw = dout; a.x = x; a.ldx = ldx; a.d = d + c0; a.ldd = ldd; a.rows = rows;
    a.n = num_rows; a.k = k; a.dout = dout - c0 < width ? dout - c0 : width;
    a.relu_x = relu_x != 0;
    a.x_vec = ldx % 4 == 0;
    a.d_vec = ldd % 4 == 0;
    a.dw_vec = dout % 4 == 0 && aligned(dw, 16);
    a.mark = take_mark();
    int rc;
    switch ((a.dout + 7) / 8) {
      case 1:  rc = weight_grad_block<1>(a, sms, s); break;
      case 2:  rc = weight_grad_block<2>(a, sms, s); break;
      case 3:  rc = weight_grad_block<3>(a, sms, s); break;
      case 4:  rc = weight_grad_block<4>(a, sms, s); break;
      case 5:  rc = weight_grad_block<5>(a, sms, s); break;
      case 6:  rc = weight_grad_block<6>(a, sms, s); break;
      case 7:  rc = weight_grad_block<7>(a, sms, s); break;
      default: rc = weight_grad_block<8>(a, sms, s); break;
    }
    if (rc != EPP_OK) return rc;
  }
  return EPP_OK;
}

static int weight_grad_impl(float *dw, const float *x, long long ldx, const float *d, long long ldd,
                            const int *row_list, int num_rows, int k, int dout, void *stream) {
  using namespace epp;
  EPP_REQUIRE(num_rows >= 0 && k >= 1 && dout >= 1, "negative size, k < 1 or dout < 1");
  if (dout > 32 || ((k + 3) / 4) * ((dout + 3) / 4) > 256) {
    set_error("eppgcn_weight_grad handles dout <= 32 and k * dout <= 4096, got k = %d, dout = %d", k, dout);
    return EPP_ERR_TOO_LARGE;
  }
  EPP_REQUIRE(dw, "null pointer");
  EPP_CUDA_TRY(cudaMemsetAsync(dw, 0, sizeof(float) * static_cast<size_t>(k) * dout, static_cast<cudaStream_t>(stream)));
  return eppgcn_weight_grad_add(dw, x, ldx, d, ldd, row_list, num_rows, k, dout, 0, stream);
}

EPP_EXPORT int eppgcn_weight_grad(float *dw, const float *x, long long ldx, const float *d, long long ldd,
                                  int num_rows, int k, int dout, void *stream) {
  return weight_grad_impl(dw, x, ldx, d, ldd, nullptr, num_rows, k, dout, stream);
}

EPP_EXPORT int eppgcn_weight_grad_rows(float *dw, const float *x, long long ldx, const float *d, long long ldd,
                                       const int *rows, int num_listed, int k, int dout, void *stream) {
  if (num_listed > 0 && !rows) {
    epp::set_error("eppgcn_weight_grad_rows: null row list");
    return EPP_ERR_BAD_ARG;
  }
  return weight_grad_impl(dw, x, ldx, d, ldd, num_listed > 0 ? rows : nullptr, num_listed, k, dout, stream);
}
