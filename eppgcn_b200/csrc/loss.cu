// Loss of the training step and its gradient, in one pass over the rows that matter:
//
//   loss = mean over labelled rows r of  logsumexp(z[r]) - z[r][y[r]]
//   grad[r] = scale[r] * (softmax(z[r]) - onehot(y[r]))            (times 1/count, applied at the end)
//
// The reference writes log_softmax over every row, gathers the labelled ones by a boolean index, takes nll_loss and
// lets autograd walk back (EPPGCN/gcn_main.py:239-240,256): nine passes over [N, classes] matrices, a sort for the
// accumulating index backward and three host synchronisations for the boolean index.  Here a labelled row is read
// once and its gradient is written once, already multiplied by the source-side factor and in the padded rows that the
// last layer's backward aggregation gathers; rows without a label are not touched (only those that the execution path
// names and the mask does not are cleared).  Bound by the sectors of the labelled rows.
//
// The mean's divisor is only known when every row has been seen.  The whole backward is linear in it, so gradients
// travel without it and mean_grads_kernel multiplies the finished weight gradients, a few thousand values.
#include "rowio.cuh"

namespace epp {
namespace {

constexpr long long kIgnoredLabel = -100;     // nll_loss's ignore_index: such rows are neither summed nor counted

// Block's share of {sum, count}; `loss` per lane, `count` per warp.
__device__ __forceinline__ void add_loss(double loss, int count, double *sums) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) loss += __shfl_xor_sync(kFull, loss, off);
  __shared__ double s_loss[8];
  __shared__ int s_count[8];
  if ((threadIdx.x & 31) == 0) {
    s_loss[threadIdx.x >> 5] = loss;
    s_count[threadIdx.x >> 5] = count;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) {
      loss += s_loss[i];
      count += s_count[i];
    }
    if (count) {
      atomicAdd(sums, loss);
      atomicAdd(sums + 1, static_cast<double>(count));
    }
  }
}

// Up to 64 columns.  A warp reads the flags of 32 rows at a time and queues the rows that have something to do; as soon
// as 32 are queued every lane takes one, whole, in registers.  Eight lanes per row with shuffles between them spent 970
// instructions on 32 rows, queued or not: 110 us on 2 M rows x 22 classes with 10 % of them labelled, 40 now (104 with half).
template <int QUADS>
__global__ void __launch_bounds__(256) masked_nll_kernel(const float *__restrict__ z, long long ldz,
                                                         const long long *__restrict__ labels,
                                                         const unsigned char *__restrict__ mask, int n, int classes,
                                                         float *__restrict__ grad, long long ldg,
                                                         const unsigned char *__restrict__ used,
                                                         const float *__restrict__ scale, double *sums, int align, const ClearList clear) {
  clear_rows(clear);
  constexpr int kUnlabelled = -1, kWrongLabel = -2;
  __shared__ int s_row[8][64], s_label[8][64];        // row | top bit where its gradient is wanted; label
  const int lane = threadIdx.x & 31, warp_in_block = threadIdx.x >> 5;
  int *const q_row = s_row[warp_in_block], *const q_label = s_label[warp_in_block];
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  double loss = 0.0;
  int count = 0;

  auto work = [&](int entry, int y) {
    const long long row = entry & 0x7fffffff;
    float v[QUADS][4];
    float factor = 0.f;
    if (y != kUnlabelled) {
      const float *p = z + row * ldz;
#pragma unroll
      for (int i = 0; i < QUADS; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = -INFINITY;
        const int have = classes - 4 * i;
        if (have <= 0) continue;
        if (align == 4) {                             // padded rows: 16 bytes even where fewer columns exist
          const float4 t = __ldg(reinterpret_cast<const float4 *>(p + 4 * i));
          v[i][0] = t.x;
          if (have > 1) v[i][1] = t.y;
          if (have > 2) v[i][2] = t.z;
          if (have > 3) v[i][3] = t.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < have) v[i][j] = __ldg(p + 4 * i + j);
        }
      }
      float top = -INFINITY, picked = 0.f, sum = 0.f;
#pragma unroll
      for (int i = 0; i < QUADS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) top = fmaxf(top, v[i][j]);
#pragma unroll
      for (int i = 0; i < QUADS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (4 * i + j >= classes) continue;
          if (4 * i + j == y) picked = v[i][j];
          v[i][j] = v[i][j] - top;
          sum += expf(v[i][j]);
        }
      const float log_sum = logf(sum);
      loss += y == kWrongLabel ? static_cast<double>(NAN) : static_cast<double>(log_sum - (picked - top));
      factor = entry < 0 && scale ? __ldg(scale + row) : 1.f;
#pragma unroll
      for (int i = 0; i < QUADS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[i][j] = 4 * i + j < classes ? (expf(v[i][j] - log_sum) - (4 * i + j == y ? 1.f : 0.f)) * factor : 0.f;
    }
    if (entry >= 0) return;
#pragma unroll
    for (int i = 0; i < QUADS; ++i)
      if (4 * i < ldg)
        *reinterpret_cast<float4 *>(grad + row * ldg + 4 * i) =
            y == kUnlabelled ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
  };

  int queued = 0;
  for (long long base = warp * kWarp; base < n; base += warps * kWarp) {
    const long long r = base + lane;
    const bool in = r < n, wanted = in && used[r] != 0;
    const long long y = in && mask[r] != 0 ? __ldg(labels + r) : kIgnoredLabel;
    const bool labelled = y != kIgnoredLabel;
    const unsigned todo = __ballot_sync(kFull, wanted || labelled);
    count += __popc(__ballot_sync(kFull, labelled));
    if (wanted || labelled) {
      const int at = queued + __popc(todo & ((1u << lane) - 1u));
      q_row[at] = static_cast<int>(static_cast<unsigned>(r) | (wanted ? 0x80000000u : 0u));
      q_label[at] = !labelled ? kUnlabelled : (y >= 0 && y < classes ? static_cast<int>(y) : kWrongLabel);
    }
    queued += __popc(todo);
    __syncwarp();
    if (queued >= kWarp) {
      work(q_row[lane], q_label[lane]);
      queued -= kWarp;
      const int moved_row = q_row[kWarp + lane], moved_label = q_label[kWarp + lane];
      __syncwarp();
      if (lane < queued) {
        q_row[lane] = moved_row;
        q_label[lane] = moved_label;
      }
      __syncwarp();
    }
  }
  if (lane < queued) work(q_row[lane], q_label[lane]);
  add_loss(loss, count, sums);
}

// More columns: a warp per row, lane l its columns 4 * (l + 32 * v) .. + 3 for v < NV.
template <int NV>
__global__ void __launch_bounds__(256) masked_nll_wide_kernel(const float *__restrict__ z, long long ldz,
                                                              const long long *__restrict__ labels,
                                                              const unsigned char *__restrict__ mask, int n, int classes,
                                                              float *__restrict__ grad, long long ldg,
                                                              const unsigned char *__restrict__ used,
                                                              const float *__restrict__ scale, double *sums, int align, const ClearList clear) {
  clear_rows(clear);
  const int lane = threadIdx.x & 31;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  double loss = 0.0;
  int count = 0;
  for (long long row = warp; row < n; row += warps) {
    const long long label = mask[row] != 0 ? __ldg(labels + row) : kIgnoredLabel;
    const bool labelled = label != kIgnoredLabel, wanted = used[row] != 0;
    if (!labelled && !wanted) continue;
    count += labelled;
    float v[NV][4];
    float top = -INFINITY, sum = 0.f, picked = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c0 = 4 * (lane + 32 * i), have = labelled ? classes - c0 : 0;
      const float *p = z + row * ldz + c0;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = -INFINITY;
      if (have > 0 && align == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
        v[i][0] = t.x;
        if (have > 1) v[i][1] = t.y;
        if (have > 2) v[i][2] = t.z;
        if (have > 3) v[i][3] = t.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < have) v[i][j] = __ldg(p + j);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) top = fmaxf(top, v[i][j]);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) top = fmaxf(top, __shfl_xor_sync(kFull, top, off));
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = 4 * (lane + 32 * i) + j;
        if (!labelled || c >= classes) continue;
        if (c == label) picked = v[i][j];
        v[i][j] = v[i][j] - top;
        sum += expf(v[i][j]);
      }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      sum += __shfl_xor_sync(kFull, sum, off);
      picked += __shfl_xor_sync(kFull, picked, off);
    }
    const float log_sum = logf(sum);
    if (labelled && lane == 0)
      loss += label >= 0 && label < classes ? static_cast<double>(log_sum - (picked - top)) : static_cast<double>(NAN);
    if (!wanted) continue;
    const float s = scale ? __ldg(scale + row) : 1.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c0 = 4 * (lane + 32 * i);
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        o[j] = labelled && c0 + j < classes ? (expf(v[i][j] - log_sum) - (c0 + j == label ? 1.f : 0.f)) * s : 0.f;
      if (c0 < ldg) *reinterpret_cast<float4 *>(grad + row * ldg + c0) = make_float4(o[0], o[1], o[2], o[3]);
    }
  }
  add_loss(loss, count, sums);
}

constexpr int kGradsPerLaunch = 12;
struct GradList {
  const float *sum[kGradsPerLaunch];
  float *grad[kGradsPerLaunch];
  int end[kGradsPerLaunch];       // running totals of the element counts
  int count;
};

// grad = sum / rows for every listed matrix, and the mean loss; without a labelled row the loss is NaN, as nll_loss's.
__global__ void __launch_bounds__(256) mean_grads_kernel(const GradList g, const double *__restrict__ sums,
                                                         float *loss) {
  const double rows = sums[1];
  const float inv = rows > 0 ? static_cast<float>(1.0 / rows) : 0.f;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (loss && i == 0) *loss = static_cast<float>(sums[0] / rows);
  int k = 0;
  while (k < g.count && i >= g.end[k]) ++k;
  if (k == g.count) return;
  const int at = i - (k ? g.end[k - 1] : 0);
  g.grad[k][at] = g.sum[k][at] * inv;
}

}  // namespace
}  // namespace epp

using namespace epp;

EPP_EXPORT int eppgcn_masked_nll(float *grad, long long grad_ld, double *sums, const float *logits, long long ld,
                                 const long long *labels, const unsigned char *mask, const unsigned char *used,
                                 const float *row_scale, int num_rows, int num_classes, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(num_rows >= 0 && num_classes >= 1, "negative size or no class");
  if (num_classes > 1024) {
    set_error("eppgcn_masked_nll handles at most 1024 classes, got %d", num_classes);
    return EPP_ERR_TOO_LARGE;
  }
  if (num_rows == 0) return EPP_OK;
  EPP_REQUIRE(grad && sums && logits && labels && mask && used, "null pointer");
  EPP_REQUIRE(ld >= num_classes, "row stride smaller than the row");
  EPP_REQUIRE(grad_ld % 4 == 0 && grad_ld >= (num_classes + 3) / 4 * 4 && aligned(grad, 16),
              "gradient rows must be 16-byte aligned and padded to a multiple of 4 floats");
  const int align = ld % 4 == 0 && ld >= (num_classes + 3) / 4 * 4 && aligned(logits, 16) ? 4 : 1;
  long long blocks = ceil_div_ll(num_rows, 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  const unsigned g = static_cast<unsigned>(blocks);
  const ClearList clear = take_clear(s);
  auto run = [&](auto kernel) {
    kernel<<<g, 256, 0, s>>>(logits, ld, labels, mask, num_rows, num_classes, grad, grad_ld, used, row_scale, sums, align,
                          clear);
  };
  // a lane holds a gradient row, padding included, while that leaves room for the warps that hide each other's loads
  if (grad_ld <= 8) run(masked_nll_kernel<2>);
  else if (grad_ld <= 16) run(masked_nll_kernel<4>);
  else if (grad_ld <= 24) run(masked_nll_kernel<6>);
  else if (grad_ld <= 32) run(masked_nll_kernel<8>);
  else if (grad_ld <= 48) run(masked_nll_kernel<12>);
  else if (grad_ld <= 64) run(masked_nll_kernel<16>);
  else if (num_classes <= 256) run(masked_nll_wide_kernel<2>);
  else run(masked_nll_wide_kernel<8>);
  EPP_CHECK_LAUNCH("masked_nll_kernel");
  return EPP_OK;
}

EPP_EXPORT int eppgcn_mean_grads(float *loss, int count, const float *const *sums_of, float *const *grads,
                                 const int *sizes, const double *sums, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(count >= 0 && loss && sums, "bad argument");
  EPP_REQUIRE(count == 0 || (sums_of && grads && sizes), "null pointer");
  for (int first = 0; first == 0 || first < count; first += kGradsPerLaunch) {
    GradList g{};
    long long total = 0;
    for (int k = first; k < count && k < first + kGradsPerLaunch; ++k) {
      EPP_REQUIRE(sums_of[k] && grads[k] && sizes[k] >= 0, "null pointer or negative size");
      total += sizes[k];
      EPP_REQUIRE(total < (1LL << 31), "gradients exceed int32");
      g.sum[g.count] = sums_of[k];
      g.grad[g.count] = grads[k];
      g.end[g.count++] = static_cast<int>(total);
    }
    const long long blocks = ceil_div_ll(total > 0 ? total : 1, 256);
    mean_grads_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(g, sums, first == 0 ? loss : nullptr);
    EPP_CHECK_LAUNCH("mean_grads_kernel");
  }
  return EPP_OK;
}
