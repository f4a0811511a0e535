// Combine kernels: moe_gather (weighted un-permute) and moe_sum.
//
// Pure streaming, bound by HBM: T * k rows in, T rows out, no reuse.  One thread owns one
// 16-byte column of one token, wherever it lies (threads are numbered across row boundaries, so
// no CTA ends in a partly filled pass over its row), and has the same column of all its k source
// rows in flight at once.  A CTA per token, a shared-memory copy of the row numbers and a loop
// over j with one load at a time before it: one token of 8 x 7168 took 11 us on one SM.
#include "common.cuh"

namespace b200moe {
namespace {

constexpr int kMaxTopK = 64;
constexpr int kAhead = 8;   // source rows in flight per thread

struct CombineParams {
  void* out;
  const void* in;
  const float* weights;       // gather
  const int32_t* row_map;     // gather
  const void* addend;         // gather, optional
  const int32_t* num_valid;   // gather, optional
  const void* ids;            // sum, optional
  int ids_dtype;
  const int32_t* expert_map;  // sum, optional
  int k, H, vecs;             // vecs: columns of V elements per row
  int64_t t0;                 // first token of this launch
  uint32_t total;             // (token, column) pairs of this launch
};

// K: rows per token when known at compile time (0: k, in batches of kAhead).
template <typename T, int V, int K, bool GATHER>
__global__ void __launch_bounds__(256) combine_kernel(CombineParams p) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait();
  pdl_trigger();
  if (i >= p.total) return;
  const uint32_t local = i / static_cast<uint32_t>(p.vecs);
  const int64_t t = p.t0 + local;
  if (GATHER && p.num_valid && t >= *p.num_valid) return;  // rows of a worst-case buffer nobody will read
  const int64_t c = static_cast<int64_t>(i - local * p.vecs) * V;
  const int k = K ? K : p.k;
  const T* in = reinterpret_cast<const T*>(p.in);
  float acc[V];
  if (GATHER && p.addend) {  // e.g. the shared expert's row of this token, weight 1
    load_f32<T, V>(reinterpret_cast<const T*>(p.addend) + t * p.H + c, acc);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = 0.f;
  }
  constexpr int B = K ? K : kAhead;
  for (int j0 = 0; j0 < k; j0 += B) {
    int64_t row[B];
    float w[B];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      row[j] = -1;
      w[j] = 1.f;
      if (K || j0 + j < k) {
        const int64_t at = t * k + j0 + j;
        if (GATHER) {
          row[j] = p.row_map[at];
          w[j] = p.weights[at];
        } else {
          row[j] = at;
          if (p.ids) {
            const int64_t id = load_index(p.ids, p.ids_dtype, at);
            if (id < 0 || (p.expert_map && p.expert_map[id] < 0)) row[j] = -1;
          }
        }
      }
    }
    Vec<T, V> v[B];
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (row[j] >= 0) v[j] = *reinterpret_cast<const Vec<T, V>*>(in + row[j] * p.H + c);
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (row[j] >= 0) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const float x = Elem<T>::to_f32(v[j].v[e]);
          acc[e] += GATHER ? w[j] * x : x;
        }
      }
  }
  store_f32<T, V>(reinterpret_cast<T*>(p.out) + t * p.H + c, acc);
}

template <typename T, int V, bool GATHER>
int launch_combine(CombineParams p, int T_, cudaStream_t st) {
  p.vecs = p.H / V;
  const int64_t most = ((1ll << 31) - 1) / p.vecs;   // tokens per launch: pair numbers stay below 2^31
  for (int64_t t0 = 0; t0 < T_; t0 += most) {
    const int64_t n = T_ - t0 < most ? T_ - t0 : most;
    p.t0 = t0;
    p.total = static_cast<uint32_t>(n * p.vecs);
    // few tokens: smaller CTAs, so that more SMs pull
    const int threads = p.total < 256u * kNumSMs ? 64 : 256;
    const dim3 grid((p.total + threads - 1) / threads);
    auto go = [&](auto kernel) { return launch_pdl("combine_kernel", kernel, grid, dim3(threads), 0, st, 1, n * p.k, p); };
    int rc;
    switch (p.k) {
      case 1: rc = go(combine_kernel<T, V, 1, GATHER>); break;
      case 2: rc = go(combine_kernel<T, V, 2, GATHER>); break;
      case 4: rc = go(combine_kernel<T, V, 4, GATHER>); break;
      case 6: rc = go(combine_kernel<T, V, 6, GATHER>); break;
      case 8: rc = go(combine_kernel<T, V, 8, GATHER>); break;
      default: rc = go(combine_kernel<T, V, 0, GATHER>); break;
    }
    if (rc != B200MOE_OK) return rc;
  }
  return B200MOE_OK;
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

static int gather_impl(void* out, const void* y, int dtype, const float* weights,
                       const int32_t* row_map, const void* addend, const int32_t* num_valid, int T,
                       int k, int H, void* stream) {
  if (T < 0 || k <= 0 || k > kMaxTopK || H <= 0) return B200MOE_INVALID_ARG;
  if (T == 0) return B200MOE_OK;
  if (!out || !y || !weights || !row_map) return B200MOE_INVALID_ARG;
  if ((H * dtype_size(dtype)) % 16 != 0) return B200MOE_INVALID_ARG;
  CombineParams p{};
  p.out = out;
  p.in = y;
  p.weights = weights;
  p.row_map = row_map;
  p.addend = addend;
  p.num_valid = num_valid;
  p.k = k;
  p.H = H;
  return B200MOE_DISPATCH_FLOAT(dtype, [&] {
    return launch_combine<scalar_t, 16 / sizeof(scalar_t), true>(p, T, as_stream(stream));
  });
}

extern "C" int b200moe_moe_gather(void* out, const void* y, int dtype, const float* weights,
                                  const int32_t* row_map, int T, int k, int H, void* stream) {
  return gather_impl(out, y, dtype, weights, row_map, nullptr, nullptr, T, k, H, stream);
}

extern "C" int b200moe_moe_gather_add(void* out, const void* y, int dtype, const float* weights,
                                      const int32_t* row_map, const void* addend, int T, int k,
                                      int H, void* stream) {
  if (!addend) return B200MOE_INVALID_ARG;
  return gather_impl(out, y, dtype, weights, row_map, addend, nullptr, T, k, H, stream);
}

extern "C" int b200moe_moe_gather_bounded(void* out, const void* y, int dtype, const float* weights,
                                          const int32_t* row_map, const int32_t* num_valid_tokens,
                                          int T, int k, int H, void* stream) {
  if (!num_valid_tokens) return B200MOE_INVALID_ARG;
  return gather_impl(out, y, dtype, weights, row_map, nullptr, num_valid_tokens, T, k, H, stream);
}

extern "C" int b200moe_moe_sum(const void* in, void* out, int dtype, int T, int k, int H,
                               const void* topk_ids, int ids_dtype, const int32_t* expert_map,
                               void* stream) {
  if (T < 0 || k <= 0 || k > kMaxTopK || H <= 0) return B200MOE_INVALID_ARG;
  if (topk_ids && !is_index_dtype(ids_dtype)) return B200MOE_INVALID_ARG;
  if (T == 0) return B200MOE_OK;
  if (!in || !out) return B200MOE_INVALID_ARG;
  CombineParams p{};
  p.out = out;
  p.in = in;
  p.ids = topk_ids;
  p.ids_dtype = ids_dtype;
  p.expert_map = expert_map;
  p.k = k;
  p.H = H;
  return B200MOE_DISPATCH_FLOAT(dtype, [&] {
    constexpr int VMAX = 16 / sizeof(scalar_t);
    if (H % VMAX == 0) return launch_combine<scalar_t, VMAX, false>(p, T, as_stream(stream));
    return launch_combine<scalar_t, 1, false>(p, T, as_stream(stream));
  });
}
