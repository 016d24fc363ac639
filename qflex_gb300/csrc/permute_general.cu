// Permutation of tensors whose dimensions are not all powers of two.
//
// Bound by HBM (16 B per element) once index arithmetic is out of the way: one
// thread per output element with 64-bit divisions by every dimension spent
// its time on those, and gathered reads used 8 bytes of every 32-byte sector.
// Here a thread moves a run of up to 16 elements that are neighbours in the
// input, so whole sectors are read; a warp's threads follow the output's
// order, so each element of the runs is stored in contiguous pieces; and the
// division is by multiplication with a precomputed factor (Granlund and
// Montgomery, Division by Invariant Integers using Multiplication, 1994), once
// per run. 12 x 15 x 7 x 24 x 10 x 27 in
// order 3 0 5 2 1 4: 92 -> 33 us (3.9 TB/s).
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "kernels.h"

namespace qfx {
namespace {

__host__ __device__ inline std::uint32_t divide(std::uint32_t n, const FastDiv& f) {
#ifdef __CUDA_ARCH__
  return (__umulhi(n, f.mul) + n) >> f.shift;
#else
  return (std::uint32_t)((((std::uint64_t)n * f.mul) >> 32) + n) >> f.shift;
#endif
}

FastDiv fast_div(std::uint32_t d) {
  FastDiv f{d, 0, 0};
  while ((1ull << f.shift) < d) ++f.shift;
  f.mul = (std::uint32_t)(((1ull << 32) * ((1ull << f.shift) - d)) / d + 1);
  return f;
}

// What the kernel takes of the schedule, for up to CAP indices: a small tensor's
// call is as long as its launch, to which 1.4 KB of arguments added 0.4 us.
template <int CAP>
struct RunPlan {
  std::uint32_t runs, last_run, run, n_div;
  FastDiv div[CAP];
  std::uint32_t div_in[CAP], div_out[CAP], run_out[16];
};

// Input and output offset of thread r's run; its length.
template <typename Plan>
__host__ __device__ inline std::uint32_t run_of(const Plan& g, std::uint32_t r, std::uint32_t* in,
                                                std::uint32_t* out) {
  std::uint32_t i = 0, o = 0, digit = 0;
  for (std::uint32_t j = 0; j < g.n_div; ++j) {
    const std::uint32_t q = divide(r, g.div[j]);
    digit = r - q * g.div[j].d;
    i += digit * g.div_in[j];
    o += digit * g.div_out[j];
    r = q;
  }
  *in = i;
  *out = o;
  // The last index numbers the runs of the input's fastest index.
  return digit + 1 == g.div[g.n_div - 1].d ? g.last_run : g.run;
}

template <int RUN, int CAP>
__global__ void __launch_bounds__(256) permute_runs_kernel(const __grid_constant__ RunPlan<CAP> g,
                                                           const float2* __restrict__ src, float2* __restrict__ dst,
                                                           std::uint64_t batch_stride) {
  src += std::uint64_t(blockIdx.y) * batch_stride;
  dst += std::uint64_t(blockIdx.y) * batch_stride;
  for (std::uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < g.runs; r += gridDim.x * blockDim.x) {
    std::uint32_t in, out;
    const std::uint32_t n = run_of(g, r, &in, &out);
    float2 v[RUN];
#pragma unroll
    for (int u = 0; u < RUN; ++u)
      if (u < n) v[u] = __ldg(src + in + u);
#pragma unroll
    for (int u = 0; u < RUN; ++u)
      if (u < n) dst[out + g.run_out[u]] = v[u];
  }
}

// Sizes from 2^31 elements: one thread per output element.
__host__ __device__ inline std::uint64_t general_source(const GeneralPerm& g, std::uint64_t o) {
  std::uint64_t in = 0;
  for (int i = int(g.rank) - 1; i >= 0; --i) {
    const std::uint64_t d = g.out_dims[i];
    const std::uint64_t q = o / d;
    in += (o - q * d) * g.in_stride[i];
    o = q;
  }
  return in;
}

__global__ void __launch_bounds__(256) permute_general_kernel(const __grid_constant__ GeneralPerm g,
                                                              const float2* __restrict__ src,
                                                              float2* __restrict__ dst,
                                                              std::uint64_t batch_stride) {
  const float2* s = src + std::uint64_t(blockIdx.y) * batch_stride;
  float2* d = dst + std::uint64_t(blockIdx.y) * batch_stride;
  for (std::uint64_t o = std::uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; o < g.size;
       o += std::uint64_t(gridDim.x) * blockDim.x)
    d[o] = __ldg(s + general_source(g, o));
}

void plan_runs(GeneralPerm* g) {
  // Small tensors need the threads more than whole sectors: of 10000 to 100000
  // elements, one launch behind the other, runs of 13 to 16 took 6.2 us, runs of
  // up to 4 take 4.2.
  const std::uint32_t most = g->size <= (1u << 17) ? 4 : 16;
  struct Dim {
    std::uint32_t d, in, out;
  };
  // The permuted indices in output order, neighbours that stay neighbours as
  // one, then fastest output index first.
  std::vector<Dim> dims;
  dims.reserve(kGeneralPermMaxRank + 1);
  std::uint64_t out = g->size;
  for (std::uint32_t i = 0; i < g->rank; ++i) {
    const std::uint32_t d = (std::uint32_t)g->out_dims[i], in = (std::uint32_t)g->in_stride[i];
    out /= d;
    if (d == 1) continue;
    if (!dims.empty() && dims.back().in == d * in)
      dims.back() = {dims.back().d * d, in, (std::uint32_t)out};
    else
      dims.push_back({d, in, (std::uint32_t)out});
  }
  if (dims.empty()) dims.push_back({1, 1, 1});
  std::reverse(dims.begin(), dims.end());
  g->run = g->last_run = 1;
  std::uint32_t chunks = 1, chunk_in = 0, chunk_out = 0;
  // The input's fastest index: in runs of up to `most` when long, else with the
  // next faster ones up to that many elements; never with the output's fastest
  // index, which the lanes follow.
  auto fastest = [&](std::uint32_t in) {
    for (std::size_t i = 1; i < dims.size(); ++i)
      if (dims[i].in == in) return i;
    return std::size_t(0);
  };
  if (std::size_t i = fastest(1)) {
    const Dim f = dims[i];
    if (f.d > most) {
      chunks = (f.d + most - 1) / most;
      g->run = (f.d + chunks - 1) / chunks;
      chunks = (f.d + g->run - 1) / g->run;
      g->last_run = f.d - g->run * (chunks - 1);
      chunk_in = g->run;
      chunk_out = g->run * f.out;
      for (std::uint32_t u = 0; u < g->run; ++u) g->run_out[u] = u * f.out;
      dims.erase(dims.begin() + i);
    } else {
      while (i) {
        const Dim e = dims[i];
        if (g->run * e.d > most) break;
        for (std::uint32_t u = g->run; u < g->run * e.d; ++u)
          g->run_out[u] = g->run_out[u % g->run] + u / g->run * e.out;
        g->run *= e.d;
        dims.erase(dims.begin() + i);
        i = fastest(g->run);
      }
      g->last_run = g->run;
    }
  }
  dims.push_back({chunks, chunk_in, chunk_out});
  std::uint32_t runs = 1;
  for (const Dim& d : dims) {
    g->div[g->n_div] = fast_div(d.d);
    g->div_in[g->n_div] = d.in;
    g->div_out[g->n_div] = d.out;
    ++g->n_div;
    runs *= d.d;
  }
  g->runs = runs;
}

}  // namespace

void make_general_perm(std::size_t rank, const std::size_t* dims, const std::size_t* new_order, GeneralPerm* g) {
  if (rank > (std::size_t)kGeneralPermMaxRank)
    throw std::string("ERROR (qflex_gb300: permute) --> at most 32 indices when a dimension is not a power of two");
  std::memset(g, 0, sizeof(*g));
  g->rank = (std::uint32_t)rank;
  std::uint64_t stride[kGeneralPermMaxRank];
  std::uint64_t size = 1;
  for (std::size_t i = rank; i-- > 0;) {
    if (dims[i] == 0) throw std::string("ERROR (qflex_gb300: permute) --> dimensions must be positive");
    stride[i] = size;
    if (dims[i] > (std::uint64_t(1) << 40) / size)
      throw std::string("ERROR (qflex_gb300: permute) --> tensor exceeds 2^40 elements");
    size *= dims[i];
  }
  bool seen[kGeneralPermMaxRank] = {};
  for (std::size_t i = 0; i < rank; ++i) {
    const std::size_t q = new_order[i];
    if (q >= rank || seen[q]) throw std::string("ERROR (qflex_gb300: permute) --> new_order is not a permutation");
    seen[q] = true;
    g->out_dims[i] = dims[q];
    g->in_stride[i] = stride[q];
  }
  g->size = size;
  if (size < (std::uint64_t(1) << 31)) plan_runs(g);
}

void permute_general_on_host(const GeneralPerm& g, const float2* src, float2* dst) {
  if (!g.runs) {
    for (std::uint64_t o = 0; o < g.size; ++o) {
      const std::uint64_t at = general_source(g, o);
      if (at >= g.size) throw std::string("ERROR (qflex_gb300: permute) --> load out of range");
      dst[o] = src[at];
    }
    return;
  }
  for (std::uint32_t r = 0; r < g.runs; ++r) {
    std::uint32_t in, out;
    const std::uint32_t n = run_of(g, r, &in, &out);
    for (std::uint32_t u = 0; u < n; ++u) {
      if (u >= 16 || in + u >= g.size || out + g.run_out[u] >= g.size)
        throw std::string("ERROR (qflex_gb300: permute) --> run out of range");
      dst[out + g.run_out[u]] = src[in + u];
    }
  }
}

template <int CAP>
static void launch_runs(const GeneralPerm& g, const float2* src, float2* dst, std::uint64_t batch_stride, dim3 grid,
                        cudaStream_t s) {
  RunPlan<CAP> p;
  p.runs = g.runs;
  p.last_run = g.last_run;
  p.run = g.run;
  p.n_div = g.n_div;
  std::copy_n(g.div, g.n_div, p.div);
  std::copy_n(g.div_in, g.n_div, p.div_in);
  std::copy_n(g.div_out, g.n_div, p.div_out);
  std::copy_n(g.run_out, 16, p.run_out);
  auto* kernel = g.run == 1   ? permute_runs_kernel<1, CAP>
                 : g.run <= 4 ? permute_runs_kernel<4, CAP>
                 : g.run <= 8 ? permute_runs_kernel<8, CAP>
                              : permute_runs_kernel<16, CAP>;
  kernel<<<grid, 256, 0, s>>>(p, src, dst, batch_stride);
}

void launch_permute_general(const GeneralPerm& g, const float2* src, float2* dst, std::uint64_t batch_stride,
                            int batch, cudaStream_t s) {
  if (g.size == 0 || batch == 0) return;
  const std::uint64_t threads = g.runs ? g.runs : g.size;
  const std::uint64_t blocks = std::min<std::uint64_t>((threads + 255) / 256, 152ull * 64ull);
  dim3 grid((unsigned)blocks, (unsigned)batch, 1);
  if (!g.runs)
    permute_general_kernel<<<grid, 256, 0, s>>>(g, src, dst, batch_stride);
  else if (g.n_div <= 8)
    launch_runs<8>(g, src, dst, batch_stride, grid, s);
  else
    launch_runs<kGeneralPermMaxRank + 1>(g, src, dst, batch_stride, grid, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    throw std::string("ERROR (qflex_gb300: launch permute_general) --> ") + cudaGetErrorString(e);
}

}  // namespace qfx
