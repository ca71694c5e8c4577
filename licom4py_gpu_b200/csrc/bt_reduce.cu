// bt_reduce.cu - on-device interior statistics and conservation sums.
//
// * bt_interior_stats: max, min and mean of a field's interior cells, the
//   global diagnostic of src/licom/mymodule/diag.py:45-75 computed where the
//   data lives (the reference copies the whole state to the host).
// * bt_conservation: total mass sum(h * da) and energy
//   sum((g h^2 / 2 + (H + h) |u|^2 / 2) * da) over the interior, where |u|^2 is
//   taken from the lon/lat components (a_c2l . (u, v)).  Each term is formed in
//   the field's precision; the sums are accumulated in float64 with
//   compensation (TwoSum) per thread and combined in a fixed order, so the result
//   is deterministic and independent of launch timing.
//
// One cluster of 16 CTAs walks the interior rows in a fixed order, each warp a
// strip of consecutive columns at a time with all its loads in flight, and
// combines through distributed shared memory: no scratch memory is used, so
// calls on any streams are independent and can be captured.  Where such a cluster
// cannot be placed (part of a GPU), a smaller one or a single CTA runs the same
// code.  Bound by the 16 SMs' share of the memory bandwidth (and by latency below C96); one CTA, as it
// was, kept a single SM waiting on one load per thread: interior statistics of a
// C384 float64 field 383 -> 18.5 us, conservation 848 -> 49 us (launch included); on a
// second stream beside a round they start like a single CTA does (C96 float64 20 us
// from call to result with 16, 30 with one).

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <string>

#include "bt_launch.cuh"
#include "bt_stencil.cuh"
#include "licom_bt.h"

namespace bt {
namespace {

namespace cg = cooperative_groups;

constexpr int kStatThreads = 1024, kConsThreads = 512;
constexpr int kRedCtas = 16;  // CTAs of the cluster at most

struct Kahan {
  double s = 0.0, c = 0.0;
  // the sum's rounding error by Knuth's TwoSum: exact like Neumaier's variant, without its comparison
  __device__ __forceinline__ void add(double x) {
    const double t = s + x, z = t - s;
    c += (s - (t - z)) + (x - z);
    s = t;
  }
  __device__ __forceinline__ void add(const Kahan& o) {
    add(o.s);
    c += o.c;
  }
  __device__ __forceinline__ double value() const { return s + c; }
};

// Runs item(row offset of column 0, first column) for this warp's strips of W
// columns: strip u is columns (u % strips) * W .. of interior row u / strips.
// CTAS: the cluster's size where it is known when compiled (0: gridDim.x).
template <int CTAS, int WARPS, int W, typename F>
__device__ __forceinline__ void for_strips(int n, F item) {
  const int m = n + 6;
  const unsigned strips = (n + W - 1) / W, total = 6u * n * strips;
  for (unsigned u = blockIdx.x * WARPS + threadIdx.x / 32; u < total; u += (CTAS ? CTAS : gridDim.x) * WARPS) {
    const unsigned row = u / strips, f = row / n, i = row - f * n;
    item(cell(f, i + kHalo, kHalo, m), (int)((u - row * strips) * W + (threadIdx.x & 31)));
  }
}

__device__ __forceinline__ Kahan warp_sum(Kahan a) {
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const Kahan b{__shfl_down_sync(0xffffffffu, a.s, w), __shfl_down_sync(0xffffffffu, a.c, w)};
    a.add(b);
  }
  return a;  // lane 0
}

// Combines the warps' values (lane 0 of each) of all CTAs in a fixed order; thread 0 of CTA 0 gets the result.
template <int CTAS, int WARPS, typename V, typename F>
__device__ __forceinline__ V cluster_combine(V v, F join) {
  __shared__ V part[WARPS];
  cg::cluster_group cl = cg::this_cluster();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x / 32] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < WARPS; ++w) join(v, part[w]);
    part[0] = v;
  }
  cl.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (int r = 1; r < (CTAS ? CTAS : (int)gridDim.x); ++r) join(v, *cl.map_shared_rank(&part[0], r));
  cl.sync();  // no CTA leaves while its shared memory is read
  return v;
}

struct StatsPart {
  double mx, mn;
  Kahan sum;
};

template <typename T, int CTAS>
__global__ void __launch_bounds__(kStatThreads) k_stats(int n, const T* F, double* out) {
  // columns per lane and strip: 32 warps with 6 loads each in flight (C384 float64 22.9 -> 18.5 us, float32 24.4 ->
  // 18.6 against 16 warps with 8)
  constexpr int K = 6;
  constexpr int A = 4;     // sums per lane: independent chains
  StatsPart p{-INFINITY, INFINITY, {}};
  Kahan sum[A];
  for_strips<CTAS, kStatThreads / 32, 32 * K>(n, [&](long o, int j) {
    T v[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (j + 32 * k < n) v[k] = F[o + j + 32 * k];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (j + 32 * k < n) {
        p.mx = fmax(p.mx, (double)v[k]);
        p.mn = fmin(p.mn, (double)v[k]);
        sum[k % A].add((double)v[k]);
      }
  });
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    p.mx = fmax(p.mx, __shfl_down_sync(0xffffffffu, p.mx, w));
    p.mn = fmin(p.mn, __shfl_down_sync(0xffffffffu, p.mn, w));
  }
#pragma unroll
  for (int k = 0; k < A; ++k) p.sum.add(sum[k]);
  p.sum = warp_sum(p.sum);
  p = cluster_combine<CTAS, kStatThreads / 32>(p, [](StatsPart& a, const StatsPart& b) {
    a.mx = fmax(a.mx, b.mx);
    a.mn = fmin(a.mn, b.mn);
    a.sum.add(b.sum);
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    out[0] = p.mx;
    out[1] = p.mn;
    out[2] = p.sum.value() / (6.0 * n * n);
  }
}

struct ConservationPart {
  Kahan mass, energy;
};

template <typename T, int CTAS>
__global__ void __launch_bounds__(kConsThreads) k_conservation(int n, const T* H, const T* U, const T* V,
                                                            const T* rda, const T* c2l, double depth,
                                                            double* out) {
  // columns per lane and strip, each with its own sums (1024 threads with 2: C384 float64 52.3 -> 55.0 us)
  constexpr int K = 3;
  ConservationPart p, q[K];
  const bool vec = (reinterpret_cast<size_t>(c2l) & 15) == 0;  // 16-byte loads (C384 float64 52.3 -> 49.1 us)
  for_strips<CTAS, kConsThreads / 32, 32 * K>(n, [&](long o, int j) {
    T h[K], u[K], v[K], r[K], C[K][4];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (j + 32 * k < n) {
        const long e = o + j + 32 * k;
        h[k] = H[e];
        u[k] = U[e];
        v[k] = V[e];
        r[k] = rda[e];
        if (vec) {
          ld_quad(c2l + 4 * e, C[k]);
        } else {
#pragma unroll
          for (int z = 0; z < 4; ++z) C[k][z] = c2l[4 * e + z];
        }
      }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (j + 32 * k < n) {
        const T da = T(1.0) / r[k];
        const T ul = C[k][0] * u[k] + C[k][1] * v[k], vl = C[k][2] * u[k] + C[k][3] * v[k];
        q[k].mass.add((double)(h[k] * da));
        const T e = (T(0.5) * T(9.8) * h[k] * h[k] + T(0.5) * (T(depth) + h[k]) * (ul * ul + vl * vl)) * da;
        q[k].energy.add((double)e);
      }
  });
#pragma unroll
  for (int k = 0; k < K; ++k) {
    p.mass.add(q[k].mass);
    p.energy.add(q[k].energy);
  }
  p.mass = warp_sum(p.mass);
  p.energy = warp_sum(p.energy);
  p = cluster_combine<CTAS, kConsThreads / 32>(p, [](ConservationPart& a, const ConservationPart& b) {
    a.mass.add(b.mass);
    a.energy.add(b.energy);
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    out[0] = p.mass.value();
    out[1] = p.energy.value();
  }
}

// The two builds of a reduction: for a cluster of kRedCtas and for any other size.
template <typename... A>
struct Builds {
  void (*full)(A...);
  void (*any)(A...);
  auto of(int ctas) const { return ctas == kRedCtas ? full : any; }
};

cudaLaunchConfig_t cluster_config(int ctas, int threads, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = ctas;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctas > 1 ? 1 : 0;  // a single CTA needs no cluster
  return cfg;
}

template <typename... A>
cudaError_t launch_on(int ctas, const Builds<A...>& k, int threads, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = cluster_config(ctas, threads, &attr);
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, k.of(ctas), args...);
}

// The largest cluster that the current device can hold: kRedCtas (more than the
// portable 8: that build opts in), else half of that and so on, at last 1.
template <typename... A>
int largest_cluster(const Builds<A...>& k, int threads) {
  const bool opted =
      cudaFuncSetAttribute(k.full, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  for (int ctas = opted ? kRedCtas : 8; ctas > 1; ctas /= 2) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config(ctas, threads, &attr);
    int held = 0;
    if (cudaOccupancyMaxActiveClusters(&held, k.of(ctas), &cfg) == cudaSuccess && held > 0) return ctas;
    cudaGetLastError();
  }
  cudaGetLastError();
  return 1;
}

// Launch on the largest cluster the device holds (asked once per device: ``known``, 0 = not yet), or on ``ctas``
// CTAs if that is not 0.  A launch that is refused all the same -- the context has fewer SMs than the device, or
// was reset -- runs on one CTA.
constexpr int kMaxDevices = 64;
template <typename... A>
cudaError_t launch_cluster(int ctas, const Builds<A...>& k, int threads, std::atomic<int>* known, cudaStream_t s,
                           A... args) {
  if (ctas > 0)
    return ctas > largest_cluster(k, threads) ? cudaErrorInvalidClusterSize
                                              : launch_on<A...>(ctas, k, threads, s, args...);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool in_range = dev >= 0 && dev < kMaxDevices;
  ctas = in_range ? known[dev].load(std::memory_order_relaxed) : 0;
  if (ctas == 0) {
    ctas = largest_cluster(k, threads);
    if (in_range) known[dev].store(ctas, std::memory_order_relaxed);
  }
  e = launch_on<A...>(ctas, k, threads, s, args...);
  if (e == cudaSuccess || ctas == 1) return e;
  cudaGetLastError();
  return launch_on<A...>(1, k, threads, s, args...);
}

template <typename T>
cudaError_t launch_stats(int ctas, int n, const void* f, void* out, cudaStream_t s) {
  static std::atomic<int> known[kMaxDevices];
  return launch_cluster<int, const T*, double*>(ctas, {k_stats<T, kRedCtas>, k_stats<T, 0>}, kStatThreads, known, s, n,
                                                (const T*)f, (double*)out);
}
template <typename T>
cudaError_t launch_conservation(int ctas, int n, const void* h, const void* u, const void* v, const void* rda,
                                const void* c2l, double depth, void* out, cudaStream_t s) {
  static std::atomic<int> known[kMaxDevices];
  return launch_cluster<int, const T*, const T*, const T*, const T*, const T*, double, double*>(
      ctas, {k_conservation<T, kRedCtas>, k_conservation<T, 0>}, kConsThreads, known, s, n, (const T*)h, (const T*)u,
      (const T*)v, (const T*)rda, (const T*)c2l, depth, (double*)out);
}

int rfail(int code, const std::string& msg) { return set_error(code, msg); }
bool ctas_ok(int ctas) { return ctas >= 0 && ctas <= kRedCtas && (ctas & (ctas - 1)) == 0; }

}  // namespace
}  // namespace bt

using namespace bt;

extern "C" {

int bt_interior_stats_on(int ctas, int n, int dtype, const void* field, void* out3, void* stream) {
  if (n < 1 || !field || !out3) return rfail(BT_EINVAL, "bt_interior_stats: bad argument");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype != BT_F64 && dtype != BT_F32)
    return rfail(BT_EINVAL, "bt_interior_stats: dtype must be BT_F64 or BT_F32");
  if (!ctas_ok(ctas)) return rfail(BT_EINVAL, "bt_interior_stats_on: ctas must be 0, 1, 2, 4, 8 or 16");
  const cudaError_t e =
      dtype == BT_F64 ? launch_stats<double>(ctas, n, field, out3, s) : launch_stats<float>(ctas, n, field, out3, s);
  if (e != cudaSuccess) return rfail(BT_ECUDA, std::string("bt_interior_stats: ") + cudaGetErrorString(e));
  return BT_OK;
}

int bt_conservation_on(int ctas, int n, int dtype, const void* h, const void* u, const void* v, const void* rda,
                       const void* a_c2l, double depth, void* out2, void* stream) {
  if (n < 1 || !h || !u || !v || !rda || !a_c2l || !out2) return rfail(BT_EINVAL, "bt_conservation: bad argument");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype != BT_F64 && dtype != BT_F32)
    return rfail(BT_EINVAL, "bt_conservation: dtype must be BT_F64 or BT_F32");
  if (!ctas_ok(ctas)) return rfail(BT_EINVAL, "bt_conservation_on: ctas must be 0, 1, 2, 4, 8 or 16");
  const cudaError_t e = dtype == BT_F64
                            ? launch_conservation<double>(ctas, n, h, u, v, rda, a_c2l, depth, out2, s)
                            : launch_conservation<float>(ctas, n, h, u, v, rda, a_c2l, depth, out2, s);
  if (e != cudaSuccess) return rfail(BT_ECUDA, std::string("bt_conservation: ") + cudaGetErrorString(e));
  return BT_OK;
}

int bt_interior_stats(int n, int dtype, const void* field, void* out3, void* stream) {
  return bt_interior_stats_on(0, n, dtype, field, out3, stream);
}

int bt_conservation(int n, int dtype, const void* h, const void* u, const void* v, const void* rda,
                    const void* a_c2l, double depth, void* out2, void* stream) {
  return bt_conservation_on(0, n, dtype, h, u, v, rda, a_c2l, depth, out2, stream);
}

}  // extern "C"
