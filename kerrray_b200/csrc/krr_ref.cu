// Kernels in the reference's operation order.  This translation unit is compiled with
// -fmad=false: every product and sum is rounded separately, as in KerrRay's Numba kernel
// (fastmath=False, src/kerrray/raytracing/backends/numba_kernel.py:466).
#include <math_constants.h>

#include "krr_launch.h"
#include "krr_quad.cuh"

namespace krr {

static cudaError_t ref_quad(const PlainArgs& a, cudaStream_t s);

cudaError_t ref_plain(bool dtype32, bool rk4, const PlainArgs& a, int block, cudaStream_t s) {
  if (a.quad) return ref_quad(a, s);
  if (dtype32) return rk4 ? run_plain<RefMode<float>, true>(a, block, s) : run_plain<RefMode<float>, false>(a, block, s);
  return rk4 ? run_plain<RefMode<double>, true>(a, block, s) : run_plain<RefMode<double>, false>(a, block, s);
}

// Launch shapes, (threads per block, minimum resident blocks per SM): the first for queues that fit
// its lanes, with the stages unrolled (neighbouring stages overlap: 100^2 photons 2.36 ms against
// 2.6 rolled), the second for longer ones, whose warps share the instruction cache, with the stages
// rolled (dp_stages_loop) at 12 warps per SM: 600^2 at rtol 1e-6 15.4 ms unrolled, 12.2 rolled at 8
// warps per SM without spills, 11.7 at 12 with, 13.0 at 16; 300^2 4.9, 4.4, 4.4, 4.7.
const Variant* ref_variants(bool dtype32, bool rk4, int* count) {
  static const Variant v64[] = {make_variant<RefMode<double>, false, 128, 1>(),
                                make_variant<RefMode<double, Stages::ROLLED>, false, 128, 3>()};
  static const Variant v64rk4[] = {make_variant<RefMode<double>, true, 128, 1>()};
  static const Variant v32[] = {make_variant<RefMode<float>, false, 128, 1>(),
                                make_variant<RefMode<float, Stages::ROLLED>, false, 128, 3>()};
  static const Variant v32rk4[] = {make_variant<RefMode<float>, true, 128, 1>()};
  *count = rk4 ? 1 : 2;
  if (dtype32) return rk4 ? v32rk4 : v32;
  return rk4 ? v64rk4 : v64;
}

cudaError_t ref_bisect(const EdgeArgs& a, cudaStream_t s) { return run_bisect<RefMode<double>, 128, 1>(a, s); }

__global__ void __launch_bounds__(128) k_trace_quad(const __grid_constant__ Params P, const Image* __restrict__ images,
                                                    int n_images, const double* __restrict__ Y0,
                                                    const long long* __restrict__ index, long long n, Outputs o, Queue* q) {
  constexpr unsigned FULL = 0xffffffffu;
  const long long i = (blockIdx.x * 128LL + threadIdx.x) >> 2;
  const bool mine = i < n;
  const long long g = mine ? (index ? index[i] : i) : (index ? index[0] : 0);  // lanes without a ray idle on the first
  const int img = images ? find_image(images, n_images, g) : 0;
  const Params& Pi = images ? images[img].P : P;
  double y0[8];
  photon_source(images, img, Y0, g, y0, mine ? q : nullptr);
  Quad ray;
  ray.start(Pi, y0, carter_initial(Pi, y0));
  if (!mine) ray.state = FAILURE;
  unsigned iters = 0;
  while (__any_sync(FULL, ray.state == RUNNING)) {
    ray.attempt(Pi, ray.state == RUNNING);
    __syncwarp();
    iters += 1;
  }
  if (mine) ray.store(o, g);
  if (q) {
    const bool counts = mine && (threadIdx.x & 3u) == 0;
    unsigned long long n_att = counts ? (unsigned long long)ray.attempts : 0, n_acc = counts ? (unsigned long long)ray.n_steps : 0;
    unsigned long long n_ret = counts ? 1 : 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      n_att += __shfl_down_sync(FULL, n_att, off);
      n_acc += __shfl_down_sync(FULL, n_acc, off);
      n_ret += __shfl_down_sync(FULL, n_ret, off);
    }
    if ((threadIdx.x & 31u) == 0 && n_ret) {
      atomicAdd(&q->retired, n_ret);
      atomicAdd(&q->attempts, n_att);
      atomicAdd(&q->accepted, n_acc);
      atomicAdd(&q->lane_iters, (unsigned long long)iters * 32ull);
      atomicAdd(&q->busy_iters, n_att);
    }
  }
}

static cudaError_t ref_quad(const PlainArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  k_trace_quad<<<(unsigned)((4 * a.n + 127) / 128), 128, 0, s>>>(a.P, a.images, a.n_images, a.Y0, a.index, a.n, a.o, a.q);
  return cudaGetLastError();
}

// Eight warps per block: at the reference order's register count one block fills an SM's
// register file, so the critical photons of the mixed pipeline hold SMs of their own.
const Variant* ref_wide_variant() {
  static const Variant v = make_variant<RefMode<double>, false, 256, 1>();
  return &v;
}

// One item per thread: where the radial potential's minimum changes sign between the ends of the
// bracket, by 8 halvings and 6 regula falsi steps (Illinois: an end kept twice counts half), which
// reach about 1e-13 M.  About 30 us whatever the study's size (one chain of 16 evaluations).
__global__ void __launch_bounds__(128) k_edge_predict(EdgeArgs a) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= a.n_items) return;
  const EdgeCase& ec = a.cases[a.item_case[i]];
  const double cphi = a.cos_phi[i], sphi = a.sin_phi[i];
  auto margin = [&](double rho) {  // > 0 captured, < 0 escapes, NaN not classified
    double y0[8], vmin, sens;
    camera_state(ec.F, ec.c_alpha + rho * cphi, ec.c_beta + rho * sphi, y0);
    if (!radial_margin(ec.P.mass, ec.P.a, ec.P.r_capture, y0, &vmin, &sens)) return CUDART_NAN;
    return vmin / sens;
  };
  double lo = a.lo[i], hi = a.hi[i];
  double f_lo = margin(lo), f_hi = margin(hi);
  double star = CUDART_NAN;
  if (f_lo >= 0.0 && f_hi < 0.0) {
    int kept = 0;  // the end the last regula falsi step left: -1 hi, +1 lo
    for (int k = 0; k < 14; ++k) {
      const double x = k < 8 ? 0.5 * (lo + hi) : lo + (hi - lo) * (f_lo / (f_lo - f_hi));
      const double f = margin(x);
      star = x;
      if (f < 0.0) {
        hi = x;
        f_hi = f;
        if (k >= 8 && kept == 1) f_lo *= 0.5;
        kept = k >= 8 ? 1 : 0;
      } else {
        lo = x;
        f_lo = f;
        if (k >= 8 && kept == -1) f_hi *= 0.5;
        kept = k >= 8 ? -1 : 0;
      }
    }
  }
  a.star[i] = star;
}

cudaError_t edge_predict(const EdgeArgs& a, cudaStream_t s) {
  if (a.n_items <= 0) return cudaSuccess;
  const int block = 128;
  k_edge_predict<<<(unsigned)((a.n_items + block - 1) / block), block, 0, s>>>(a);
  return cudaGetLastError();
}

// Warp-aggregated append of the flagged lanes' global indices to list (count in q->flagged).
__device__ __forceinline__ void append_flagged(bool flag, long long g, long long* list, Queue* q) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned mask = __ballot_sync(FULL, flag);
  if (mask) {
    const unsigned lane = threadIdx.x & 31u;
    const int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if ((int)lane == leader) base = atomicAdd(&q->flagged, (unsigned long long)__popc(mask));
    base = __shfl_sync(FULL, base, leader);
    if (flag) list[base + __popc(mask & ((1u << lane) - 1u))] = g;
  }
}

// The trace order: long photons from the front, short ones from the back, in any order within the
// two (no result depends on it).  A captured photon takes two to three times an escaping one's steps
// (the momenta grow towards the horizon), one that escapes within kOrderNear of the edge up to twice
// as many as one far out; what cannot be classified goes with the long ones.  Rows in random order,
// a few per lane, otherwise mix long and short photons in every warp and leave the last long ones to
// run on alone: 100k random rays, rtol 1e-8, in fast64 2.28 -> 1.72 ms, in reference order 8.2 ->
// 6.7; float32 at 1e-5 2.43 -> 2.02; mixed at 1e-6 1.03 -> 0.73; 30k rays 4-11 % less, 1M rays 4-7 %;
// twelve 160^2 images of one tolerance 10 %.  Below the resident lanes, and on one image, whose rows
// come and go like this by themselves, nothing or a few per cent more (order_wanted).  One atomic
// per block of 256 and end.
constexpr double kOrderNear = 1.0;  // M

__global__ void __launch_bounds__(256) k_trace_order(const __grid_constant__ OrderArgs a) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ unsigned n_long[8], n_short[8];
  __shared__ unsigned long long base_long, base_short;
  const long long g = blockIdx.x * 256LL + threadIdx.x;
  const bool valid = g < a.total;
  bool is_long = false;
  if (valid) {
    const int img = a.images ? find_image(a.images, a.n_images, g) : 0;
    const Params& P = a.images ? a.images[img].P : a.P;
    double y0[8], vmin, sens;
    photon_source(a.images, img, a.Y0, g, y0, nullptr);
    is_long = !(radial_margin(P.mass, P.a, P.r_capture, y0, &vmin, &sens) && vmin < 0.0 &&
                -vmin > kOrderNear * P.mass * sens);
  }
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
  const unsigned ml = __ballot_sync(FULL, valid && is_long), ms = __ballot_sync(FULL, valid && !is_long);
  if (lane == 0) {
    n_long[warp] = __popc(ml);
    n_short[warp] = __popc(ms);
  }
  __syncthreads();
  unsigned before_long = 0, before_short = 0, all_long = 0, all_short = 0;
  for (unsigned w = 0; w < 8; ++w) {
    before_long += w < warp ? n_long[w] : 0;
    before_short += w < warp ? n_short[w] : 0;
    all_long += n_long[w];
    all_short += n_short[w];
  }
  if (threadIdx.x == 0) {
    base_long = atomicAdd(&a.q->order_front, (unsigned long long)all_long);
    base_short = atomicAdd(&a.q->order_back, (unsigned long long)all_short);
  }
  __syncthreads();
  if (valid) {
    const long long at = is_long ? (long long)base_long + before_long + __popc(ml & below)
                                 : a.total - 1 - ((long long)base_short + before_short + __popc(ms & below));
    a.order[at] = g;
  }
}

cudaError_t trace_order(const OrderArgs& a, cudaStream_t s) {
  if (a.total <= 0) return cudaSuccess;
  k_trace_order<<<(unsigned)((a.total + 255) / 256), 256, 0, s>>>(a);
  return cudaGetLastError();
}

__global__ void k_risk_prepass(const Image* __restrict__ images, int n_images, long long total,
                               const double* __restrict__ Y0, unsigned char* __restrict__ risk,
                               long long* __restrict__ list, Queue* q, long long* __restrict__ near_list,
                               Queue* q_near) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  bool critical = false, near = false;
  if (g < total) {
    const int img = find_image(images, n_images, g);
    const Params& P = images[img].P;
    double y0[8];
    photon_source(images, img, Y0, g, y0, q);
    const int cls = radial_risk(P.mass, P.a, P.r_capture, y0, risk_band(P.mass, P.rtol),
                                near_list ? near_band(P.mass) : 0.0);
    risk[g] = (unsigned char)cls;
    critical = cls == RISK_CRITICAL;
    near = cls == RISK_NEAR;
  }
  append_flagged(critical, g, list, q);
  if (near_list) append_flagged(near, g, near_list, q_near);
}

__global__ void k_check_risk(const Image* __restrict__ images, int n_images, long long total,
                             const unsigned char* __restrict__ risk, const long long* __restrict__ state,
                             long long* __restrict__ list, Queue* q, int recheck) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  bool flag = false;
  if (g < total) {
    const int cls = risk[g];
    const long long st = state[g];
    if (cls == RISK_ESCAPE || cls == RISK_NEAR) flag = st != ESCAPED;
    else if (cls == RISK_CAPTURE) flag = st != CAPTURED;
    else if (cls == RISK_RECHECK) flag = recheck != 0;
  }
  append_flagged(flag, g, list, q);
}

cudaError_t risk_prepass(const Image* images, int n_images, long long total, const double* Y0, unsigned char* risk,
                         long long* list, Queue* q, long long* near_list, Queue* q_near, cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
  const int block = 256;  // a multiple of 32: the append is warp-aggregated
  k_risk_prepass<<<(unsigned)((total + block - 1) / block), block, 0, s>>>(images, n_images, total, Y0, risk, list, q,
                                                                          near_list, q_near);
  return cudaGetLastError();
}

cudaError_t check_risk(const Image* images, int n_images, long long total, const unsigned char* risk,
                       const long long* state, long long* list, Queue* q, bool recheck, cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
  const int block = 256;
  k_check_risk<<<(unsigned)((total + block - 1) / block), block, 0, s>>>(images, n_images, total, risk, state, list, q,
                                                                        recheck ? 1 : 0);
  return cudaGetLastError();
}

__global__ void k_flag_boundary(const Image* __restrict__ images, int n_images, long long total,
                                const long long* __restrict__ state, long long* __restrict__ list, Queue* q) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  bool flag = false;
  if (g < total) {
    const Image& im = images[find_image(images, n_images, g)];
    const long long n = im.res;
    const long long p = g - im.offset + im.first;  // pixel of the image's grid
    const long long i = p / n, j = p - (p / n) * n;
    const long long s = state[g];
    flag = !(s == ESCAPED || s == CAPTURED);
    for (int di = -1; di <= 1 && !flag; ++di) {
      for (int dj = -1; dj <= 1 && !flag; ++dj) {
        const long long ii = i + di, jj = j + dj;
        if ((di == 0 && dj == 0) || ii < 0 || ii >= n || jj < 0 || jj >= n) continue;
        const long long q = ii * n + jj - im.first;  // the neighbour's row of this launch, if traced in it
        if (q < 0 || q >= im.count) continue;
        flag = state[im.offset + q] != s;
      }
    }
  }
  append_flagged(flag, g, list, q);
}

cudaError_t flag_boundary(const Image* images, int n_images, long long total, const long long* state, long long* list,
                          Queue* q, cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
  const int block = 256;  // a multiple of 32: the append is warp-aggregated
  k_flag_boundary<<<(unsigned)((total + block - 1) / block), block, 0, s>>>(images, n_images, total, state, list, q);
  return cudaGetLastError();
}

// Camera kernel: one image point per thread.
__global__ void k_camera_states(Frame F, double fov, long long res, const double* __restrict__ alpha,
                                const double* __restrict__ beta, long long n, double* __restrict__ Y0, int* err) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a, b;
  if (alpha) {
    a = alpha[i];
    b = beta[i];
  } else {
    pixel_alpha_beta(fov, res, i, a, b);
  }
  double y0[8];
  if (camera_state(F, a, b, y0) != 0 && err) atomicCAS(err, 0, 6);
#pragma unroll
  for (int c = 0; c < 8; ++c) Y0[i * 8 + c] = y0[c];
}

cudaError_t camera_states(const Frame& F, double fov, long long res, const double* alpha, const double* beta,
                          long long n, double* Y0, int* err, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int block = 256;
  k_camera_states<<<(unsigned)((n + block - 1) / block), block, 0, s>>>(F, fov, res, alpha, beta, n, Y0, err);
  return cudaGetLastError();
}

}  // namespace krr
