// energy.cu -- FP64 energy and momentum diagnostics on the device.
// Restates the softened potential energy and kinetic energy of
// scripts/nbody_physics/energy.py:146-192 (PE = -sum_{i<j} m_i m_j /
// sqrt(r^2 + eps^2), KE = sum m v^2 / 2; the reference has unit masses) with
// masses, plus linear and angular momentum.  Deterministic: per-CTA tree sums,
// then CTA partials added in order.
//
// Each pair is taken once: body i has the partners i + 1, ..., i + h (modulo n),
// h = (n - 1) / 2, and for even n the first half of the bodies i + n / 2 too, so
// every body has the same share.  A CTA's 128 bodies i0 + b and the partners
// i0 + v: the pair counts where 1 <= v - b <= h, which cuts off the corners of
// the first and last 128 partners.
//
// The FP64 pair sum is bound by the FP64 pipe (IEEE square root and division,
// about 23 operations a pair), so it runs in fixed point on the integer pipes
// (fixpair.cuh), the partners split over the CTAs of a cluster; the FP64 loop is
// left for systems without a fixed-point grid.  N = 16384: 14.8 ms with every
// pair twice in FP64 on one CTA per 128 bodies, 1.13 ms in fixed point, 0.65
// ms with each pair once (a call with the result's copy 0.69).
#include "force.cuh"

namespace gb {
namespace {

constexpr int kT = 128;
// CTAs of the pair kernel on an SM: with every pair twice N = 16384 took 1.21 ms
// at 5, 1.16 at 6, 1.13 at 7, 1.16 at 8 (135 cycles of a sub-partition per 32
// terms, ~95 instructions)
constexpr int kCtasPerSm = 7;

// Body i's sum of [m_j] / r over its partners v in [vb, ve), in FP64.
__device__ __noinline__ double pot_f64(const double* __restrict__ pos, long long n, long long i0,
                                       long long vb, long long ve, long long span, double eps2,
                                       const double* __restrict__ masses, double* sh) {
  const int b = threadIdx.x;
  const long long i = i0 + b;
  double xi = 0, yi = 0, zi = 0, phi = 0.0;
  if (i < n) {
    xi = pos[3 * i];
    yi = pos[3 * i + 1];
    zi = pos[3 * i + 2];
  }
  for (long long v0 = vb; v0 < ve; v0 += kT) {
    const int cnt = (int)min((long long)kT, ve - v0);
    __syncthreads();
    if (b < cnt) {
      const long long j = (i0 + v0 + b) % n;
      sh[4 * b] = pos[3 * j];
      sh[4 * b + 1] = pos[3 * j + 1];
      sh[4 * b + 2] = pos[3 * j + 2];
      sh[4 * b + 3] = masses ? masses[j] : 1.0;
    }
    __syncthreads();
    for (int k = 0; k < cnt; ++k) {
      const long long d = v0 + k - b;
      if (d < 1 || d > span) continue;
      const double dx = sh[4 * k] - xi, dy = sh[4 * k + 1] - yi, dz = sh[4 * k + 2] - zi;
      phi += sh[4 * k + 3] / sqrt(dx * dx + dy * dy + dz * dz + eps2);
    }
  }
  return phi;
}

// The same in fixed point on the grid of ex; close pairs in FP64.
template <int MASSES>
__device__ __noinline__ double pot_fx(const double* __restrict__ pos, long long n, long long i0,
                                      long long vb, long long ve, long long span, double eps2,
                                      const double* __restrict__ masses, int ex, int em,
                                      FxBody* rec, const FxRow* tab) {
  constexpr bool MASS = MASSES != kFxEqual, CLASSES = MASSES == kFxClasses;
  const int b = threadIdx.x;
  const long long i = min(i0 + b, n - 1);
  const Fx96 xi = fx_from_double(pos[3 * i], ex), yi = fx_from_double(pos[3 * i + 1], ex),
             zi = fx_from_double(pos[3 * i + 2], ex);
  const float eps2f = fx_eps2f(eps2, ex);
  __int128 tot = 0;
  double near = 0.0;
  for (long long v0 = vb; v0 < ve; v0 += kT) {
    const int cnt = (int)min((long long)kT, ve - v0);
    fx_stage<MASSES>(rec, pos, masses, (i0 + v0 + b) % n, cnt, ex, em, kT, b, 0);
    // the tile's partner k counts where 0 <= k - first < span
    const long long first = b + 1 - v0;
    for (int c = 0, end; c < cnt; c = end) {
      end = min(cnt, c + kFxChunk);
      int run = cnt, cls = 0;
      if (CLASSES) {
        run = fx_tag_end(rec[c].tag);
        cls = fx_tag_class(rec[c].tag);
        end = min(end, run);
      }
      const bool light = CLASSES && cls == kFxClassFp64;
      unsigned mask = 0;
      FxAcc a = {};
#pragma unroll 2
      for (int k = c; k < end; ++k) {
        const int at = CLASSES ? fx_tag_index(rec[k].tag) : k;
        const bool on = (unsigned long long)(at - first) < (unsigned long long)span;
        const int norm = fx_term_pot<MASS>(rec[k], xi, yi, zi, eps2f, tab, on, a);
        mask = (mask << 1) | (on && (light || norm > kFxMaxK) ? 1u : 0u);
      }
      if (!light) fx_fold(tot, a);
      while (mask) {  // close pairs
        const int k = end - 32 + __clz(mask);
        mask &= ~(0x80000000u >> __clz(mask));
        const long long j = (i0 + v0 + (CLASSES ? fx_tag_index(rec[k].tag) : k)) % n;
        const double dx = pos[3 * j] - pos[3 * i], dy = pos[3 * j + 1] - pos[3 * i + 1],
                     dz = pos[3 * j + 2] - pos[3 * i + 2];
        near += (MASS ? masses[j] : 1.0) / sqrt(dx * dx + dy * dy + dz * dz + eps2);
      }
      if (CLASSES && end == run) {  // the class's sum in the tile
        near += fx_to_double(tot, fx_out_exp_pot(ex) + fx_class_exp(em, cls) + 2);
        tot = 0;
      }
    }
  }
  return fx_to_double(tot, fx_out_exp_pot(ex) + (MASS ? fx_class_exp(em, 0) + 2 : 0)) + near;
}

__global__ void __launch_bounds__(kT, kCtasPerSm)
    energy_partial_kernel(const double* __restrict__ x, long long n, double eps2, double mass,
                          const double* __restrict__ masses, double* __restrict__ partial) {
  __shared__ __align__(16) unsigned char sh_raw[f64_smem_bytes<kT>()];
  __shared__ double part[kT];
  __shared__ double red[8][kT];
  const ClusterInfo ci = cluster_info();
  const long long i0 = ci.itile * kT, i = i0 + threadIdx.x;
  const double* pos = x;
  const double* vel = x + 3 * n;
  double xi = 0, yi = 0, zi = 0;
  if (i < n) {
    xi = pos[3 * i];
    yi = pos[3 * i + 1];
    zi = pos[3 * i + 2];
  }
  const long long h = (n - 1) / 2, even = 1 - n % 2;
  const long long span = i < n ? h + (even && i < n / 2 ? 1 : 0) : 0;  // partners of the body
  long long vb, ve;
  j_chunk(h + even + kT, ci.rank, ci.size, kFxChunk, vb, ve);
  FxBody* rec = reinterpret_cast<FxBody*>(sh_raw);
  FxRow* tab = reinterpret_cast<FxRow*>(rec + kT);
  int ex, em;
  bool classes;
  FxShape shape;
  if (fx_grid(pos, n, min(i, n - 1), (i0 + vb) % n, min(n, ve - vb), eps2, masses,
              reinterpret_cast<int*>(tab + kFxRows), kT, threadIdx.x, 0, &ex, &em, &classes, &shape)) {
    if (threadIdx.x < kFxRows) tab[threadIdx.x] = fx_row(threadIdx.x, eps2, ex);
    part[threadIdx.x] =
        !masses ? pot_fx<kFxEqual>(pos, n, i0, vb, ve, span, eps2, nullptr, ex, 0, rec, tab)
        : !classes
            ? pot_fx<kFxOneClass>(pos, n, i0, vb, ve, span, eps2, masses, ex, em, rec, tab)
            : pot_fx<kFxClasses>(pos, n, i0, vb, ve, span, eps2, masses, ex, em, rec, tab);
  } else {
    part[threadIdx.x] = pot_f64(pos, n, i0, vb, ve, span, eps2, masses,
                                reinterpret_cast<double*>(sh_raw));
  }
  // rank 0 adds the ranks' sums in rank order
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  double phi = 0.0;
  if (ci.rank == 0) {
    phi = cluster_sum(cl, part, threadIdx.x, ci.size);
    if (!masses) phi *= mass;
    phi = -phi;
  }
  cl.sync();
  if (ci.rank != 0) return;
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (i < n) {
    const double mi = masses ? masses[i] : mass;
    const double vx = vel[3 * i], vy = vel[3 * i + 1], vz = vel[3 * i + 2];
    v[0] = 0.5 * mi * (vx * vx + vy * vy + vz * vz);
    v[1] = mi * phi;
    v[2] = mi * vx;
    v[3] = mi * vy;
    v[4] = mi * vz;
    v[5] = mi * (yi * vz - zi * vy);
    v[6] = mi * (zi * vx - xi * vz);
    v[7] = mi * (xi * vy - yi * vx);
  }
  for (int c = 0; c < 8; ++c) red[c][threadIdx.x] = v[c];
  __syncthreads();
  for (int st = kT / 2; st > 0; st /= 2) {
    if ((int)threadIdx.x < st)
      for (int c = 0; c < 8; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x < 8) partial[ci.itile * 8 + threadIdx.x] = red[threadIdx.x][0];
}

// One warp per quantity: lanes over the CTAs' partials, then a tree (one thread
// adding them one after the other waited for a load and an FP64 addition each).
__global__ void __launch_bounds__(256)
    energy_final_kernel(const double* __restrict__ partial, int nb, double* __restrict__ out) {
  const int c = threadIdx.x / 32, lane = threadIdx.x % 32;
  double s = 0.0;
#pragma unroll 4
  for (int b = lane; b < nb; b += 32) s += partial[b * 8 + c];
#pragma unroll
  for (int off = 16; off >= 1; off /= 2) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) out[c] = s;
}

}  // namespace
}  // namespace gb

using namespace gb;

extern "C" size_t gb_nbody_energy_workspace_bytes(int64_t n) {
  if (n < 1) return 0;
  return (size_t)((n + kT - 1) / kT) * 8 * sizeof(double);
}

// out_dev[0] = kinetic, [1] = potential, [2..4] = linear momentum,
// [5..7] = angular momentum (about the origin).
extern "C" int gb_nbody_energy_f64(const double* x, int64_t n, double softening, double mass,
                                   const double* masses, void* work, size_t work_bytes,
                                   double* out_dev, gb_stream_t stream) {
  if (!x || n < 1 || !work || !out_dev || !(softening >= 0.0)) return GB_ERR_INVALID_ARGUMENT;
  if (!masses && !(mass > 0.0)) return GB_ERR_INVALID_ARGUMENT;
  if (work_bytes < gb_nbody_energy_workspace_bytes(n)) return GB_ERR_CAPACITY;
  cudaStream_t s = as_cuda(stream);
  const int nb = (int)((n + kT - 1) / kT);
  double* partial = reinterpret_cast<double*>(work);
  // CTAs per 128 bodies: the split with the shortest time, waves of resident
  // CTAs over the split (N = 16384, 5 CTAs per SM: 1.21 ms at 5, one wave of
  // 640, against 1.29 ms at 8, whose second wave is a third full).
  ForceGeom g{};
  g.T = kT;
  g.P = 1;
  const long long slots = (long long)kCtasPerSm * num_sms();
  const auto waves = [&](long long p) { return ((long long)nb * p + slots - 1) / slots; };
  for (int p = 2; p <= 8; ++p)
    if (waves(p) * g.P < waves(g.P) * p) g.P = p;
  g.n_itiles = nb;
  long long nn = n;
  double eps2 = softening * softening;
  void* args[] = {(void*)&x, (void*)&nn, (void*)&eps2, (void*)&mass, (void*)&masses,
                  (void*)&partial};
  GB_TRY(launch_cluster((const void*)energy_partial_kernel, g, 0, s, args));
  energy_final_kernel<<<1, 256, 0, s>>>(partial, nb, out_dev);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}
