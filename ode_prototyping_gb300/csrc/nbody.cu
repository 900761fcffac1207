// nbody.cu -- standalone right-hand-side entry points (FP64 and mixed).
// Replaces NBodyODE<double, 6N>::operator() / acc() (src/ode/NBodyODE.hpp:31-46)
// and its two kernels nbody_init_dxdt_kernel (:51-56) and nbody_acc_kernel
// (:68-133), which the reference runs as one thread per unordered pair with
// six FP64 atomicAdds; here each body's sum is owned by one lane group.
#include "force.cuh"
#include "sortpack.cuh"

namespace gb {

// Argument checks shared by the right-hand-side entry points (also the
// allocation-free one in noalloc.cu).
int validate_nbody(const void* a, const void* b, long long n, double softening, double mass,
                   const double* masses) {
  if (!a || !b || n < 1) return GB_ERR_INVALID_ARGUMENT;
  if (!(softening >= 0.0) || !std::isfinite(softening)) return GB_ERR_INVALID_ARGUMENT;
  if (!masses && !(mass > 0.0)) return GB_ERR_INVALID_ARGUMENT;
  return GB_OK;
}

namespace {

enum { kModeRhs = 0, kModeAccWrite = 1, kModeAccAdd = 2 };

// AFTER: the launch overlaps the kernel before it in the stream.  For grids of
// at most 4 CTAs per SM, whose launches are short (N = 257 FP64 10.25 -> 8.96 us
// a call, 3001 1846 -> 1807 us for 16 steps of leapfrog; N = 4096 mixed 28.7 -> 24.7
// us); beyond that the loops run 0.3-0.6 % faster with their pointers left
// __restrict__ (N = 16384 FP64, 100003 mixed).  A kernel of at most kFewCtas CTAs,
// half the SMs, lets the next one's wait beside it; more of them leave the next kernel's
// unevenly spread over the SMs (3001: 2088 us for the 16 steps where they may).
constexpr unsigned kFewCtas = 76;
constexpr int kAfterCtasPerSm = 4;
// FX: with fixed-point pair terms, and registers for 4 CTAs of 128 threads on an SM
// (N = 16384 1.66 ms, 1.88 at 5; 162 registers and 3 CTAs where the compiler is left
// to itself, 13 % slower).  Without them, for the calls that ask for the
// reference's order, a kernel has the registers of the FP64 loop alone (N = 5000, 4
// ranks of 8 lanes: 2.49 ms with those of the fixed-point one, whose 4 CTAs an SM
// need a third wave, 2.25 so).
template <int T, int L, bool AFTER = false, bool FX = true>
__global__ void __launch_bounds__(T, FX ? 4 * 128 / T : 0) rhs_f64_kernel(const double* __restrict__ pos,
                                                    const double* __restrict__ vel,
                                                    double* __restrict__ out_vel,
                                                    double* __restrict__ out_acc, long long n,
                                                    double eps2, double mass,
                                                    const double* __restrict__ masses, int mode,
                                                    int pair) {
  constexpr int BI = T / L;
  __shared__ __align__(16) unsigned char sh_raw[FX ? f64_smem_bytes<T>() : 32 * T];
  __shared__ double part[BI][3];
  if constexpr (AFTER) {
    after_previous(pos, vel, out_vel, out_acc, masses);
    if (gridDim.x <= kFewCtas) let_next_in();
  }
  const ClusterInfo ci = cluster_info();
  const long long i0 = ci.itile * BI;
  long long jb, je;
  j_chunk(n, ci.rank, ci.size, T, jb, je);
  force_f64_cta<T, L, FX>(pos, n, i0, jb, je, eps2, masses, sh_raw, part, pair);
  cluster_combine<BI>(part, ci.rank, ci.size);
  if (ci.rank != 0) return;
  const long long nb = min((long long)BI, n - i0);
  for (int e = threadIdx.x; e < 3 * nb; e += T) {
    const long long g = 3 * i0 + e;
    double a = part[e / 3][e % 3];
    if (!masses) a = dmul(a, mass);
    if (mode == kModeRhs) {
      out_vel[g] = vel[g];
      out_acc[g] = a;
    } else if (mode == kModeAccWrite) {
      out_acc[g] = a;
    } else {
      out_acc[g] = dadd(out_acc[g], a);
    }
  }
}

__device__ __forceinline__ PackedBody pack_row(const double* __restrict__ pos,
                                               const double* __restrict__ masses, double cx,
                                               double cy, double cz, long long i) {
  const float w = masses ? (float)masses[i] : 1.0f;
  return pack_body(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], cx, cy, cz, w);
}

// Centroid of n bodies: 1024 chains (body t, t + 1024, ... added in order), then
// a tree over the chains.  Bound by the FP64 pipe, 3 n adds: one CTA of 1024
// threads took 9.4 us at N = 4096 and 93 us at 100003, so a cluster of 8 CTAs
// holds 128 chains each and its first CTA, thread t with chains t, t + 128, ...,
// runs the tree, the same additions.  PACK: the cluster then packs the
// bodies itself (it saves the launch of the packing kernel; up to
// kFusedPackBodies, where eight SMs are as fast as a launch).
constexpr int kCentroidCtas = 8;
constexpr long long kFusedPackBodies = 4096;
template <bool PACK>
__global__ void __cluster_dims__(kCentroidCtas, 1, 1) __launch_bounds__(128)
    centroid_kernel(const double* __restrict__ pos, const double* __restrict__ masses, long long n,
                    double* c_out, PackedBody* out) {
  after_previous(pos, masses, c_out, out);
  let_next_in();
  __shared__ double chain[3][128];
  __shared__ double cen[3];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), t = threadIdx.x;
  double v[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (long long i = rank * 128 + t; i < n; i += 1024) {
    v[0] += pos[3 * i];
    v[1] += pos[3 * i + 1];
    v[2] += pos[3 * i + 2];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) chain[c][t] = v[c];
  cl.sync();
  if (rank == 0) {
    double w[3][8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const double(*rc)[128] = cl.map_shared_rank(chain, r);
#pragma unroll
      for (int c = 0; c < 3; ++c) w[c][r] = rc[c][t];
    }
#pragma unroll
    for (int st = 4; st >= 1; st /= 2)  // chains 512, 256 and 128 apart
#pragma unroll
      for (int r = 0; r < st; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) w[c][r] += w[c][r + st];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; ++c) chain[c][t] = w[c][0];
    __syncthreads();
    for (int st = 64; st > 0; st /= 2) {
      if (t < st) {
#pragma unroll
        for (int c = 0; c < 3; ++c) chain[c][t] += chain[c][t + st];
      }
      __syncthreads();
    }
    if (t < 3) {
      cen[t] = chain[t][0] / (double)n;
      c_out[t] = cen[t];
    }
  }
  cl.sync();
  if (PACK) {
    const double* c = cl.map_shared_rank(cen, 0);
    const double cx = c[0], cy = c[1], cz = c[2];
    for (long long i = rank * 128 + t; i < n; i += 1024)
      out[i] = pack_row(pos, masses, cx, cy, cz, i);
    cl.sync();  // rank 0's centroid stays until every CTA has read it
  }
}

__global__ void pack_kernel(const double* __restrict__ pos, const double* __restrict__ masses,
                            const double* __restrict__ c, long long n, PackedBody* out) {
  after_previous(pos, masses, c, out);
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = pack_row(pos, masses, c[0], c[1], c[2], i);
}

// Registers: the one-lane packed loop (large systems) runs fastest with 56, 9
// CTAs of 128 threads on an SM (N = 100003 4.79 ms, 4.88 with those of 5; in one
// sweep, ms: 4.62 at 9, 4.68 at 8, 4.80 at 10, 4.87 at 5, 5.2 at 6 and 7; the same
// order at 16384 and 65536), the other forms,
// whose launches are shorter, with what 5 CTAs leave.
template <int T, int L, int BPT, bool PACKED, bool AFTER = false>
__global__ void __launch_bounds__(T, (PACKED && L == 1 && BPT == 1 ? 9 : 5) * 128 / T)
    rhs_mixed_kernel(const PackedBody* __restrict__ packed, const double* __restrict__ vel,
                     double* __restrict__ out_vel, double* __restrict__ out_acc, long long n,
                     float eps2, double mass, int uniform_mass) {
  if constexpr (AFTER) after_previous(packed, vel, out_vel, out_acc);
  constexpr int BI = (T / L) * BPT;
  constexpr int SH = PACKED ? jp_smem_bytes<T>() : (int)sizeof(PackedBody) * T;
  __shared__ __align__(16) unsigned char sh_raw[SH];
  __shared__ double part[BI][3];
  const ClusterInfo ci = cluster_info();
  const long long i0 = ci.itile * BI;
  long long jb, je;
  j_chunk(n, ci.rank, ci.size, T, jb, je);
  if constexpr (PACKED) {
    static_assert(BPT == 1 || BPT == 2, "packed loop: one or two bodies per thread");
    force_mixed_cta_jp<T, L, BPT>(packed, n, i0, jb, je, eps2, sh_raw, part);
  } else {
    PackedBody* sh = reinterpret_cast<PackedBody*>(sh_raw);
    if (uniform_mass)
      force_mixed_cta<T, L, BPT, true>(packed, n, i0, jb, je, eps2, sh, part);
    else
      force_mixed_cta<T, L, BPT, false>(packed, n, i0, jb, je, eps2, sh, part);
  }
  cluster_combine<BI>(part, ci.rank, ci.size);
  if (ci.rank != 0) return;
  const long long nb = min((long long)BI, n - i0);
  for (int e = threadIdx.x; e < 3 * nb; e += T) {
    const long long g = 3 * i0 + e;
    double a = part[e / 3][e % 3];
    if (uniform_mass) a = dmul(a, mass);
    out_vel[g] = vel[g];
    out_acc[g] = a;
  }
}

template <int T, bool FX>
const void* pick_f64(int L) {
  switch (L) {
    case 1: return (const void*)rhs_f64_kernel<T, 1, false, FX>;
    case 2: return (const void*)rhs_f64_kernel<T, 2, false, FX>;
    case 4: return (const void*)rhs_f64_kernel<T, 4, false, FX>;
    case 8: return (const void*)rhs_f64_kernel<T, 8, false, FX>;
    default: return nullptr;
  }
}
const void* pick_f64(const ForceGeom& g, bool fx) {
  switch (g.T) {
    case 64: return fx ? pick_f64<64, true>(g.L) : pick_f64<64, false>(g.L);
    case 128: return fx ? pick_f64<128, true>(g.L) : pick_f64<128, false>(g.L);
    case 256: return fx ? pick_f64<256, true>(g.L) : pick_f64<256, false>(g.L);
    default: return nullptr;
  }
}

// The kernel whose launch overlaps the one before it, for the geometries that the
// library picks itself, or null.
bool may_overlap(const ForceGeom& g) {
  return g.n_itiles * g.P <= (long long)kAfterCtasPerSm * num_sms();
}
template <bool FX>
const void* pick_f64_after(const ForceGeom& g) {
  if (g.T != 128 || !may_overlap(g)) return nullptr;
  switch (g.L) {
    case 2: return (const void*)rhs_f64_kernel<128, 2, true, FX>;
    case 4: return (const void*)rhs_f64_kernel<128, 4, true, FX>;
    case 8: return (const void*)rhs_f64_kernel<128, 8, true, FX>;
    default: return nullptr;
  }
}
template <int BPT, bool PACKED>
const void* pick_mixed_after_L(int L) {
  switch (L) {
    case 1: return (const void*)rhs_mixed_kernel<128, 1, BPT, PACKED, true>;
    case 2: return (const void*)rhs_mixed_kernel<128, 2, BPT, PACKED, true>;
    case 4: return (const void*)rhs_mixed_kernel<128, 4, BPT, PACKED, true>;
    default: return nullptr;
  }
}
const void* pick_mixed_after(const ForceGeom& g, bool packed) {
  if (g.T != 128 || !may_overlap(g)) return nullptr;
  if (packed && g.BPT == 1) return pick_mixed_after_L<1, true>(g.L);
  if (!packed && g.BPT == 2) return pick_mixed_after_L<2, false>(g.L);
  return nullptr;
}

template <int T, int BPT, bool PACKED>
const void* pick_mixed_L(int L) {
  switch (L) {
    case 1: return (const void*)rhs_mixed_kernel<T, 1, BPT, PACKED>;
    case 2: return (const void*)rhs_mixed_kernel<T, 2, BPT, PACKED>;
    case 4: return (const void*)rhs_mixed_kernel<T, 4, BPT, PACKED>;
    case 8: return (const void*)rhs_mixed_kernel<T, 8, BPT, PACKED>;
    default: return nullptr;
  }
}

// packed: the f32x2 path (pairs of bodies per thread, uniform masses)
template <int T>
const void* pick_mixed(int L, int BPT, bool packed = false) {
  if (packed && T <= 128 && BPT == 1) return pick_mixed_L<T, 1, true>(L);
  if (packed && T <= 128 && BPT == 2) return pick_mixed_L<T, 2, true>(L);
  switch (BPT) {
    case 1: return pick_mixed_L<T, 1, false>(L);
    case 2: return pick_mixed_L<T, 2, false>(L);
    default: return nullptr;
  }
}

// The packed loops run for uniform masses unless the tiling asks for the
// scalar loop (mixed_variant == 1).
bool use_packed(const gb_force_tiling* tiling, int BPT, const double* masses) {
  return (BPT == 1 || BPT == 2) && !masses && !(tiling && tiling->mixed_variant == 1);
}

int run_f64(const double* pos, const double* vel, double* out_vel, double* out_acc, long long n,
            double softening, double mass, const double* masses, int mode,
            const gb_force_tiling* tiling, cudaStream_t s) {
  ForceGeom g = choose_geom(n, GB_PREC_F64, tiling, 0);
  double eps2 = softening * softening;
  // Fixed-point pair terms (fixpair.cuh: closer to the exact sum than the
  // reference's operation order, and 14 times as fast at N = 16384) unless the
  // tiling asks for that order, or fixes the launch geometry, with it the
  // order of the sums, and says nothing else.
  const int want = tiling ? tiling->f64_pair : 0;
  const bool own_geom = tiling && (tiling->j_split > 0 || tiling->lanes > 0 ||
                                   tiling->bodies_per_cta > 0);
  int pair = want == 1                   ? kPairFixedFast
             : want == 0 && !own_geom ? kPairFixedIeee
                                      : kPairIeee;
  const bool fx = pair != kPairIeee;
  const void* k = pick_f64(g, fx);
  if (!k) return GB_ERR_UNSUPPORTED;
  void* args[] = {(void*)&pos, (void*)&vel, (void*)&out_vel, (void*)&out_acc, (void*)&n,
                  (void*)&eps2, (void*)&mass, (void*)&masses, (void*)&mode, (void*)&pair};
  const void* ka = fx ? pick_f64_after<true>(g) : pick_f64_after<false>(g);
  return launch_cluster(ka ? ka : k, g, 0, s, args, ka != nullptr);
}

}  // namespace

// Right-hand side for the integrator's start-up (initial step estimate): FP64
// with the integrator's tiling, or mixed from an already packed state.
int rhs_for_start(int prec, const double* x, double* dxdt, long long n, double softening,
                  double mass, const double* masses, const PackedBody* packed, int exact,
                  const gb_force_tiling* tiling, cudaStream_t s) {
  if (prec == GB_PREC_F64) {
    gb_force_tiling t = {};
    if (tiling) t = *tiling;
    if (exact) {
      t.j_split = 1;
      t.lanes = 1;
    }
    return run_f64(x, x + 3 * n, dxdt, dxdt + 3 * n, n, softening, mass, masses, kModeRhs, &t,
                   s);
  }
  ForceGeom g = choose_geom(n, GB_PREC_MIXED, tiling, 0, masses == nullptr);
  const void* k = nullptr;
  switch (g.T) {
    case 64: k = pick_mixed<64>(g.L, g.BPT, use_packed(tiling, g.BPT, masses)); break;
    case 128: k = pick_mixed<128>(g.L, g.BPT, use_packed(tiling, g.BPT, masses)); break;
    case 256: k = pick_mixed<256>(g.L, g.BPT, use_packed(tiling, g.BPT, masses)); break;
  }
  if (!k) return GB_ERR_UNSUPPORTED;
  const double* vel = x + 3 * n;
  double* out_vel = dxdt;
  double* out_acc = dxdt + 3 * n;
  float eps2 = (float)(softening * softening);
  int uniform = masses ? 0 : 1;
  void* args[] = {(void*)&packed, (void*)&vel,  (void*)&out_vel, (void*)&out_acc,
                  (void*)&n,      (void*)&eps2, (void*)&mass,    (void*)&uniform};
  return launch_cluster(k, g, 0, s, args);
}

int launch_cluster(const void* kernel, const ForceGeom& g, size_t smem, cudaStream_t s,
                   void** args, bool after) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(g.n_itiles * g.P), 1, 1);
  cfg.blockDim = dim3((unsigned)g.T, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)g.P;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = after && overlaps(s) ? 2 : 1;
  if (g.P > 8) {
    // clusters above 8 CTAs are opt-in per kernel; the attribute is set on
    // the first (uncaptured) launch and persists
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    GB_CUDA_TRY(cudaStreamIsCapturing(s, &cs));
    if (cs == cudaStreamCaptureStatusNone)
      GB_CUDA_TRY(
          cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  GB_CUDA_TRY(cudaLaunchKernelExC(&cfg, kernel, args));
  return GB_OK;
}

ForceGeom choose_geom(long long n, int precision, const gb_force_tiling* tiling, int exact,
                      bool uniform_masses) {
  ForceGeom g;
  g.T = 128;
  g.L = 1;
  g.P = 1;
  g.BPT = 1;
  g.variant = 0;
  const int sms = num_sms();
  if (exact) {
    g.L = 1;
    g.P = 1;
  } else if (precision == GB_PREC_F64) {
    if (n >= 4096) {
      // 8 cluster ranks and lanes for about 2048 CTAs of 128 threads, so that
      // the pair loop balances across the SMs.  Chosen with FP64 terms (a stage,
      // ms: N = 16384 23.9 at 8 x 2 against 25.5 at 4 x 1; 4096 1.51 at 8 x 8
      // against 1.60 at 8 x 2) and kept for the fixed-point terms (1.67 and 0.137).
      int L = 1;
      while (L < 8 && (long long)L * 2 * n <= 32768) L *= 2;
      g.P = 8;
      g.L = L;
    } else if (n < 768) {
      // a few pairs a lane: lanes rather than ranks (fixed-point terms, N = 257
      // 12.6 us against 14.9 with 8 ranks x 4 lanes, 512 12.5 against 16.8, 1024
      // 17.1 against 16.8)
      g.P = 4;
      g.L = 8;
    } else {
      // Aim for ~8 resident warps per SM over the whole grid.
      long long want = (long long)sms * 8 * 32;
      long long lp = (want + n - 1) / n;
      int P = 1;
      while (P < 8 && P < lp) P *= 2;
      int L = 1;
      while (L < 4 && (long long)P * L < lp) L *= 2;
      g.P = P;
      g.L = L;
    }
  } else {
    int v = tiling ? tiling->mixed_variant : 0;
    if (v < 1 || v > 3) v = kDefaultMixedVariant;
    if (!uniform_masses) v = 1;
    g.variant = v;
    g.BPT = v == 3 ? 1 : 2;
    // ~32 warps' worth of two-body threads per SM, each lane pair-loop at
    // least ~256 partners long; lanes only when the cluster split leaves the
    // grid well short of that (measured with the partner-pair loop: N = 4096
    // runs fastest at 8 ranks x 2 lanes, N = 16384 at 8 x 1, N = 65536 at 4 x 1).
    long long want = (long long)sms * 16 * 32 * 2;
    long long lp = (want + n - 1) / n;
    int P = 1;
    while (P < 8 && P < lp && n / (2 * P) >= 256) P *= 2;
    int L = 1;
    const int lmax = g.BPT == 1 ? 2 : 4;
    while (L < lmax && 2LL * P * L < lp && n / (2 * P * L) >= 128) L *= 2;
    g.P = P;
    g.L = L;
  }
  if (tiling) {
    if (tiling->j_split > 0) g.P = tiling->j_split;
    if (tiling->lanes > 0) g.L = tiling->lanes;
    if (tiling->bodies_per_cta > 0) {
      // bodies per CTA = (T / L) * BPT
      int t = tiling->bodies_per_cta * g.L / g.BPT;
      g.T = t <= 64 ? 64 : (t <= 128 ? 128 : 256);
    }
  }
  // the packed loops stage 2T partners per tile: 128 threads per CTA
  if (precision == GB_PREC_MIXED && g.variant != 1 && !exact) g.T = 128;
  const long long per_cta = g.bodies_per_cta();
  g.n_itiles = (n + per_cta - 1) / per_cta;
  return g;
}

}  // namespace gb

using namespace gb;

extern "C" int gb_nbody_rhs_f64(const double* x, double* dxdt, int64_t n, double softening,
                                double mass, const double* masses, const gb_force_tiling* tiling,
                                gb_stream_t stream) {
  GB_TRY(validate_nbody(x, dxdt, n, softening, mass, masses));
  return run_f64(x, x + 3 * n, dxdt, dxdt + 3 * n, n, softening, mass, masses, kModeRhs, tiling,
                 as_cuda(stream));
}

extern "C" int gb_nbody_acc_f64(const double* pos, double* acc, int64_t n, double softening,
                                double mass, const double* masses, int32_t accumulate,
                                const gb_force_tiling* tiling, gb_stream_t stream) {
  GB_TRY(validate_nbody(pos, acc, n, softening, mass, masses));
  return run_f64(pos, nullptr, nullptr, acc, n, softening, mass, masses,
                 accumulate ? kModeAccAdd : kModeAccWrite, tiling, as_cuda(stream));
}

namespace gb {
// Mixed-precision right-hand side into caller-located scratch: `packed`
// (n PackedBody records, 16-byte aligned) and `c` (3 doubles).  Both
// gb_nbody_rhs_mixed (workspace from the caller) and
// gb_nbody_rhs_mixed_noalloc (workspace inside the library) run through it,
// so the two give identical bits; allocates nothing.
int mixed_rhs_into(const double* x, double* dxdt, long long n, double softening, double mass,
                   const double* masses, PackedBody* packed, double* c,
                   const gb_force_tiling* tiling, cudaStream_t s) {
  if (n <= kFusedPackBodies) {
    GB_CUDA_TRY(launch_after(centroid_kernel<true>, kCentroidCtas, 128, s, x, masses, n, c, packed));
  } else {
    GB_CUDA_TRY(launch_after(centroid_kernel<false>, kCentroidCtas, 128, s, x, nullptr, n, c, nullptr));
    GB_CUDA_TRY(launch_after(pack_kernel, (unsigned)((n + 255) / 256), 256, s, x, masses, c, n, packed));
  }
  ForceGeom g = choose_geom(n, GB_PREC_MIXED, tiling, 0, masses == nullptr);
  const void* k = nullptr;
  switch (g.T) {
    case 64: k = pick_mixed<64>(g.L, g.BPT, use_packed(tiling, g.BPT, masses)); break;
    case 128: k = pick_mixed<128>(g.L, g.BPT, use_packed(tiling, g.BPT, masses)); break;
    case 256: k = pick_mixed<256>(g.L, g.BPT, use_packed(tiling, g.BPT, masses)); break;
  }
  if (!k) return GB_ERR_UNSUPPORTED;
  const double* vel = x + 3 * n;
  double* out_vel = dxdt;
  double* out_acc = dxdt + 3 * n;
  float eps2 = (float)(softening * softening);
  int uniform = masses ? 0 : 1;
  void* args[] = {(void*)&packed, (void*)&vel,  (void*)&out_vel, (void*)&out_acc,
                  (void*)&n,      (void*)&eps2, (void*)&mass,    (void*)&uniform};
  const void* ka = pick_mixed_after(g, use_packed(tiling, g.BPT, masses));
  return launch_cluster(ka ? ka : k, g, 0, s, args, ka != nullptr);
}
}  // namespace gb

namespace gb {
namespace {

// Mixed-precision right-hand side on Morton-sorted tiles (near hi/lo path
// plus the tile-centroid far path); rows are written back in body order.
template <int T, int L, bool UNIFORM>
__global__ void __launch_bounds__(T, 1024 / T)
    rhs_sorted_kernel(const PackedBody* __restrict__ near, const float4* __restrict__ far,
                      const TileMeta* __restrict__ meta, const int* __restrict__ perm,
                      const double* __restrict__ vel, double* __restrict__ out_vel,
                      double* __restrict__ out_acc, long long n, float eps2, double mass) {
  __shared__ __align__(16) PackedBody sh[T];
  __shared__ double part[T][3];
  const ClusterInfo ci = cluster_info();
  long long jb, je;
  j_chunk(n, ci.rank, ci.size, T, jb, je);
  force_mixed_sorted_cta<T, L, L, UNIFORM>(near, far, meta, n, ci.itile, jb, je, eps2, sh, part);
  cluster_combine<T>(part, ci.rank, ci.size);
  if (ci.rank != 0) return;
  const long long i = ci.itile * T + threadIdx.x;
  if (i >= n) return;
  const long long id = perm[i];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    out_vel[3 * id + c] = vel[3 * id + c];
    out_acc[3 * id + c] = UNIFORM ? dmul(part[threadIdx.x][c], mass) : part[threadIdx.x][c];
  }
}

struct SortedWork {
  PackedBody* near;
  float4* far;
  TileMeta* meta;
  SortBuffers sb;
  double* cref;
  size_t total;
};

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

SortedWork sorted_layout(long long n, void* base) {
  const long long nt = (n + 127) / 128;
  char* p = static_cast<char*>(base);
  SortedWork w;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = p ? p + off : nullptr;
    off += align256(bytes);
    return q;
  };
  w.near = reinterpret_cast<PackedBody*>(take((size_t)n * sizeof(PackedBody)));
  w.far = reinterpret_cast<float4*>(take((size_t)n * sizeof(float4)));
  w.meta = reinterpret_cast<TileMeta*>(take((size_t)nt * sizeof(TileMeta)));
  w.sb.perm = reinterpret_cast<int*>(take((size_t)n * sizeof(int)));
  w.sb.vals = reinterpret_cast<int*>(take((size_t)n * sizeof(int)));
  w.sb.keys = reinterpret_cast<unsigned long long*>(take((size_t)n * 8));
  w.sb.keys_alt = reinterpret_cast<unsigned long long*>(take((size_t)n * 8));
  w.sb.bbox = reinterpret_cast<double*>(take(8 * sizeof(double)));
  w.cref = reinterpret_cast<double*>(take(4 * sizeof(double)));
  w.sb.cub_bytes = sort_temp_bytes(n);
  w.sb.cub_temp = take(w.sb.cub_bytes);
  w.total = off;
  return w;
}

template <int T, int L>
const void* pick_rhs_sorted(bool uniform) {
  return uniform ? (const void*)rhs_sorted_kernel<T, L, true>
                 : (const void*)rhs_sorted_kernel<T, L, false>;
}

}  // namespace
}  // namespace gb

extern "C" size_t gb_nbody_mixed_sorted_workspace_bytes(int64_t n) {
  return n < 1 ? 0 : gb::sorted_layout(n, nullptr).total;
}

extern "C" int gb_nbody_rhs_mixed_sorted(const double* x, double* dxdt, int64_t n,
                                         double softening, double mass, const double* masses,
                                         void* work, size_t work_bytes,
                                         const gb_force_tiling* tiling, gb_stream_t stream) {
  using namespace gb;
  GB_TRY(validate_nbody(x, dxdt, n, softening, mass, masses));
  if (!(softening > 0.0) || !work || (reinterpret_cast<uintptr_t>(work) & 255u))
    return GB_ERR_INVALID_ARGUMENT;
  SortedWork w = sorted_layout(n, work);
  if (work_bytes < w.total) return GB_ERR_CAPACITY;
  cudaStream_t s = as_cuda(stream);
  centroid_kernel<false><<<kCentroidCtas, 128, 0, s>>>(x, nullptr, n, w.cref, nullptr);
  GB_CUDA_TRY(cudaGetLastError());
  const long long nt = (n + 127) / 128;
  GB_TRY(sort_and_pack(x, nullptr, 0, n, w.sb, masses, w.cref, w.near, w.far, w.meta, nullptr,
                       nt, 128, s));
  ForceGeom g = choose_geom(n, GB_PREC_MIXED, tiling, 0, masses == nullptr);
  g.T = 128;
  if (g.L > 2) g.L = 2;
  g.BPT = g.L;
  g.n_itiles = nt;
  const void* k = g.L == 1 ? pick_rhs_sorted<128, 1>(masses == nullptr)
                           : pick_rhs_sorted<128, 2>(masses == nullptr);
  const PackedBody* near = w.near;
  const float4* far = w.far;
  const TileMeta* meta = w.meta;
  const int* perm = w.sb.perm;
  const double* vel = x + 3 * n;
  double* out_vel = dxdt;
  double* out_acc = dxdt + 3 * n;
  float eps2 = (float)(softening * softening);
  long long nn = n;
  void* args[] = {(void*)&near, (void*)&far, (void*)&meta, (void*)&perm, (void*)&vel,
                  (void*)&out_vel, (void*)&out_acc, (void*)&nn, (void*)&eps2, (void*)&mass};
  return launch_cluster(k, g, 0, s, args);
}

extern "C" size_t gb_nbody_mixed_workspace_bytes(int64_t n) {
  if (n < 1) return 0;
  // packed bodies + reference point (3 doubles), 256-byte aligned pieces
  size_t packed = ((size_t)n * sizeof(PackedBody) + 255) / 256 * 256;
  return packed + 256;
}

extern "C" int gb_nbody_rhs_mixed(const double* x, double* dxdt, int64_t n, double softening,
                                  double mass, const double* masses, void* work,
                                  const gb_force_tiling* tiling, gb_stream_t stream) {
  GB_TRY(validate_nbody(x, dxdt, n, softening, mass, masses));
  if (!work || (reinterpret_cast<uintptr_t>(work) & 15u)) return GB_ERR_INVALID_ARGUMENT;
  if (!(softening > 0.0)) return GB_ERR_INVALID_ARGUMENT;
  PackedBody* packed = reinterpret_cast<PackedBody*>(work);
  const size_t packed_bytes = ((size_t)n * sizeof(PackedBody) + 255) / 256 * 256;
  double* c = reinterpret_cast<double*>(reinterpret_cast<char*>(work) + packed_bytes);
  return mixed_rhs_into(x, dxdt, n, softening, mass, masses, packed, c, tiling, as_cuda(stream));
}
