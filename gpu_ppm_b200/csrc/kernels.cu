// Engine kernels: work planner, persistent integrand (NSX FP32 and blackbody
// FP64/FP32 variants) and SIMT response folds.
//
// Two forms.  Batches whose rings fill the GPU run from tiles: a CTA per tile does
// all of the steps below.  Small ones (a single profile, a served batch) and
// blackbody spectra run from ring records: ring_kernel does steps 1 to 5 once a
// ring, the *_rec kernels do step 6 for a ring's phase nodes, any CTA taking any
// node, and sum_parts_kernel adds the stored node sums.  NSX results are the same
// bits in both forms; blackbody results agree to about 1e-16 (FP64 sums in another
// order), FP32 blackbody ones to some units of 2^-23 times E / kT.
//
// Integrand structure (one CTA per tile = candidate elements of one ring of
// one spot of one profile; CTAs pull tiles from a device queue, except in the
// blackbody kernel's fused point-source mode, where CTA b takes profile b's
// point spots without a planner):
//   1. ring geometry                      cpu/devarshi24st_cpu.cpp:90-124
//   2. active-element compaction by warp ballot + prefix (deterministic order)
//                                         gpu/devarshi24st_gpu.cu:196-212
//   3. two lensing rows of each table staged in shared memory, FP64 sweep of
//      the fine phases                    cpu/devarshi24st_cpu.cpp:126-193
//   4. gap fill / wrap                    cpu/devarshi24st_cpu.cpp:195-212
//   5. NSX (logT, logg) slice pre-reduced into shared memory (FP32)
//                                         gpu/devarshi24st_gpu.cu:323-351
//   6. deposit: rounds of phase points (FP64 phase, hunt, lerps, mu weights),
//      visible ones compacted into records; per record the mu-contracted slice
//      becomes per-cell cubic polynomials in log(E/kT), evaluated for the
//      observed energies with per-bin partial sums in registers (no
//      per-element atomics); a bin's partial sums are flushed once into the
//      FP64 flux pool                     cpu/devarshi24st_cpu.cpp:214-241
//      Home-cell kernel (default): each lane owns the energies of a few NSX
//      cells and builds their cubics in registers from shuffled slice rows,
//      two records at a time.
//      Pooled-polynomial kernel (grids with > 16 energies in one cell): one
//      warp per point writes the cubics to shared memory, one thread per
//      energy reads its cell's cubic.
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "kernels.cuh"

namespace ppm {
namespace {

// Barrier of one warp set of n threads (a multiple of 32): the warp itself for
// a one-warp set, else named barrier 1 + set.
__device__ __forceinline__ void set_sync(int set, int n) {
  if (n == 32)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(1 + set), "r"(n) : "memory");
}

// 16-byte asynchronous copy from global to shared memory.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace
}  // namespace ppm

#include "rec_loop.cuh"

namespace ppm {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr double kTwoPi = 2. * kPi;
constexpr int kSlotBytes = 48;  // bytes per batch point (SoA)
constexpr int kBbPass = 128;        // blackbody from ring records: energies per pass
constexpr int kPhaseMajorMaxE = 4;  // blackbody grids of at most this many energies take the phase-major walk

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Block-wide ordered compaction: returns this thread's slot among flagged
// threads (or -1) and the total through *total.  Uses scratch[32].
__device__ __forceinline__ int block_compact(bool flag, int* scratch, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  unsigned b = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) scratch[warp] = __popc(b);
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int w = 0; w < nw; ++w) {
      int c = scratch[w];
      scratch[w] = run;
      run += c;
    }
    scratch[32] = run;
  }
  __syncthreads();
  int pos = flag ? scratch[warp] + __popc(b & lanemask_lt()) : -1;
  *total = scratch[32];
  return pos;
}

struct SmemPtrs {
  unsigned short* j;  // active elements' indices in the ring (at most 4 N_side = 32768)
  double *P, *F, *Z, *MU, *mu;
  float* S;
  double* rows;
  unsigned char* batch;
  float4* Q;
  float* H;
  unsigned short* hidx;  // home-cell kernel: bracket table of phase_o (see node_point_tab)
};

__device__ __forceinline__ SmemPtrs carve(unsigned char* sm, const IntegrandShape& S) {
  SmemPtrs s;
  s.j = (unsigned short*)(sm + S.off_j);
  s.P = (double*)(sm + S.off_P);
  s.F = (double*)(sm + S.off_F);
  s.Z = (double*)(sm + S.off_Z);
  s.MU = (double*)(sm + S.off_MU);
  s.mu = (double*)(sm + S.off_mu);
  s.S = (float*)(sm + S.off_S);
  s.rows = (double*)(sm + S.off_rows);
  s.batch = sm + S.off_batch;
  s.Q = (float4*)(sm + S.off_Q);
  s.H = (float*)(sm + S.off_Q + (S.nsx ? S.pb * S.cells * 16 : 0));
  s.hidx = (unsigned short*)(sm + S.off_hidx);
  return s;
}

// Stages the two lensing rows of each table and sweeps the fine phases: returns
// whether the ring is dropped (fine sample 0 or n_fine - 1 invisible,
// cpu/devarshi24st_cpu.cpp:195); if not, P/F/Z/MU hold the filled and wrapped
// arrays.  s_g is visible to all threads; block barriers inside.
__device__ __forceinline__ bool ring_sweep(const KernelArgs& a, const DevProfile& p, const SmemPtrs& s,
                                           const RingGeom& s_g, int* s_int, bool nsx) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const DevLens& L = a.lens;
  if (tid == 0) {
    s_int[40] = p.n_fine + 1;  // invisible min
    s_int[41] = -1;            // invisible max
  }
  // stage the two lensing rows of each table
  const int ncp = L.n_cp, nca = L.n_ca, iu = s_g.i_u;
  double* r = s.rows;
  for (int k = tid; k < 2 * ncp; k += nt) {
    int row = k / ncp, col = k - row * ncp;
    r[k] = L.ca[(size_t)(iu + row) * ncp + col];
    r[2 * ncp + k] = L.lf[(size_t)(iu + row) * ncp + col];
  }
  for (int k = tid; k < 2 * nca; k += nt) {
    int row = k / nca, col = k - row * nca;
    r[4 * ncp + k] = L.cdt[(size_t)(iu + row) * nca + col];
  }
  __syncthreads();
  LensRows rows{r, r + ncp, r + 2 * ncp, r + 3 * ncp, r + 4 * ncp, r + 4 * ncp + nca};
  const RingGeom g = s_g;
  const int nf = p.n_fine;
  for (int i = tid; i < nf; i += nt) {
    double F, Z, P, MU;
    if (sweep_sample(p, L, g, rows, i, nsx, F, Z, P, MU)) {
      s.F[i] = F;
      s.Z[i] = Z;
      s.P[i] = P;
      s.MU[i] = MU;
    } else {
      s.F[i] = 0;
      s.Z[i] = -1;
      s.P[i] = -1;
      s.MU[i] = 0;
      atomicMin(&s_int[40], i);
      atomicMax(&s_int[41], i);
    }
  }
  __syncthreads();
  const int inv_min = s_int[40], inv_max = s_int[41];
  if (inv_min == 0 || inv_max == nf - 1) return true;
  if (inv_min <= inv_max) {
    const int beg = inv_min - 1, end = inv_max + 1;
    const double p0 = s.P[beg], p1 = s.P[end], z0 = s.Z[beg], z1 = s.Z[end];
    for (int i = inv_min + tid; i <= inv_max; i += nt) {
      s.P[i] = p0 + (p1 - p0) * ((double)(i - beg) / (end - beg));
      s.Z[i] = z0 + (z1 - z0) * ((double)(i - beg) / (end - beg));
    }
  }
  __syncthreads();
  if (tid == 0) {
    s.F[nf] = s.F[0];
    s.Z[nf] = s.Z[0];
    s.P[nf] = 1.0 + s.P[0];
    s.MU[nf] = s.MU[0];
  }
  __syncthreads();
  return false;
}

// Steps 1-4 for one tile.  Returns the number of active elements (0 = nothing to do).
// On return (non-zero), P/F/Z/MU hold the filled fine-phase arrays and s_g the ring geometry.
__device__ int tile_prologue(const KernelArgs& a, const DevProfile& p, const DevSpot& sp, const Tile& tile,
                             const SmemPtrs& s, RingGeom& s_g, int* s_int, bool nsx) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const bool point = sp.kind == 1;
  const DevLens& L = a.lens;
  if (tid == 0) {
    double cos_t = point ? sp.cos_theta_pt : p.ring[3 * tile.ring];
    double dOmega = point ? sp.dOmega_pt : p.dOmega_hp;
    ring_geometry(p, L, cos_t, dOmega, nsx, s_g);
  }
  // compaction of active elements over the candidate range
  int n_act = 0;
  if (point) {
    if (tid == 0) s.j[0] = 0;
    n_act = 1;
  } else {
    const int N = p.n_side, ring = tile.ring;
    const double c2 = p.ring[3 * ring + 1], s2 = p.ring[3 * ring + 2];
    const int n_c = tile.j1 - tile.j0;
    for (int k0 = 0; k0 < n_c; k0 += nt) {
      int k = k0 + tid;
      bool flag = false;
      if (k < n_c) flag = in_spot(sp, c2, s2, healpix_phi(N, ring, tile.j0 + k));
      int tot;
      int pos = block_compact(flag, s_int, &tot);
      if (flag) s.j[n_act + pos] = (unsigned short)(tile.j0 + k);
      n_act += tot;
      __syncthreads();
    }
  }
  __syncthreads();
  if (n_act == 0) return 0;
  // counted by the tiles of the first node range only; a ring counts once, by the first of its tiles to
  // find active elements.  In the fused point-source mode no planner has dropped the ring yet: the counting
  // waits for the sweep's drop test below
  auto count_ring = [&]() {
    atomicAdd(&p.stats[0], (unsigned long long)n_act);
    const unsigned bit = 1u << (tile.ring & 31);
    if (!(atomicOr(&p.ring_seen[tile.spot * p.ring_words + (tile.ring >> 5)], bit) & bit))
      atomicAdd(&p.stats[1], 1ull);
    if (s_g.u_clamped && tile.first) atomicAdd(&p.stats[4], 1ull);
  };
  const bool fused = a.n_fused > 0;
  if (tid == 0) {
    if (tile.u0 == 0 && !fused) count_ring();
  }
  const bool dropped = ring_sweep(a, p, s, s_g, s_int, nsx);
  if (fused && tid == 0) {
    if (!dropped) {
      count_ring();
    } else {  // the planner's count of a dropped ring (plan_kernel)
      atomicAdd(&p.stats[1], 1ull);
      atomicAdd(&p.stats[2], 1ull);
      atomicAdd(&p.stats[5], (unsigned long long)n_act);
    }
  }
  return dropped ? 0 : n_act;
}

// Ring range of disk 1 in element index j: up to two [j_lo, j_hi] ranges
// (with a one-element margin) that contain every active element.
__device__ int candidate_ranges(const DevSpot& s, int N, int i, double c2, double s2, int jmax, int r[2][2]) {
  const double A = s.s1 * s2, B = s.c1 * c2;
  bool full = false;
  double w = 0.0;
  if (A < 1e-12) {
    if (B > s.cos_ar1 - 1e-9)
      full = true;
    else
      return 0;
  } else {
    const double qv = (s.cos_ar1 - B) / A;
    if (qv > 1.0 + 1e-9) return 0;
    if (qv <= -1.0)
      full = true;
    else
      w = acos(fmin(qv, 1.0)) + 1e-7;
    if (w >= kPi) full = true;
  }
  if (full) {
    r[0][0] = 1;
    r[0][1] = jmax;
    return 1;
  }
  const int ii = i > 2 * N ? 4 * N - i : i;
  const double sh = ii < N ? 0.5 : 0.5 * ((ii - N + 1) % 2);
  const double dphi = kTwoPi / jmax;
  const double jc = s.ph1 / dphi + sh, jw = w / dphi;
  long long jlo = (long long)floor(jc - jw) - 1, jhi = (long long)ceil(jc + jw) + 1;
  const long long len = jhi - jlo + 1;
  if (len >= jmax) {
    r[0][0] = 1;
    r[0][1] = jmax;
    return 1;
  }
  long long m = ((jlo - 1) % jmax + jmax) % jmax + 1;  // jlo mapped into [1, jmax]
  if (m + len - 1 <= jmax) {
    r[0][0] = (int)m;
    r[0][1] = (int)(m + len - 1);
    return 1;
  }
  r[0][0] = (int)m;
  r[0][1] = jmax;
  r[1][0] = 1;
  r[1][1] = (int)(m + len - 1 - jmax);
  return 2;
}

// Phase node u = bin * n_gl + GL point (u = bin when n_gl = 0): its bin, its
// phase ppt and GL weight (cpu/devarshi24st_cpu.cpp:214-219).  width: 1. / n_bins.
__device__ __forceinline__ void node_phase(int n_gl, double width, int u, int& bin, double& ppt, double& wgl) {
  if (n_gl > 0) {
    bin = u / n_gl;
    const int g = u - bin * n_gl;
    const double lb = bin * width, ub = (bin + 1) * width;
    ppt = 0.5 * (lb + ub + c_gl_nodes[n_gl * (n_gl - 1) / 2 + g] * (ub - lb));
    wgl = 0.5 * 1. * c_gl_weights[n_gl * (n_gl - 1) / 2 + g];
  } else {
    bin = u;
    ppt = bin * width;
    wgl = 1.0;
  }
}
__device__ __forceinline__ void node_phase(const DevProfile& p, int u, int& bin, double& ppt, double& wgl) {
  node_phase(p.n_gl, 1. / p.n_bins, u, bin, ppt, wgl);
}

// Active element jj of the tile at phase ppt: patch phase, hunt and lerps in
// FP64 (cpu/devarshi24st_cpu.cpp:220-229).  Returns flux/I (0 = skip).
__device__ __forceinline__ double node_point(const DevProfile& p, const SmemPtrs& s, const RingPhi& rp, bool point,
                                             int jj, double ppt, double& z, double& mu) {
  const double phi = point ? 0.0 : rp.dphi * (s.j[jj] - rp.jofs);
  const double phase_shift = phi / kTwoPi;
  // fmod(x, 1) of x = ppt + phase_shift + 1 in [1, 3): x - floor(x) is the same exact value
  const double xph = ppt + phase_shift + 1.;
  double patch = xph - floor(xph);
  if (patch < s.P[0]) patch += 1.;
  double af;
  const int i = vhunt(s.P, p.n_fine + 1, patch, af);
  const double flux = (1 - af) * s.F[i] + af * s.F[i + 1];
  if (flux == 0) return 0.0;
  z = (1 - af) * s.Z[i] + af * s.Z[i + 1];
  mu = (1 - af) * s.MU[i] + af * s.MU[i + 1];
  return flux;
}

// Phase point q of the tile's node range (node u0 + q / n_act, element q % n_act).
__device__ __forceinline__ double phase_point(const DevProfile& p, const SmemPtrs& s, const RingPhi& rp, bool point,
                                              int n_act, int u0, int q, int& bin, double& wgl, double& z, double& mu) {
  const int du = q / n_act, jj = q - du * n_act;
  double ppt;
  node_phase(p, u0 + du, bin, ppt, wgl);
  return node_point(p, s, rp, point, jj, ppt, z, mu);
}

// phase_point's arithmetic for one element at phase point i_pp, for the
// blackbody kernel's point-wise path, with the per-tile and per-element terms
// (n = n_fine + 1, phase_o[0], 1 / n_bins, the element's phase shift
// phi / 2 pi) computed once by the caller.  When the tile's phase_o is
// non-decreasing (mono), the bracket is hunted from `hint`, this thread's
// previous one, which gives vhunt's bracket exactly, and the fraction uses
// the tile's reciprocal interval widths inv_dp when given (within an ulp of
// vhunt's division).
__device__ __forceinline__ double phase_point_at(const SmemPtrs& s, int n, double P0, const double* inv_dp, int n_gl,
                                                 double inv_bins, double phase_shift, int i_pp, bool mono, int& hint,
                                                 int& bin, double& wgl, double& z) {
  int g = 0;
  if (n_gl > 0) {
    bin = i_pp / n_gl;
    g = i_pp - bin * n_gl;
  } else {
    bin = i_pp;
  }
  double ppt;
  if (n_gl > 0) {
    const double width = inv_bins;
    const double lb = bin * width, ub = (bin + 1) * width;
    ppt = 0.5 * (lb + ub + c_gl_nodes[n_gl * (n_gl - 1) / 2 + g] * (ub - lb));
    wgl = 0.5 * 1. * c_gl_weights[n_gl * (n_gl - 1) / 2 + g];
  } else {
    ppt = bin * inv_bins;
    wgl = 1.0;
  }
  const double xph = ppt + phase_shift + 1.;
  double patch = xph - floor(xph);
  if (patch < P0) patch += 1.;
  double af;
  int i;
  if (mono) {
    hint = hunt_from(s.P, n, patch, hint);
    i = clampi(hint, 0, n - 2);
    af = inv_dp ? (patch - s.P[i]) * inv_dp[i] : (patch - s.P[i]) / (s.P[i + 1] - s.P[i]);
  } else {
    i = vhunt(s.P, n, patch, af);
  }
  const double flux = (1 - af) * s.F[i] + af * s.F[i + 1];
  if (flux == 0) return 0.0;
  z = (1 - af) * s.Z[i] + af * s.Z[i + 1];
  return flux;
}

// ---------------------------------------------------------------------------
template <int NE_T, int MINB>
__global__ void __launch_bounds__(MINB == 1 ? 512 : 320, MINB) integrand_nsx_kernel(const KernelArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  const IntegrandShape& S = a.shape;
  const SmemPtrs s = carve(sm, S);
  __shared__ RingGeom s_g;
  __shared__ int s_int[48];
  __shared__ int s_tile;
  __shared__ float s_tapw[16];
  __shared__ int s_tapo[16];
  __shared__ int s_ntap;
  const int tid = threadIdx.x, nt = blockDim.x;
  const DevNsx& X = a.nsx;
  const int nE = X.nE, nmu = X.nmu, cells = S.cells, HN = cells + 3;

  // point records, one slot per thread: {c, fP, bin, G0} packed for one broadcast load,
  // plus the mu stencil start and weights
  float4* r_pk = (float4*)s.batch;
  int* r_imu = (int*)(r_pk + nt);
  float* r_w = (float*)(r_imu + nt);  // [4][nt]

  for (;;) {
    __syncthreads();
    if (tid == 0) s_tile = atomicAdd(a.queue.next, 1);
    __syncthreads();
    const int t = s_tile;
    if (t >= *a.queue.n_tiles || t >= a.queue.capacity) break;
    const Tile tile = a.queue.tiles[t];
    const DevProfile& p = a.profiles[tile.profile];
    const DevSpot& sp = p.spot[tile.spot];
    const bool point = sp.kind == 1;
    const int n_act = tile_prologue(a, p, sp, tile, s, s_g, s_int, true);
    if (n_act == 0) continue;
    const RingPhi rp = point ? RingPhi{0.0, 0.0} : healpix_ring_phi(p.n_side, tile.ring);

    // ---- step 5: (logT, logg) pre-reduction of the NSX table into S[E][mu]
    if (tid == 0) {
      const bool cubic = (p.interp == 0 || p.interp == 1 || p.interp == 2);
      double lg = s_g.logg, ag;
      s_int[45] = (lg < X.g_min || lg > X.g_max) ? 1 : 0;
      s_int[44] = 0;
      int ig = uhunt(lg, X.g_min, X.g_max, X.ng, ag);
      double wg[4];
      int ig0, ngt;
      if (cubic) {
        ig0 = clampi(ig - 1, 0, X.ng - 4);
        cubic_lagrange(wg, lg, uhunt_at(X.g_min, X.g_max, X.ng, ig0), uhunt_at(X.g_min, X.g_max, X.ng, ig0 + 1),
                       uhunt_at(X.g_min, X.g_max, X.ng, ig0 + 2), uhunt_at(X.g_min, X.g_max, X.ng, ig0 + 3));
        ngt = 4;
      } else {
        ig0 = ig;
        wg[0] = 1 - ag;
        wg[1] = ag;
        ngt = 2;
      }
      int n = 0;
      for (int jt = 0; jt < sp.nT_taps; ++jt)
        for (int jg = 0; jg < ngt; ++jg) {
          s_tapw[n] = (float)(sp.wT[jt] * wg[jg]);
          s_tapo[n] = (sp.iT[jt] * X.ng + ig0 + jg) * X.slice_stride;
          ++n;
        }
      s_ntap = n;
    }
    for (int k = tid; k < nmu; k += nt) s.mu[k] = X.mu[k];
    for (int k = tid; k < 4 * (nmu - 3); k += nt) s.mu[nmu + k] = X.mu_den[k];
    __syncthreads();
    {
      const int n4 = X.slice_stride >> 2, ntap = s_ntap;
      float4* S4 = (float4*)s.S;
      for (int k = tid; k < n4; k += nt) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < ntap; ++q) {
          const float4 v = __ldg((const float4*)(X.data + s_tapo[q]) + k);
          const float w = s_tapw[q];
          acc.x = fmaf(w, v.x, acc.x);
          acc.y = fmaf(w, v.y, acc.y);
          acc.z = fmaf(w, v.z, acc.z);
          acc.w = fmaf(w, v.w, acc.w);
        }
        S4[k] = acc;
      }
    }
    __syncthreads();

    // ---- step 6: deposit
    const DevGrid& G = p.grid;
    const int n_e = G.n_e;
    int rE[NE_T];
    float fE[NE_T];
    float acc[NE_T];
#pragma unroll
    for (int k = 0; k < NE_T; ++k) {
      const int e = tid + k * nt;
      const bool ok = e < n_e;
      rE[k] = ok ? G.rE[e] : 0;
      fE[k] = ok ? G.fE[e] : 0.f;
      acc[k] = 0.f;
    }
    const int mode = p.interp;
    const bool cubicE = mode != 4;
    const bool sg = mode == 1;
    const double mu_min = s.mu[nmu - 1];
    const int n_pp = tile.u1 - tile.u0;  // the tile's phase nodes
    const int n_pts = n_pp * n_act;
    int cur_bin = -1;
    double* flux_base = a.flux + p.flux_off;
    const double out_scale = sp.out_scale;

    double* comp_base = a.comp ? a.comp + p.flux_off : nullptr;
    auto flush = [&]() {
#pragma unroll
      for (int k = 0; k < NE_T; ++k) {
        const int e = tid + k * nt;
        if (e < n_e && acc[k] != 0.f) {
          const size_t o = (size_t)cur_bin * n_e + e;
          comp_add(flux_base + o, comp_base ? comp_base + o : nullptr, (double)acc[k] * out_scale * G.invE[e]);
        }
        acc[k] = 0.f;
      }
    };

    const int lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    const double* den = s.mu + nmu;  // [nmu - 3][4] reciprocal Lagrange denominators
    for (int q0 = 0; q0 < n_pts; q0 += nt) {
      // stage A: every thread evaluates one phase point (FP64); visible ones are
      // compacted, in order, into the point records
      bool vis = false, clamped = false;
      float c = 0.f, fP = 0.f;
      int G0 = 0, bin = 0, imu = 0;
      float w4[4] = {0.f, 0.f, 0.f, 0.f};
      const int q = q0 + tid;
      if (q < n_pts) {
        double wgl, z = 0, mu = 0;
        const double flux = phase_point(p, s, rp, point, n_act, tile.u0, q, bin, wgl, z, mu);
        if (flux != 0.0) {
          vis = true;
          if (mu < mu_min) mu = mu_min;
          c = (float)(flux * wgl);
          const double tP = (log10(z) - sp.l10kT - X.E_min) * X.inv_dE;
          const double fl = floor(tP);
          fP = (float)(tP - fl);
          if (fP >= 1.f) fP = 0.99999994f;
          G0 = G.iE_min + (int)fl;
          clamped = (G.tE_lo + tP < 0.0) || (G.tE_hi + tP > (double)(nE - 1)) || sp.T_clamped || s_int[45];
          // mu weights (cpu/nsx.hpp:173-321)
          double am;
          const int im = vhunt(s.mu, nmu, mu, am);
          const bool linear_mu = (mode == 4) || ((mode == 2 || mode == 3) && im >= nmu - 5);
          int start;
          if (linear_mu) {
            start = min(im, nmu - 4);
            const int o = im - start;
#pragma unroll
            for (int k = 0; k < 4; ++k) w4[k] = k == o ? (float)(1 - am) : (k == o + 1 ? (float)am : 0.f);
          } else {
            start = clampi(im - 1, 0, nmu - 4);
            const double x0 = s.mu[start], x1 = s.mu[start + 1], x2 = s.mu[start + 2], x3 = s.mu[start + 3];
            const double* r = den + 4 * start;
            w4[0] = (float)((mu - x1) * (mu - x2) * (mu - x3) * r[0]);
            w4[1] = (float)((mu - x0) * (mu - x2) * (mu - x3) * r[1]);
            w4[2] = (float)((mu - x0) * (mu - x1) * (mu - x3) * r[2]);
            w4[3] = (float)((mu - x0) * (mu - x1) * (mu - x2) * r[3]);
          }
          imu = start;
        }
      }
      int nv;
      const int slot = block_compact(vis, s_int, &nv);
      if (vis) {
        r_pk[slot] = make_float4(c, fP, __int_as_float(bin), __int_as_float(G0));
        r_imu[slot] = imu;
#pragma unroll
        for (int k = 0; k < 4; ++k) r_w[k * nt + slot] = w4[k];
        if (clamped) atomicAdd(&s_int[44], 1);
      }
      __syncthreads();
      if (tid == 0) {
        if (nv) atomicAdd(&p.stats[3], (unsigned long long)nv);
        if (s_int[44]) atomicAdd(&p.stats[4], (unsigned long long)s_int[44]);
        s_int[44] = 0;
      }

      for (int s0 = 0; s0 < nv; s0 += S.pb) {
        const int nb = min(S.pb, nv - s0);
        // stage B: one warp per point builds the mu-contracted rows H and the
        // per-cell cubic polynomials Q (Newton form rewritten in the cell fraction)
        for (int b = warp; b < nb; b += 2 * nwarps) {
          // two points per warp, interleaved for instruction-level parallelism
          const int bB = b + nwarps;
          const bool has2 = bB < nb;
          const int recA = s0 + b, recB = s0 + (has2 ? bB : b);
          const int G0a = __float_as_int(r_pk[recA].w), G0b = __float_as_int(r_pk[recB].w);
          const int ima = r_imu[recA], imb = r_imu[recB];
          const float wa0 = r_w[recA], wa1 = r_w[nt + recA], wa2 = r_w[2 * nt + recA], wa3 = r_w[3 * nt + recA];
          const float wb0 = r_w[recB], wb1 = r_w[nt + recB], wb2 = r_w[2 * nt + recB], wb3 = r_w[3 * nt + recB];
          const int kHa = clampi(G0a - 1, 0, nE - 4), kHb = clampi(G0b - 1, 0, nE - 4);
          float* Ha = s.H + b * HN;
          float* Hb = s.H + bB * HN;
          for (int kk = lane; kk < HN; kk += 32) {
            const int ka = kHa + kk, kb = kHb + kk;
            float ha = 0.f, hb = 0.f;
            if (ka < nE) {
              const float* row = s.S + ka * nmu + ima;
              ha = fmaf(wa3, row[3], fmaf(wa2, row[2], fmaf(wa1, row[1], wa0 * row[0])));
            }
            if (has2 && kb < nE) {
              const float* row = s.S + kb * nmu + imb;
              hb = fmaf(wb3, row[3], fmaf(wb2, row[2], fmaf(wb1, row[1], wb0 * row[0])));
            }
            Ha[kk] = ha;
            if (has2) Hb[kk] = hb;
          }
          __syncwarp();
          for (int pt = 0; pt < (has2 ? 2 : 1); ++pt) {
            const int G0x = pt ? G0b : G0a, kH0 = pt ? kHb : kHa;
            const float* H = pt ? Hb : Ha;
            float4* Qb = s.Q + (pt ? bB : b) * cells;
            for (int cc = lane; cc < cells; cc += 32) {
              const int gcell = G0x + cc;
              float4 Qv;
              if (gcell < 0) {
                Qv = make_float4(H[0 - kH0], 0.f, 0.f, 0.f);
              } else if (gcell > nE - 2) {
                Qv = make_float4(H[nE - 1 - kH0], 0.f, 0.f, 0.f);
              } else if (cubicE) {
                const int ie = clampi(gcell - 1, 0, nE - 4);
                const int off = gcell - ie;
                const float h0 = H[ie - kH0], h1 = H[ie - kH0 + 1], h2 = H[ie - kH0 + 2], h3 = H[ie - kH0 + 3];
                const float d1 = h1 - h0, d2 = h2 - 2.f * h1 + h0, d3 = h3 - 3.f * h2 + 3.f * h1 - h0;
                const float c3 = d3 * (1.f / 6.f);
                if (off == 1)
                  Qv = make_float4(h1, d1 + 0.5f * d2 - c3, 0.5f * d2, c3);
                else if (off == 0)
                  Qv = make_float4(h0, d1 - 0.5f * d2 + d3 * (1.f / 3.f), 0.5f * d2 - 0.5f * d3, c3);
                else
                  Qv = make_float4(h2, d1 + 1.5f * d2 + d3 * (1.f / 3.f), 0.5f * d2 + 0.5f * d3, c3);
              } else {
                const float h0 = H[gcell - kH0], h1 = H[gcell - kH0 + 1];
                Qv = make_float4(h0, h1 - h0, 0.f, 0.f);
              }
              Qb[cc] = Qv;
            }
          }
        }
        __syncthreads();

        // stage C: every thread integrates its energies over the sub-batch; two
        // points of the same bin are interleaved for instruction-level parallelism
        for (int b = 0; b < nb;) {
          const float4 r0 = r_pk[s0 + b];
          const int bin0 = __float_as_int(r0.z);
          if (bin0 != cur_bin) {
            if (cur_bin >= 0) flush();
            cur_bin = bin0;
          }
          const float4* Q0 = s.Q + b * cells;
          bool two = false;
          float4 r1 = r0;
          if (b + 1 < nb) {
            r1 = r_pk[s0 + b + 1];
            two = __float_as_int(r1.z) == bin0;
          }
          if (two) {
            const float4* Q1 = Q0 + cells;
#pragma unroll
            for (int k = 0; k < NE_T; ++k) {
              float t0 = fE[k] + r0.y, t1 = fE[k] + r1.y;
              const int k0 = t0 >= 1.f, k1 = t1 >= 1.f;
              t0 = k0 ? t0 - 1.f : t0;
              t1 = k1 ? t1 - 1.f : t1;
              const float4 qa = Q0[rE[k] + k0], qb = Q1[rE[k] + k1];
              float ia = fmaf(fmaf(fmaf(qa.w, t0, qa.z), t0, qa.y), t0, qa.x);
              float ib = fmaf(fmaf(fmaf(qb.w, t1, qb.z), t1, qb.y), t1, qb.x);
              if (sg) {
                ia = fmaxf(ia, 0.f);
                ib = fmaxf(ib, 0.f);
              }
              acc[k] = fmaf(r1.x, ib, fmaf(r0.x, ia, acc[k]));
            }
            b += 2;
          } else {
#pragma unroll
            for (int k = 0; k < NE_T; ++k) {
              float t0 = fE[k] + r0.y;
              const int k0 = t0 >= 1.f;
              t0 = k0 ? t0 - 1.f : t0;
              const float4 qa = Q0[rE[k] + k0];
              float ia = fmaf(fmaf(fmaf(qa.w, t0, qa.z), t0, qa.y), t0, qa.x);
              if (sg) ia = fmaxf(ia, 0.f);
              acc[k] = fmaf(r0.x, ia, acc[k]);
            }
            b += 1;
          }
        }
        __syncthreads();
      }
    }
    if (cur_bin >= 0) flush();
  }
}

// ---------------------------------------------------------------------------
// Home-cell NSX integrand.
//
// For a phase point with cell origin G0 and cell fraction fP, energy e falls
// in NSX cell G0 + rE[e] + carry (carry = fE[e] + fP >= 1).  Every lane owns
// one home cell r = rE (32 per warp) and the few energies whose rE is r, so
// per point it needs the cubic polynomials of cells G0 + r and G0 + r + 1,
// i.e. the mu-contracted slice H at G0 + r - 1 .. G0 + r + 3: each lane
// contracts the first and the last of these rows and takes the three between
// from its neighbours by warp shuffles.
// Polynomials and partial sums stay in registers; a warp set of cell_warps
// warps covers every cell of a point, and the CTA's warp sets take the
// point records in contiguous runs, each keeping its own per-bin partial sums.
//
// The polynomial of a cell is the one the pooled kernel builds (4-point
// Lagrange stencil clamped at the table ends, cpu/nsx.hpp:187-225, written
// as Newton differences in the cell fraction); outside the logEkT axis the
// edge value is held (cpu/hunt.hpp:98-121 clamps the coordinate).
// Lanes of a warp that only supply slice rows to their neighbours (no home
// cells): a lane needs rows up to C + 3 past its first, i.e. own rows of the
// next (C + 3) / C lanes.
template <int C>
__host__ __device__ constexpr int halo_lanes() {
  return (C + 3) / C;
}

// Packed FP32 pairs (.f32x2: one instruction for two lanes of arithmetic, each
// rounded as the scalar instruction rounds).  The home-cell kernel packs two
// point records: lo = record A, hi = record B.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void upk(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Groups of the energy slots of a cell whose side of the carry is known together (at most `most`: pair_slots has a
// variant for each, and a kernel whose warps run apart keeps its code small for the instruction cache).
__host__ __device__ constexpr int slot_groups(int maxe, int most) {
  return maxe <= most ? maxe : (maxe == 3 ? 3 : most);
}

// Cubic q.x + t (q.y + t (q.z + t q.w)) of one cell for both records of a pair.
struct Cubic2 {
  f32x2 x, y, z, w;
};
__device__ __forceinline__ f32x2 cubic_at(const Cubic2& q, f32x2 t) {
  return fma2(fma2(fma2(q.w, t, q.z), t, q.y), t, q.x);
}

// Slice rows seen by one lane for a pair of point records.  The lane owns C
// consecutive cells starting at cell g (= G0 + first cell of the lane) and
// needs the cubics of cells g .. g + C, i.e. rows g - 1 .. g + C + 2 of the
// mu-contracted slice: window h[j] = row g - 1 + j, j = 0 .. C + 3.  The lane
// contracts rows j < C itself; row j >= C is own row j mod C of lane
// lane + j / C (the last halo_lanes<C>() lanes of the warp own no cells).
// ra / rb: row g - 1, column imu of each record.
template <int C>
__device__ __forceinline__ void pair_window(const float* ra, const float* rb, int ldS, f32x2 w0, f32x2 w1, f32x2 w2,
                                            f32x2 w3, f32x2 (&h)[C + 4]) {
#pragma unroll
  for (int j = 0; j < C; ++j, ra += ldS, rb += ldS)
    h[j] = fma2(w3, pk(ra[3], rb[3]), fma2(w2, pk(ra[2], rb[2]), fma2(w1, pk(ra[1], rb[1]), mul2(w0, pk(ra[0], rb[0])))));
#pragma unroll
  for (int j = C; j < C + 4; ++j) h[j] = __shfl_down_sync(0xffffffffu, h[j % C], j / C);
}

// Cubics of the C + 1 cells whose stencils are window rows i .. i + 3 (the
// cell between rows i + 1 and i + 2), in the cell fraction t: the Newton form
// about row i + 1 rewritten as q0 + t (q1 + t (q2 + t q3)), from forward
// differences shared by neighbouring cells.
template <int C>
__device__ __forceinline__ void window_cubics(const f32x2 (&h)[C + 4], Cubic2 (&Q)[C + 1]) {
  const f32x2 half = pk(0.5f, 0.5f), sixth = pk(1.f / 6.f, 1.f / 6.f);
  f32x2 d1[C + 3], d2[C + 2], d3[C + 1];
#pragma unroll
  for (int j = 0; j < C + 3; ++j) d1[j] = sub2(h[j + 1], h[j]);
#pragma unroll
  for (int j = 0; j < C + 2; ++j) d2[j] = sub2(d1[j + 1], d1[j]);
#pragma unroll
  for (int j = 0; j < C + 1; ++j) d3[j] = sub2(d2[j + 1], d2[j]);
#pragma unroll
  for (int i = 0; i <= C; ++i) {
    Q[i].x = h[i + 1];
    Q[i].z = mul2(half, d2[i]);
    Q[i].w = mul2(d3[i], sixth);
    Q[i].y = sub2(fma2(half, d2[i], d1[i]), Q[i].w);
  }
}

// Cubics of cells lo .. lo + 2 (either record) become the constant x; cell `mid`
// takes the x of a neighbouring cell.  ga / gb: the lane's first cell.
template <int C>
__device__ __forceinline__ void hold_cells(Cubic2 (&Q)[C + 1], int ga, int gb, int lo, int mid) {
  auto hold = [](f32x2& v, bool a, bool b) {
    float va, vb;
    upk(v, va, vb);
    v = pk(a ? 0.f : va, b ? 0.f : vb);
  };
#pragma unroll
  for (int i = 0; i <= C; ++i) {
    const bool a = (unsigned)(ga + i - lo) <= 2u, b = (unsigned)(gb + i - lo) <= 2u;
    float na, nb, xa, xb;
    upk(i < C ? Q[i + 1].x : Q[i > 0 ? i - 1 : 0].x, na, nb);
    upk(Q[i].x, xa, xb);
    Q[i].x = pk(ga + i == mid ? na : xa, gb + i == mid ? nb : xb);
    hold(Q[i].y, a, b);
    hold(Q[i].z, a, b);
    hold(Q[i].w, a, b);
  }
}

// Adds one pair of records to a lane's energies.  The split coordinate of an
// energy is t = fE + fP; its cell is the home cell below 1 and the next one, at
// t - 1, above.  KG says which case each group of slots is in, for every cell
// and both records: groups below KG lie below 1, groups above KG at or above 1,
// and group KG is decided slot by slot (both cubics, the result selected);
// KG = -1 decides every slot and sets negative intensities to 0 if sg.  MG slots per group.
template <int MAXE, int C, int MG, int KG>
__device__ __forceinline__ void pair_slots(const Cubic2 (&Q)[C + 1], const float (&fE)[C][MAXE], float fPa, float fPb,
                                           float ca, float cb, bool has_b, bool sg, float (&acc)[C][MAXE]) {
  const f32x2 m1 = pk(-1.f, -1.f);
#pragma unroll
  for (int i = 0; i < C; ++i) {
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
      const int kg = k / MG;
      const float ta = fE[i][k] + fPa, tb = fE[i][k] + fPb;
      const f32x2 t0 = pk(ta, tb);
      float va, vb;
      if (KG >= 0 && kg < KG) {
        upk(cubic_at(Q[i], t0), va, vb);
      } else if (KG >= 0 && kg > KG) {
        upk(cubic_at(Q[i + 1], add2(t0, m1)), va, vb);
      } else {
        float a0, b0, a1, b1;
        upk(cubic_at(Q[i], t0), a0, b0);
        upk(cubic_at(Q[i + 1], add2(t0, m1)), a1, b1);
        va = ta >= 1.f ? a1 : a0;
        vb = tb >= 1.f ? b1 : b0;
      }
      if (KG < 0) {
        va = sg && !(va >= 0.f) ? 0.f : va;
        vb = sg && !(vb >= 0.f) ? 0.f : vb;
      }
      float s = fmaf(ca, va, acc[i][k]);
      if (has_b) s = fmaf(cb, vb, s);
      acc[i][k] = s;
    }
  }
}

// Fills a context (one thread); MAXE slots a cell.
template <int MAXE, int MOST>
__device__ __forceinline__ void fill_ctx(ChunkCtx& c, const DevProfile& p, const DevSpot& sp, int ring, int n_act,
                                         bool mono, bool held) {
  constexpr int NG = slot_groups(MAXE, MOST), MG = MAXE / NG;
  const RingPhi rp = sp.kind == 1 ? RingPhi{0.0, 0.0} : healpix_ring_phi(p.n_side, ring);
  c.dphi = rp.dphi;
  c.jofs = rp.jofs;
  c.l10kT = sp.l10kT;
  c.width = 1. / p.n_bins;
  c.n_gl = p.n_gl;
  c.tE_lo = p.grid.tE_lo;
  c.tE_hi = p.grid.tE_hi;
  c.out_scale = sp.out_scale;
  c.flux_off = p.flux_off;
  c.perm = p.grid.perm;
  c.cell_first = p.grid.cell_first;
  c.fEs = p.grid.fEs;
  c.invE = p.grid.invE;
  c.stats = p.stats;
  c.part = nullptr;
  c.n_act = n_act;
  c.n_nodes = p.n_bins * max(p.n_gl, 1);
  c.u_ofs = 0;
  c.n_fine = p.n_fine;
  c.n_e = p.n_e;
  c.span = p.grid.span;
  c.iE_min = p.grid.iE_min;
  c.mode = p.interp;
  c.mono = mono;
  c.held = held;
  for (int g = 0; g < NG; ++g) {
    float lo = 2.f, hi = -1.f;
    for (int k = g * MG; k < (g + 1) * MG; ++k) {
      lo = fminf(lo, p.grid.slot_lo[k]);
      hi = fmaxf(hi, p.grid.slot_hi[k]);
    }
    c.glo[g] = lo;
    c.ghi[g] = hi;
  }
}

// A phase node taken by a warp set: its number, bin, phase and weight.
struct Node {
  int node, bin;
  double ppt, wgl;
};

// walk_bracket from a bracket that is right or at most two too low for almost every x (the table's: phase_o's widths
// differ from 1 / n_fine by the delays' few per cent): two steps without a branch, the walk where a lane needs it.
// All lanes of a warp call it.  lo, hi: xx at the bracket's ends.
__device__ __forceinline__ int near_bracket(const double* xx, int n, double x, int i, double& lo, double& hi) {
  i += x >= xx[i + 1] && i < n - 2 ? 1 : 0;
  i += x >= xx[i + 1] && i < n - 2 ? 1 : 0;
  lo = xx[i];
  hi = xx[i + 1];
  if (__any_sync(0xffffffffu, (x < lo && i > 0) || (x >= hi && i < n - 2))) {
    i = walk_bracket(xx, n, x, i);
    lo = xx[i];
    hi = xx[i + 1];
  }
  return i;
}

// (out of line: the deposit's code is kept small for the instruction cache)
__device__ __noinline__ int vhunt_call(const double* xx, int n, double x, double& a) { return vhunt(xx, n, x, a); }

// Element jj of the chunk at phase ppt: patch phase, hunt and lerps in FP64
// (cpu/devarshi24st_cpu.cpp:220-229).  Returns flux/I (0 = skip; z and mu are then
// not meant).  hidx[k] is vhunt's bracket of phase_o[0] + k / n_fine: on a
// non-decreasing phase_o (mono) the bracket of the patch phase is next to its table
// entry and is vhunt's bracket exactly.  All lanes of a warp call it (jj past the
// last element: the last one's values).
__device__ __forceinline__ double node_point_tab(const ChunkCtx& c, const ChunkBufs& b, int jj, double ppt, double& z,
                                                 double& mu) {
  const double phi = c.dphi * (b.j[min(jj, c.n_act - 1)] - c.jofs);
  const double phase_shift = phi / kTwoPi;
  // fmod(x, 1) of x = ppt + phase_shift + 1 in [1, 3): x - floor(x) is the same exact value
  const double xph = ppt + phase_shift + 1.;
  double patch = xph - floor(xph);
  patch = patch < b.P[0] ? patch + 1. : patch;
  const int n = c.n_fine + 1;
  double af;
  int i;
  if (c.mono) {
    const int k = clampi((int)((patch - b.P[0]) * c.n_fine), 0, c.n_fine);
    double lo, hi;
    i = near_bracket(b.P, n, patch, b.hidx[k], lo, hi);
    af = (patch - lo) / (hi - lo);
  } else {
    i = vhunt_call(b.P, n, patch, af);
  }
  z = (1 - af) * b.Z[i] + af * b.Z[i + 1];
  mu = (1 - af) * b.MU[i] + af * b.MU[i + 1];
  return (1 - af) * b.F[i] + af * b.F[i + 1];
}

// vhunt's bracket on the descending mu axis (cpu/hunt.hpp:14-66), walked to from
// the bracket stored for the value's uniform cell (kMuHints of them, behind the
// axis and the reciprocal denominators).
__device__ __forceinline__ int mu_bracket(const double* mu_s, int nmu, double scale, double x, double& a) {
  const unsigned short* hint = (const unsigned short*)(mu_s + 5 * nmu);
  int i = hint[clampi((int)((mu_s[0] - x) * scale), 0, kMuHints - 1)];
#pragma unroll 1
  while (i > 0 && !(x < mu_s[i])) --i;
#pragma unroll 1
  while (i < nmu - 2 && x < mu_s[i + 1]) ++i;
  a = (x - mu_s[i]) / (mu_s[i + 1] - mu_s[i]);
  return i;
}

// Loads the mu axis, its reciprocal denominators and brackets (all threads).
__device__ __forceinline__ void load_mu(const DevNsx& X, double* mu_s) {
  const int tid = threadIdx.x, nt = blockDim.x, nmu = X.nmu;
  for (int k = tid; k < nmu; k += nt) mu_s[k] = X.mu[k];
  for (int k = tid; k < 4 * (nmu - 3); k += nt) mu_s[nmu + k] = X.mu_den[k];
  unsigned short* hint = (unsigned short*)(mu_s + 5 * nmu);
  for (int k = tid; k < kMuHints; k += nt) {
    double a_unused;
    hint[k] = (unsigned short)vhunt(X.mu, nmu, X.mu[0] - k / X.mu_scale, a_unused);
  }
}

// Where a thread stands: its warp set, its lane's first home cell, the set's record space.
template <int C>
struct SetPlace {
  static constexpr int kOwners = 32 - halo_lanes<C>();  // lanes with home cells
  int lane, warp, set, ST, st, r0;                      // ST: threads of a set, st: this thread's index in it
  float* srec;
  __device__ __forceinline__ SetPlace(const IntegrandShape& S, float* rec) {
    const int tid = threadIdx.x;
    lane = tid & 31;
    warp = tid >> 5;
    set = warp / S.cell_warps;
    ST = 32 * S.cell_warps;
    st = tid - set * ST;
    r0 = ((warp - set * S.cell_warps) * kOwners + lane) * C;
    srec = rec + (kPairFloats / 2) * set * ST;
  }
};

// The lane's energy fractions: per home cell, MAXE energy slots.
template <int MAXE, int C>
__device__ __forceinline__ void lane_fractions(const ChunkCtx& c, const SetPlace<C>& w, float (&fE)[C][MAXE]) {
#pragma unroll
  for (int i = 0; i < C; ++i) {
    const int rc = w.r0 + i;
    const bool own = w.lane < SetPlace<C>::kOwners && rc < c.span;
    const int e0 = own ? c.cell_first[rc] : 0;
    const int cnt = own ? min(c.cell_first[rc + 1] - e0, MAXE) : 0;
#pragma unroll
    for (int k = 0; k < MAXE; ++k) fE[i][k] = k < cnt ? c.fEs[e0 + k] : 0.f;
  }
}

// The deposit of one phase node of a chunk by one warp set.  The set walks the
// elements jj = 0 .. n_act - 1 in order, 32 x cell_warps at a time: every
// thread evaluates one point (FP64), the visible points are compacted in order
// into the set's records, and every lane adds each record to its energies' FP32
// partial sums; at the end the sums are stored or flushed with compensated FP64
// atomics.  A node's sums thus depend on the chunk's elements and the node only,
// not on which set or CTA takes it or what else is in the batch.  wcnt: per-warp
// counts of a set of several warps; n_vis, n_clamped: the warp's visible and
// clamped points are added.
template <int MAXE, int C, int MOST>
__device__ __forceinline__ void deposit_node(const KernelArgs& a, const ChunkCtx& c, const ChunkBufs& b, const Node& nd,
                                             const double* mu_s, const SetPlace<C>& w, const float (&fE)[C][MAXE],
                                             int* wcnt, unsigned& n_vis, unsigned& n_clamped) {
  const IntegrandShape& S = a.shape;
  const DevNsx& X = a.nsx;
  const int nE = X.nE, nmu = X.nmu, ldS = S.ldS;
  const int lane = w.lane, warp = w.warp, set = w.set, ST = w.ST, st = w.st, r0 = w.r0;
  constexpr int kOwners = SetPlace<C>::kOwners;
  // point records in pairs, kPairFloats floats each: {c}, {fP}, {w0}..{w3}, {row base}, {16 G0 + slot-group mask},
  // {imu}, every field as (record A, record B)
  float* srec = w.srec;
  constexpr int NG = slot_groups(MAXE, MOST), MG = MAXE / NG;  // slot groups, slots per group
  const float* Sx = b.Sx;
  // the lane's first row, past a record's row base (no cell needs rows past G0 + span + 2)
  const char* const Sl = (const char*)(Sx + min(r0, c.span + 3) * ldS);
  const int mode = c.mode, n_act = c.n_act, n_e = c.n_e;
  const double* den = mu_s + nmu;  // [nmu - 3][4] reciprocal Lagrange denominators
  float acc[C][MAXE];
#pragma unroll
  for (int i = 0; i < C; ++i)
#pragma unroll
    for (int k = 0; k < MAXE; ++k) acc[i][k] = 0.f;
#pragma unroll 1
  for (int jb = 0; jb < n_act; jb += ST) {
    // every thread evaluates one element at the node (FP64); the visible
    // ones are compacted, in element order, into the set's records
    bool vis = false, clamped = false;
    float cw = 0.f, fP = 0.f;
    int G0 = 0, imu = 0;
    float w4[4] = {0.f, 0.f, 0.f, 0.f};
    const int jj = jb + st;
    {
      double z = 0, mu = 0;
      const double flux = node_point_tab(c, b, jj, nd.ppt, z, mu);
      if (jj < n_act && flux != 0.0) {
        vis = true;
        if (mu < mu_s[nmu - 1]) mu = mu_s[nmu - 1];
        cw = (float)(flux * nd.wgl);
        const double tP = (log10(z) - c.l10kT - X.E_min) * X.inv_dE;
        const double fl = floor(tP);
        fP = (float)(tP - fl);
        if (fP >= 1.f) fP = 0.99999994f;
        G0 = c.iE_min + (int)fl;
        clamped = (c.tE_lo + tP < 0.0) || (c.tE_hi + tP > (double)(nE - 1)) || c.held;
        // mu weights (cpu/nsx.hpp:173-321)
        double am;
        const int im = mu_bracket(mu_s, nmu, X.mu_scale, mu, am);
        const bool linear_mu = (mode == 4) || ((mode == 2 || mode == 3) && im >= nmu - 5);
        int start;
        if (linear_mu) {
          start = min(im, nmu - 4);
          const int o = im - start;
#pragma unroll
          for (int k = 0; k < 4; ++k) w4[k] = k == o ? (float)(1 - am) : (k == o + 1 ? (float)am : 0.f);
        } else {
          start = clampi(im - 1, 0, nmu - 4);
          const double x0 = mu_s[start], x1 = mu_s[start + 1], x2 = mu_s[start + 2], x3 = mu_s[start + 3];
          const double* rd = den + 4 * start;
          w4[0] = (float)((mu - x1) * (mu - x2) * (mu - x3) * rd[0]);
          w4[1] = (float)((mu - x0) * (mu - x2) * (mu - x3) * rd[1]);
          w4[2] = (float)((mu - x0) * (mu - x1) * (mu - x3) * rd[2]);
          w4[3] = (float)((mu - x0) * (mu - x1) * (mu - x2) * rd[3]);
        }
        imu = start;
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, vis);
    const unsigned bal_clamped = __ballot_sync(0xffffffffu, clamped);
    n_vis += __popc(bal);
    n_clamped += __popc(bal_clamped);
    int nv, slot;
    if (S.cell_warps == 1) {
      nv = __popc(bal);
      slot = __popc(bal & lanemask_lt());
    } else {
      const int w = st >> 5;
      if (lane == 0) wcnt[warp] = __popc(bal);
      set_sync(set, ST);
      int before = 0;
      nv = 0;
      for (int k = 0; k < S.cell_warps; ++k) {
        const int cw = wcnt[set * S.cell_warps + k];
        before += k < w ? cw : 0;
        nv += cw;
      }
      slot = before + __popc(bal & lanemask_lt());
    }
    if (vis) {
      // which slot group holds the energies whose cell is decided slot by slot: bit k is set where every
      // slot of the groups below k lies below the carry and every slot of the groups above k past it
      unsigned mask = 0;
#pragma unroll
      for (int k = 0; k < NG; ++k) {
        bool ok = true;
#pragma unroll
        for (int j = 0; j < NG; ++j) ok = ok && (j == k || (j < k ? c.ghi[j] + fP < 1.f : c.glo[j] + fP >= 1.f));
        mask |= ok ? 1u << k : 0u;
      }
      G0 = max(-(1 << 16), min(G0, 1 << 16));  // far past either end: the same held value
      auto put = [&](int at, float cc) {
        float* r = srec + (at >> 1) * kPairFloats + (at & 1);
        r[0] = cc;
        r[2] = fP;
        r[4] = w4[0];
        r[6] = w4[1];
        r[8] = w4[2];
        r[10] = w4[3];
        r[12] = __int_as_float(4 * ((G0 - 1) * ldS + imu));
        r[14] = __int_as_float(G0 * 16 + (int)mask);
        r[16] = __int_as_float(imu);
      };
      put(slot, cw);
      if (slot == nv - 1 && !(slot & 1)) put(slot + 1, 0.f);  // fills the last pair (its sums are skipped)
    }
    // whether a record of this step may reach past a table end (rows G0 - 1 .. G0 + span + C + 1 are read,
    // cells G0 .. G0 + span are in use); the same for every lane: the warp's votes, or both ends for sets of
    // several warps
    bool step_hi = true, step_lo = true;
    if (S.cell_warps == 1) {
      step_hi = __any_sync(0xffffffffu, vis && G0 + c.span >= nE - (C > 1 ? C : 1));
      step_lo = __any_sync(0xffffffffu, vis && G0 <= -1);
    }
    set_sync(set, ST);
    const int nrec = __reduce_max_sync(0xffffffffu, nv);
    const int flags = (step_hi ? 16 : 0) | (step_lo ? 32 : 0) | (mode == 4 ? 64 : 0) | (mode == 1 ? 128 : 0);
    const int variants = mode == 1 ? 0 : 15;
#pragma unroll 1
    for (int q = 0; q < nrec; q += 2) {
      const float* r = srec + (q >> 1) * kPairFloats;
      const float4 rc = *(const float4*)r;
      const int4 rg = *(const int4*)(r + 12);
      const ulonglong2 w01 = *(const ulonglong2*)(r + 4), w23 = *(const ulonglong2*)(r + 8);
      // what the pair needs, as one vote (uniform over the warp, so that the branches below need no divergence
      // bookkeeping): bits 0..3 slot-group variants that serve both records, 4 and 5 rows past the high or low
      // end, 6 linear in energy, 7 negative intensities become 0
      const unsigned um = __ballot_sync(0xffffffffu, (((rg.z & rg.w & variants) | flags) >> (lane & 7)) & 1) & 255u;
      f32x2 h[C + 4];
      const float *ra = (const float*)(Sl + rg.x), *rb = (const float*)(Sl + rg.y);
      if (um & 0x30u) {
        // rows past either end repeat (C of them are stored past rows -1 and nE): the lane's first row is
        // clamped so that all C rows exist
        const int2 im = *(const int2*)(r + 16);
        ra = Sx + min(max((rg.z >> 4) + r0 - 1, -1 - C), nE + 1) * ldS + im.x;
        rb = Sx + min(max((rg.w >> 4) + r0 - 1, -1 - C), nE + 1) * ldS + im.y;
      }
      pair_window<C>(ra, rb, ldS, w01.x, w01.y, w23.x, w23.y, h);
      Cubic2 Q[C + 1];
      window_cubics<C>(h, Q);
      if (um & 0xf0u) {
        if (um & 0x40u) {
#pragma unroll
          for (int i = 0; i <= C; ++i) Q[i] = Cubic2{h[i + 1], sub2(h[i + 2], h[i + 1]), pk(0.f, 0.f), pk(0.f, 0.f)};
        }
        // cells past an end hold the end value.  A cell four or more rows past
        // an end reads four equal rows, so its cubic is that constant already;
        // the three cells next to each end become constants here.  Their value
        // is the x of a cubic (the x of cell k is row k): of the cell itself,
        // except for cell nE and cell -1, whose rows are the extrapolated ones;
        // they take the x of a neighbouring cell, row nE + 1 or nE - 1 (both
        // hold H[nE - 1]), row 0 or row -2 (H[0]).
        if (um & 0x10u) hold_cells<C>(Q, (rg.z >> 4) + r0, (rg.w >> 4) + r0, nE - 1, nE);
        if (um & 0x20u) hold_cells<C>(Q, (rg.z >> 4) + r0, (rg.w >> 4) + r0, -3, -1);
      }
      const bool has_b = q + 1 < nrec;
      if (um & 1u)
        pair_slots<MAXE, C, MG, 0>(Q, fE, rc.z, rc.w, rc.x, rc.y, has_b, (um & 0x80u) != 0, acc);
      else if (um & 2u)
        pair_slots<MAXE, C, MG, 1>(Q, fE, rc.z, rc.w, rc.x, rc.y, has_b, (um & 0x80u) != 0, acc);
      else if (NG > 2 && (um & 4u))
        pair_slots<MAXE, C, MG, (NG > 2 ? 2 : 0)>(Q, fE, rc.z, rc.w, rc.x, rc.y, has_b, (um & 0x80u) != 0, acc);
      else if (NG > 3 && (um & 8u))
        pair_slots<MAXE, C, MG, (NG > 3 ? 3 : 0)>(Q, fE, rc.z, rc.w, rc.x, rc.y, has_b, (um & 0x80u) != 0, acc);
      else
        pair_slots<MAXE, C, MG, -1>(Q, fE, rc.z, rc.w, rc.x, rc.y, has_b, (um & 0x80u) != 0, acc);
    }
    set_sync(set, ST);  // the records are rewritten by the next step
  }
  // the node's partial sums into the flux pool
  const int bin = nd.bin;
  double* flux_base = a.flux + c.flux_off;
  double* comp_base = a.comp ? a.comp + c.flux_off : nullptr;
  const double out_scale = c.out_scale;
  // through the set's record space, so that consecutive threads add to consecutive energies (one 32-byte sector
  // serves four atomics) and kFlush atomics of a thread are in flight at once
  constexpr int kFlush = 5;
  const int cap = (kPairFloats / 2) * ST;
  for (int base = 0; base < n_e; base += cap) {
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const int rc = r0 + i;
      const bool own = lane < kOwners && rc < c.span;
      const int e0 = own ? c.cell_first[rc] : 0;
      const int cnt = own ? min(c.cell_first[rc + 1] - e0, MAXE) : 0;
#pragma unroll
      for (int k = 0; k < MAXE; ++k)
        if (k < cnt && (unsigned)(e0 + k - base) < (unsigned)cap) srec[e0 + k - base] = acc[i][k];
    }
    set_sync(set, ST);
    const int lim = min(cap, n_e - base);
    if (c.part) {
      float* out = c.part + (size_t)nd.node * n_e + base;
      for (int q = st; q < lim; q += ST) out[q] = srec[q];
      set_sync(set, ST);
      continue;
    }
    for (int q0 = st; q0 < lim; q0 += kFlush * ST) {
      double v[kFlush], old[kFlush];
      int o[kFlush];
#pragma unroll
      for (int u = 0; u < kFlush; ++u) {
        const int q = q0 + u * ST;
        v[u] = 0.0;
        o[u] = -1;
        if (q < lim && srec[q] != 0.f) {
          const int e = c.perm[base + q];
          o[u] = bin * n_e + e;
          v[u] = (double)srec[q] * out_scale * c.invE[e];
        }
      }
      if (comp_base) {
#pragma unroll
        for (int u = 0; u < kFlush; ++u)
          if (o[u] >= 0) old[u] = atomicAdd(flux_base + o[u], v[u]);
#pragma unroll
        for (int u = 0; u < kFlush; ++u)
          if (o[u] >= 0) comp_error(comp_base + o[u], old[u], v[u]);
      } else {
#pragma unroll
        for (int u = 0; u < kFlush; ++u)
          if (o[u] >= 0) atomicAdd(flux_base + o[u], v[u]);
      }
    }
    set_sync(set, ST);
  }
}

// (logT, logg) taps of the slice at one ring's gravity: weights and table offsets (one thread).
__device__ __forceinline__ int nsx_taps(const DevNsx& X, const DevProfile& p, const DevSpot& sp, double lg, float* tapw,
                                        int* tapo) {
  const bool cubic = (p.interp == 0 || p.interp == 1 || p.interp == 2);
  double ag;
  int ig = uhunt(lg, X.g_min, X.g_max, X.ng, ag);
  double wg[4];
  int ig0, ngt;
  if (cubic) {
    ig0 = clampi(ig - 1, 0, X.ng - 4);
    cubic_lagrange(wg, lg, uhunt_at(X.g_min, X.g_max, X.ng, ig0), uhunt_at(X.g_min, X.g_max, X.ng, ig0 + 1),
                   uhunt_at(X.g_min, X.g_max, X.ng, ig0 + 2), uhunt_at(X.g_min, X.g_max, X.ng, ig0 + 3));
    ngt = 4;
  } else {
    ig0 = ig;
    wg[0] = 1 - ag;
    wg[1] = ag;
    ngt = 2;
  }
  int n = 0;
  for (int jt = 0; jt < sp.nT_taps; ++jt)
    for (int jg = 0; jg < ngt; ++jg) {
      tapw[n] = (float)(sp.wT[jt] * wg[jg]);
      tapo[n] = (sp.iT[jt] * X.ng + ig0 + jg) * X.slice_stride;
      ++n;
    }
  return n;
}

// Reduces the NSX table into S[E][mu] (row stride ldS, Sx = row 0, in shared or
// global memory); all threads of the block, block barriers inside.
__device__ __forceinline__ void build_slice(const DevNsx& X, int ldS, int C, const float* tapw, const int* tapo,
                                            int ntap, float* Sx) {
  const int tid = threadIdx.x, nt = blockDim.x, nE = X.nE, nmu = X.nmu;
  const int n_el = nE * nmu;
  if (ldS == nmu) {
    const int n4 = (n_el + 3) >> 2;
    float4* S4 = (float4*)Sx;
    for (int k = tid; k < n4; k += nt) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int q = 0; q < ntap; ++q) {
        const float4 v = __ldg((const float4*)(X.data + tapo[q]) + k);
        const float w = tapw[q];
        acc.x = fmaf(w, v.x, acc.x);
        acc.y = fmaf(w, v.y, acc.y);
        acc.z = fmaf(w, v.z, acc.z);
        acc.w = fmaf(w, v.w, acc.w);
      }
      S4[k] = acc;
    }
  } else {
    for (int k = tid; k < n_el; k += nt) {
      float acc = 0.f;
      for (int q = 0; q < ntap; ++q) acc = fmaf(tapw[q], __ldg(X.data + tapo[q] + k), acc);
      const int row = k / nmu;
      Sx[row * ldS + (k - row * nmu)] = acc;
    }
  }
  __syncthreads();
  // rows -1 and nE: the cubic through the first (last) four rows, one row
  // further out; the C rows past them: copies of rows 0 and nE - 1
  for (int k = tid; k < 2 * nmu; k += nt) {
    const int top = k >= nmu, m = top ? k - nmu : k;
    const float* a = Sx + (top ? (nE - 1) * ldS : 0) + m;
    const int st = top ? -ldS : ldS;
    Sx[(top ? nE : -1) * ldS + m] = fmaf(4.f, a[0], fmaf(-6.f, a[st], fmaf(4.f, a[2 * st], -a[3 * st])));
    for (int j = 1; j <= C; ++j) Sx[(top ? nE + j : -1 - j) * ldS + m] = a[0];
  }
  __syncthreads();
}

// The bracket table of phase_o for node_point_tab (hidx in shared or global
// memory), used where phase_o is non-decreasing: returns whether it is (a block
// barrier; the table is complete after the next one).  walk_bracket gives vhunt's
// bracket there, a step or two from entry k.
__device__ __forceinline__ bool phase_table(const double* P, int n_fine, unsigned short* hidx) {
  const int tid = threadIdx.x, nt = blockDim.x;
  bool ok = true;
  for (int k = tid; k < n_fine; k += nt) ok &= P[k + 1] >= P[k];
  if (__syncthreads_and(ok) == 0) return false;
  for (int k = tid; k <= n_fine; k += nt)
    hidx[k] = (unsigned short)walk_bracket(P, n_fine + 1, P[0] + (double)k / n_fine, min(k, n_fine - 1));
  return true;
}

// Home-cell kernel over the planner's tiles: every tile computes its ring's
// sweep and slice itself; its phase nodes u in [u0, u1) go to the warp sets one
// at a time through a shared counter.  For batches with rings enough to fill the
// GPU, and for ppm_profile_noalloc.
template <int MAXE, int C, int NTMAX, int MINB>
__global__ void __launch_bounds__(NTMAX, MINB) integrand_nsx_cell_kernel(const KernelArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  const SmemPtrs s = carve(sm, a.shape);
  __shared__ RingGeom s_g;
  __shared__ int s_int[48];
  __shared__ int s_tile;
  __shared__ float s_tapw[16];
  __shared__ int s_tapo[16];
  __shared__ int s_ntap;
  __shared__ ChunkCtx s_ctx;
  __shared__ Node s_node[16];
  __shared__ int s_next[16], s_wcnt[16];
  const int tid = threadIdx.x;
  const DevNsx& X = a.nsx;
  const int ldS = a.shape.ldS;
  float* const Sx = s.S + slice_row0(ldS, C);
  const SetPlace<C> w(a.shape, (float*)s.batch);
  load_mu(X, s.mu);  // (visible after the barriers of the first tile)

  for (;;) {
    __syncthreads();
    if (tid == 0) s_tile = atomicAdd(a.queue.next, 1);
    __syncthreads();
    const int t = s_tile;
    if (t >= *a.queue.n_tiles || t >= a.queue.capacity) break;
    const Tile tile = a.queue.tiles[t];
    const DevProfile& p = a.profiles[tile.profile];
    const DevSpot& sp = p.spot[tile.spot];
    const int n_act = tile_prologue(a, p, sp, tile, s, s_g, s_int, true);
    if (n_act == 0) continue;
    if (tid == 0) {
      s_int[46] = tile.u0;  // next phase node of the deposit
      s_ntap = nsx_taps(X, p, sp, s_g.logg, s_tapw, s_tapo);
    }
    const bool mono = phase_table(s.P, p.n_fine, s.hidx);
    if (tid == 0)
      fill_ctx<MAXE, 4>(s_ctx, p, sp, tile.ring, n_act, mono, sp.T_clamped || s_g.logg < X.g_min || s_g.logg > X.g_max);
    build_slice(X, ldS, C, s_tapw, s_tapo, s_ntap, Sx);
    const ChunkBufs bufs{s.j, s.P, s.F, s.Z, s.MU, s.hidx, Sx};
    float fE[C][MAXE];
    lane_fractions<MAXE, C>(s_ctx, w, fE);
    unsigned n_vis = 0, n_clamped = 0;
    for (;;) {
      if (w.st == 0) {
        const int u = atomicAdd(&s_int[46], 1);
        s_next[w.set] = u;
        if (u < tile.u1) {
          Node& nd = s_node[w.set];
          nd.node = u;
          node_phase(p, u, nd.bin, nd.ppt, nd.wgl);
        }
      }
      set_sync(w.set, w.ST);
      if (s_next[w.set] >= tile.u1) break;
      deposit_node<MAXE, C, 4>(a, s_ctx, bufs, s_node[w.set], s.mu, w, fE, s_wcnt, n_vis, n_clamped);
    }
    if (w.lane == 0) {
      if (n_vis) atomicAdd(&p.stats[3], (unsigned long long)n_vis);
      if (n_clamped) atomicAdd(&p.stats[4], (unsigned long long)n_clamped);
    }
  }
}

// ---------------------------------------------------------------------------
// Ring records: the home-cell path of batches with few rings (single profiles,
// small batches), whose nodes have to be spread over many CTAs.  ring_kernel
// does each ring's planning, sweep and slice once and leaves them in global
// memory (L2); integrand_nsx_rec_kernel's CTAs load a ring's record and take its
// phase nodes one at a time from the chunk's counter in global memory.

// One CTA per (profile, spot, ring).  Bound by latency, a chain of block barriers (geometry, arcs, rows, sweep, gap
// fill, slice): 14 us for 48 rings, 30 for 412, 62 for 819, of which the plan alone took 16 before.
template <bool NSX>
__global__ void __launch_bounds__(256) ring_kernel(const KernelArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  const IntegrandShape& S = a.shape;
  const RingWork& W = a.rings;
  const SmemPtrs s = carve(sm, S);
  __shared__ RingGeom s_g;
  __shared__ int s_int[48];
  __shared__ int s_first;
  __shared__ int s_range[2][2], s_nr;
  __shared__ float s_tapw[16];
  __shared__ int s_tapo[16];
  __shared__ int s_ntap;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int job = blockIdx.x;
  if (job == 0 && tid == 0) W.ctr[W.rec_cap] = make_int4(0, 0, 0, 0);
  // the job's profile, in [first, last): an nt-fold search, none for one profile, a step up to nt of them (every CTA
  // over every spot would be profiles^2: 16384 point sources took 2.8 ms in this kernel)
  int first = 0;
  for (int last = W.n_profiles; last - first > 1;) {
    const int step = (last - first + nt - 1) / nt, k = first + tid * step, k1 = min(k + step, last);
    if (k < last && a.profiles[k].spot[0].job0 <= job && (k1 == last || job < a.profiles[k1].spot[0].job0)) s_first = k;
    __syncthreads();
    first = s_first;
    last = min(first + step, last);
    __syncthreads();
  }
  const DevProfile& p = a.profiles[first];
  const int spot = job - p.spot[0].job0 < ring_jobs(p.spot[0]) ? 0 : 1;
  const DevSpot& sp = p.spot[spot];
  const bool point = sp.kind == 1;
  const int ring = point ? 0 : sp.i_lo + job - sp.job0;
  const DevLens& L = a.lens;
  const double z = point ? sp.cos_theta_pt : p.ring[3 * ring];
  const double c2 = point ? 0.0 : p.ring[3 * ring + 1], s2 = point ? 0.0 : p.ring[3 * ring + 2];
  if (tid == 0) {
    ring_geometry(p, L, z, point ? sp.dOmega_pt : p.dOmega_hp, NSX, s_g);
  }
  if (tid == 32) {
    int r[2][2] = {{0, 0}, {0, 0}};
    s_nr = point ? 1 : candidate_ranges(sp, p.n_side, ring, c2, s2, healpix_jmax(p.n_side, ring), r);
    for (int k = 0; k < 2; ++k) {
      s_range[k][0] = r[k][0];
      s_range[k][1] = r[k][1];
    }
  }
  __syncthreads();
  const int nr = s_nr;
  if (nr == 0) return;
  const bool dropped = ring_sweep(a, p, s, s_g, s_int, NSX);
  if (NSX && tid == nt - 1) s_ntap = nsx_taps(a.nsx, p, sp, s_g.logg, s_tapw, s_tapo);
  // the ring's image: the sweep as it lies in shared memory, the bracket table, the slice
  unsigned char* const img = W.data + (size_t)job * W.stride;
  const bool mono = !dropped && phase_table(s.P, p.n_fine, (unsigned short*)(img + W.off_hidx));
  if (!NSX && !dropped) {  // MU is not needed: reciprocal widths of the phase_o intervals in its place
    __syncthreads();
    for (int k = tid; k < p.n_fine; k += nt) s.MU[k] = 1.0 / (s.P[k + 1] - s.P[k]);
  }
  const RingPhi rp = point ? RingPhi{0.0, 0.0} : healpix_ring_phi(p.n_side, ring);
  // active elements, one record per chunk of candidates
  int n_ring = 0;
  bool first_chunk = true;
  for (int k = 0; k < nr; ++k) {
    const int j_end = point ? 1 : s_range[k][1] + 1;
    for (int j0 = point ? 0 : s_range[k][0]; j0 < j_end; j0 += W.chunk, first_chunk = false) {
      const int n_c = min(W.chunk, j_end - j0);
      int n_act = 0;
      for (int k0 = 0; k0 < n_c; k0 += nt) {
        const int c = k0 + tid;
        const bool flag = c < n_c && (point || in_spot(sp, c2, s2, healpix_phi(p.n_side, ring, j0 + c)));
        int tot;
        const int pos = block_compact(flag, s_int, &tot);
        if (flag) s.j[n_act + pos] = (unsigned short)(j0 + c);
        n_act += tot;
        __syncthreads();
      }
      n_ring += n_act;
      if (n_act == 0 || dropped) continue;
      if (tid == 0) {
        const int at = atomicAdd(W.n_recs, 1), lo = atomicAdd(W.list_next, (n_act + 7) & ~7);
        const int nth = (int)atomicAdd(p.ring_seen, 1u);
        s_int[43] = lo;
        const bool held = NSX && (sp.T_clamped || s_g.logg < a.nsx.g_min || s_g.logg > a.nsx.g_max);
        const int tasks = p.n_bins * max(p.n_gl, 1) * (NSX ? 1 : (p.n_e + kBbPass - 1) / kBbPass);
        if (at < W.rec_cap && lo + n_act <= W.list_cap) {
          W.recs[at] = RingRec{first, spot, ring, job, n_act, lo, tasks, (mono ? 1 : 0) | (held ? 2 : 0)};
          W.ctr[at] = make_int4(0, 0, tasks, n_act);
        } else {
          s_int[43] = -1;
          atomicOr(a.queue.overflow, 1);
        }
        W.by_profile[W.per_job * p.spot[0].job0 + nth] = s_int[43] >= 0 ? 2 * at + spot : INT_MAX;
        if (s_g.u_clamped && first_chunk) atomicAdd(&p.stats[4], 1ull);
      }
      __syncthreads();
      const int lo = s_int[43];
      if (lo >= 0)
        for (int c = tid; c < n_act; c += nt) {
          if (NSX)
            ((unsigned short*)W.lists)[lo + c] = s.j[c];
          else  // the element's phase shift phi / 2 pi
            ((double*)W.lists)[lo + c] = (point ? 0.0 : rp.dphi * (s.j[c] - rp.jofs)) / kTwoPi;
        }
      __syncthreads();
    }
  }
  if (n_ring == 0) return;
  if (tid == 0) {  // a dropped ring is counted, with its elements, only if it holds active elements (as plan_kernel)
    atomicAdd(&p.stats[dropped ? 5 : 0], (unsigned long long)n_ring);
    atomicAdd(&p.stats[1], 1ull);
    if (dropped) {
      atomicAdd(&p.stats[2], 1ull);
      if (s_g.u_clamped && !point) atomicAdd(&p.stats[4], 1ull);
    }
  }
  if (dropped) return;
  const int n16 = (S.off_mu - S.off_P) >> 4;
  for (int k = tid; k < n16; k += nt) ((float4*)img)[k] = ((const float4*)(sm + S.off_P))[k];
  if (NSX)
    build_slice(a.nsx, S.ldS, S.cpl, s_tapw, s_tapo, s_ntap, (float*)(img + W.off_slice) + slice_row0(S.ldS, S.cpl));
}

// Work of the home-cell NSX kernel: one node at a time.  Bound by the FMA pipe and the register file's ports, as over
// tiles.  What a node is added to no longer shows: its sums are stored, not added atomically.  N_side 256, two spots,
// 64 bins x 2 nodes, 300 energies: 1071 us with plan and sum from tiles, 973 with rings and sum from records.
template <int MAXE, int C, int NTMAX>
struct NsxWork : SetPlace<C> {
  const KernelArgs& a;
  const double* mu_s;
  Node* s_node;
  int* wcnt;
  float fE[C][MAXE];
  unsigned n_vis = 0, n_clamped = 0;
  __device__ __forceinline__ NsxWork(const KernelArgs& args, unsigned char* sm, Node* nodes_, int* wcnt_)
      : SetPlace<C>(args.shape, (float*)(sm + args.shape.rec_off_batch)), a(args),
        mu_s((const double*)(sm + args.shape.rec_off_mu)), s_node(nodes_), wcnt(wcnt_) {}
  __device__ __forceinline__ void fill(ChunkCtx& c, const DevProfile& p, const DevSpot& sp, const RingRec& q) {
    fill_ctx<MAXE, 2>(c, p, sp, q.ring, q.n_act, (q.flags & 1) != 0, (q.flags & 2) != 0);
    c.take = 1;
    c.u_mod = c.n_nodes;
  }
  __device__ __forceinline__ void enter(const ChunkCtx& c) { lane_fractions<MAXE, C>(c, *this, fE); }
  __device__ __forceinline__ void nodes(const ChunkCtx& c, const ChunkBufs& b, int u) {
    Node& nd = s_node[this->set];
    if (this->st == 0) {
      nd.node = u + c.u_ofs < c.n_nodes ? u + c.u_ofs : u + c.u_ofs - c.n_nodes;
      node_phase(c.n_gl, c.width, nd.node, nd.bin, nd.ppt, nd.wgl);
    }
    set_sync(this->set, this->ST);
    deposit_node<MAXE, C, 2>(a, c, b, nd, mu_s, *this, fE, wcnt, n_vis, n_clamped);
  }
  __device__ __forceinline__ void count(int profile) {  // the warp's counters to the profile it leaves
    if (this->lane == 0 && profile >= 0) {
      if (n_vis) atomicAdd(&a.profiles[profile].stats[3], (unsigned long long)n_vis);
      if (n_clamped) atomicAdd(&a.profiles[profile].stats[4], (unsigned long long)n_clamped);
    }
    n_vis = n_clamped = 0;
  }
};

template <int MAXE, int C, int NTMAX>
__global__ void __launch_bounds__(NTMAX, 1) integrand_nsx_rec_kernel(const KernelArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ Node s_node[NTMAX / 32];
  __shared__ int s_wcnt[NTMAX / 32];
  load_mu(a.nsx, (double*)(sm + a.shape.rec_off_mu));
  NsxWork<MAXE, C, NTMAX> w(a, sm, s_node, s_wcnt);
  rec_loop<NTMAX>(a, sm, w);
}

// ---------------------------------------------------------------------------
// Blackbody integrand from ring records.  A warp takes `take` phase nodes of a
// chunk at a time and walks a node's elements 32 at a time, a point per lane.
// Few energies (at most kPhaseMajorMaxE): the lane evaluates its point at each.
// More: the visible points are compacted into the warp's records and the lanes
// own the energies (c.lanes of them, up to four each; the lane groups take the
// records in turn), kBbPass energies a pass, each pass a task of its own.  The
// sums are FP64 in every arithmetic; a node's are combined over the lanes and
// stored.  Bound by issue and latency (51 % of the issue slots, the FP64 pipe at
// 16 %; 32 us for 48 rings, 64 energies, 32 x 2 nodes): the point's bracket walk
// and the node's bookkeeping.  That spectrum takes 458 us a call from tiles, 96
// from records; where each form is used: Engine::bb_records.
// FP32 arithmetic keeps the form of the tile kernel's path for the grid's size.
template <typename Real>
struct BbWork {
  const KernelArgs& a;
  int lane, set, st;
  static constexpr int ST = 32;
  double2* rec;
  unsigned n_vis = 0;
  __device__ __forceinline__ BbWork(const KernelArgs& args, unsigned char* sm) : a(args) {
    lane = st = threadIdx.x & 31;
    set = threadIdx.x >> 5;
    rec = (double2*)(sm + args.shape.rec_off_batch) + 32 * set;
  }
  __device__ __forceinline__ void fill(ChunkCtx& c, const DevProfile& p, const DevSpot& sp, const RingRec& q) {
    fill_ctx<1, 1>(c, p, sp, q.ring, q.n_act, (q.flags & 1) != 0, false);
    c.kT = sp.kT;
    c.E = p.grid.E;
    const int passes = (p.n_e + kBbPass - 1) / kBbPass;
    c.per_pass = (p.n_e + passes - 1) / passes;
    c.u_mod = c.n_nodes;
    c.n_nodes *= passes;  // as ring_kernel counted the chunk's tasks
    // nodes per take: about 2048 points, but takes for every warp several times over
    const long long tasks = (long long)min(*a.rings.n_recs, a.rings.rec_cap) * c.n_nodes;
    const long long per_take = min((long long)c.u_mod / 8, 2048ll / max(q.n_act, 8));
    c.take = (int)max(1ll, min(per_take, tasks / (gridDim.x * (blockDim.x / 8))));
    int ll = 0;
    if (c.per_pass > kPhaseMajorMaxE)
      while (ll < 5 && (1 << ll) < c.per_pass) ++ll;
    c.lanes_log = ll;
  }
  // few energies: nodes at a time, this lane's node among them and its (first) element
  int m = 1, sub = 0, jl = 0;
  __device__ __forceinline__ void enter(const ChunkCtx& c) {
    m = c.n_act <= 16 ? 32 / c.n_act : 1;
    sub = m > 1 ? lane / c.n_act : 0;
    jl = lane - sub * c.n_act;
    if (m == 1) jl = lane;
  }
  __device__ __forceinline__ void count(int profile) {
    n_vis = __reduce_add_sync(0xffffffffu, n_vis);
    if (lane == 0 && profile >= 0 && n_vis) atomicAdd(&a.profiles[profile].stats[3], (unsigned long long)n_vis);
    n_vis = 0;
  }
  // Ibb without its constant, times the point's flux (cpu/unit.hpp:28-31).  divide: E / kT as a division, as the tile
  // kernel's path for more than 64 energies has it (one rounding less), else by the reciprocal.
  static __device__ __forceinline__ double planck(Real cb, Real zb, Real E, Real kT, Real inv_kT, bool divide) {
    const Real Ee = E * zb;
    return (double)(cb * (Ee * Ee * Ee / expm1(divide ? Ee / kT : Ee * inv_kT)));
  }
  // The same of two points, in one block, so that the two evaluations overlap and share their constants; hidden points
  // have c = 0 and z = 1.  A point's value is its own: what the other lanes hold depends on the batch.
  static __device__ __forceinline__ double planck_pair(double ca, double za, double cb, double zb, double E,
                                                       double inv_kT) {
    const double ea = E * za, eb = E * zb;
    return ca * (ea * ea * ea / expm1(ea * inv_kT)) + cb * (eb * eb * eb / expm1(eb * inv_kT));
  }
  // The bracket and fraction of element jj's patch phase (node_point_tab, with the element's phase shift from the
  // chunk's list and, unless divide, the reciprocal interval widths from the ring's image).  All lanes call it.
  static __device__ __forceinline__ int bracket(const ChunkCtx& c, const ChunkBufs& b, int jj, double ppt, bool divide,
                                                double& af) {
    const double xph = ppt + ((const double*)b.j)[min(jj, c.n_act - 1)] + 1.;
    // x - floor(x) for x in [1, 3]: the same exact value
    double patch = xph - (xph >= 3.0 ? 3.0 : (xph >= 2.0 ? 2.0 : 1.0));
    const double P0 = b.P[0];
    patch = patch < P0 ? patch + 1. : patch;
    if (!c.mono) return vhunt_call(b.P, c.n_fine + 1, patch, af);
    double lo, hi;
    const int k = clampi((int)((patch - P0) * c.n_fine), 0, c.n_fine);
    const int i = near_bracket(b.P, c.n_fine + 1, patch, b.hidx[k], lo, hi);
    af = divide ? (patch - lo) / (hi - lo) : (patch - lo) * b.MU[i];
    return i;
  }
  // flux/I and redshift of element jj where `on` (else 0 and 1)
  static __device__ __forceinline__ double point(const ChunkCtx& c, const ChunkBufs& b, int jj, bool on, double ppt,
                                                 bool divide, double& z) {
    double af;
    const int i = bracket(c, b, jj, ppt, divide, af);
    // (fused as the tile kernel's two paths are compiled)
    const double g = 1 - af;
    const double flux = divide ? __fma_rn(af, b.F[i + 1], g * b.F[i]) : __fma_rn(g, b.F[i], af * b.F[i + 1]);
    const double zz = g * b.Z[i] + af * b.Z[i + 1];
    on = on && flux != 0.0;
    z = on ? zz : 1.0;
    return on ? flux : 0.0;
  }
  // one point at the grid's few energies, in FP32 arithmetic: the phase-major walk's form (pm_walk)
  static __device__ __forceinline__ void point_few32(const ChunkCtx& c, const ChunkBufs& b, int jj, bool on, double ppt,
                                                     double wgl, const float* E, int n_e, float inv_kT, double* acc,
                                                     unsigned& vis) {
    double afd;
    const int i = bracket(c, b, jj, ppt, false, afd);
    const float af = (float)afd;
    const float f0 = (float)b.F[i], flux = fmaf(af, (float)b.F[i + 1] - f0, f0);
    if (!on || flux == 0.f) return;
    const float z0 = (float)b.Z[i], zb = fmaf(af, (float)b.Z[i + 1] - z0, z0), cb = flux * (float)wgl;
    ++vis;
#pragma unroll
    for (int e = 0; e < kPhaseMajorMaxE; ++e) {
      if (e >= n_e) break;
      const float Ee = E[e] * zb, x = Ee * inv_kT;
      acc[e] += (double)(cb * __fdividef(Ee * Ee * Ee, x > 0.5f ? __expf(x) - 1.f : expm1f(x)));
    }
  }
  // a node's sum of energy e
  __device__ __forceinline__ void store(const ChunkCtx& c, int v, int bin, int e, double sum) {
    if (c.part) {
      ((double*)c.part)[(size_t)v * c.n_e + e] = sum;
    } else if (sum != 0.0) {
      const size_t o = (size_t)c.flux_off + (size_t)bin * c.n_e + e;
      comp_add(a.flux + o, a.comp ? a.comp + o : nullptr, sum * c.out_scale * c.invE[e]);
    }
  }
  // few energies: m nodes at a time (rings of few elements), else two elements a lane
  __device__ __forceinline__ void nodes_few(const ChunkCtx& c, const ChunkBufs& b, int u0) {
    const int u_end = min(u0 + c.take, c.n_nodes), ne = c.n_e, n_act = c.n_act;
    const Real inv_kT = (Real)1 / (Real)c.kT;
    Real E[kPhaseMajorMaxE];
#pragma unroll
    for (int k = 0; k < kPhaseMajorMaxE; ++k) E[k] = k < ne ? (Real)c.E[k] : (Real)1;
    const bool few32 = std::is_same<Real, float>::value && c.mono;
    for (int u = u0; u < u_end; u += m) {
      const bool live = sub < m && u + sub < u_end;
      int v = u + (live ? sub : 0) + c.u_ofs, bin;
      v -= v >= c.u_mod ? c.u_mod : 0;
      double ppt, wgl;
      node_phase(c.n_gl, c.width, v, bin, ppt, wgl);
      double acc[kPhaseMajorMaxE] = {0.0, 0.0, 0.0, 0.0};
      for (int jb = 0; jb < n_act; jb += 64) {
        const int ja = jb + jl, jc = ja + 32;
        const bool on_a = live && ja < n_act, on_b = m == 1 && jc < n_act;
        if (few32) {
          point_few32(c, b, ja, on_a, ppt, wgl, (const float*)E, ne, (float)inv_kT, acc, n_vis);
          if (m == 1) point_few32(c, b, jc, on_b, ppt, wgl, (const float*)E, ne, (float)inv_kT, acc, n_vis);
          continue;
        }
        double za = 1.0, zb = 1.0, ca = 0.0, cb = 0.0;
        const double fa = point(c, b, ja, on_a, ppt, false, za);
        double fb = 0.0;
        if (m == 1) fb = point(c, b, jc, on_b, ppt, false, zb);
        n_vis += (fa != 0.0 ? 1u : 0u) + (fb != 0.0 ? 1u : 0u);
        ca = fa * wgl;
        cb = fb * wgl;
#pragma unroll
        for (int k = 0; k < kPhaseMajorMaxE; ++k)
          if (k < ne) {
            if constexpr (std::is_same<Real, double>::value) {
              acc[k] += m == 1 ? planck_pair(ca, za, cb, zb, E[k], inv_kT) : planck(ca, za, E[k], 0.0, inv_kT, false);
            } else {
              if (fa != 0.0) acc[k] += planck((Real)ca, (Real)za, E[k], (Real)0, inv_kT, false);
              if (fb != 0.0) acc[k] += planck((Real)cb, (Real)zb, E[k], (Real)0, inv_kT, false);
            }
          }
      }
      for (int off = 1; off < 32; off <<= 1) {
        const bool same = m == 1 || (lane + off < 32 && jl + off < n_act);
#pragma unroll
        for (int k = 0; k < kPhaseMajorMaxE; ++k)
          if (k < ne) {
            const double o = __shfl_down_sync(0xffffffffu, acc[k], off);
            if (same) acc[k] += o;
          }
      }
      if (live && (m == 1 ? lane == 0 : jl == 0))
#pragma unroll
        for (int k = 0; k < kPhaseMajorMaxE; ++k)
          if (k < ne) store(c, v, bin, k, acc[k]);
    }
  }
  __device__ __forceinline__ void nodes(const ChunkCtx& c, const ChunkBufs& b, int u0) {
    if (c.lanes_log == 0) {
      nodes_few(c, b, u0);
      return;
    }
    const int u_end = min(u0 + c.take, c.n_nodes);
    const Real kT = (Real)c.kT, inv_kT = (Real)1 / kT;
    const int ll = c.lanes_log, ln = 1 << ll, grp = lane >> ll, el = lane & (ln - 1), n_grp = 32 >> ll;
    const bool divide = c.n_e > 64;
    for (int u = u0; u < u_end; ++u) {
      int pass = 0, v = u;
      while (v >= c.u_mod) {
        v -= c.u_mod;
        ++pass;
      }
      const int e0 = pass * c.per_pass, ne = min(c.per_pass, c.n_e - e0), ke = (ne + ln - 1) >> ll;
      v += c.u_ofs;
      v -= v >= c.u_mod ? c.u_mod : 0;
      int bin;
      double ppt, wgl;
      node_phase(c.n_gl, c.width, v, bin, ppt, wgl);
      Real E[4];
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int e = el + (k << ll);
        E[k] = e < ne ? (Real)c.E[e0 + e] : (Real)1;
      }
      for (int jb = 0; jb < c.n_act; jb += 32) {
        const int jj = jb + lane;
        double flux = 0.0, z = 0;
        flux = point(c, b, jj, jj < c.n_act, ppt, divide, z);
        const unsigned bal = __ballot_sync(0xffffffffu, flux != 0.0);
        if (flux != 0.0) {
          rec[__popc(bal & lanemask_lt())] = make_double2(flux * wgl, z);
          n_vis += pass == 0 ? 1u : 0u;
        }
        __syncwarp();
        const int nv = __popc(bal);
        for (int q = grp; q < nv; q += n_grp) {
          const double2 r = rec[q];
          const Real cb = (Real)r.x, zb = (Real)r.y;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < ke) acc[k] += planck(cb, zb, E[k], kT, inv_kT, divide);
        }
        __syncwarp();
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        if (off >= ln)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < ke) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int e = el + (k << ll);
        if (grp == 0 && e < ne) store(c, v, bin, e0 + e, acc[k]);
      }
    }
  }
};

template <typename Real>
__global__ void __launch_bounds__(kBbRecThreads, 1) integrand_bb_rec_kernel(const KernelArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  BbWork<Real> w(a, sm);
  rec_loop<kBbRecThreads>(a, sm, w);
}

// ---------------------------------------------------------------------------
// The blackbody phase-major walk over the tile's elements jj0 .. jj1 - 1 at one
// phase node (phase ppt, weight wgl): adds each visible element's Ibb at the
// grid's first NE energies (NE = 1, or up to n_e) into acc and returns the
// number of visible elements.  The patch phase and its phase_o bracket are
// FP64 in every arithmetic, the bracket hunted from the previous element's.
// FP64 arithmetic lerps F and Z in FP64 and divides exactly; FP32 arithmetic
// lerps the tile's FP32 copies of F and Z and divides with the fast
// reciprocal.
template <typename Real, int NE>
__device__ __forceinline__ unsigned pm_walk(const SmemPtrs& s, const double* inv_dp, const float* F32, const float* Z32,
                                            const double* shift_s, const Real* E_s, int n_e, Real inv_kT, double ppt,
                                            double wgl, int jj0, int jj1, int n_fp, double P0, double* acc) {
  unsigned n_vis = 0;
  int hint = -1;
  double prev = -1.0;  // below every patch phase
  for (int jj = jj0; jj < jj1; ++jj) {
    const double xph = ppt + shift_s[jj] + 1.;
    // x - floor(x) for x in [1, 3]: the same exact value
    double patch = xph - (xph >= 3.0 ? 3.0 : (xph >= 2.0 ? 2.0 : 1.0));
    if (patch < P0) patch += 1.;
    // phase_o[i] is phase i / n_fine plus a small time-of-flight delay: the
    // first element's bracket is walked to from that guess, the others' from
    // the previous bracket by unit steps (none or one for the next element;
    // from the first bracket when the patch phase wraps past phase_o[0] + 1).
    // On a non-decreasing phase_o the walk stops at vhunt's bracket: the
    // largest i <= n - 2 with phase_o[i] <= patch, or 0.
    if (patch < prev) hint = 0;
    prev = patch;
    if (hint < 0) hint = clampi((int)((patch - P0) * (n_fp - 1)), 0, n_fp - 2);
    hint = walk_bracket(s.P, n_fp, patch, hint);
    const int i = hint;
    Real cb, zb;
    if constexpr (std::is_same<Real, float>::value) {
      const float af = (float)((patch - s.P[i]) * inv_dp[i]);
      const float f0 = F32[i];
      const float flux = fmaf(af, F32[i + 1] - f0, f0);
      if (flux == 0.f) continue;
      const float z0 = Z32[i];
      zb = fmaf(af, Z32[i + 1] - z0, z0);
      cb = flux * (float)wgl;
    } else {
      const double af = (patch - s.P[i]) * inv_dp[i];
      const double flux = (1 - af) * s.F[i] + af * s.F[i + 1];
      if (flux == 0) continue;
      zb = (1 - af) * s.Z[i] + af * s.Z[i + 1];
      cb = flux * wgl;
    }
    ++n_vis;
#pragma unroll
    for (int e = 0; e < NE; ++e)
      if (NE == 1 || e < n_e) {
        const Real Ee = E_s[e] * zb;
        Real v;  // Ibb without its constant
        if constexpr (std::is_same<Real, float>::value) {
          // e^x - 1: the fast exponential where x > 0.5 (no cancellation there), expm1f below
          const float x = Ee * inv_kT;
          v = cb * __fdividef(Ee * Ee * Ee, x > 0.5f ? __expf(x) - 1.f : expm1f(x));
        } else {
          v = cb * (Ee * Ee * Ee / expm1(Ee * inv_kT));
        }
        acc[e] += (double)v;
      }
  }
  return n_vis;
}

// Fused point-source mode: the first point spot k >= k0 of the profile inside the batch's ring window, or
// n_spots (the tile's own sweep then makes plan_kernel's ring-drop test, tile_prologue).
__device__ __forceinline__ int fused_next_spot(const DevProfile& pf, int k0) {
  int k = k0;
  while (k < pf.n_spots && pf.spot[k].i_lo > pf.spot[k].i_hi) ++k;
  return k;
}

template <typename Real, int NE_T>
__global__ void __launch_bounds__(512, 2) integrand_bb_kernel(const KernelArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  const IntegrandShape& S = a.shape;
  const SmemPtrs s = carve(sm, S);
  __shared__ RingGeom s_g;
  __shared__ int s_int[48];
  __shared__ int s_tile;
  const int tid = threadIdx.x, nt = blockDim.x;
  double* b_c = (double*)s.batch;  // point records, one slot per thread
  double* b_z = b_c + nt;
  int* b_bin = (int*)(b_z + nt);

  // fused point-source mode: this CTA's profile starts from zero flux and counters (ordered before the tiles'
  // atomics by the barrier at the top of the loop); each point spot is planned here as the planner would
  if (a.n_fused > 0) {
    if ((int)blockIdx.x >= a.n_fused) return;
    const DevProfile& pf = a.profiles[blockIdx.x];
    const long long n_flux = (long long)pf.n_bins * pf.n_e;
    for (long long k = tid; k < n_flux; k += nt) a.flux[pf.flux_off + k] = 0.0;
    for (int k = tid; k < kStats; k += nt) pf.stats[k] = 0ull;
    for (int k = tid; k < kMaxSpots * pf.ring_words; k += nt) pf.ring_seen[k] = 0u;
    if (tid == 0) s_tile = -1;  // the spot last taken
  }
  __shared__ Tile s_tile_rec;  // the tile taken (fused mode: built here)
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      if (a.n_fused > 0) {
        const DevProfile& pf = a.profiles[blockIdx.x];
        const int k = fused_next_spot(pf, s_tile + 1);
        s_tile = k;
        s_int[47] = k < pf.n_spots ? 1 : 0;
        s_tile_rec = Tile{(int)blockIdx.x, (short)k, 1, 0, 0, 1, 0, (short)(pf.n_bins * max(pf.n_gl, 1))};
      } else {
        const int t = atomicAdd(a.queue.next, 1);
        const bool live = t < *a.queue.n_tiles && t < a.queue.capacity;
        s_int[47] = live ? 1 : 0;
        if (live) s_tile_rec = a.queue.tiles[t];
      }
    }
    __syncthreads();
    if (!s_int[47]) break;
    const Tile tile = s_tile_rec;
    const DevProfile& p = a.profiles[tile.profile];
    const DevSpot& sp = p.spot[tile.spot];
    const bool point = sp.kind == 1;
    const int n_act = tile_prologue(a, p, sp, tile, s, s_g, s_int, false);
    if (n_act == 0) continue;
    const RingPhi rp = point ? RingPhi{0.0, 0.0} : healpix_ring_phi(p.n_side, tile.ring);

    const DevGrid& G = p.grid;
    const int n_e = G.n_e;
    // partial sums in FP64 in every arithmetic (the FP32 integrand's values are summed exactly enough that the
    // grouping of the points does not show)
    Real E[NE_T];
    double acc[NE_T];
#pragma unroll
    for (int k = 0; k < NE_T; ++k) {
      const int e = tid + k * nt;
      E[k] = e < n_e ? (Real)G.E[e] : (Real)1;
      acc[k] = 0;
    }
    const Real kT = (Real)sp.kT;
    const int n_pp = tile.u1 - tile.u0;  // the tile's phase nodes
    const int n_pts = n_pp * n_act;
    int cur_bin = -1;
    double* flux_base = a.flux + p.flux_off;
    double* comp_base = a.comp ? a.comp + p.flux_off : nullptr;
    const double out_scale = sp.out_scale;
    auto flush = [&]() {
#pragma unroll
      for (int k = 0; k < NE_T; ++k) {
        const int e = tid + k * nt;
        if (e < n_e && acc[k] != 0.0) {
          const size_t o = (size_t)cur_bin * n_e + e;
          comp_add(flux_base + o, comp_base ? comp_base + o : nullptr, acc[k] * out_scale * G.invE[e]);
        }
        acc[k] = 0;
      }
    };
    // Few energies (at most a quarter of the threads): every thread walks a
    // run of consecutive phase points of one element and evaluates each at all
    // energies, instead of the compacted points being walked serially by the
    // threads that own energies.  The lanes of a warp hold consecutive elements
    // at the same phase point, and each thread hunts its next bracket in
    // phase_o from the last one.
    if (n_e * 4 <= nt) {
      const int n_fine = p.n_fine;
      bool ok = true;
      for (int i = tid; i < n_fine; i += nt) ok &= s.P[i + 1] >= s.P[i];
      const bool mono = __syncthreads_and(ok) != 0;
      // per tile, in the lensing-row space the sweep no longer needs: reciprocal
      // phase_o interval widths, the energies and 1/E (when they fit)
      double* inv_dp = (double*)s.rows;
      Real* E_s = (Real*)(inv_dp + n_fine);
      double* invE_s = (double*)(((uintptr_t)(E_s + n_e) + 7) & ~(uintptr_t)7);
      const bool staged = (long)((unsigned char*)(invE_s + n_e) - (unsigned char*)s.rows) <= (long)(S.total - S.off_rows);
      // the phase-major walk also stages each active element's phase shift phi / 2 pi (one division per element
      // per tile instead of one per element and node)
      double* shift_s = invE_s + n_e;
      // FP32 arithmetic: FP32 copies of the fine-phase F and Z after them
      float* F32 = (float*)(shift_s + n_act);
      float* Z32 = F32 + (n_fine + 1);
      const bool fp32 = std::is_same<Real, float>::value;
      const bool pm = n_e <= kPhaseMajorMaxE && mono &&
                      (long)((unsigned char*)(fp32 ? (void*)(Z32 + n_fine + 1) : (void*)(shift_s + n_act)) -
                             (unsigned char*)s.rows) <= (long)(S.total - S.off_rows);
      if (staged) {
        if (mono)
          for (int i = tid; i < n_fine; i += nt) inv_dp[i] = 1.0 / (s.P[i + 1] - s.P[i]);
        for (int e = tid; e < n_e; e += nt) {
          E_s[e] = (Real)G.E[e];
          invE_s[e] = G.invE[e];
        }
        if (pm) {
          for (int jj = tid; jj < n_act; jj += nt) shift_s[jj] = (point ? 0.0 : rp.dphi * (s.j[jj] - rp.jofs)) / kTwoPi;
          if (fp32)
            for (int i = tid; i <= n_fine; i += nt) {
              F32[i] = (float)s.F[i];
              Z32[i] = (float)s.Z[i];
            }
        }
      }
      __syncthreads();
      const double* inv_dp_use = (staged && mono) ? inv_dp : nullptr;
      const int n_fp = n_fine + 1;
      const double P0 = s.P[0];
      const Real inv_kT = (Real)1 / kT;
      if (pm && staged) {
        // Phase-major walk (the os1 light curves: one energy).  A thread walks
        // a contiguous segment of the tile's active elements at one phase
        // point, then at a second one.  The elements' azimuths increase along the ring, so the
        // point's patch phase moves monotonically from one element to the
        // next (wrapping once past 1) and its phase_o bracket is hunted from
        // the previous element's: vhunt's bracket exactly, as phase_o is
        // non-decreasing.  The point's sums stay in FP64 registers; one atomic
        // per energy flushes them at the end of the segment.
        const int n_gl = p.n_gl;
        const double inv_bins = 1. / p.n_bins;
        // Work items pair node k with node k + H, H = ceil(nodes / 2), half a
        // rotation later, on one segment: an element seen at one of the two
        // phases is often hidden at the other, so the pairs cost about the
        // same and the warps finish together.  Each item ends with one
        // compensated atomic per energy, whose returned value the thread
        // waits for, so the items are kept few and long.
        const int H = (n_pp + 1) / 2;
        const int segs = max(1, min(n_act, nt / max(1, H)));
        const double scale = out_scale;
        const int lane = tid & 31;
        unsigned int n_vis = 0;
        for (int it = tid; it < H * segs; it += nt) {
          const int seg = it / H;
          const int jj0 = (int)((long long)n_act * seg / segs), jj1 = (int)((long long)n_act * (seg + 1) / segs);
          for (int half = 0; half < 2; ++half) {
            const int kk = it % H + half * H;
            if (kk >= n_pp) break;
            const int k = tile.u0 + kk;
            int bin, g = 0;
            if (n_gl > 0) {
              bin = k / n_gl;
              g = k - bin * n_gl;
            } else {
              bin = k;
            }
            double ppt, wgl;
            if (n_gl > 0) {
              const double lb = bin * inv_bins, ub = (bin + 1) * inv_bins;
              ppt = 0.5 * (lb + ub + c_gl_nodes[n_gl * (n_gl - 1) / 2 + g] * (ub - lb));
              wgl = 0.5 * 1. * c_gl_weights[n_gl * (n_gl - 1) / 2 + g];
            } else {
              ppt = bin * inv_bins;
              wgl = 1.0;
            }
            double acc[kPhaseMajorMaxE];
#pragma unroll
            for (int e = 0; e < kPhaseMajorMaxE; ++e) acc[e] = 0.0;
            n_vis += n_e == 1 ? pm_walk<Real, 1>(s, inv_dp, F32, Z32, shift_s, E_s, n_e, inv_kT, ppt, wgl, jj0, jj1,
                                                 n_fp, P0, acc)
                              : pm_walk<Real, kPhaseMajorMaxE>(s, inv_dp, F32, Z32, shift_s, E_s, n_e, inv_kT, ppt, wgl,
                                                               jj0, jj1, n_fp, P0, acc);
#pragma unroll
            for (int e = 0; e < kPhaseMajorMaxE; ++e)
              if (e < n_e && acc[e] != 0.0) {
                const size_t o = (size_t)bin * n_e + e;
                comp_add(flux_base + o, comp_base ? comp_base + o : nullptr, acc[e] * scale * invE_s[e]);
              }
          }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) n_vis += __shfl_down_sync(0xffffffffu, n_vis, off);
        if (lane == 0 && n_vis) atomicAdd(&p.stats[3], (unsigned long long)n_vis);
        continue;
      }
      const int runs = max(1, min(n_pp, nt / n_act));  // runs of phase points per element
      const int per_run = (n_pp + runs - 1) / runs;
      const int n_items = n_act * runs;
      const int lane = tid & 31;
      const int n_gl = p.n_gl;
      const double inv_bins = 1. / p.n_bins;
      const double scale = out_scale;
      unsigned int n_vis = 0;
      for (int it0 = 0; it0 < n_items; it0 += nt) {
        const int it = it0 + tid;
        const bool live = it < n_items;
        const int jj = live ? it % n_act : 0;
        const int pp0 = live ? (it / n_act) * per_run : 0;
        const int pp1 = live ? min(n_pp, pp0 + per_run) : 0;
        const double phase_shift = (point ? 0.0 : rp.dphi * (s.j[jj] - rp.jofs)) / kTwoPi;
        int hint = -1;
        for (int k = 0; k < per_run; ++k) {  // the same trip count on every lane
          int bin = INT_MAX;  // lanes without a point: a bin after every real one
          double c = 0, zz = 0;
          bool vis = false;
          if (pp0 + k < pp1) {
            double wgl, z = 0;
            const double flux =
                phase_point_at(s, n_fp, P0, inv_dp_use, n_gl, inv_bins, phase_shift, tile.u0 + pp0 + k, mono, hint, bin,
                               wgl, z);
            if (flux != 0.0) {
              vis = true;
              c = flux * wgl;
              zz = z;
            }
          }
          n_vis += vis ? 1u : 0u;
          // bins never decrease along the lanes (consecutive elements of one run
          // share the phase point; later runs have later points; lanes without a
          // point come last), so the lanes of one bin are one run of lanes, summed
          // by a segmented shuffle reduction into the run's first lane
          const int prev_bin = __shfl_up_sync(0xffffffffu, bin, 1);
          const bool head = (lane == 0 || prev_bin != bin) && bin != INT_MAX;
          const Real cb = (Real)c, zb = (Real)zz;
          for (int e = 0; e < n_e; ++e) {
            double v = 0;
            if (vis) {
              const Real Ee = (staged ? E_s[e] : (Real)G.E[e]) * zb;
              v = (double)(cb * (Ee * Ee * Ee / expm1(Ee * inv_kT)));  // Ibb without its constant (in out_scale)
            }
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
              const double o = __shfl_down_sync(0xffffffffu, v, off);
              const int ob = __shfl_down_sync(0xffffffffu, bin, off);
              if (lane + off < 32 && ob == bin) v += o;
            }
            if (head && v != 0.0) {
              const size_t o = (size_t)bin * n_e + e;
              comp_add(flux_base + o, comp_base ? comp_base + o : nullptr,
                       v * scale * (staged ? invE_s[e] : G.invE[e]));
            }
          }
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) n_vis += __shfl_down_sync(0xffffffffu, n_vis, off);
      if (lane == 0 && n_vis) atomicAdd(&p.stats[3], (unsigned long long)n_vis);
      continue;
    }
    for (int q0 = 0; q0 < n_pts; q0 += nt) {
      bool vis = false;
      double c = 0, zz = 0;
      int bin = 0;
      const int q = q0 + tid;
      if (q < n_pts) {
        double wgl, z = 0, mu = 0;
        const double flux = phase_point(p, s, rp, point, n_act, tile.u0, q, bin, wgl, z, mu);
        if (flux != 0.0) {
          vis = true;
          c = flux * wgl;
          zz = z;
        }
      }
      int n_batch;
      const int slot = block_compact(vis, s_int, &n_batch);
      if (vis) {
        b_c[slot] = c;
        b_z[slot] = zz;
        b_bin[slot] = bin;
      }
      if (tid == 0 && n_batch) atomicAdd(&p.stats[3], (unsigned long long)n_batch);
      __syncthreads();
      for (int b = 0; b < n_batch; ++b) {
        const int bb = b_bin[b];
        if (bb != cur_bin) {
          if (cur_bin >= 0) flush();
          cur_bin = bb;
        }
        const Real cb = (Real)b_c[b], zb = (Real)b_z[b];
#pragma unroll
        for (int k = 0; k < NE_T; ++k) {
          // Ibb(E, kT) = Ibb_constant E^3 / expm1(E / kT) (cpu/unit.hpp:28-31); the constant is in out_scale
          const Real Ee = E[k] * zb;
          const Real I = Ee * Ee * Ee / expm1(Ee / kT);
          acc[k] += (double)(cb * I);
        }
      }
      __syncthreads();
    }
    if (cur_bin >= 0) flush();
  }
}

// ---------------------------------------------------------------------------
// Whether the ring is skipped because fine sample 0 or n_fine-1 is invisible
// (cpu/devarshi24st_cpu.cpp:195), evaluated with the sweep's own arithmetic.
__device__ bool ring_dropped(const DevProfile& p, const DevLens& L, const RingGeom& g, bool nsx) {
  LensRows rows;
  lens_rows_global(L, g.i_u, rows);
  double F, Z, P, MU;
  if (!sweep_sample(p, L, g, rows, 0, nsx, F, Z, P, MU)) return true;
  if (!sweep_sample(p, L, g, rows, p.n_fine - 1, nsx, F, Z, P, MU)) return true;
  return false;
}

__device__ __forceinline__ void push_tile(const WorkQueue& q, const Tile& t) {
  const int k = atomicAdd(q.n_tiles, 1);
  if (k < q.capacity)
    q.tiles[k] = t;
  else
    atomicOr(q.overflow, 1);
}

// One CTA per (profile, spot, ring block): a spot's rings are shared by
// ring_blocks CTAs, so that a small batch plans on many SMs at once.  Every
// chunk of a ring's candidate range becomes ceil(nodes / nodes_per_tile) tiles,
// one per range of phase nodes.
__global__ void plan_kernel(const DevProfile* profiles, int n_profiles, const DevLens L, const WorkQueue q, int chunk,
                            int nodes_per_tile, int ring_blocks) {
  const int ps = blockIdx.x / ring_blocks, rb = blockIdx.x - ps * ring_blocks;
  const int pi = ps / kMaxSpots, si = ps % kMaxSpots;
  if (pi >= n_profiles) return;
  const DevProfile& p = profiles[pi];
  if (si >= p.n_spots) return;
  const DevSpot& sp = p.spot[si];
  const bool nsx = p.atmosphere == 0;
  const int n_nodes = p.n_bins * max(p.n_gl, 1);
  const int npt = nodes_per_tile > 0 ? min(nodes_per_tile, n_nodes) : n_nodes;
  auto push_nodes = [&](Tile t) {
    for (int u = 0; u < n_nodes; u += npt) {
      t.u0 = (short)u;
      t.u1 = (short)min(u + npt, n_nodes);
      push_tile(q, t);
    }
  };
  if (sp.kind == 1) {
    if (sp.i_lo > sp.i_hi || rb != 0) return;  // outside the batch's ring window, or another block's
    if (threadIdx.x == 0) {
      RingGeom g;
      ring_geometry(p, L, sp.cos_theta_pt, sp.dOmega_pt, false, g);
      if (ring_dropped(p, L, g, nsx)) {
        atomicAdd(&p.stats[1], 1ull);
        atomicAdd(&p.stats[2], 1ull);
        atomicAdd(&p.stats[5], 1ull);
      } else {
        push_nodes(Tile{pi, (short)si, 1, 0, 0, 1, 0, 0});
      }
    }
    return;
  }
  const int N = p.n_side;
  for (int i = sp.i_lo + rb * (int)blockDim.x + (int)threadIdx.x; i <= sp.i_hi; i += ring_blocks * (int)blockDim.x) {
    const double z = p.ring[3 * i], c2 = p.ring[3 * i + 1], s2 = p.ring[3 * i + 2];
    const int jmax = healpix_jmax(N, i);
    int r[2][2];
    const int nr = candidate_ranges(sp, N, i, c2, s2, jmax, r);
    if (nr == 0) continue;
    RingGeom g;
    ring_geometry(p, L, z, p.dOmega_hp, false, g);
    if (ring_dropped(p, L, g, nsx)) {
      // count the ring (and its elements) only if it holds active elements
      long long na = 0;
      for (int k = 0; k < nr; ++k)
        for (int j = r[k][0]; j <= r[k][1]; ++j) na += in_spot(sp, c2, s2, healpix_phi(N, i, j)) ? 1 : 0;
      if (na) {
        atomicAdd(&p.stats[1], 1ull);
        atomicAdd(&p.stats[2], 1ull);
        atomicAdd(&p.stats[5], (unsigned long long)na);
        if (g.u_clamped) atomicAdd(&p.stats[4], 1ull);
      }
      continue;
    }
    bool first = true;
    for (int k = 0; k < nr; ++k)
      for (int j0 = r[k][0]; j0 <= r[k][1]; j0 += chunk) {
        const int j1 = min(j0 + chunk, r[k][1] + 1);
        push_nodes(Tile{pi, (short)si, (short)(first ? 1 : 0), i, j0, j1, 0, 0});
        first = false;
      }
  }
}

// ---------------------------------------------------------------------------
template <typename Real>
__global__ void fold_simt_kernel(const FoldJob* jobs, const double* rsp, int n_ch, int n_e, int n_bins,
                                 const double* flux, double* counts) {
  constexpr int TC = 16, TB = 16, TK = 32;
  __shared__ Real sr[TC][TK + 1];
  __shared__ Real sf[TB][TK + 1];
  const FoldJob job = jobs[blockIdx.z];
  const int c0 = blockIdx.x * TC, b0 = blockIdx.y * TB;
  const int tx = threadIdx.x % TB, ty = threadIdx.x / TB;  // tx: bin, ty: channel
  const double* F = flux + job.flux_off;
  Real acc = 0;
  for (int k0 = 0; k0 < n_e; k0 += TK) {
    for (int idx = threadIdx.x; idx < TC * TK; idx += blockDim.x) {
      const int cc = idx / TK, kk = idx % TK;
      const int c = c0 + cc, k = k0 + kk;
      sr[cc][kk] = (c < n_ch && k < n_e) ? (Real)rsp[(size_t)c * n_e + k] : (Real)0;
    }
    for (int idx = threadIdx.x; idx < TB * TK; idx += blockDim.x) {
      const int bb = idx / TK, kk = idx % TK;
      const int b = b0 + bb, k = k0 + kk;
      sf[bb][kk] = (b < n_bins && k < n_e) ? (Real)F[(size_t)b * n_e + k] : (Real)0;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < TK; ++kk) acc += sr[ty][kk] * sf[tx][kk];
    __syncthreads();
  }
  const int c = c0 + ty, b = b0 + tx;
  if (c < n_ch && b < n_bins) counts[job.counts_off + (size_t)c * n_bins + b] = (double)acc * job.alpha;
}

}  // namespace

// ---------------------------------------------------------------------------
IntegrandShape make_shape(bool nsx, int nt, int ne_t, int pb, int max_cand, int n_fine, int n_cp, int n_ca, int nE,
                          int nmu, int cells, bool cellk, int cpl) {
  IntegrandShape s{};
  s.nsx = nsx;
  s.cellk = (nsx && cellk) ? 1 : 0;
  s.nt = nt;
  s.ne_t = ne_t;
  s.pb = pb;
  s.max_cand = max_cand;
  s.n_fine = n_fine;
  s.n_cp = n_cp;
  s.n_ca = n_ca;
  s.nE = nsx ? nE : 0;
  s.nmu = nsx ? nmu : 0;
  s.cells = nsx ? cells : 0;
  auto al = [](long v) { return (int)((v + 15) / 16 * 16); };
  int off = 0;
  s.off_j = off;
  off += al((long)max_cand * 2);
  const long nf1 = n_fine + 1;
  s.off_P = off;
  off += al(nf1 * 8);
  s.off_F = off;
  off += al(nf1 * 8);
  s.off_Z = off;
  off += al(nf1 * 8);
  s.off_MU = off;
  off += al(nf1 * 8);
  s.off_mu = off;
  off += nsx ? al((long)nmu * 8 * 5 + (s.cellk ? 2 * kMuHints : 0)) : 0;
  s.off_S = off;
  const int rows = al((long)(4 * n_cp + 2 * n_ca) * 8);
  if (s.cellk) {
    // home-cell kernel: odd row stride; the lensing rows (used only by the
    // sweep, before the slice is built) share the slice's space; 80 bytes per pair of point records
    s.ldS = nmu | 1;
    // rows -1 - cpl .. nE + cpl, row 0 16-byte aligned
    const int slice = al(((long)(((cpl + 1) * s.ldS + 3) & ~3) + (long)(nE + cpl + 1) * s.ldS) * 4);
    s.off_rows = off;
    off += slice > rows ? slice : rows;
    s.off_union = off;
    s.off_batch = off;
    s.off_Q = off;
    off += al((long)nt * (kPairFloats / 2) * 4);
    s.off_hidx = off;
    off += al((long)nf1 * 2);
    s.total = off;
    s.ring_bytes = s.off_rows + rows;
    return s;
  }
  s.ldS = nmu;
  // the slice is stored with the table's 16-byte aligned stride
  const long slice = nsx ? ((long)nE * nmu + 3) / 4 * 4 : 0;
  off += al(slice * 4);
  s.off_union = off;
  const int batch = al((long)nt * kSlotBytes);
  const int qbuf = nsx ? al((long)pb * cells * 16) + al((long)pb * (cells + 3) * 4) : 0;
  s.off_rows = off;
  s.off_batch = off;
  s.off_Q = off + batch;
  off += rows > batch + qbuf ? rows : batch + qbuf;
  s.total = off;
  s.ring_bytes = s.off_rows + rows;
  return s;
}

namespace {
// home-cell kernels: (energy slots per cell, cells per lane) as compiled, two register budgets each: two CTAs per
// SM (96 registers, nothing of the record loop spilled) up to kCellThreads threads, one up to 512
#define PPM_CELL_SHAPES(X) X(2, 1) X(2, 2) X(2, 3) X(3, 1) X(3, 2) X(3, 3) X(4, 1) X(4, 2) X(4, 3) X(8, 1) X(8, 2) X(16, 1)

void* kernel_for(const IntegrandShape& s, int precision) {
  if (s.nsx && s.cellk) {
    const bool two = s.minb >= 2 && s.nt <= kCellThreads;
#define PPM_CELL(E, C)                                                                                            \
  if (s.maxe_t == E && s.cpl == C) {                                                                              \
    if (s.rec)                                                                                                    \
      return (void*)integrand_nsx_rec_kernel<E, C, rec_threads(E)>;                                               \
    return two ? (void*)integrand_nsx_cell_kernel<E, C, kCellThreads, 2> : (void*)integrand_nsx_cell_kernel<E, C, 512, 1>; \
  }
    PPM_CELL_SHAPES(PPM_CELL)
#undef PPM_CELL
    return nullptr;
  }
  if (s.nsx) {
    const bool two = s.minb >= 2;
    switch (s.ne_t) {
      case 1: return two ? (void*)integrand_nsx_kernel<1, 2> : (void*)integrand_nsx_kernel<1, 1>;
      case 2: return two ? (void*)integrand_nsx_kernel<2, 2> : (void*)integrand_nsx_kernel<2, 1>;
      default: return (void*)integrand_nsx_kernel<4, 1>;
    }
  }
  if (s.rec) return precision == 1 ? (void*)integrand_bb_rec_kernel<double> : (void*)integrand_bb_rec_kernel<float>;
  if (precision == 1) {
    switch (s.ne_t) {
      case 1: return (void*)integrand_bb_kernel<double, 1>;
      case 2: return (void*)integrand_bb_kernel<double, 2>;
      default: return (void*)integrand_bb_kernel<double, 4>;
    }
  }
  switch (s.ne_t) {
    case 1: return (void*)integrand_bb_kernel<float, 1>;
    case 2: return (void*)integrand_bb_kernel<float, 2>;
    default: return (void*)integrand_bb_kernel<float, 4>;
  }
}
}  // namespace

namespace {
constexpr int kOnceSlots = 4, kOnceDevices = 64;
std::mutex g_once_mu;
bool g_once_done[kOnceSlots][kOnceDevices];
}  // namespace

cudaError_t once_per_device(int slot, cudaError_t (*set_up)()) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (slot < 0 || slot >= kOnceSlots || dev < 0 || dev >= kOnceDevices) return set_up();
  std::lock_guard<std::mutex> lk(g_once_mu);
  if (g_once_done[slot][dev]) return cudaSuccess;
  e = set_up();
  if (e == cudaSuccess) g_once_done[slot][dev] = true;
  return e;
}

namespace {
// every integrand variant gets the largest dynamic shared-memory allowance of the current device
cudaError_t set_integrand_smem() {
#define PPM_CELL(E, C)                                                                            \
  (void*)integrand_nsx_cell_kernel<E, C, 512, 1>, (void*)integrand_nsx_cell_kernel<E, C, kCellThreads, 2>, \
      (void*)integrand_nsx_rec_kernel<E, C, rec_threads(E)>,
  void* fns[] = {PPM_CELL_SHAPES(PPM_CELL)(void*) ring_kernel<true>, (void*)ring_kernel<false>,
                 (void*)integrand_bb_rec_kernel<double>, (void*)integrand_bb_rec_kernel<float>,
                 (void*)integrand_nsx_kernel<1, 1>, (void*)integrand_nsx_kernel<1, 2>,
                 (void*)integrand_nsx_kernel<2, 1>, (void*)integrand_nsx_kernel<2, 2>, (void*)integrand_nsx_kernel<4, 1>,
                 (void*)integrand_bb_kernel<double, 1>, (void*)integrand_bb_kernel<double, 2>,
                 (void*)integrand_bb_kernel<double, 4>, (void*)integrand_bb_kernel<float, 1>,
                 (void*)integrand_bb_kernel<float, 2>, (void*)integrand_bb_kernel<float, 4>};
#undef PPM_CELL
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  for (void* f : fns) {
    cudaFuncAttributes at{};
    e = cudaFuncGetAttributes(&at, f);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)at.sharedSizeBytes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace

cudaError_t configure_integrand_smem(const IntegrandShape&) { return once_per_device(0, set_integrand_smem); }

int max_active_ctas(const IntegrandShape& s) {
  // the occupancy query costs as much as a launch: the answers are kept, one for each kernel and launch size
  static std::mutex m;
  static std::map<std::tuple<int, void*, int, int>, int> known;
  int n = 0, dev = 0;
  void* f = kernel_for(s, s.bb_fp64);
  if (!f || cudaGetDevice(&dev) != cudaSuccess) return 0;
  const auto key = std::make_tuple(dev, f, s.nt, s.total);
  {
    std::lock_guard<std::mutex> lk(m);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, s.nt, s.total) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lk(m);
  if (known.size() > 1024) known.clear();
  known[key] = n;
  return n;
}

cudaError_t launch_plan(const DevProfile* profiles, int n_profiles, const DevLens& lens, const WorkQueue& q, int chunk,
                        int nodes_per_tile, cudaStream_t st) {
  if (n_profiles <= 0) return cudaSuccess;
  // a few profiles: up to 32 CTAs share each spot's rings (4N - 1 of them at most)
  const int ring_blocks = std::max(1, std::min(32, 64 / n_profiles));
  plan_kernel<<<n_profiles * kMaxSpots * ring_blocks, 128, 0, st>>>(profiles, n_profiles, lens, q, chunk,
                                                                      nodes_per_tile, ring_blocks);
  return cudaGetLastError();
}

namespace {
// flux += comp: the compensation pool's rounding errors back into the flux pool before the fold
__global__ void add_comp_kernel(double* __restrict__ flux, const double* __restrict__ comp, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    flux[i] += comp[i];
}
}  // namespace

cudaError_t launch_add_comp(double* flux, const double* comp, long long n, int sm_count, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const long long blocks = std::min<long long>((n + 255) / 256, (long long)sm_count * 8);
  add_comp_kernel<<<(unsigned)blocks, 256, 0, st>>>(flux, comp, n);
  return cudaGetLastError();
}

namespace {
constexpr int kSumThreads = 256, kSumQ = 32, kSumUnroll = 12, kSumList = 6 * kSumThreads;

__device__ __forceinline__ void dd_add(double& s, double& c, double x) {
  // (intrinsics: x is a product, which must not be contracted into the sum)
  const double t = __dadd_rn(s, x), bb = __dsub_rn(t, s);
  c = __dadd_rn(c, __dadd_rn(__dsub_rn(s, __dsub_rn(t, bb)), __dsub_rn(x, bb)));
  s = t;
}

// The flux of one (profile, bin) from its chunks' node sums (T: float in t_E order for NSX, double in energy order
// for blackbody): grid (bins, energy tiles of Q, profiles from p0 on), Q energies x kSumThreads / Q segments of chunks.
// Double-double sums: the exact sum to about 1e-32, in any order of the records, as the pool's compensated atomics
// give it; what the atomics added is included.  Bound by the read of the node sums, from L2 for a single profile:
// 125 MB in 69 us with 12 loads in flight a thread and 256-thread blocks (512 threads, 8 loads: 83 to 108; 1024
// threads, one after the other: 177), of an 1080 us call.
template <typename T>
__global__ void __launch_bounds__(kSumThreads) sum_parts_kernel(const KernelArgs a, int Q, int p0) {
  const RingWork& W = a.rings;
  const DevProfile& p = a.profiles[p0 + (int)blockIdx.z];
  const int bin = blockIdx.x, n_e = p.n_e, segs = kSumThreads / Q;
  const int ql = threadIdx.x % Q, seg = threadIdx.x / Q, q = blockIdx.y * Q + ql;
  if (bin >= p.n_bins || blockIdx.y * Q >= n_e) return;
  // the profile's (record, GL node) rows, in units of 4 bytes: the first spot's from the front, the second's from the
  // back of the list
  __shared__ unsigned s_ofs[kSumList];
  __shared__ int s_n[kMaxSpots];
  __shared__ double s_s[kSumThreads], s_c[kSumThreads];
  const int n_recs = (int)*p.ring_seen;
  const int* const recs = W.by_profile + (size_t)W.per_job * p.spot[0].job0;
  const int e = q < n_e ? (std::is_same<T, float>::value ? p.grid.perm[q] : q) : 0;
  const double invE = q < n_e ? p.grid.invE[e] : 0.0;
  const int n_gl = max(p.n_gl, 1);
  const double scale0 = p.spot[0].out_scale, scale1 = p.spot[1].out_scale;
  const float* const src = (const float*)((const T*)W.parts + (size_t)bin * n_gl * n_e + min(q, n_e - 1));
  double s = 0.0, c = 0.0;
  for (int r0 = 0; r0 < n_recs; r0 += kSumThreads) {
    __syncthreads();
    if (threadIdx.x < kMaxSpots) s_n[threadIdx.x] = 0;
    __syncthreads();
    const int entry = r0 + (int)threadIdx.x < n_recs ? recs[r0 + threadIdx.x] : 2 * W.part_cap, r = entry >> 1;
    if (r < W.part_cap) {
      const int sp = entry & 1, at = atomicAdd(&s_n[sp], n_gl);
      for (int g = 0; g < n_gl; ++g)
        s_ofs[sp ? kSumList - 1 - (at + g) : at + g] =
            (unsigned)(r * W.part_stride) + (unsigned)(g * n_e * (int)(sizeof(T) / 4));
    }
    __syncthreads();
    const int n0 = s_n[0], n = n0 + s_n[1];
    for (int k0 = seg; k0 < n; k0 += kSumUnroll * segs) {
      T v[kSumUnroll];  // (loads in flight together)
#pragma unroll
      for (int u = 0; u < kSumUnroll; ++u) {
        const int k = k0 + u * segs;
        v[u] = k < n ? __ldcg((const T*)(src + s_ofs[k < n0 ? k : kSumList - 1 - (k - n0)])) : (T)0;
      }
#pragma unroll
      for (int u = 0; u < kSumUnroll; ++u)
        dd_add(s, c, __dmul_rn(__dmul_rn((double)v[u], k0 + u * segs < n0 ? scale0 : scale1), invE));
    }
  }
  s_s[threadIdx.x] = s;
  s_c[threadIdx.x] = c;
  for (int half = segs / 2; half > 0; half /= 2) {
    __syncthreads();
    if (seg < half) {
      dd_add(s, c, s_s[threadIdx.x + half * Q]);
      c += s_c[threadIdx.x + half * Q];
      s_s[threadIdx.x] = s;
      s_c[threadIdx.x] = c;
    }
  }
  if (seg == 0 && q < n_e) {
    const size_t o = (size_t)p.flux_off + (size_t)bin * n_e + e;
    dd_add(s, c, a.flux[o]);
    c += a.comp[o];
    a.comp[o] = 0.0;
    a.flux[o] = s + c;
  }
}
}  // namespace

cudaError_t launch_sum_parts(const KernelArgs& a, int bins_max, int ne_max, cudaStream_t st) {
  int Q = 1;
  while (Q < kSumQ && Q < ne_max) Q <<= 1;
  for (int p0 = 0; p0 < a.rings.n_profiles; p0 += kSumProfiles) {
    const dim3 grid(bins_max, (ne_max + Q - 1) / Q, std::min(kSumProfiles, a.rings.n_profiles - p0));
    if (a.shape.nsx)
      sum_parts_kernel<float><<<grid, kSumThreads, 0, st>>>(a, Q, p0);
    else
      sum_parts_kernel<double><<<grid, kSumThreads, 0, st>>>(a, Q, p0);
  }
  return cudaGetLastError();
}

cudaError_t launch_rings(const KernelArgs& a, cudaStream_t st) {
  if (a.rings.n_jobs <= 0) return cudaSuccess;
  if (a.shape.nsx)
    ring_kernel<true><<<a.rings.n_jobs, 256, a.shape.ring_bytes, st>>>(a);
  else
    ring_kernel<false><<<a.rings.n_jobs, 256, a.shape.ring_bytes, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_integrand(const KernelArgs& a, int grid, cudaStream_t st) {
  if (grid <= 0) return cudaSuccess;
  const IntegrandShape& s = a.shape;
  void* f = nullptr;
  f = kernel_for(s, s.bb_fp64);
  void* args[] = {(void*)&a};
  return cudaLaunchKernel(f, dim3(grid), dim3(s.nt), args, s.total, st);
}

cudaError_t launch_fold_simt(const FoldJob* jobs, int n_jobs, const double* rsp, int n_ch, int n_e, int n_bins,
                             const double* flux, double* counts, bool fp64, cudaStream_t st) {
  if (n_jobs <= 0) return cudaSuccess;
  dim3 grid((n_ch + 15) / 16, (n_bins + 15) / 16, n_jobs);
  if (fp64)
    fold_simt_kernel<double><<<grid, 256, 0, st>>>(jobs, rsp, n_ch, n_e, n_bins, flux, counts);
  else
    fold_simt_kernel<float><<<grid, 256, 0, st>>>(jobs, rsp, n_ch, n_e, n_bins, flux, counts);
  return cudaGetLastError();
}

}  // namespace ppm
