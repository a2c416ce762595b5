// Jacobi relaxation of the Poisson equation on the voxel grid.
//
// Reference mode (gpu_hartree_iteration, kernel_hartree.cu:85-171):
//     V'(interior) = (xm + xp + yp + ym + zp + zm - Q/h) / 6,  V' = 0 on the outer shell,
// summed in that order so FP32 results match the reference update.
// Dirichlet mode (new): V'(interior) = (sum of 6 neighbours + 4 pi h^2 rho) / 6, evaluated as an
// increment of V, and the outer shell keeps its given values.
//
// Three kernels, all one launch for every sweep and all with the same update, so their results are
// identical; they differ in where the field lives and who waits for whom:
//   persistent  any grid: the field in L2 (three fields up to 192^3 = 85 MB stay there), a work item
//               is four consecutive x points, a grid barrier between sweeps (persistent.cuh);
//   plane       nz <= the SM count, planes of up to 16384 points: one CTA per plane, values in
//               registers and shared memory, only z neighbours through L2, each CTA waiting for its two
//               neighbours' publications;
//   cluster     up to 4096 points a plane, 64 planes: one 16-CTA thread-block cluster, the field in
//               the CTAs' shared memory, z neighbours through distributed shared memory, the hardware
//               cluster barrier between sweeps (the best for the smallest grids).
// V and its copy are rewritten by other CTAs between sweeps, so they are read through L2
// (ld.global.cg), never through the non-coherent L1 paths.  On sweeps that feed a
// convergence check each CTA sums |V' - V| in FP64 over its points and the CTA sums are added in
// CTA order, so the residual is deterministic, and every CTA takes the same stop decision.  Every wait is
// bounded: it raises an error flag after the library's wait limit (2 s unless qmt_set_wait_limit_ns changed it).
#include "mol.cuh"
#include "persistent.cuh"
#include "reduce.cuh"
#include "sm100.cuh"

namespace qmt {

constexpr int JX = 32, JY = 8;
constexpr int JAC_THREADS = JX * JY;
constexpr int JAC_BLOCKS_PER_SM = 4;

struct JacobiArgs {
  int nx, ny, nz;
  float h, src_scale;
  const float* Q;
  float* V;            // start value in, result out
  float* T;            // second buffer
  int vec4;            // nx % 4 == 0 and 16-byte aligned V, T, Q: groups of four x points
  int max_sweeps, check_every;
  double tol;
  double* part;        // per-CTA partial sums
  unsigned long long* bar;   // grid-barrier counter
  unsigned long long* pub;   // plane kernel: sweeps published by each plane
  uint64_t wait_ns;    // limit of a grid-barrier wait before the solve gives up
  double* res;         // [0] residual of the last check
  int* out;            // [0] sweeps done, [1] status: 0 running/cap, 1 converged, 2 not finite, 3 barrier timeout
};

template <bool DIRICHLET>
__device__ __forceinline__ float jac_source(float q, float h, float src_scale) {
  if constexpr (!DIRICHLET) return q / h;
  else return __fmul_rn(src_scale, q);
}

// Update of one point from its six neighbours (in the reference's summation order) and its
// source term.
template <bool DIRICHLET>
__device__ __forceinline__ float jac_point(float xm, float xp, float yp, float ym, float zp, float zm, float src,
                                           float vc, bool edge) {
  if constexpr (!DIRICHLET) {
    float s = xm + xp;
    s = s + yp;
    s = s + ym;
    s = s + zp;
    s = s + zm;
    s = s - src;
    return edge ? 0.f : s / 6.0f;
  } else {
    // increment form V + (sum (nb - V) + 4 pi h^2 rho) / 6: the FP32 rounding of 1/6 and of the
    // neighbour sum then scale only the increment, which vanishes at convergence.  (The direct
    // form (sum nb + 4 pi h^2 rho) * fp32(1/6) biases every sweep the same way; over 2000 sweeps
    // of a 64^3 grid the smooth error modes amplify that to ~1e-5 relative, against ~4e-8 here.)
    const float s = ((xm - vc) + (xp - vc)) + ((yp - vc) + (ym - vc)) + ((zp - vc) + (zm - vc));
    return edge ? vc : fmaf(__fadd_rn(s, src), 1.0f / 6.0f, vc);
  }
}


// One sweep src -> dst.  Work items are groups of four consecutive x points (float4 loads of
// the row, the four neighbouring rows and Q, scalar loads of the two x halo values), spread over
// all CTAs; every load of a group is independent, so many are in flight per thread.  Returns
// this thread's FP64 sum |dst - src| when `resid` is set.
template <bool DIRICHLET>
__device__ double sweep(const JacobiArgs& a, const float* src, float* dst, bool resid, const GridWalk& wk) {
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int64_t row = nx, plane = (int64_t)nx * ny;
  const int64_t nthreads = (int64_t)gridDim.x * JAC_THREADS;
  const int64_t tid = (int64_t)blockIdx.x * JAC_THREADS + threadIdx.y * JX + threadIdx.x;
  double dsum = 0.0;
  if (a.vec4) {
    const int nxq = nx >> 2;
    const int64_t ngroups = (int64_t)nxq * ny * nz;
    int xq = wk.x, y = wk.y, z = wk.z;
    for (int64_t gi = tid; gi < ngroups; gi += nthreads) {
      const int x0 = xq * 4;
      const int64_t b = z * plane + (int64_t)y * row + x0;
      const float4 c = ldcg4(src + b);
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 ym = y > 0 ? ldcg4(src + b - row) : zero;
      const float4 yp = y + 1 < ny ? ldcg4(src + b + row) : zero;
      const float4 zm = z > 0 ? ldcg4(src + b - plane) : zero;
      const float4 zp = z + 1 < nz ? ldcg4(src + b + plane) : zero;
      const float4 q4 = __ldg(reinterpret_cast<const float4*>(a.Q + b));
      const float4 q = make_float4(jac_source<DIRICHLET>(q4.x, a.h, a.src_scale),
                                   jac_source<DIRICHLET>(q4.y, a.h, a.src_scale),
                                   jac_source<DIRICHLET>(q4.z, a.h, a.src_scale),
                                   jac_source<DIRICHLET>(q4.w, a.h, a.src_scale));
      const float xl = x0 > 0 ? __ldcg(src + b - 1) : 0.f;
      const float xr = x0 + 4 < nx ? __ldcg(src + b + 4) : 0.f;
      const bool eyz = y == 0 || y == ny - 1 || z == 0 || z == nz - 1;
      float4 o;
      o.x = jac_point<DIRICHLET>(xl, c.y, yp.x, ym.x, zp.x, zm.x, q.x, c.x, eyz || x0 == 0);
      o.y = jac_point<DIRICHLET>(c.x, c.z, yp.y, ym.y, zp.y, zm.y, q.y, c.y, eyz || x0 + 1 == nx - 1);
      o.z = jac_point<DIRICHLET>(c.y, c.w, yp.z, ym.z, zp.z, zm.z, q.z, c.z, eyz || x0 + 2 == nx - 1);
      o.w = jac_point<DIRICHLET>(c.z, xr, yp.w, ym.w, zp.w, zm.w, q.w, c.w, eyz || x0 + 3 == nx - 1);
      __stcg(reinterpret_cast<float4*>(dst + b), o);
      if (resid)
        dsum += (fabs((double)o.x - (double)c.x) + fabs((double)o.y - (double)c.y)) +
                (fabs((double)o.z - (double)c.z) + fabs((double)o.w - (double)c.w));
      grid_step(wk, nxq, ny, xq, y, z);
    }
  } else {
    const int64_t n = plane * nz;
    int x = wk.x, y = wk.y, z = wk.z;
    for (int64_t g = tid; g < n; g += nthreads) {
      const float vc = __ldcg(src + g);
      const float xm = x > 0 ? __ldcg(src + g - 1) : 0.f;
      const float xp = x + 1 < nx ? __ldcg(src + g + 1) : 0.f;
      const float ym = y > 0 ? __ldcg(src + g - row) : 0.f;
      const float yp = y + 1 < ny ? __ldcg(src + g + row) : 0.f;
      const float zm = z > 0 ? __ldcg(src + g - plane) : 0.f;
      const float zp = z + 1 < nz ? __ldcg(src + g + plane) : 0.f;
      const bool edge = x == 0 || x == nx - 1 || y == 0 || y == ny - 1 || z == 0 || z == nz - 1;
      const float o =
          jac_point<DIRICHLET>(xm, xp, yp, ym, zp, zm, jac_source<DIRICHLET>(__ldg(a.Q + g), a.h, a.src_scale), vc, edge);
      __stcg(dst + g, o);
      if (resid) dsum += fabs((double)o - (double)vc);
      grid_step(wk, nx, ny, x, y, z);
    }
  }
  return dsum;
}

template <bool DIRICHLET>
__global__ void __launch_bounds__(JAC_THREADS, JAC_BLOCKS_PER_SM) jacobi_persistent_kernel(JacobiArgs a) {
  __shared__ double sh[JAC_THREADS / 32];
  const unsigned nb = gridDim.x;
  int* flag = a.out + 2;
  double delta = INFINITY;
  int sweeps = 0, pairs = 0, status = 0;
  const int lin = threadIdx.y * JX + threadIdx.x;
  unsigned long long round = 0;
  const GridWalk wk = grid_walk(a.vec4 ? a.nx >> 2 : a.nx, a.ny, gridDim.x * JAC_THREADS, blockIdx.x * JAC_THREADS + lin);
  while (sweeps + 2 <= a.max_sweeps) {
    ++pairs;
    const bool check = pairs % a.check_every == 0 || sweeps + 4 > a.max_sweeps;
    sweep<DIRICHLET>(a, a.V, a.T, false, wk);
    if (!grid_barrier(a.bar, round, flag, nb, a.wait_ns)) {
      status = 3;
      break;
    }
    const double ds = sweep<DIRICHLET>(a, a.T, a.V, check, wk);
    sweeps += 2;
    if (!check) {
      if (!grid_barrier(a.bar, round, flag, nb, a.wait_ns)) {
        status = 3;
        break;
      }
      continue;
    }
    // FP64 residual: warp tree, warps in order, CTAs in order
    double v = ds;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((lin & 31) == 0) sh[lin >> 5] = v;
    __syncthreads();
    if (lin == 0) {
      double r = 0.0;
      for (int w = 0; w < JAC_THREADS / 32; ++w) r += sh[w];
      __stcg(a.part + blockIdx.x, r);
    }
    if (!grid_barrier(a.bar, round, flag, nb, a.wait_ns)) {
      status = 3;
      break;
    }
    if (blockIdx.x == 0 && lin == 0) {
      double r = 0.0;
      for (unsigned b = 0; b < nb; ++b) r += __ldcg(a.part + b);
      __stcg(a.res, r);
    }
    if (!grid_barrier(a.bar, round, flag, nb, a.wait_ns)) {
      status = 3;
      break;
    }
    delta = __ldcg(a.res);
    if (!isfinite(delta)) {
      status = 2;
      break;
    }
    if (delta <= a.tol) {
      status = 1;
      break;
    }
  }
  if (blockIdx.x == 0 && lin == 0) {
    a.out[0] = sweeps;
    a.out[1] = status;
    __stcg(a.res + 1, delta);
  }
}

// ---- plane kernel ------------------------------------------------------------------------------
// One CTA per plane z (nz <= the SM count): the plane's values stay in its threads' registers and, for the
// x and y neighbours, in shared memory; the charges stay in shared memory; only the planes themselves go
// through L2, for the CTAs of z - 1 and z + 1.  No grid barrier: CTA z publishes the number of sweeps it
// has stored, and starts the next one when its two neighbours have published as many (they have then
// also read what the next store overwrites).  Per sweep 12 B per point of L2 traffic (two planes read,
// one written) against 28 of the persistent kernel, and the waiting time of two neighbours against all
// CTAs'.  The x and y part of the update is formed before the wait.
constexpr int JAC_PLANE_THREADS = 1024;
constexpr int JAC_PLANE_MAX_G = 4;   // groups of four points per thread: planes of up to 16384 points

// The update in two parts: the x and y neighbours, then z and the source (jac_point's order).
template <bool DIRICHLET>
__device__ __forceinline__ float jac_xy(float xm, float xp, float yp, float ym, float vc) {
  if constexpr (!DIRICHLET) return ((xm + xp) + yp) + ym;
  else return ((xm - vc) + (xp - vc)) + ((yp - vc) + (ym - vc));
}
template <bool DIRICHLET>
__device__ __forceinline__ float jac_z(float part, float zp, float zm, float src, float vc, bool edge) {
  if constexpr (!DIRICHLET) {
    const float s = ((part + zp) + zm) - src;
    return edge ? 0.f : s / 6.0f;
  } else {
    const float s = part + ((zp - vc) + (zm - vc));
    return edge ? vc : fmaf(__fadd_rn(s, src), 1.0f / 6.0f, vc);
  }
}

template <bool DIRICHLET, int G>
__global__ void __launch_bounds__(JAC_PLANE_THREADS, 1) jacobi_plane_kernel(JacobiArgs a) {
  extern __shared__ float4 pbuf[];
  __shared__ double red[JAC_PLANE_THREADS / 32];
  __shared__ int ok_s;
  const int nx = a.nx, ny = a.ny, nz = a.nz, nxq = nx >> 2, ng = nxq * ny;
  const int t = threadIdx.x, lane = t & 31, z = blockIdx.x;
  int* flag = a.out + 2;
  float4* val = pbuf;         // the plane's values
  float4* src = pbuf + ng;    // its source terms
  const int64_t plane = (int64_t)nx * ny, base = z * plane;
  float4 v[G];
  uint32_t edges = 0;         // per group: bit 0 whole row is edge, bit 1 x low, bit 2 x high, bit 3 y low, bit 4 y high
#pragma unroll
  for (int k = 0; k < G; ++k) {
    const int g = t + k * JAC_PLANE_THREADS;
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g < ng) {
      const int y = g / nxq, xq = g - y * nxq;
      v[k] = __ldcg(reinterpret_cast<const float4*>(a.V + base) + g);
      const float4 q4 = __ldg(reinterpret_cast<const float4*>(a.Q + base) + g);
      src[g] = make_float4(jac_source<DIRICHLET>(q4.x, a.h, a.src_scale), jac_source<DIRICHLET>(q4.y, a.h, a.src_scale),
                           jac_source<DIRICHLET>(q4.z, a.h, a.src_scale), jac_source<DIRICHLET>(q4.w, a.h, a.src_scale));
      val[g] = v[k];
      uint32_t e = 0;
      if (y == 0 || y == ny - 1 || z == 0 || z == nz - 1) e |= 1u;
      if (xq == 0) e |= 2u;
      if (xq == nxq - 1) e |= 4u;
      if (y == 0) e |= 8u;
      if (y == ny - 1) e |= 16u;
      edges |= e << (8 * k);
    }
  }
  __syncthreads();
  int sweeps = 0, pairs = 0, status = 0;
  unsigned long long round = 0;
  double delta = INFINITY;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  while (sweeps + 2 <= a.max_sweeps) {
    ++pairs;
    const bool check = pairs % a.check_every == 0 || sweeps + 4 > a.max_sweeps;
    double ds = 0.0;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const float* from = half == 0 ? a.V : a.T;
      float* to = half == 0 ? a.T : a.V;
      const bool resid = check && half == 1;
      // x and y neighbours from this CTA's plane
      float4 p[G];
#pragma unroll
      for (int k = 0; k < G; ++k) {
        const int g = t + k * JAC_PLANE_THREADS;
        const uint32_t e = edges >> (8 * k);
        const float4 c = v[k];
        const float wl = __shfl_up_sync(0xffffffffu, c.w, 1), xr0 = __shfl_down_sync(0xffffffffu, c.x, 1);
        if (g < ng) {
          const float4 ym = e & 8u ? zero : val[g - nxq], yp = e & 16u ? zero : val[g + nxq];
          const float xl = e & 2u ? 0.f : (lane == 0 ? val[g - 1].w : wl);
          const float xr = e & 4u ? 0.f : (lane == 31 ? val[g + 1].x : xr0);
          p[k].x = jac_xy<DIRICHLET>(xl, c.y, yp.x, ym.x, c.x);
          p[k].y = jac_xy<DIRICHLET>(c.x, c.z, yp.y, ym.y, c.y);
          p[k].z = jac_xy<DIRICHLET>(c.y, c.w, yp.z, ym.z, c.z);
          p[k].w = jac_xy<DIRICHLET>(c.z, xr, yp.w, ym.w, c.w);
        }
      }
      // the neighbouring planes have stored sweep `sweeps + half`
      if (t == 0) ok_s = 1;
      __syncthreads();
      if (t < 2) {
        const int zn = t == 0 ? z - 1 : z + 1;
        if (zn >= 0 && zn < nz && !wait_count(a.pub + zn, (unsigned long long)(sweeps + half), flag, a.wait_ns)) {
          atomicOr(a.pub + z, kGaveUp);   // passes it on
          ok_s = 0;
        }
      }
      __syncthreads();
      if (!ok_s) {
        status = 3;
        break;
      }
#pragma unroll
      for (int k = 0; k < G; ++k) {
        const int g = t + k * JAC_PLANE_THREADS;
        if (g < ng) {
          const uint32_t e = edges >> (8 * k);
          const float4 zm = z > 0 ? __ldcg(reinterpret_cast<const float4*>(from + base - plane) + g) : zero;
          const float4 zp = z + 1 < nz ? __ldcg(reinterpret_cast<const float4*>(from + base + plane) + g) : zero;
          const float4 s4 = src[g], c = v[k];
          const bool er = e & 1u, elo = e & 2u, ehi = e & 4u;
          float4 o;
          o.x = jac_z<DIRICHLET>(p[k].x, zp.x, zm.x, s4.x, c.x, er || elo);
          o.y = jac_z<DIRICHLET>(p[k].y, zp.y, zm.y, s4.y, c.y, er);
          o.z = jac_z<DIRICHLET>(p[k].z, zp.z, zm.z, s4.z, c.z, er);
          o.w = jac_z<DIRICHLET>(p[k].w, zp.w, zm.w, s4.w, c.w, er || ehi);
          __stcg(reinterpret_cast<float4*>(to + base) + g, o);
          val[g] = o;
          v[k] = o;
          if (resid)
            ds += (fabs((double)o.x - (double)c.x) + fabs((double)o.y - (double)c.y)) +
                  (fabs((double)o.z - (double)c.z) + fabs((double)o.w - (double)c.w));
        }
      }
      __syncthreads();   // the plane's stores before its publication, its values before the next reads
      if (t == 0)
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(a.pub + z) : "memory");
    }
    if (status) break;
    sweeps += 2;
    if (!check) continue;
    // FP64 residual: warp tree, warps in order, planes in order; every CTA adds the same partials in
    // the same order and takes the same decision
    for (int o = 16; o > 0; o >>= 1) ds += __shfl_xor_sync(0xffffffffu, ds, o);
    if (lane == 0) red[t >> 5] = ds;
    __syncthreads();
    if (t == 0) {
      double r = 0.0;
      for (int w = 0; w < JAC_PLANE_THREADS / 32; ++w) r += red[w];
      __stcg(a.part + z, r);
    }
    if (!grid_barrier(a.bar, round, flag, gridDim.x, a.wait_ns)) {
      status = 3;
      break;
    }
    if (t < 32) {
      double r = 0.0;
      for (int b = t; b < nz; b += 32) r += __ldcg(a.part + b);
      for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
      if (t == 0) red[0] = r;
    }
    __syncthreads();
    delta = red[0];
    // the partials may be overwritten only when every CTA has read them: the next check is at least one
    // publication of the neighbours away, but not of all CTAs
    if (!grid_barrier(a.bar, round, flag, gridDim.x, a.wait_ns)) {
      status = 3;
      break;
    }
    if (!isfinite(delta)) {
      status = 2;
      break;
    }
    if (delta <= a.tol) {
      status = 1;
      break;
    }
  }
  if (z == 0 && t == 0) {
    a.out[0] = sweeps;
    a.out[1] = status;
    __stcg(a.res + 1, delta);
  }
}

// ---- single-cluster kernel ---------------------------------------------------------------------
constexpr int JAC_CLUSTER = 16;          // CTAs of the cluster (a non-portable size)
constexpr int JAC_CLUSTER_THREADS = 1024;

// One cluster; CTA c owns planes [c P, c P + np) of the grid.  Thread t owns the four-point group
// (xq, y) = (t % nxq, t / nxq) of every plane of the slab.  Shared memory: buf[2][P][ny][nxq]
// float4 (the field before / after a sweep).  Launched only when nx % 4 == 0, nxq * ny <= 1024,
// ceil(nz / 16) <= P <= 4 and V, Q 16-byte aligned (checked on the host).
template <bool DIRICHLET, int P>
__global__ void __launch_bounds__(JAC_CLUSTER_THREADS, 1) jacobi_cluster_kernel(JacobiArgs a) {
  extern __shared__ float4 jbuf[];
  __shared__ double red[JAC_CLUSTER_THREADS / 32];
  __shared__ double part;
  __shared__ int stop_s;
  const int nx = a.nx, ny = a.ny, nz = a.nz, nxq = nx >> 2;
  const int t = threadIdx.x, lane = t & 31;
  const bool act = t < nxq * ny;
  const int xq = act ? t % nxq : 0, y = act ? t / nxq : 0;
  const uint32_t c = sm100::cluster_cta_rank(), ncta = gridDim.x;
  const int z0 = (int)c * P;
  const int np = max(0, min(P, nz - z0));
  const int pstride = nxq * ny;                 // float4 per plane
  float4* buf0 = jbuf;
  float4* buf1 = jbuf + (size_t)P * pstride;
  const int own = y * nxq + xq;
  float4 v[P], q[P];
#pragma unroll
  for (int k = 0; k < P; ++k) {
    v[k] = q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act && k < np) {
      const int64_t g = ((int64_t)(z0 + k) * ny + y) * nx + xq * 4;
      v[k] = __ldcg(reinterpret_cast<const float4*>(a.V + g));
      const float4 q4 = __ldg(reinterpret_cast<const float4*>(a.Q + g));   // source terms, once
      q[k] = make_float4(jac_source<DIRICHLET>(q4.x, a.h, a.src_scale), jac_source<DIRICHLET>(q4.y, a.h, a.src_scale),
                         jac_source<DIRICHLET>(q4.z, a.h, a.src_scale), jac_source<DIRICHLET>(q4.w, a.h, a.src_scale));
      buf0[k * pstride + own] = v[k];
    }
  }
  const bool ey = y == 0 || y == ny - 1;
  const bool xlo = xq == 0, xhi = xq == nxq - 1;
  // shuffles give the x neighbours within a warp; at a warp's first / last lane the group beside
  // it (same row) belongs to another warp and is read from shared memory
  const bool left_smem = !xlo && lane == 0, right_smem = !xhi && lane == 31;
  sm100::cluster_barrier();
  int sweeps = 0, pairs = 0, status = 0;
  double delta = INFINITY;
  while (sweeps + 2 <= a.max_sweeps) {
    ++pairs;
    const bool check = pairs % a.check_every == 0 || sweeps + 4 > a.max_sweeps;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      float4* src = half == 0 ? buf0 : buf1;
      float4* dst = half == 0 ? buf1 : buf0;
      const bool resid = check && half == 1;
      double ds = 0.0;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 below = zero, above = zero;
      if (act && np > 0) {
        if (z0 > 0) below = sm100::cluster_load_f4(src + (P - 1) * pstride + own, c - 1);
        if (z0 + np < nz) above = sm100::cluster_load_f4(src + own, c + 1);
      }
      float4 prev = below;
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const float4 cen = v[k];
        const float wl = __shfl_up_sync(0xffffffffu, cen.w, 1);
        const float xr0 = __shfl_down_sync(0xffffffffu, cen.x, 1);
        if (k < np && act) {
          const float4* pl = src + k * pstride;
          const float4 ym = y > 0 ? pl[own - nxq] : zero;
          const float4 yp = y + 1 < ny ? pl[own + nxq] : zero;
          const float4 zp = k + 1 < np ? v[k + 1] : above;
          const float4 zm = prev;
          const float xl = xlo ? 0.f : (left_smem ? pl[own - 1].w : wl);
          const float xr = xhi ? 0.f : (right_smem ? pl[own + 1].x : xr0);
          const int z = z0 + k;
          const bool eyz = ey || z == 0 || z == nz - 1;
          float4 o;
          o.x = jac_point<DIRICHLET>(xl, cen.y, yp.x, ym.x, zp.x, zm.x, q[k].x, cen.x, eyz || xlo);
          o.y = jac_point<DIRICHLET>(cen.x, cen.z, yp.y, ym.y, zp.y, zm.y, q[k].y, cen.y, eyz || xq * 4 + 1 == nx - 1);
          o.z = jac_point<DIRICHLET>(cen.y, cen.w, yp.z, ym.z, zp.z, zm.z, q[k].z, cen.z, eyz || xq * 4 + 2 == nx - 1);
          o.w = jac_point<DIRICHLET>(cen.z, xr, yp.w, ym.w, zp.w, zm.w, q[k].w, cen.w, eyz || xhi);
          if (resid)
            ds += (fabs((double)o.x - (double)cen.x) + fabs((double)o.y - (double)cen.y)) +
                  (fabs((double)o.z - (double)cen.z) + fabs((double)o.w - (double)cen.w));
          prev = cen;
          v[k] = o;
          dst[k * pstride + own] = o;
        }
      }
      sm100::cluster_barrier();   // every read of src done, every write of dst visible cluster-wide
      if (resid) {
        // FP64 residual: warp tree, warps in order, CTAs in rank order -- every CTA adds the same
        // partials in the same order, so all take the same decision
        for (int o = 16; o > 0; o >>= 1) ds += __shfl_xor_sync(0xffffffffu, ds, o);
        if (lane == 0) red[t >> 5] = ds;
        __syncthreads();
        if (t == 0) {
          double r = 0.0;
          for (int w = 0; w < JAC_CLUSTER_THREADS / 32; ++w) r += red[w];
          part = r;
        }
        sm100::cluster_barrier();
        if (t == 0) {
          double r = 0.0;
          for (uint32_t b = 0; b < ncta; ++b) r += sm100::cluster_load_f64(&part, b);
          delta = r;
          stop_s = !isfinite(r) ? 2 : (r <= a.tol ? 1 : 0);
        }
        __syncthreads();
      }
    }
    sweeps += 2;
    if (check) {
      status = stop_s;
      if (status != 0) break;
    }
  }
  // no CTA may leave while another can still read its shared memory
  sm100::cluster_barrier();
#pragma unroll
  for (int k = 0; k < P; ++k)
    if (act && k < np)
      __stcg(reinterpret_cast<float4*>(a.V + ((int64_t)(z0 + k) * ny + y) * nx + xq * 4), v[k]);
  if (c == 0 && t == 0) {
    a.out[0] = sweeps;
    a.out[1] = status;
    a.res[1] = delta;
  }
}

// Groups per thread of the plane kernel for this grid, or 0 where it does not apply or is not the faster
// one: one CTA per plane, all resident at once.  Its sweep takes about 1.2 us + 1.05 us per group of
// 1024 x 4 points of a plane, whatever nz; the grid-barrier kernel's 2.2 us + 2.3 us per million points
// (Dirichlet, us per sweep, plane / grid barrier: 64^3 2.1 / 2.6, 120x56x56 2.8 / 3.2, 128x64x128 2.9 / 4.9,
// 96x96x64 3.9 / 4.0, 96x128x120 4.5 / 5.9, 128^3 5.4 / 6.9, 128x120x88 5.2 / 5.7, 128x128x48 5.3 / 4.7).
static int plane_groups(const JacobiArgs& a, int nsm) {
  if (!a.vec4 || a.nz > nsm) return 0;
  const int64_t ng = (int64_t)(a.nx / 4) * a.ny, n = 4 * ng * a.nz;
  const int64_t g = (ng + JAC_PLANE_THREADS - 1) / JAC_PLANE_THREADS;
  static const int64_t least[JAC_PLANE_MAX_G + 1] = {0, 0, 300000, 550000, 1300000};
  return g <= JAC_PLANE_MAX_G && n >= least[g] ? (int)g : 0;
}

template <bool DIRICHLET, int G>
static qmt_status launch_plane(JacobiArgs& a, cudaStream_t s, bool* launched) {
  auto kern = jacobi_plane_kernel<DIRICHLET, G>;
  const size_t smem = 2ull * (a.nx / 4) * a.ny * sizeof(float4);
  QMT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  void* params[] = {&a};
  QMT_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3(a.nz), dim3(JAC_PLANE_THREADS), params, smem, s));
  note_launches(1);
  *launched = true;
  return QMT_OK;
}

template <bool DIRICHLET>
static qmt_status try_plane(JacobiArgs& a, int G, cudaStream_t s, bool* launched) {
  switch (G) {
    case 1: return launch_plane<DIRICHLET, 1>(a, s, launched);
    case 2: return launch_plane<DIRICHLET, 2>(a, s, launched);
    case 3: return launch_plane<DIRICHLET, 3>(a, s, launched);
    case 4: return launch_plane<DIRICHLET, 4>(a, s, launched);
    default: return QMT_OK;
  }
}

static int g_jacobi_path = 0;   // 0 automatic, 1 grid barrier per sweep, 2 single cluster

// Planes per CTA of the cluster kernel for this grid (1, 2 or 4), or 0 if it does not apply.
static int cluster_planes(int nx, int ny, int nz, const float* rho, const float* v) {
  if (nx % 4 || (nx / 4) * ny > JAC_CLUSTER_THREADS || nz < 2) return 0;
  if ((reinterpret_cast<uintptr_t>(rho) | reinterpret_cast<uintptr_t>(v)) % 16) return 0;
  const int need = (nz + JAC_CLUSTER - 1) / JAC_CLUSTER;
  int P = 1;
  while (P < need) P *= 2;
  if (P > 4) return 0;   // eight planes of values and sources do not fit in a thread's registers
  const size_t smem = 2ull * P * (size_t)nx * ny * sizeof(float);
  if (smem > 200u * 1024u) return 0;
  return P;
}

template <bool DIRICHLET, int P>
static qmt_status launch_cluster(JacobiArgs& a, cudaStream_t s, bool* launched) {
  *launched = false;
  auto kern = jacobi_cluster_kernel<DIRICHLET, P>;
  const size_t smem = 2ull * P * (size_t)a.nx * a.ny * sizeof(float);
  const int ncta = std::min(JAC_CLUSTER, (a.nz + P - 1) / P);
  QMT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  QMT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ncta);
  cfg.blockDim = dim3(JAC_CLUSTER_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ncta;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nclusters = 0;
  if (cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) != cudaSuccess || nclusters < 1) {
    cudaGetLastError();   // the persistent kernel takes the solve
    return QMT_OK;
  }
  QMT_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  note_launches(1);
  *launched = true;
  return QMT_OK;
}

template <bool DIRICHLET>
static qmt_status try_cluster(JacobiArgs& a, int P, cudaStream_t s, bool* launched) {
  switch (P) {
    case 1: return launch_cluster<DIRICHLET, 1>(a, s, launched);
    case 2: return launch_cluster<DIRICHLET, 2>(a, s, launched);
    case 4: return launch_cluster<DIRICHLET, 4>(a, s, launched);
    default: *launched = false; return QMT_OK;
  }
}

template <bool DIRICHLET>
static qmt_status run_jacobi(int nx, int ny, int nz, float step, const float* rho, float* v, float* t,
                             int max_sweeps, int check_every, double tol, int* sweeps_out,
                             double* delta_out, cudaStream_t s) {
  if (nx < 1 || ny < 1 || nz < 1 || !(step > 0.f) || !rho || !v || !t || max_sweeps < 0 || check_every < 1)
    return fail(QMT_BAD_ARG, "bad Jacobi arguments");
  const int nsm = sm_count();
  int per_sm = 0;
  auto kern = jacobi_persistent_kernel<DIRICHLET>;
  QMT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, JAC_THREADS, 0));
  if (per_sm < 1) return fail(QMT_CUDA_ERR, "Jacobi kernel does not fit on an SM");
  per_sm = std::min(per_sm, JAC_BLOCKS_PER_SM);
  const int64_t capacity = (int64_t)nsm * per_sm;

  JacobiArgs a{};
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.h = DIRICHLET ? 0.f : step;
  a.src_scale = DIRICHLET ? (float)(4.0 * 3.14159265358979323846 * (double)step * step) : 0.f;
  a.Q = rho;
  a.V = v;
  a.T = t;
  a.vec4 = (nx % 4 == 0) && ((reinterpret_cast<uintptr_t>(rho) | reinterpret_cast<uintptr_t>(v) |
                                reinterpret_cast<uintptr_t>(t)) % 16 == 0);
  a.max_sweeps = max_sweeps;
  a.check_every = check_every;
  a.tol = tol;
  a.wait_ns = wait_limit_ns();
  const int64_t items = a.vec4 ? (int64_t)(nx / 4) * ny * nz : (int64_t)nx * ny * nz;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((items + JAC_THREADS - 1) / JAC_THREADS, capacity));

  // scratch: CTA partial sums, barrier words, residuals, status words, publications (grows, never freed)
  static thread_local DevBuf scratch;
  const size_t part_bytes = ((size_t)std::max(grid, nsm) * sizeof(double) + 255) / 256 * 256;
  const size_t word_bytes = 256 + (size_t)nsm * sizeof(unsigned long long);
  qmt_status st = scratch.reserve(part_bytes + word_bytes);
  if (st) return st;
  uint8_t* base = scratch.as<uint8_t>();
  a.part = reinterpret_cast<double*>(base);
  a.res = reinterpret_cast<double*>(base + part_bytes);          // [0] check sum, [1] last residual
  a.bar = reinterpret_cast<unsigned long long*>(base + part_bytes + 64);
  a.pub = reinterpret_cast<unsigned long long*>(base + part_bytes + 256);
  a.out = reinterpret_cast<int*>(base + part_bytes + 128);        // [0] sweeps, [1] status, [2] flag
  QMT_CUDA(cudaMemsetAsync(base + part_bytes, 0, word_bytes, s));
  if (max_sweeps >= 2) {
    bool done = false;
    // automatic: the cluster kernel for grids of up to 32768 points (32^3: 1.4 us per sweep against 1.8 of
    // the plane and 2.1 of the grid-barrier kernel; 40^3, four planes a CTA: 2.7, 1.9, 2.2), else the
    // plane kernel where plane_groups has it, else the grid-barrier kernel
    const bool small = (int64_t)nx * ny * nz <= 32768;
    const bool want_cluster = g_jacobi_path == 2 || (g_jacobi_path == 0 && small);
    const int P = want_cluster ? cluster_planes(nx, ny, nz, rho, v) : 0;
    if (P > 0 && (st = try_cluster<DIRICHLET>(a, P, s, &done))) return st;
    const int G = !done && g_jacobi_path == 0 ? plane_groups(a, nsm) : 0;
    if (G && (st = try_plane<DIRICHLET>(a, G, s, &done))) return st;
    if (g_jacobi_path == 2 && !done)
      return fail(QMT_BAD_ARG, "the single-cluster Jacobi kernel does not apply to this grid or device");
    if (!done) {
      void* params[] = {&a};
      QMT_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(JX, JY), params, 0, s));
      note_launches(1);
    }
  }
  int out[3] = {0, 0, 0};
  double res[2] = {0.0, INFINITY};
  QMT_CUDA(cudaMemcpyAsync(out, a.out, sizeof(out), cudaMemcpyDeviceToHost, s));
  QMT_CUDA(cudaMemcpyAsync(res, a.res, sizeof(res), cudaMemcpyDeviceToHost, s));
  QMT_CUDA(cudaStreamSynchronize(s));
  const double delta = max_sweeps >= 2 ? res[1] : INFINITY;
  if (sweeps_out) *sweeps_out = out[0];
  if (delta_out) *delta_out = delta;
  if (out[1] == 3 || out[2]) return fail(QMT_CUDA_ERR, "Jacobi grid barrier timed out");
  if (out[1] == 2) return fail(QMT_NAN, "Jacobi residual is not finite");
  if (out[1] != 1 && tol > 0) return fail(QMT_NOT_CONVERGED, "Jacobi stopped at its sweep cap");
  return QMT_OK;
}

}  // namespace qmt

using namespace qmt;

extern "C" qmt_status qmt_jacobi(int nx, int ny, int nz, float step, const float* rho_dev, float* v_dev,
                                 float* t_dev, int max_sweeps, int check_every, double tol, int* sweeps_out,
                                 double* delta_out, void* stream) {
  return run_jacobi<false>(nx, ny, nz, step, rho_dev, v_dev, t_dev, max_sweeps, check_every, tol, sweeps_out,
                           delta_out, as_stream(stream));
}

extern "C" qmt_status qmt_jacobi_dirichlet(int nx, int ny, int nz, float step, const float* rho_dev, float* v_dev,
                                           float* t_dev, int max_sweeps, int check_every, double tol,
                                           int* sweeps_out, double* delta_out, void* stream) {
  return run_jacobi<true>(nx, ny, nz, step, rho_dev, v_dev, t_dev, max_sweeps, check_every, tol, sweeps_out,
                          delta_out, as_stream(stream));
}

extern "C" qmt_status qmt_set_jacobi_path(int mode) {
  if (mode < 0 || mode > 2)
    return fail(QMT_BAD_ARG, "Jacobi path must be 0 (automatic), 1 (grid barrier per sweep) or 2 (single cluster)");
  g_jacobi_path = mode;
  return QMT_OK;
}
