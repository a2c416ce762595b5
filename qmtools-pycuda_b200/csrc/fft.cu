// FFT Poisson solves with an in-house FFT.
//
// Reference semantics (QMTools.Compute_hartree_fft, qmtools/qmtools.py:2578-2639):
//   gpu_add_nuclear_charge (kernel_fft.cu:23-79) builds, in Angstrom units,
//       RHS = -( -q/h^3 + sum_A Z_A g_sigma(r - R_A) [r^2 <= (cutoff sigma)^2] ) / EPS0,
//   a periodic FFT, V_hat = -RHS_hat / (4 pi^2 |k|^2) with V_hat(0) = 0
//   (gpu_poisson_frequency_solve, kernel_fft.cu:82-107), an inverse FFT scaled by 1/N and the
//   real part returned in C order (i*NY*NZ + j*NZ + k) in volts.  The reference called cuFFT
//   through scikit-cuda, whose import is commented out (qmtools/qmtools.py:16).
// Free-space variant (new): the same charge density, convolved with the Hockney Green's
//   function 1/(4 pi EPS0 |r|) on a zero-padded grid of at least 2n per axis (sizes with
//   factors 2, 3, 5, 7), G(0) = voxel-cube average of 1/|r|; G_hat is real and even, so only
//   its octant [0, M/2]^3 is stored, cached per (M, h, device).
//
// 1D transforms are mixed-radix FFTs of batches of lines in shared memory, twiddles from a
// per-length table computed in FP64 on the host: in place with one butterfly of up to 10 points per
// thread where the length has no prime above 7, Stockham stages (self-sorting) for the others; 256- and
// 128-point lines (the padded axes of 128- and 64-voxel boxes) take register kernels instead (16 x 16
// and 16 x 8 four-step, one shared-memory exchange per transform).  A solve is five passes over an
// x-fastest complex work grid:
//   1. x forward, with the RHS assembled on the fly from q and the nuclei (only lines and
//      elements inside the physical box are non-zero: y < ny, z < nz, x < nx);
//   2. y forward on the z < nz planes (elements y >= ny are zero and not read);
//   3. z forward, multiply by G_hat (or the periodic k-space factor), z inverse, store z < nz;
//   4. y inverse on the z < nz planes, store y < ny;
//   5. x inverse, 1/M^3, real part written straight into the C-order output (x < nx).
// The right-hand side is real, so passes 2 to 4 run over the x frequencies up to Mx / 2 only and pass 5
// reads the others as their conjugates (256^3 padded: 190 -> 125 us a solve,
// 180 x 210 x 192: 278 -> 195 us).
// With the zero padding the solve moves about 1.3 full-grid passes instead of 6.
#include <algorithm>
#include <map>
#include <tuple>

#include <mutex>

#include "mol.cuh"

namespace qmt {

constexpr double EPS0 = 0.0055263494;       // e/(V*Ang), kernel_fft.cu:18
constexpr double R_BOHR = 0.529177211;      // kernel_fft.cu:17
constexpr double CUBE_INV_R = 2.3800772417; // h * <1/|r|> over a voxel cube
constexpr double PI = 3.14159265358979323846;
constexpr int FFT_MAXFAC = 16;
constexpr int FFT_MAXLEN = 2048;

// Plan of the in-place line kernel: radices, and per stage the distance of a butterfly's elements (L over the
// radices up to and including this one) with its exact multiply-high divisor (as in Plan1D below).
constexpr int LINE_MAXFAC = 5;
struct LinePlan {
  int nfac;               // 0: the length has a prime factor above 7
  int fac[LINE_MAXFAC], sub[LINE_MAXFAC];
  unsigned m_sub[LINE_MAXFAC];
};

struct Plan1D {
  int L;
  int nfac;
  int fac[FFT_MAXFAC];
  // per stage: Ns (product of the earlier radices) and exact multiply-high divisors
  // ceil(2^32 / d) for d = L / R and d = Ns (dividends stay below 2^16, divisors <= 2048;
  // d == 1 does not fit in 32 bits and is handled without the multiply)
  int ns[FFT_MAXFAC];
  unsigned m_nbf[FFT_MAXFAC], m_ns[FFT_MAXFAC];
  unsigned m_len;   // ceil(2^32 / L)
  LinePlan lp;
};

__device__ __forceinline__ unsigned fdiv(unsigned n, unsigned m) { return __umulhi(n, m); }

static bool factorize(int L, Plan1D& p) {
  p.L = L;
  p.nfac = 0;
  int n = L;
  for (int r : {4, 2, 3, 5, 7})
    while (n % r == 0) {
      if (p.nfac >= FFT_MAXFAC) return false;
      p.fac[p.nfac++] = r;
      n /= r;
    }
  for (int r = 11; n > 1; r += 2)
    while (n % r == 0) {
      if (p.nfac >= FFT_MAXFAC) return false;
      p.fac[p.nfac++] = r;
      n /= r;
    }
  return true;
}

static bool nice(int n) {
  for (int r : {2, 3, 5, 7})
    while (n % r == 0) n /= r;
  return n == 1;
}

static int nice_at_least(int n) {
  while (!nice(n)) ++n;
  return n;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// table entry m: exp(-2 pi i m / L); conjugated for the inverse direction
__device__ __forceinline__ float2 twid(const float2* tw, int m, bool inv) {
  const float2 t = tw[m];
  return inv ? make_float2(t.x, -t.y) : t;
}

// One radix-R butterfly of a Stockham stage (twiddle, DFT_R, scatter to sorted position).
template <int R>
__device__ __forceinline__ void radix_stage(const float2* __restrict__ s, float2* __restrict__ d, int j, int k,
                                            int idxD, int nbf, int Ns, const float2* tw, int L, bool inv) {
  const int step = L / (Ns * R);
  float2 v[R];
  v[0] = s[j];
#pragma unroll
  for (int q = 1; q < R; ++q) v[q] = cmul(s[j + q * nbf], twid(tw, k * q * step, inv));
  if constexpr (R == 2) {
    d[idxD] = cadd(v[0], v[1]);
    d[idxD + Ns] = csub(v[0], v[1]);
  } else if constexpr (R == 4) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    const float2 b0 = cadd(v[1], v[3]), b1 = csub(v[1], v[3]);
    // b1 times exp(-+ i pi/2): forward -i, inverse +i
    const float2 b1r = inv ? make_float2(-b1.y, b1.x) : make_float2(b1.y, -b1.x);
    d[idxD] = cadd(a0, b0);
    d[idxD + Ns] = cadd(a1, b1r);
    d[idxD + 2 * Ns] = csub(a0, b0);
    d[idxD + 3 * Ns] = csub(a1, b1r);
  } else {
    float2 w[R];
#pragma unroll
    for (int m = 0; m < R; ++m) w[m] = twid(tw, m * (L / R), inv);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      float2 acc = v[0];
#pragma unroll
      for (int p = 1; p < R; ++p) acc = cadd(acc, cmul(v[p], w[(p * q) % R]));
      d[idxD + q * Ns] = acc;
    }
  }
}

// Transforms nb lines of length plan.L held in `src` (ping-pong with `dst`); the pointer
// holding the result is returned in *result.
__device__ void fft_lines_smem(float2* src, float2* dst, const Plan1D& plan, int nb, const float2* tw, bool inv,
                               float2** result) {
  const int L = plan.L;
  for (int st = 0; st < plan.nfac; ++st) {
    const int R = plan.fac[st];
    const int nbf = L / R;
    const int Ns = plan.ns[st];
    const unsigned mnbf = plan.m_nbf[st], mns = plan.m_ns[st];
    for (int w = threadIdx.x; w < nb * nbf; w += blockDim.x) {
      const int b = nbf == 1 ? w : (int)fdiv((unsigned)w, mnbf), j = w - b * nbf;
      const float2* s = src + b * L;
      float2* d = dst + b * L;
      const int jq = Ns == 1 ? j : (int)fdiv((unsigned)j, mns);
      const int k = j - jq * Ns;
      const int idxD = jq * Ns * R + k;
      switch (R) {
        case 2: radix_stage<2>(s, d, j, k, idxD, nbf, Ns, tw, L, inv); break;
        case 3: radix_stage<3>(s, d, j, k, idxD, nbf, Ns, tw, L, inv); break;
        case 4: radix_stage<4>(s, d, j, k, idxD, nbf, Ns, tw, L, inv); break;
        case 5: radix_stage<5>(s, d, j, k, idxD, nbf, Ns, tw, L, inv); break;
        case 7: radix_stage<7>(s, d, j, k, idxD, nbf, Ns, tw, L, inv); break;
        default: {
          const int step = L / (Ns * R);
          for (int q = 0; q < R; ++q) {
            float2 acc = make_float2(0.f, 0.f);
            for (int p = 0; p < R; ++p) {
              float2 x = s[j + p * nbf];
              if (p) x = cmul(x, twid(tw, k * p * step, inv));
              acc = cadd(acc, cmul(x, twid(tw, ((p * q) % R) * (L / R), inv)));
            }
            d[idxD + q * Ns] = acc;
          }
        }
      }
    }
    __syncthreads();
    float2* t = src;
    src = dst;
    dst = t;
  }
  *result = src;
}

enum { PASS_PLAIN = 0, PASS_X_RHS = 1, PASS_Z_MUL = 2, PASS_X_OUT = 3 };

struct PassArgs {
  Plan1D plan;
  int64_t n1, s1, s2, se, nlines;   // line l: base (l % n1)*s1 + (l / n1)*s2, element e at + e*se
  int lload, lstore;                // elements >= lload are zero; only e < lstore are stored
  int B;                            // lines per CTA
  int inv;                          // direction of the (first) transform
  float scale;
  const float2* tw;
  float2* data;
  // RHS assembly (PASS_X_RHS): lines are (y, z) with n1 = ny
  MolView mol;
  const float* q;
  int nx, ny, nz;
  float h_ang, ox, oy, oz, norm, i2s2, cut2;
  int periodic;
  // multiply (PASS_Z_MUL): lines are (x, y) with n1 = Mx
  const float* gsym;
  int Mx, My, Mz;
  // C-order real output (PASS_X_OUT): lines are (z, y) with n1 = nz
  float* out;
};

// Periodic k-space factor (kernel_fft.cu:90-104): k in cycles/Ang, negative frequencies above N/2 - 1, k = 0 -> 0.
__device__ __forceinline__ float k_factor(const PassArgs& a, int x, int y, int z) {
  const float kx = (x > a.Mx / 2 - 1 ? (float)(x - a.Mx) : (float)x) / (a.Mx * a.h_ang);
  const float ky = (y > a.My / 2 - 1 ? (float)(y - a.My) : (float)y) / (a.My * a.h_ang);
  const float kz = (z > a.Mz / 2 - 1 ? (float)(z - a.Mz) : (float)z) / (a.Mz * a.h_ang);
  const double k2 = (double)(kx * kx + ky * ky + kz * kz);
  return (x == 0 && y == 0 && z == 0) ? 0.f : (float)(-1.0 / (4.0 * PI * PI * k2));
}

// On an odd axis that rule makes (N - 1) / 2 a negative frequency, so the factors of k and -k differ.  The
// real part of a transform over all frequencies averages them, which half of the spectrum has to do itself.
__device__ __forceinline__ float periodic_factor(const PassArgs& a, int x, int y, int z) {
  const float f = k_factor(a, x, y, z);
  if (((a.Mx | a.My | a.Mz) & 1) == 0) return f;
  return 0.5f * (f + k_factor(a, x ? a.Mx - x : 0, y ? a.My - y : 0, z ? a.Mz - z : 0));
}

// Element e of the line at `base`.  The last pass transforms spectra of real lines, of which the work grid
// holds the elements up to L / 2: the others are their conjugates.
template <int MODE>
__device__ __forceinline__ float2 load_elem(const PassArgs& a, int64_t base, int e) {
  if constexpr (MODE == PASS_X_OUT) {
    const int L = a.plan.L;
    const float2 v = a.data[base + (e > L / 2 ? L - e : e)];
    return e > L / 2 ? make_float2(v.x, -v.y) : v;
  } else {
    return a.data[base + (int64_t)e * a.se];
  }
}

template <int N>
struct Int { static constexpr int value = N; };
// ---- right-hand side of an x line (y, z) ----
__device__ __forceinline__ void load_atoms(const PassArgs& a, float* sat) {
  for (int i = threadIdx.x; i < a.mol.natoms; i += blockDim.x) {
    sat[4 * i] = a.mol.coords[3 * i] * (float)R_BOHR;
    sat[4 * i + 1] = a.mol.coords[3 * i + 1] * (float)R_BOHR;
    sat[4 * i + 2] = a.mol.coords[3 * i + 2] * (float)R_BOHR;
    sat[4 * i + 3] = (float)a.mol.types[i];
  }
}

__device__ __forceinline__ float electrons_at(const PassArgs& a, int x, int y, int z) {
  return a.q[x + (int64_t)y * a.nx + (int64_t)z * a.nx * a.ny] / (-a.h_ang * a.h_ang * a.h_ang);
}

// Adds the Gaussian nuclei to the charge densities rho(line, x) of nb staged lines (y, z).  A warp per line, a
// nucleus per lane for the (y, z) distance, then the lanes over the voxels within the cut-off in x; an element
// stays with one lane and the nuclei come in their order.  With every voxel's thread running over a list of its line's
// nuclei, and a thread per line making that list, the nuclei were half of this pass (20 of them, 168^3: 35 of 93 us).
template <class Rho>
__device__ __forceinline__ void add_nuclei(const PassArgs& a, const float* sat, int nb, const int* ly, const int* lz,
                                           Rho rho) {
  const int lane = threadIdx.x & 31;
  const float cut = sqrtf(a.cut2) * 1.0001f;
  for (int b = threadIdx.x >> 5; b < nb; b += blockDim.x >> 5) {
    const float py = a.oy + (ly[b] + 0.5f) * a.h_ang, pz = a.oz + (lz[b] + 0.5f) * a.h_ang;
    for (int at0 = 0; at0 < a.mol.natoms; at0 += 32) {
      const int mine = at0 + lane;
      bool near = false;
      if (mine < a.mol.natoms) {
        const float cy = py - sat[4 * mine + 1], cz = pz - sat[4 * mine + 2];
        near = cy * cy + cz * cz <= a.cut2 * 1.0001f;   // superset of the per-voxel test below
      }
      for (unsigned m = __ballot_sync(0xffffffffu, near); m; m &= m - 1) {
        const float* c = sat + 4 * (at0 + __ffs(m) - 1);
        const float cy = py - c[1], cz = pz - c[2], mid = (c[0] - a.ox) / a.h_ang - 0.5f, half = cut / a.h_ang + 1.f;
        const int lo = (int)fminf(fmaxf(floorf(mid - half), 0.f), (float)a.nx);
        const int hi = (int)fmaxf(fminf(ceilf(mid + half), (float)(a.nx - 1)), -1.f);
        for (int x = (lo & ~31) + lane; x <= hi; x += 32) {
          const float cx = a.ox + (x + 0.5f) * a.h_ang - c[0];
          const float r2 = cx * cx + cy * cy + cz * cz;
          if (x >= lo && r2 <= a.cut2) rho(b, x) += c[3] * a.norm * expf(-r2 * a.i2s2);
        }
      }
    }
  }
}

// Charge density to the right-hand side that is transformed.
__device__ __forceinline__ float rhs_of(const PassArgs& a, float rho) {
  return a.periodic ? (float)(-(double)rho / EPS0) : rho * a.h_ang * a.h_ang * a.h_ang;
}

template <int MODE>
__global__ void __launch_bounds__(256) fft_pass_kernel(const PassArgs a) {
  extern __shared__ float2 fsm[];
  const int L = a.plan.L;
  float2* tw = fsm;
  float2* b0 = fsm + L;
  float2* b1 = b0 + (size_t)a.B * L;
  float* sat = reinterpret_cast<float*>(b1 + (size_t)a.B * L);   // atoms (PASS_X_RHS)
  for (int i = threadIdx.x; i < L; i += blockDim.x) tw[i] = a.tw[i];
  if constexpr (MODE == PASS_X_RHS) {
    load_atoms(a, sat);
  }
  const int64_t l0 = (int64_t)blockIdx.x * a.B;
  const int64_t rem = a.nlines - l0;
  const int nb = rem < a.B ? (int)rem : a.B;
  const bool lines_adjacent = a.s1 == 1;
  // per-line data, computed once per CTA (B <= 16 lines)
  __shared__ int64_t lbase[16];          // element 0 of the line in the work grid / output
  __shared__ int lx[16], ly[16];         // the line's two grid coordinates (RHS, multiply, output)
  __syncthreads();   // twiddles and nuclei are in shared memory
  if (threadIdx.x < nb) {
    const int b = threadIdx.x;
    const int64_t l = l0 + b;
    const int c0 = (int)(l % a.n1), c1 = (int)(l / a.n1);
    lx[b] = c0;
    ly[b] = c1;
    lbase[b] = (int64_t)c0 * a.s1 + (int64_t)c1 * a.s2;
  }
  __syncthreads();
  // ---- load ----
  auto load_one = [&](int b, int e) {
    float2 v = make_float2(0.f, 0.f);
    if (e < a.lload) {
      if constexpr (MODE == PASS_X_RHS) {
        v.x = electrons_at(a, e, lx[b], ly[b]);
      } else {
        v = load_elem<MODE>(a, lbase[b], e);
      }
    }
    b0[b * L + e] = v;
  };
  if (lines_adjacent) {
    // 16 adjacent lines side by side: one 128-byte row of the grid per element index
    const int b = threadIdx.x & 15;
    for (int e = threadIdx.x >> 4; e < L; e += 16)
      if (b < nb) load_one(b, e);
  } else {
    for (int b = 0; b < nb; ++b)
      for (int e = threadIdx.x; e < L; e += blockDim.x) load_one(b, e);
  }
  __syncthreads();
  if constexpr (MODE == PASS_X_RHS) {
    add_nuclei(a, sat, nb, lx, ly, [&](int b, int x) -> float& { return b0[b * L + x].x; });
    __syncthreads();
    for (int i = threadIdx.x; i < nb * L; i += blockDim.x) b0[i].x = rhs_of(a, b0[i].x);
    __syncthreads();
  }
  float2* res;
  fft_lines_smem(b0, b1, a.plan, nb, tw, a.inv != 0, &res);
  if constexpr (MODE == PASS_Z_MUL) {
    const int hx = a.Mx / 2 + 1, hy = a.My / 2 + 1;
    for (int i = threadIdx.x; i < nb * L; i += blockDim.x) {
      const int b = (int)fdiv((unsigned)i, a.plan.m_len), kz = i - b * L;
      const int x = lx[b], y = ly[b];
      float f;
      if (a.periodic) {
        f = periodic_factor(a, x, y, kz);
      } else {
        const int gx = min(x, a.Mx - x), gy = min(y, a.My - y), gz = min(kz, a.Mz - kz);
        f = __ldg(a.gsym + gx + (int64_t)hx * (gy + (int64_t)hy * gz));
      }
      float2 v = res[b * L + kz];
      res[b * L + kz] = make_float2(v.x * f, v.y * f);
    }
    __syncthreads();
    float2* other = res == b0 ? b1 : b0;
    fft_lines_smem(res, other, a.plan, nb, tw, a.inv == 0, &res);
  }
  // ---- store ----
  auto store_one = [&](int b, int e) {
    const float2 v = res[b * L + e];
    if constexpr (MODE == PASS_X_OUT) {
      // line (z = lx, y = ly) along x into the C-order output
      a.out[(int64_t)e * a.ny * a.nz + (int64_t)ly[b] * a.nz + lx[b]] = v.x * a.scale;
    } else {
      a.data[lbase[b] + (int64_t)e * a.se] = make_float2(v.x * a.scale, v.y * a.scale);
    }
  };
  if (lines_adjacent || MODE == PASS_X_OUT) {
    const int b = threadIdx.x & 15;
    for (int e = threadIdx.x >> 4; e < a.lstore; e += 16)
      if (b < nb) store_one(b, e);
  } else {
    for (int b = 0; b < nb; ++b)
      for (int e = threadIdx.x; e < a.lstore; e += blockDim.x) store_one(b, e);
  }
}

// ---- lines in place, one butterfly per thread ------------------------------------------------
//
// Lengths whose primes are 2, 3, 5 and 7 (every padded axis).  B = 16 lines per CTA (4 above 704 points, so that
// an SM holds two blocks), stored element by element with the lines side by side, B + 1 float2 apart: a half-warp
// reads one element of 16 lines, so global rows are 128 bytes, shared memory has no bank conflicts, a twiddle is
// one broadcast and the butterfly index needs no division by B.  The radices go up to 10 (12 and 16 save some
// lengths a stage, but their registers cost a block per SM: 100^3 padded 115 -> 137 us), a length takes two or three
// stages, and the stages are decimation in frequency in place: one buffer and one barrier each.  The first stage
// reads its elements from the grid and the last writes to it at the digit-reversed frequency; the z pass multiplies
// by the kernel in the registers of the last stage, which are the inputs of the first stage back (the transposed
// algorithm, frequencies in the same digit-reversed places), so a three-stage line crosses shared memory four times
// there and back instead of fourteen.  Inverse transforms swap the two components on the way in and out.
// Bound by issue (57 % of the slots in the z pass) and by the latency of the first loads.  Padded solves, kernels
// alone, before and after: 88 x 104 x 96 182 -> 85 us, 168^3 1021 -> 334 us, 48^3 64 -> 44 us.
template <int N>
struct Roots {   // cos and sin of 2 pi k / N
  float c[N], s[N];
  __host__ __device__ constexpr Roots() : c{}, s{} {
    for (int k = 0; k < N; ++k) {
      // series at an angle folded to [-pi, pi]
      const double x = 2 * PI * (2 * k > N ? k - N : k) / N;
      double t = 1, cs = 0, sn = 0;
      for (int i = 0; i < 40; i += 2) {
        cs += t;
        sn += t * x / (i + 1);
        t *= -x * x / ((i + 1) * (i + 2));
      }
      c[k] = (float)cs;
      s[k] = (float)sn;
    }
  }
};

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]);

// R = N1 N2 points as N2 transforms of N1 points and N1 of N2.
template <int N1, int N2>
__device__ __forceinline__ void dft_split(float2 (&v)[N1 * N2]) {
  constexpr int R = N1 * N2;
  constexpr Roots<R> w;
  float2 u[N2][N1];
#pragma unroll
  for (int b = 0; b < N2; ++b) {
#pragma unroll
    for (int i = 0; i < N1; ++i) u[b][i] = v[N2 * i + b];
    dft<N1>(u[b]);
#pragma unroll
    for (int k = 1; k < N1; ++k) {
      if (b * k == 0) continue;
      if (4 * b * k == R) u[b][k] = make_float2(u[b][k].y, -u[b][k].x);
      else u[b][k] = cmul(u[b][k], make_float2(w.c[b * k % R], -w.s[b * k % R]));
    }
  }
#pragma unroll
  for (int k = 0; k < N1; ++k) {
    float2 z[N2];
#pragma unroll
    for (int b = 0; b < N2; ++b) z[b] = u[b][k];
    dft<N2>(z);
#pragma unroll
    for (int b = 0; b < N2; ++b) v[k + N1 * b] = z[b];
  }
}

// Forward R-point DFT in registers, natural order.
template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
  if constexpr (R == 2) {
    const float2 t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
  } else if constexpr (R == 4) {
    const float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = make_float2(t1.x + t3.y, t1.y - t3.x);
    v[3] = make_float2(t1.x - t3.y, t1.y + t3.x);
  } else if constexpr (R == 3 || R == 5 || R == 7) {
    // elements k and R - k share their cosines and their sines up to the sign
    constexpr Roots<R> w;
    constexpr int H = (R - 1) / 2;
    float2 t[H], d[H], x0 = v[0];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      t[k] = cadd(v[k + 1], v[R - 1 - k]);
      d[k] = csub(v[k + 1], v[R - 1 - k]);
      v[0] = cadd(v[0], t[k]);
    }
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      float2 e = x0, o = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < H; ++k) {
        const float c = w.c[(k + 1) * q % R], sn = w.s[(k + 1) * q % R];
        e = make_float2(e.x + c * t[k].x, e.y + c * t[k].y);
        o = make_float2(o.x + sn * d[k].x, o.y + sn * d[k].y);
      }
      v[q] = make_float2(e.x + o.y, e.y - o.x);
      v[R - q] = make_float2(e.x - o.y, e.y + o.x);
    }
  } else if constexpr (R == 6) dft_split<3, 2>(v);
  else if constexpr (R == 8) dft_split<4, 2>(v);
  else if constexpr (R == 9) dft_split<3, 3>(v);
  else if constexpr (R == 10) dft_split<5, 2>(v);
}

__device__ __forceinline__ float2 swapped(float2 v) { return make_float2(v.y, v.x); }

template <int MODE, int B>
__global__ void __launch_bounds__(256, 4) fft_line_kernel(const PassArgs a) {
  extern __shared__ float2 fsm[];
  constexpr int P = B + 1, lb = B == 16 ? 4 : 2;
  const int L = a.plan.L, T = blockDim.x, nf = a.plan.lp.nfac;
  const int Rl = a.plan.lp.fac[nf - 1], Nl = L / Rl;
  float2* const tw = fsm;
  float2* const buf = fsm + L;
  unsigned short* const rev = reinterpret_cast<unsigned short*>(buf + (size_t)L * P);   // frequency of block p
  unsigned short* const place = rev + L;   // where frequency e stands in the buffer
  float* const sat = reinterpret_cast<float*>(place + L);   // atoms (PASS_X_RHS); 2 L shorts before it
  for (int i = threadIdx.x; i < L; i += T) tw[i] = a.tw[i];
  if constexpr (MODE == PASS_X_RHS) load_atoms(a, sat);
  for (int p = threadIdx.x; p < Nl; p += T) {
    int k = 0, w = 1, pos = p * Rl;
    for (int i = 0; i < nf - 1; ++i) {
      const int d = (int)fdiv((unsigned)pos, a.plan.lp.m_sub[i]);
      pos -= d * a.plan.lp.sub[i];
      k += d * w;
      w *= a.plan.lp.fac[i];
    }
    rev[p] = (unsigned short)k;
    if constexpr (MODE == PASS_PLAIN || MODE == PASS_X_RHS)
      for (int m = 0; m < Rl; ++m) place[k + m * Nl] = (unsigned short)(p * Rl + m);
  }
  const unsigned l0 = blockIdx.x * B, rem = (unsigned)a.nlines - l0;   // at most 2048^2 lines
  const int nb = rem < B ? (int)rem : B;
  __shared__ int64_t lbase[B];          // element 0 of the line in the work grid
  __shared__ int lx[B], ly[B];          // the line's two grid coordinates
  if (threadIdx.x < nb) {
    const int i = threadIdx.x;
    const unsigned l = l0 + i, c1 = l / (unsigned)a.n1, c0 = l - c1 * (unsigned)a.n1;
    lx[i] = (int)c0;
    ly[i] = (int)c1;
    lbase[i] = (int64_t)c0 * a.s1 + (int64_t)c1 * a.s2;
  }
  __syncthreads();
  const bool inv = a.inv != 0;
  const bool adjacent = a.s1 == 1;
  const int b = threadIdx.x & (B - 1);   // the blocks are multiples of 32 threads
  const bool live = b < nb;
  float2* const line = MODE == PASS_X_RHS ? nullptr : a.data + (live ? lbase[b] : 0);

  // a stage of radix R: Load(element) and Store(element, butterfly, digit, value)
  auto stage = [&](auto rc, int i, bool down, auto load, auto store) {
    constexpr int R = decltype(rc)::value;
    const int sub = a.plan.lp.sub[i], ts = L / (sub * R), items = (L / R) << lb;
    const unsigned msub = a.plan.lp.m_sub[i];
    for (int w = threadIdx.x; w < items; w += T) {
      const int it = w >> lb, p = sub == 1 ? it : (int)fdiv((unsigned)it, msub), j = it - p * sub;
      const int base = p * sub * R + j;
      float2 v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = load(base + q * sub);
      if (!down && sub > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmul(v[q], tw[j * q * ts]);
      }
      dft<R>(v);
      if (down && sub > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmul(v[q], tw[j * q * ts]);
      }
#pragma unroll
      for (int q = 0; q < R; ++q) store(base + q * sub, it, q, v[q]);
    }
  };
  auto with_radix = [&](int i, auto f) {
    switch (a.plan.lp.fac[i]) {
      case 2: f(Int<2>()); break;
      case 3: f(Int<3>()); break;
      case 4: f(Int<4>()); break;
      case 5: f(Int<5>()); break;
      case 6: f(Int<6>()); break;
      case 7: f(Int<7>()); break;
      case 8: f(Int<8>()); break;
      case 9: f(Int<9>()); break;
      default: f(Int<10>()); break;
    }
    __syncthreads();
  };
  auto from_buf = [&](int e) { return buf[e * P + b]; };
  auto to_buf = [&](int e, int, int, float2 v) { buf[e * P + b] = v; };

  // ---- first stage, or the lines into the buffer where they are not side by side in the grid ----
  int i0 = 0;   // first stage still to do
  if (MODE == PASS_X_RHS || !adjacent) {
    auto put = [&](int bb, int e, float2 v) { buf[e * P + bb] = inv ? swapped(v) : v; };
    const float2 zero = make_float2(0.f, 0.f);
    constexpr int AHEAD = B < 8 ? B : 8;   // reads in flight per thread
    for (int e = threadIdx.x; e < L; e += T)
      for (int b0 = 0; b0 < B; b0 += AHEAD) {
        float2 v[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          v[u] = zero;
          if (b0 + u < nb && e < a.lload) {
            if constexpr (MODE == PASS_X_RHS) v[u].x = electrons_at(a, e, lx[b0 + u], ly[b0 + u]);
            else v[u] = load_elem<MODE>(a, lbase[b0 + u], e);
          }
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) put(b0 + u, e, v[u]);
      }
    __syncthreads();
    if constexpr (MODE == PASS_X_RHS) {
      add_nuclei(a, sat, nb, lx, ly, [&](int bb, int x) -> float& { return buf[x * P + bb].x; });
      __syncthreads();
      auto from_rho = [&](int e) { return make_float2(rhs_of(a, buf[e * P + b].x), 0.f); };
      with_radix(0, [&](auto rc) { stage(rc, 0, true, from_rho, to_buf); });
      i0 = 1;
    }
  } else if constexpr (MODE == PASS_PLAIN || MODE == PASS_Z_MUL) {
    auto from_grid = [&](int e) {
      float2 v = make_float2(0.f, 0.f);
      if (live && e < a.lload) v = line[(int64_t)e * a.se];
      return inv ? swapped(v) : v;
    };
    with_radix(0, [&](auto rc) { stage(rc, 0, true, from_grid, to_buf); });
    i0 = 1;
  }
  const bool staged_out = MODE == PASS_X_RHS || (MODE == PASS_PLAIN && !adjacent);
  for (int i = i0; i < nf - (staged_out ? 0 : 1); ++i)
    with_radix(i, [&](auto rc) { stage(rc, i, true, from_buf, to_buf); });

  auto to_grid = [&](int e, float2 v) {
    if (inv) v = swapped(v);
    if (live && e < a.lstore) line[(int64_t)e * a.se] = make_float2(v.x * a.scale, v.y * a.scale);
  };
  if constexpr (MODE == PASS_X_RHS || MODE == PASS_PLAIN) {
    if (staged_out) {
      for (int bb = 0; bb < nb; ++bb)
        for (int e = threadIdx.x; e < a.lstore; e += T) {
          float2 v = buf[place[e] * P + bb];
          if (inv) v = swapped(v);
          a.data[lbase[bb] + (int64_t)e * a.se] = make_float2(v.x * a.scale, v.y * a.scale);
        }
      return;
    }
  }
  if constexpr (MODE == PASS_PLAIN) {
    with_radix(nf - 1, [&](auto rc) {
      stage(rc, nf - 1, true, from_buf, [&](int, int it, int q, float2 v) { to_grid(rev[it] + q * Nl, v); });
    });
  } else if constexpr (MODE == PASS_X_OUT) {
    // line (z = lx, y = ly) along x into the C-order output: adjacent lines are adjacent in z
    const int64_t row = (int64_t)a.ny * a.nz;
    float* const out = a.out + (live ? (int64_t)ly[b] * a.nz + lx[b] : 0);
    with_radix(nf - 1, [&](auto rc) {
      stage(rc, nf - 1, true, from_buf, [&](int, int it, int q, float2 v) {
        const int e = rev[it] + q * Nl;
        if (live && e < a.lstore) out[e * row] = (inv ? v.y : v.x) * a.scale;
      });
    });
  } else if constexpr (MODE == PASS_Z_MUL) {
    const int hx = a.Mx / 2 + 1, hy = a.My / 2 + 1;
    const int x = live ? lx[b] : 0, y = live ? ly[b] : 0;
    const float* const g =
        a.periodic ? nullptr : a.gsym + min(x, a.Mx - x) + (int64_t)hx * min(y, a.My - y);
    const int64_t gz = (int64_t)hx * hy;
    with_radix(nf - 1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int w = threadIdx.x; w < Nl << lb; w += T) {
        const int it = w >> lb, k0 = rev[it];
        float2 v[R];
        float f[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int kz = k0 + q * Nl;
          f[q] = a.periodic ? periodic_factor(a, x, y, kz) : __ldg(g + gz * min(kz, L - kz));
        }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = from_buf(it * R + q);
        dft<R>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = make_float2(v[q].y * f[q], v[q].x * f[q]);   // swapped for the way back
        dft<R>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) to_buf(it * R + q, 0, 0, v[q]);
      }
    });
    for (int i = nf - 2; i > 0; --i)
      with_radix(i, [&](auto rc) { stage(rc, i, false, from_buf, to_buf); });
    auto back = [&](int e, float2 v) { to_grid(e, swapped(v)); };
    with_radix(0, [&](auto rc) {
      stage(rc, 0, false, from_buf, [&](int e, int, int, float2 v) { back(e, v); });
    });
  }
}

// ---- 256- and 128-point lines in registers -----------------------------------------------
// Four-step transforms with every thread holding 16 elements e = t + TPL m (m = 0..15) of its
// line, TPL = L / 16 threads per line, 256 / TPL lines per CTA: the 16-point DFT over m, the
// twiddle W_L^(t k1), one exchange through shared memory, then the DFTs over t.  L = 256: thread
// t forms the 16-point DFT of k1 = t (16 values); L = 128: the two 8-point DFTs of k1 = t and
// t + 8.  Either way the thread then holds X[t + TPL m'] in register m', the same element pattern
// as its input, so global loads and stores are issued 16 per thread back to back.
struct Tw16 {
  float2 w1, w2, w3, w6, w9;   // W16^p = table entry (L/16) p (conjugated for the inverse)
};

template <int L>
__device__ __forceinline__ Tw16 tw16(const float2* tw, bool inv) {
  constexpr int st = L / 16;
  return Tw16{twid(tw, st, inv), twid(tw, 2 * st, inv), twid(tw, 3 * st, inv), twid(tw, 6 * st, inv),
              twid(tw, 9 * st, inv)};
}

// In-place 4-point DFT (forward: W4 = -i; inverse: +i).
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3, bool inv) {
  const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = csub(a1, a3);
  const float2 t3r = inv ? make_float2(-t3.y, t3.x) : make_float2(t3.y, -t3.x);
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = cadd(t1, t3r);
  a3 = csub(t1, t3r);
}

// 16-point DFT of x[0..15] (4 x 4), result in natural order.
__device__ __forceinline__ void dft16(float2 (&x)[16], const Tw16& w, bool inv) {
#pragma unroll
  for (int m2 = 0; m2 < 4; ++m2) dft4(x[m2], x[4 + m2], x[8 + m2], x[12 + m2], inv);
  // x[m2 + 4 k1] holds the m2-th partial DFT at k1: twiddle W16^(m2 k1)
  x[5] = cmul(x[5], w.w1);
  x[9] = cmul(x[9], w.w2);
  x[13] = cmul(x[13], w.w3);
  x[6] = cmul(x[6], w.w2);
  x[10] = inv ? make_float2(-x[10].y, x[10].x) : make_float2(x[10].y, -x[10].x);   // W16^4 = -+i
  x[14] = cmul(x[14], w.w6);
  x[7] = cmul(x[7], w.w3);
  x[11] = cmul(x[11], w.w6);
  x[15] = cmul(x[15], w.w9);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) dft4(x[4 * k1], x[4 * k1 + 1], x[4 * k1 + 2], x[4 * k1 + 3], inv);
  // x[4 k1 + k2] holds X[k1 + 4 k2]
  float2 y[16];
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) y[k1 + 4 * k2] = x[4 * k1 + k2];
#pragma unroll
  for (int k = 0; k < 16; ++k) x[k] = y[k];
}

// 8-point DFT of y[0..7] (even/odd 4-point DFTs), result in natural order; w1, w3 = W8^1, W8^3.
__device__ __forceinline__ void dft8(float2 (&y)[8], float2 w1, float2 w3, bool inv) {
  float2 a0 = y[0], a1 = y[2], a2 = y[4], a3 = y[6];
  float2 b0 = y[1], b1 = y[3], b2 = y[5], b3 = y[7];
  dft4(a0, a1, a2, a3, inv);
  dft4(b0, b1, b2, b3, inv);
  b1 = cmul(b1, w1);
  b2 = inv ? make_float2(-b2.y, b2.x) : make_float2(b2.y, -b2.x);   // W8^2 = -+i
  b3 = cmul(b3, w3);
  y[0] = cadd(a0, b0);
  y[1] = cadd(a1, b1);
  y[2] = cadd(a2, b2);
  y[3] = cadd(a3, b3);
  y[4] = csub(a0, b0);
  y[5] = csub(a1, b1);
  y[6] = csub(a2, b2);
  y[7] = csub(a3, b3);
}

// Exchange-buffer geometry per length: element (k1, t) of line b at b S + k1 R + t.  R and S are
// chosen so that neither thread mapping (lines or elements fastest) has bank conflicts.
template <int L> struct RegFft;
template <> struct RegFft<256> {
  static constexpr int TPL = 16, LINES = 16, R = 17, S_MAX = 273;
  static __device__ __forceinline__ int S(bool) { return 273; }
};
template <> struct RegFft<128> {
  static constexpr int TPL = 8, LINES = 32, R = 9, S_MAX = 152;
  static __device__ __forceinline__ int S(bool bfast) { return bfast ? 143 : 152; }
};

// One transform of the thread's line b (thread t of it); `buf` is the CTA's exchange buffer,
// free on entry (the barrier below orders it after earlier readers).
template <int L>
__device__ __forceinline__ void fft_regs(float2 (&x)[16], const float2* tw, float2* buf, int b, int t, int S,
                                         bool inv) {
  constexpr int R = RegFft<L>::R;
  const Tw16 w = tw16<L>(tw, inv);
  dft16(x, w, inv);
#pragma unroll
  for (int k1 = 1; k1 < 16; ++k1) x[k1] = cmul(x[k1], twid(tw, (t * k1) & (L - 1), inv));
  __syncthreads();
#pragma unroll
  for (int k1 = 0; k1 < 16; ++k1) buf[b * S + k1 * R + t] = x[k1];
  __syncthreads();
  if constexpr (L == 256) {
#pragma unroll
    for (int u = 0; u < 16; ++u) x[u] = buf[b * S + t * R + u];
    dft16(x, w, inv);
  } else {
    const float2 w1 = twid(tw, L / 8, inv), w3 = twid(tw, 3 * L / 8, inv);
    float2 ya[8], yb[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      ya[u] = buf[b * S + t * R + u];
      yb[u] = buf[b * S + (t + 8) * R + u];
    }
    dft8(ya, w1, w3, inv);
    dft8(yb, w1, w3, inv);
#pragma unroll
    for (int k2 = 0; k2 < 8; ++k2) {
      x[2 * k2] = ya[k2];       // X[t + 16 k2]     = element t + 8 (2 k2)
      x[2 * k2 + 1] = yb[k2];   // X[t + 8 + 16 k2] = element t + 8 (2 k2 + 1)
    }
  }
}

template <int MODE, int L>
__global__ void __launch_bounds__(256) fft_reg_pass_kernel(const PassArgs a) {
  constexpr int TPL = RegFft<L>::TPL, LINES = RegFft<L>::LINES;
  extern __shared__ float2 fsm[];
  float2* tw = fsm;
  float2* buf = fsm + L;
  float* sat = reinterpret_cast<float*>(buf + LINES * RegFft<L>::S_MAX);   // atoms (PASS_X_RHS)
  for (int i = threadIdx.x; i < L; i += blockDim.x) tw[i] = a.tw[i];
  if constexpr (MODE == PASS_X_RHS) {
    load_atoms(a, sat);
  }
  const int64_t l0 = (int64_t)blockIdx.x * LINES;
  const int64_t rem = a.nlines - l0;
  const int nb = rem < LINES ? (int)rem : LINES;
  __shared__ int64_t lbase[LINES];
  __shared__ int lx[LINES], ly[LINES];
  __syncthreads();
  if (threadIdx.x < nb) {
    const int bb = threadIdx.x;
    const int64_t l = l0 + bb;
    const int c0 = (int)(l % a.n1), c1 = (int)(l / a.n1);
    lx[bb] = c0;
    ly[bb] = c1;
    lbase[bb] = (int64_t)c0 * a.s1 + (int64_t)c1 * a.s2;
  }
  __syncthreads();
  // lines adjacent in memory: a half-warp spans 16 lines at one element; lines contiguous: it
  // spans consecutive elements of one (L = 256) or two (L = 128) lines
  const bool bfast = a.s1 == 1;
  const int b = bfast ? (int)(threadIdx.x % LINES) : (int)(threadIdx.x / TPL);
  const int t = bfast ? (int)(threadIdx.x / LINES) : (int)(threadIdx.x % TPL);
  const int S = RegFft<L>::S(bfast);
  const bool live = b < nb;
  float2 x[16];
  if constexpr (MODE == PASS_X_RHS) {
    float* const rho = reinterpret_cast<float*>(buf);   // line b, voxel e at b (L + 1) + e
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int e = t + TPL * m;
      rho[b * (L + 1) + e] = live && e < a.lload ? electrons_at(a, e, lx[b], ly[b]) : 0.f;
    }
    __syncthreads();
    add_nuclei(a, sat, nb, lx, ly, [&](int bb, int e) -> float& { return rho[bb * (L + 1) + e]; });
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = make_float2(rhs_of(a, rho[b * (L + 1) + t + TPL * m]), 0.f);
  } else {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int e = t + TPL * m;
      x[m] = live && e < a.lload ? load_elem<MODE>(a, lbase[b], e) : make_float2(0.f, 0.f);
    }
  }
  fft_regs<L>(x, tw, buf, b, t, S, a.inv != 0);
  if constexpr (MODE == PASS_Z_MUL) {
    const int hx = a.Mx / 2 + 1, hy = a.My / 2 + 1;
    const int xg = lx[b], yg = ly[b];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int kz = t + TPL * m;
      float f;
      if (a.periodic) {
        f = periodic_factor(a, xg, yg, kz);
      } else {
        const int gx = min(xg, a.Mx - xg), gy = min(yg, a.My - yg), gz = min(kz, a.Mz - kz);
        f = live ? __ldg(a.gsym + gx + (int64_t)hx * (gy + (int64_t)hy * gz)) : 0.f;
      }
      x[m] = make_float2(x[m].x * f, x[m].y * f);
    }
    fft_regs<L>(x, tw, buf, b, t, S, a.inv == 0);
  }
  if constexpr (MODE == PASS_X_OUT) {
    // line (z = lx, y = ly) along x into the C-order output: regroup through shared memory so
    // that a warp writes consecutive z of one x
    constexpr int S2 = L + 1;
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; ++m) buf[b * S2 + t + TPL * m] = x[m];
    __syncthreads();
    const int bo = (int)(threadIdx.x % LINES);
    if (bo < nb)
      for (int e = (int)(threadIdx.x / LINES); e < a.lstore; e += TPL)
        a.out[(int64_t)e * a.ny * a.nz + (int64_t)ly[bo] * a.nz + lx[bo]] = buf[bo * S2 + e].x * a.scale;
  } else {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int e = t + TPL * m;
      if (live && e < a.lstore)
        a.data[lbase[b] + (int64_t)e * a.se] = make_float2(x[m].x * a.scale, x[m].y * a.scale);
    }
  }
}

// ---- Green's function ----------------------------------------------------------------
__global__ void green_kernel(float2* __restrict__ g, int Mx, int My, int Mz, float h_ang) {
  const int64_t n = (int64_t)Mx * My * Mz;
  const double pref = 1.0 / (4.0 * PI * EPS0);
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx % Mx, j = (idx / Mx) % My, k = idx / ((int64_t)Mx * My);
    const double x = (double)min(i, Mx - i) * h_ang, y = (double)min(j, My - j) * h_ang,
                 z = (double)min(k, Mz - k) * h_ang;
    const double r = sqrt(x * x + y * y + z * z);
    const double v = r > 0 ? pref / r : pref * CUBE_INV_R / h_ang;
    g[idx] = make_float2((float)v, 0.f);
  }
}

__global__ void green_octant_kernel(const float2* __restrict__ g, int Mx, int My, int Mz, float* __restrict__ out) {
  const int ox = Mx / 2 + 1, oy = My / 2 + 1, oz = Mz / 2 + 1;
  const int64_t n = (int64_t)ox * oy * oz;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx % ox, j = (idx / ox) % oy, k = idx / ((int64_t)ox * oy);
    out[idx] = g[i + j * Mx + k * (int64_t)Mx * My].x;
  }
}

// ---- host ------------------------------------------------------------------------------------
static unsigned grid_blocks(int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)sm_count() * 16); }

struct GreenEntry {
  DevBuf* buf;
  uint64_t used;        // last use, for least-recently-used eviction
  size_t bytes;
  cudaEvent_t ready;    // recorded after the build, on the stream that built it
  bool built;           // `ready` seen complete: later solves need no wait (and, inside a CUDA-graph
                        // capture, make no event call)
};

// Device-side caches shared by all calls: twiddle tables per (length, device), transformed
// Green's functions per (padded shape, step, device) up to GREEN_CACHE_BYTES of octants, and one
// growing scratch grid per device for building them.  `tw_mu` guards the twiddles and `green_mu`
// the rest; building a Green's function takes green_mu and then (through its FFT passes) tw_mu,
// never the other way round.  No host synchronisation in steady state: a solve on another
// stream waits for a cached octant's `ready` event on the device, and a build waits for the
// previous build's use of the scratch grid (`tmp_done`) the same way.  (Growing the scratch and
// evicting an entry past GREEN_CACHE_BYTES free device memory with cudaFree, which does
// synchronise the device: a workload of many new shapes pays that per new shape.)
constexpr size_t GREEN_CACHE_BYTES = (size_t)4 << 30;
struct DevCache {
  std::mutex tw_mu, green_mu;
  std::map<std::tuple<int, int>, DevBuf*> tw;                         // (L, device)
  std::map<std::tuple<int, int, int, float, int>, GreenEntry> green;  // (Mx, My, Mz, h, device)
  std::map<int, DevBuf*> green_tmp;                                   // device -> scratch
  std::map<int, cudaEvent_t> tmp_done;                                // device -> last build's end
  size_t green_bytes = 0;
  uint64_t clock = 0;
};
static DevCache& cache() {
  static DevCache c;
  return c;
}

static qmt_status twiddles(int L, const float2** out) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(cache().tw_mu);
  DevBuf*& b = cache().tw[std::make_tuple(L, dev)];
  if (!b) {
    std::vector<float2> h(L);
    for (int m = 0; m < L; ++m) {
      const double a = -2.0 * PI * (double)m / (double)L;
      h[m] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    b = new DevBuf();
    qmt_status st = b->reserve(L * sizeof(float2));
    if (st) {
      delete b;
      b = nullptr;
      return st;
    }
    // synchronous: the table is shared by every stream (built once per length and device)
    QMT_CUDA(cudaMemcpy(b->ptr, h.data(), L * sizeof(float2), cudaMemcpyHostToDevice));
  }
  *out = b->as<float2>();
  return QMT_OK;
}

template <int MODE>
static qmt_status launch_mode(const PassArgs& a, unsigned blocks, size_t smem, cudaStream_t s) {
  QMT_CUDA(cudaFuncSetAttribute(fft_pass_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  fft_pass_kernel<MODE><<<blocks, 256, smem, s>>>(a);
  QMT_CHECK_LAUNCH("fft_pass_kernel");
  return QMT_OK;
}

template <int MODE, int L>
static qmt_status launch_mode_reg(const PassArgs& a, unsigned blocks, size_t smem, cudaStream_t s) {
  QMT_CUDA(cudaFuncSetAttribute(fft_reg_pass_kernel<MODE, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  fft_reg_pass_kernel<MODE, L><<<blocks, 256, smem, s>>>(a);
  QMT_CHECK_LAUNCH("fft_reg_pass_kernel");
  return QMT_OK;
}

template <int L>
static qmt_status launch_pass_reg(int mode, PassArgs a, cudaStream_t s) {
  constexpr int LINES = RegFft<L>::LINES;
  a.B = LINES;
  size_t smem = ((size_t)L + (size_t)LINES * RegFft<L>::S_MAX) * sizeof(float2);
  if (mode == PASS_X_RHS) smem += 16 * (size_t)a.mol.natoms;
  const unsigned blocks = (unsigned)((a.nlines + LINES - 1) / LINES);
  if (blocks == 0) return QMT_OK;
  switch (mode) {
    case PASS_PLAIN: return launch_mode_reg<PASS_PLAIN, L>(a, blocks, smem, s);
    case PASS_X_RHS: return launch_mode_reg<PASS_X_RHS, L>(a, blocks, smem, s);
    case PASS_Z_MUL: return launch_mode_reg<PASS_Z_MUL, L>(a, blocks, smem, s);
    default: return launch_mode_reg<PASS_X_OUT, L>(a, blocks, smem, s);
  }
}

template <int MODE, int B>
static qmt_status launch_mode_lines(const PassArgs& a, unsigned blocks, int threads, size_t smem, cudaStream_t s) {
  QMT_CUDA(cudaFuncSetAttribute(fft_line_kernel<MODE, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  fft_line_kernel<MODE, B><<<blocks, threads, smem, s>>>(a);
  QMT_CHECK_LAUNCH("fft_line_kernel");
  return QMT_OK;
}

template <int B>
static qmt_status launch_pass_lines(int mode, const PassArgs& a, cudaStream_t s) {
  const int L = a.plan.L;
  size_t smem = (size_t)L * ((2 + B) * sizeof(float2) + 2 * sizeof(unsigned short));
  if (mode == PASS_X_RHS) smem += 16 * (size_t)a.mol.natoms;
  const unsigned blocks = (unsigned)((a.nlines + B - 1) / B);
  if (blocks == 0) return QMT_OK;
  // the block size that leaves the fewest threads idle in the last round of each stage; four blocks of at least
  // 192 (with 128 and fewer idle threads a 336-point solve took 393 us, with these 334)
  int threads = 256, best = 1 << 30;
  for (int t = 256; t >= 192; t -= 32) {
    int cost = 0;
    for (int i = 0; i < a.plan.lp.nfac; ++i) {
      const int items = L / a.plan.lp.fac[i] * B;
      cost += (items + t - 1) / t * t * a.plan.lp.fac[i];
    }
    if (cost < best) {
      best = cost;
      threads = t;
    }
  }
  switch (mode) {
    case PASS_PLAIN: return launch_mode_lines<PASS_PLAIN, B>(a, blocks, threads, smem, s);
    case PASS_X_RHS: return launch_mode_lines<PASS_X_RHS, B>(a, blocks, threads, smem, s);
    case PASS_Z_MUL: return launch_mode_lines<PASS_Z_MUL, B>(a, blocks, threads, smem, s);
    default: return launch_mode_lines<PASS_X_OUT, B>(a, blocks, threads, smem, s);
  }
}

static qmt_status launch_pass(int mode, PassArgs a, cudaStream_t s) {
  a.B = std::max(1, std::min(16, 12288 / a.plan.L));
  const float2* tw;
  qmt_status st = twiddles(a.plan.L, &tw);
  if (st) return st;
  a.tw = tw;
  // Register kernels for their two lengths (128^3 padded 125 us; the in-place kernel takes 190).  The in-place
  // kernel where there are two stages to take (88 x 104 x 96 padded: 181 us by the kernel below, 85 by it); a single
  // radix, up to 10 points, gains nothing there (3 x 2 x 2: 19 us below, 26), and other primes need it.
  if (a.plan.L == 256) return launch_pass_reg<256>(mode, a, s);
  if (a.plan.L == 128) return launch_pass_reg<128>(mode, a, s);
  if (a.plan.lp.nfac > 1)
    return a.plan.L <= 704 ? launch_pass_lines<16>(mode, a, s) : launch_pass_lines<4>(mode, a, s);
  size_t smem = ((size_t)a.plan.L * (1 + 2 * a.B)) * sizeof(float2);
  if (mode == PASS_X_RHS) smem += 16 * (size_t)a.mol.natoms;
  const unsigned blocks = (unsigned)((a.nlines + a.B - 1) / a.B);
  if (blocks == 0) return QMT_OK;
  switch (mode) {
    case PASS_PLAIN: return launch_mode<PASS_PLAIN>(a, blocks, smem, s);
    case PASS_X_RHS: return launch_mode<PASS_X_RHS>(a, blocks, smem, s);
    case PASS_Z_MUL: return launch_mode<PASS_Z_MUL>(a, blocks, smem, s);
    default: return launch_mode<PASS_X_OUT>(a, blocks, smem, s);
  }
}

// Fewest stages of radices up to 10, then the smallest sum of the radices (work per element); larger radices
// first.  No plan (nfac 0) if the length has another prime.
static LinePlan line_plan(int L) {
  constexpr int radices[] = {10, 9, 8, 7, 6, 5, 4, 3, 2};
  LinePlan best{};
  int best_sum = 0, pick[LINE_MAXFAC];
  auto search = [&](auto&& self, int left, int depth, int first, int sum) -> void {
    if (left == 1) {
      if (best.nfac == 0 || depth < best.nfac || sum < best_sum) {
        best.nfac = depth;
        best_sum = sum;
        std::copy(pick, pick + depth, best.fac);
      }
      return;
    }
    const int limit = best.nfac ? best.nfac : LINE_MAXFAC;
    if (depth == limit) return;
    for (int i = first; i < (int)(sizeof(radices) / sizeof(int)); ++i)
      if (left % radices[i] == 0) {
        pick[depth] = radices[i];
        self(self, left / radices[i], depth + 1, i, sum + radices[i]);
      }
  };
  search(search, L, 0, 0, 0);
  int n = L;
  for (int i = 0; i < best.nfac; ++i) {
    n /= best.fac[i];
    best.sub[i] = n;
    best.m_sub[i] = n > 1 ? (unsigned)(((1ull << 32) + (uint64_t)n - 1) / (uint64_t)n) : 0u;
  }
  return best;
}

static qmt_status plan_of(int L, Plan1D& p) {
  if (L < 2 || L > FFT_MAXLEN) return fail(QMT_BAD_ARG, "FFT line length out of range");
  if (!factorize(L, p)) return fail(QMT_BAD_ARG, "FFT size has too many factors");
  p.m_len = (unsigned)(((1ull << 32) + (uint64_t)L - 1) / (uint64_t)L);
  int ns = 1;
  for (int i = 0; i < p.nfac; ++i) {
    if (p.fac[i] > 127) return fail(QMT_BAD_ARG, "FFT size has a prime factor above 127");
    const uint64_t nbf = (uint64_t)(L / p.fac[i]);
    p.ns[i] = ns;
    p.m_nbf[i] = nbf > 1 ? (unsigned)(((1ull << 32) + nbf - 1) / nbf) : 0u;
    p.m_ns[i] = ns > 1 ? (unsigned)(((1ull << 32) + (uint64_t)ns - 1) / (uint64_t)ns) : 0u;
    ns *= p.fac[i];
  }
  p.lp = line_plan(L);
  return QMT_OK;
}

// Hockney G_hat octant for (Mx, My, Mz, h): one unpruned forward 3D transform, cached.
static qmt_status green_hat(int Mx, int My, int Mz, float h_ang, const Plan1D& px, const Plan1D& py,
                            const Plan1D& pz, const float** out, cudaStream_t s) {
  int dev = 0;
  cudaGetDevice(&dev);
  auto key = std::make_tuple(Mx, My, Mz, h_ang, dev);
  DevCache& c = cache();
  std::lock_guard<std::mutex> lock(c.green_mu);
  auto it = c.green.find(key);
  if (it != c.green.end()) {
    GreenEntry& e = it->second;
    e.used = ++c.clock;
    if (!e.built) {
      if (cudaEventQuery(e.ready) == cudaSuccess) e.built = true;
      else QMT_CUDA(cudaStreamWaitEvent(s, e.ready, 0));   // still being built on another stream, maybe
    }
    *out = e.buf->as<float>();
    return QMT_OK;
  }
  const int64_t M = (int64_t)Mx * My * Mz;
  DevBuf*& tmp = c.green_tmp[dev];
  if (!tmp) tmp = new DevBuf();
  cudaEvent_t& tmp_done = c.tmp_done[dev];
  if (!tmp_done) QMT_CUDA(cudaEventCreateWithFlags(&tmp_done, cudaEventDisableTiming));
  // growing the scratch frees the old one (cudaFree waits for its users); otherwise the previous
  // build's use of it is ordered before this one on the device
  qmt_status st = tmp->reserve(M * sizeof(float2));   // grows only: no allocation in steady state
  if (st) return st;
  QMT_CUDA(cudaStreamWaitEvent(s, tmp_done, 0));
  float2* g = tmp->as<float2>();
  green_kernel<<<grid_blocks(M), 256, 0, s>>>(g, Mx, My, Mz, h_ang);
  QMT_CHECK_LAUNCH("green_kernel");
  PassArgs a{};
  a.data = g;
  a.scale = 1.f;
  a.inv = 0;
  a.plan = px; a.n1 = My; a.s1 = Mx; a.s2 = (int64_t)Mx * My; a.se = 1; a.nlines = (int64_t)My * Mz;
  a.lload = a.lstore = Mx;
  if ((st = launch_pass(PASS_PLAIN, a, s))) return st;
  a.plan = py; a.n1 = Mx; a.s1 = 1; a.s2 = (int64_t)Mx * My; a.se = Mx; a.nlines = (int64_t)Mx * Mz;
  a.lload = a.lstore = My;
  if ((st = launch_pass(PASS_PLAIN, a, s))) return st;
  a.plan = pz; a.n1 = Mx; a.s1 = 1; a.s2 = Mx; a.se = (int64_t)Mx * My; a.nlines = (int64_t)Mx * My;
  a.lload = a.lstore = Mz;
  if ((st = launch_pass(PASS_PLAIN, a, s))) return st;
  auto* gb = new DevBuf();
  const int64_t no = (int64_t)(Mx / 2 + 1) * (My / 2 + 1) * (Mz / 2 + 1);
  if ((st = gb->reserve(no * sizeof(float)))) {
    delete gb;
    return st;
  }
  green_octant_kernel<<<grid_blocks(no), 256, 0, s>>>(g, Mx, My, Mz, gb->as<float>());
  QMT_CHECK_LAUNCH("green_octant_kernel");
  QMT_CUDA(cudaEventRecord(tmp_done, s));
  cudaEvent_t ready;
  QMT_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
  QMT_CUDA(cudaEventRecord(ready, s));
  const size_t nbytes = (size_t)no * sizeof(float);
  while (!c.green.empty() && c.green_bytes + nbytes > GREEN_CACHE_BYTES) {
    auto lru = c.green.begin();
    for (auto e = c.green.begin(); e != c.green.end(); ++e)
      if (e->second.used < lru->second.used) lru = e;
    lru->second.buf->release();   // cudaFree waits for kernels still reading it
    delete lru->second.buf;
    cudaEventDestroy(lru->second.ready);
    c.green_bytes -= lru->second.bytes;
    c.green.erase(lru);
  }
  c.green[key] = GreenEntry{gb, ++c.clock, nbytes, ready, false};
  c.green_bytes += nbytes;
  *out = gb->as<float>();
  return QMT_OK;
}

static qmt_status fft_poisson(qmt_mol* mol, int nx, int ny, int nz, float step, float ox, float oy, float oz,
                              float sigma, float cutoff, int padded, int Mx, int My, int Mz, const float* q_dev,
                              float* out_dev, cudaStream_t s);

}  // namespace qmt

using namespace qmt;

extern "C" qmt_status qmt_fft_poisson(qmt_mol* mol, int nx, int ny, int nz, float step, float ox, float oy,
                                      float oz, float sigma, float cutoff, int padded, const float* q_dev,
                                      float* out_dev, void* stream) {
  if (nx < 2 || ny < 2 || nz < 2) return fail(QMT_BAD_ARG, "bad FFT Poisson arguments");
  const int Mx = padded ? nice_at_least(2 * nx) : nx;
  const int My = padded ? nice_at_least(2 * ny) : ny;
  const int Mz = padded ? nice_at_least(2 * nz) : nz;
  return fft_poisson(mol, nx, ny, nz, step, ox, oy, oz, sigma, cutoff, padded ? 1 : 0, Mx, My, Mz, q_dev, out_dev,
                     as_stream(stream));
}

extern "C" qmt_status qmt_fft_poisson_padded(qmt_mol* mol, int nx, int ny, int nz, float step, float ox, float oy,
                                             float oz, float sigma, float cutoff, int mx, int my, int mz,
                                             const float* q_dev, float* out_dev, void* stream) {
  if (nx < 2 || ny < 2 || nz < 2 || mx < 2 * nx || my < 2 * ny || mz < 2 * nz)
    return fail(QMT_BAD_ARG, "padded FFT lengths must be at least twice the grid");
  return fft_poisson(mol, nx, ny, nz, step, ox, oy, oz, sigma, cutoff, 1, mx, my, mz, q_dev, out_dev,
                     as_stream(stream));
}

namespace qmt {

static qmt_status fft_poisson(qmt_mol* mol, int nx, int ny, int nz, float step, float ox, float oy, float oz,
                              float sigma, float cutoff, int padded, int Mx, int My, int Mz, const float* q_dev,
                              float* out_dev, cudaStream_t s) {
  if (!mol || !q_dev || !out_dev || nx < 2 || ny < 2 || nz < 2 || !(step > 0.f) || !(sigma > 0.f) || cutoff < 0)
    return fail(QMT_BAD_ARG, "bad FFT Poisson arguments");
  if (mol->natoms > 4096) return fail(QMT_BAD_ARG, "too many atoms");
  Plan1D px, py, pz;
  qmt_status st;
  if ((st = plan_of(Mx, px)) || (st = plan_of(My, py)) || (st = plan_of(Mz, pz))) return st;
  const int64_t M = (int64_t)Mx * My * Mz;
  // work grid: x-fastest, only the planes z < nz and (the right-hand side is real) the x frequencies up to
  // Mx / 2 are ever touched; rows are padded to whole 32-byte sectors where the spectrum has the elements
  const int hx = Mx / 2 + 1, Hx = (hx + 3) / 4 * 4 <= Mx ? (hx + 3) / 4 * 4 : hx;
  if ((st = mol->d_work.reserve((int64_t)Hx * My * nz * sizeof(float2)))) return st;
  float2* c = mol->d_work.as<float2>();
  const float h_ang = (float)(step / ANG2BOR);
  const float* gsym = nullptr;
  if (padded && (st = green_hat(Mx, My, Mz, h_ang, px, py, pz, &gsym, s))) return st;

  PassArgs a{};
  a.data = c;
  a.mol = mol->view();
  a.q = q_dev;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.h_ang = h_ang;
  a.ox = (float)(ox / ANG2BOR);
  a.oy = (float)(oy / ANG2BOR);
  a.oz = (float)(oz / ANG2BOR);
  a.norm = 1.0f / (sigma * sigma * sigma * 2.0f * (float)PI * sqrtf(2.0f * (float)PI));
  a.i2s2 = 1.0f / (2.0f * sigma * sigma);
  a.cut2 = (cutoff * sigma) * (cutoff * sigma);
  a.periodic = padded ? 0 : 1;
  a.gsym = gsym;
  a.Mx = Mx;
  a.My = My;
  a.Mz = Mz;
  a.out = out_dev;
  a.scale = 1.f;
  // 1. x forward with the RHS: lines (y < ny, z < nz), elements x < nx non-zero
  a.plan = px; a.n1 = ny; a.s1 = Hx; a.s2 = (int64_t)Hx * My; a.se = 1; a.nlines = (int64_t)ny * nz;
  a.lload = nx; a.lstore = Hx; a.inv = 0;
  if ((st = launch_pass(PASS_X_RHS, a, s))) return st;
  // 2. y forward on the planes z < nz: lines (x < Hx, z < nz), elements y < ny non-zero
  a.plan = py; a.n1 = Hx; a.s1 = 1; a.s2 = (int64_t)Hx * My; a.se = Hx; a.nlines = (int64_t)Hx * nz;
  a.lload = ny; a.lstore = My;
  if ((st = launch_pass(PASS_PLAIN, a, s))) return st;
  // 3. z forward, kernel multiply, z inverse: lines (x < Hx, y < My), store z < nz
  a.plan = pz; a.n1 = Hx; a.s1 = 1; a.s2 = Hx; a.se = (int64_t)Hx * My; a.nlines = (int64_t)Hx * My;
  a.lload = nz; a.lstore = nz;
  if ((st = launch_pass(PASS_Z_MUL, a, s))) return st;
  // 4. y inverse on the planes z < nz, store y < ny
  a.plan = py; a.n1 = Hx; a.s1 = 1; a.s2 = (int64_t)Hx * My; a.se = Hx; a.nlines = (int64_t)Hx * nz;
  a.lload = My; a.lstore = ny; a.inv = 1;
  if ((st = launch_pass(PASS_PLAIN, a, s))) return st;
  // 5. x inverse, 1/M^3, real part into the C-order output: lines (z < nz, y < ny)
  a.plan = px; a.n1 = nz; a.s1 = (int64_t)Hx * My; a.s2 = Hx; a.se = 1; a.nlines = (int64_t)ny * nz;
  a.lload = Mx; a.lstore = nx; a.inv = 1; a.scale = (float)(1.0 / (double)M);
  return launch_pass(PASS_X_OUT, a, s);
}

}  // namespace qmt
