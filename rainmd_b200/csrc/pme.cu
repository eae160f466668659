// Particle-mesh Ewald reciprocal space for a batch of systems.
//
// Same mathematics and conventions as RainMD's pme.js:137-345 / cpu/forces/pme.js:76-259:
// B-spline spreading with grid index (floor(u) + k - order + 1) mod K, signed frequencies,
// wave vectors from the ROWS of the inverse box, moduli dividing the kernel, the factor 2
// folded into the convolved grid, an unnormalised inverse transform, and no 1/2 in the
// force gather. The spline order is a template parameter (4 or 5).
//
// B200 design (not the reference's pass structure):
//   spread   ORDER^2 threads per atom, 64-bit fixed-point integer atomics (deterministic);
//   z pass   R2C: two real z-lines packed as one complex line, FFT in shared memory,
//            split into two half spectra, stored plane by plane (kz outermost); also converts
//            fixed point -> f32 and zeroes the fixed grid for the next step;
//   planes   forward y and x FFTs, the Ewald convolution (with the FP64 energy partial) and the
//            inverse x and y FFTs of a whole kz plane in one kernel: one block a plane for small
//            planes, a thread-block cluster a plane (distributed shared memory) for larger ones;
//   z pass   C2R back to a real f32 grid; gather four threads per atom.
// Lines are transformed by two register-resident DFTs a point (fft.cuh). Measured on one B200,
// the reciprocal kernels run back to back, against the radix-4 Stockham passes over a spectrum
// with kz innermost that these replaced: 32^3 27.9 -> 22.8 us, 64^3 49.2 -> 38.2, 108^3
// 139 -> 80, 144^3 360 -> 170, a batch of 24 grids of 24^3-48^3 106 -> 80. What they gained from:
// a plane's rows are contiguous (they were strided by the kz lines: one 32-byte sector a value),
// the r2c pass issues all its loads before it clears the grid, and a transform is two steps
// instead of three or four.
// Planes beyond the cluster's shared memory, and axes without two factors (243, 384 and those
// above 400 points), take passes of their own, y, x with the convolution, y (and z), with a
// mixed-radix (4, 2, 3, 5) Stockham autosort; lines filled by a transpose are padded to n + 1.
// A host-built task table gives each block a set of lines (or a plane) of one system, so
// systems with different grid sizes run in the same launch.
#include <algorithm>
#include <climits>

#include <cooperative_groups.h>

#include "common.cuh"
#include "fft.cuh"
#include "kernels.h"

namespace rmd {

namespace cg = cooperative_groups;

__device__ __forceinline__ int fast_div(int x, FastDiv f) {
  return (int)((__umulhi((uint32_t)x, f.magic) + (uint32_t)x) >> f.shift);
}

template <int R>
__device__ __forceinline__ void stockham_stage(const float2 *__restrict__ in, float2 *__restrict__ out,
                                               int lines, int N, int ld, int Ns, const float2 *tw,
                                               bool inv, FastDiv per_line_div, FastDiv span_div) {
  const int per_line = N / R;
  const int stride_tw = N / (Ns * R);
  for (int idx = threadIdx.x; idx < lines * per_line; idx += blockDim.x) {
    const int line = fast_div(idx, per_line_div), j = idx - line * per_line;
    const float2 *src = in + line * ld;
    float2 v[R];
    const int jq = fast_div(j, span_div);
    const int k = j - jq * Ns;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[j + r * per_line];
#pragma unroll
    for (int r = 1; r < R; ++r) {
      float2 w = tw[k * r * stride_tw];
      if (inv) w.y = -w.y;
      v[r] = cmul(v[r], w);
    }
    dft_small<R>(v, inv);
    float2 *dst = out + line * ld + jq * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[r * Ns] = v[r];
  }
}

// Transform `lines` lines of length N held in a, line l starting at a + l * ld (ld >= N;
// lines filled by a transpose use ld = N + 1 so that the transposing accesses, which step
// by ld, fall in different shared-memory banks); returns the buffer holding the result. The
// twiddles tw are read as given (global or shared memory).
__device__ float2 *fft_stages(float2 *a, float2 *b, int lines, int N, int ld, const FftAxis &ax,
                              const float2 *tw, bool inv) {
  int Ns = 1;
  for (int st = 0; st < ax.nstages; ++st) {
    const int R = ax.radix[st];
    __syncthreads();
    const FastDiv pl = ax.per_line[st], sp = ax.span[st];
    if (R == 4) stockham_stage<4>(a, b, lines, N, ld, Ns, tw, inv, pl, sp);
    else if (R == 2) stockham_stage<2>(a, b, lines, N, ld, Ns, tw, inv, pl, sp);
    else if (R == 3) stockham_stage<3>(a, b, lines, N, ld, Ns, tw, inv, pl, sp);
    else stockham_stage<5>(a, b, lines, N, ld, Ns, tw, inv, pl, sp);
    Ns *= R;
    float2 *t = a;
    a = b;
    b = t;
  }
  __syncthreads();
  return a;
}

// Twiddle tables up to this length are read from shared memory.
constexpr int TW_CACHE = 512;

// fft_stages with the axis's twiddles first copied to shared memory, so the stages read them
// without a global round trip after each barrier (longer tables stay in global memory).
__device__ float2 *fft_lines(float2 *a, float2 *b, int lines, int N, int ld, const FftAxis &ax,
                             const float2 *tw, bool inv) {
  __shared__ float2 tw_cache[TW_CACHE];
  if (N <= TW_CACHE) {
    __syncthreads();  // a previous transform in this block has finished with the cache
    for (int k = threadIdx.x; k < N; k += blockDim.x) tw_cache[k] = tw[k];
    tw = tw_cache;    // visible after the barrier that opens the first stage
  }
  return fft_stages(a, b, lines, N, ld, ax, tw, inv);
}

constexpr int FFT_SMEM = 2048;  // complex values per buffer per block

// ------------------------------------------------------------------------ spreading
// Grid index v in [-n, 2 n) wrapped into [0, n): the spline's points lie within an order (<= n) of
// the atom's own grid point. (An integer modulo is some twenty instructions, three a thread and
// half of this kernel's before.)
__device__ __forceinline__ int wrap_near(int v, int n) {
  if (v < 0) v += n;
  return v >= n ? v - n : v;
}

// ORDER*ORDER threads per atom: thread (ky, kz) adds the ORDER points of one x-line, so the ORDER
// threads of a ky add consecutive z points together: a warp's atomic instruction covers rows of
// 8 * ORDER bytes, one or two sectors each, where a thread a (kx, ky) touched 32 sectors an
// instruction. Each thread recomputes the atom's splines (cheap) so no cross-thread exchange is
// needed. With the gather's wrapped indices below, the reciprocal kernels at 250,000 atoms on 144^3 went from
// 170 to 133 us, at 23,558 on 64^3 from 38.2 to 32.8. At 23,558 atoms (9.7 us cold, 14.2 before) its warps wait for
// the atoms' records (long scoreboard 9.7 of them an issue); the L2's atomic input is busy 19% of the time.
template <int ORDER>
__global__ void k_spread(const float4 *__restrict__ posq, const int *__restrict__ sys_of_atom,
                         const DevSys *__restrict__ sys, unsigned long long *__restrict__ fixed_grid,
                         int n_atoms) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(t / (ORDER * ORDER));
  const bool valid = i < n_atoms;
  const DevSys &s = sys[valid ? sys_of_atom[i] : 0];
  const int nx = s.grid[0], ny = s.grid[1], nz = s.grid[2];
  unsigned long long *grid = fixed_grid + s.grid_base;
  chain_begin();  // (DevSys::grid and grid_base never change; positions and box do)
  if (!valid) return;
  const int ky = (int)(t % (ORDER * ORDER)) / ORDER, kz = (int)(t % ORDER);
  const float4 p = posq[i];
  if (p.w == 0.f) return;
  float w[3][ORDER], dw[3][ORDER];
  int base[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float f = p.x * s.recip[d] + p.y * s.recip[3 + d] + p.z * s.recip[6 + d];
    const float scaled = (f - floorf(f)) * (float)s.grid[d];
    const float fl = floorf(scaled);
    base[d] = (int)fl;
    bspline<ORDER>(scaled - fl, w[d], dw[d]);
  }
  float wy = 0.f, wz = 0.f;
#pragma unroll
  for (int k = 0; k < ORDER; ++k) {
    if (k == ky) wy = w[1][k];
    if (k == kz) wz = w[2][k];
  }
  const int iy = wrap_near(base[1] + ky - ORDER + 1, ny);
  const int iz = wrap_near(base[2] + kz - ORDER + 1, nz);
  grid += (long long)iy * nz + iz;
#pragma unroll
  for (int kx = 0; kx < ORDER; ++kx) {
    const int ix = wrap_near(base[0] + kx - ORDER + 1, nx);
    atomicAdd(grid + (long long)ix * ny * nz, to_fixed(p.w * w[0][kx] * wy * wz));
  }
}

// -------------------------------------------------------------- z pass, forward (R2C)
__global__ void __launch_bounds__(256) k_fft_z_r2c(const FftTask *__restrict__ tasks,
                                                   const DevSys *__restrict__ sys,
                                                   const FftPlan *__restrict__ plans,
                                                   const float2 *__restrict__ twiddles,
                                                   unsigned long long *__restrict__ fixed_grid,
                                                   float2 *__restrict__ half) {
  chain_begin();
  __shared__ float2 bufa[FFT_SMEM], bufb[FFT_SMEM];
  const FftTask t = tasks[blockIdx.x];
  const DevSys &s = sys[t.sys];
  const FftPlan &pl = plans[t.sys];
  const int N = s.grid[2], nzh = N / 2 + 1;
  const int nlines = s.grid[0] * s.grid[1];
  const int M = t.count;
  unsigned long long *g = fixed_grid + s.grid_base;
  for (int idx = threadIdx.x; idx < M * N; idx += blockDim.x) {
    const int p = fast_div(idx, pl.axis[2].n_div), k = idx - p * N;
    const int l = 2 * (t.first + p);
    unsigned long long *ra = g + (long long)l * N + k;
    const bool two = l + 1 < nlines;
    // both values read before either is cleared for the next step's spreading
    const unsigned long long va = ra[0];
    const unsigned long long vb = two ? ra[N] : 0ull;
    ra[0] = 0ull;
    if (two) ra[N] = 0ull;
    bufa[idx] = make_float2(from_fixed(va), two ? from_fixed(vb) : 0.f);
  }
  float2 *r = fft_lines(bufa, bufb, M, N, N, pl.axis[2], twiddles + pl.axis[2].tw_base, false);
  float2 *h = half + s.half_base;
  for (int idx = threadIdx.x; idx < M * nzh; idx += blockDim.x) {
    const int p = fast_div(idx, pl.axis[2].half_div), k = idx - p * nzh;
    const int l = 2 * (t.first + p);
    const float2 z = r[p * N + k];
    const float2 zc = r[p * N + (N - k) % N];
    // A = (Z + conj(Zc))/2, B = -i (Z - conj(Zc))/2
    const float2 a = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
    const float2 b = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
    h[(long long)k * nlines + l] = a;
    if (l + 1 < nlines) h[(long long)k * nlines + l + 1] = b;
  }
}

// -------------------------------------------------------------- z pass, inverse (C2R)
__global__ void __launch_bounds__(256) k_fft_z_c2r(const FftTask *__restrict__ tasks,
                                                   const DevSys *__restrict__ sys,
                                                   const FftPlan *__restrict__ plans,
                                                   const float2 *__restrict__ twiddles,
                                                   const float2 *__restrict__ half,
                                                   float *__restrict__ real_grid) {
  chain_begin();
  __shared__ float2 bufa[FFT_SMEM], bufb[FFT_SMEM];
  const FftTask t = tasks[blockIdx.x];
  const DevSys &s = sys[t.sys];
  const FftPlan &pl = plans[t.sys];
  const int N = s.grid[2], nzh = N / 2 + 1;
  const int nlines = s.grid[0] * s.grid[1];
  const int M = t.count;
  const float2 *h = half + s.half_base;
  for (int idx = threadIdx.x; idx < M * N; idx += blockDim.x) {
    const int p = fast_div(idx, pl.axis[2].n_div), k = idx - p * N;
    const int l = 2 * (t.first + p);
    const bool has_b = l + 1 < nlines;
    float2 a, b;
    if (k < nzh) {
      a = h[(long long)k * nlines + l];
      b = has_b ? h[(long long)k * nlines + l + 1] : make_float2(0.f, 0.f);
      if (k == 0 || 2 * k == N) {
        a.y = 0.f;
        b.y = 0.f;
      }
    } else {
      a = h[(long long)(N - k) * nlines + l];
      b = has_b ? h[(long long)(N - k) * nlines + l + 1] : make_float2(0.f, 0.f);
      a.y = -a.y;
      b.y = -b.y;
    }
    bufa[idx] = make_float2(a.x - b.y, a.y + b.x);  // A + iB
  }
  float2 *r = fft_lines(bufa, bufb, M, N, N, pl.axis[2], twiddles + pl.axis[2].tw_base, true);
  float *g = real_grid + s.grid_base;
  for (int idx = threadIdx.x; idx < M * N; idx += blockDim.x) {
    const int p = fast_div(idx, pl.axis[2].n_div), k = idx - p * N;
    const int l = 2 * (t.first + p);
    const float2 z = r[idx];
    g[(long long)l * N + k] = z.x;
    if (l + 1 < nlines) g[(long long)(l + 1) * N + k] = z.y;
  }
}

// ------------------------------------------------------ y pass (either direction, in place)
// A task is `count` consecutive x rows of plane kz = `fixed`: one contiguous run of the plane.
__global__ void __launch_bounds__(256) k_fft_y(const FftTask *__restrict__ tasks,
                                               const DevSys *__restrict__ sys,
                                               const FftPlan *__restrict__ plans,
                                               const float2 *__restrict__ twiddles,
                                               float2 *__restrict__ half, int inverse) {
  chain_begin();
  __shared__ float2 bufa[FFT_SMEM], bufb[FFT_SMEM];
  const FftTask t = tasks[blockIdx.x];
  const DevSys &s = sys[t.sys];
  const FftPlan &pl = plans[t.sys];
  const int nx = s.grid[0], ny = s.grid[1], M = t.count;
  float2 *h = half + s.half_base + ((long long)t.fixed * nx + t.first) * ny;
  for (int idx = threadIdx.x; idx < ny * M; idx += blockDim.x) bufa[idx] = h[idx];
  float2 *r = fft_lines(bufa, bufb, M, ny, ny, pl.axis[1], twiddles + pl.axis[1].tw_base, inverse != 0);
  for (int idx = threadIdx.x; idx < ny * M; idx += blockDim.x) h[idx] = r[idx];
}

// The Ewald convolution along a line of kx at fixed ky and kz (signed frequencies): the wave
// vector is (kx, ky, kz) times the rows of the inverse box, of which the entries above the diagonal
// are zero (the box is reduced), so only its kx part changes along the line. mod_yz: the product
// of the y and z moduli. With ENERGY the point's energy and virial terms are added; `weight` counts
// the point and its mirror image. The zero wave vector gives zero.
struct ConvolveLine {
  float r0, r3, r6, cy, cz, mod_yz, factor, pref;
  __device__ __forceinline__ ConvolveLine(const DevSys &s, int ky, int kz, float mod) {
    r0 = s.recip[0];
    r3 = s.recip[3];
    r6 = s.recip[6];
    cy = (float)ky * s.recip[4];
    cz = (float)ky * s.recip[7] + (float)kz * s.recip[8];
    mod_yz = mod;
    factor = s.pme_factor;
    pref = s.pme_pref;
  }
  template <bool ENERGY>
  __device__ __forceinline__ void apply(float2 &v, int kx, float mod_x, double weight, double &energy,
                                        double &virial) const {
    const float fx = (float)kx;
    const float x = fx * r0, y = fmaf(fx, r3, cy), z = fmaf(fx, r6, cz);
    const float m2 = x * x + y * y + z * z;
    const float kernel = m2 != 0.f ? __expf(-factor * m2) / (m2 * (mod_x * mod_yz)) : 0.f;
    if (ENERGY) {
      const double ek = weight * 0.5 * (double)pref * (double)kernel * ((double)v.x * v.x + (double)v.y * v.y);
      energy += ek;
      virial += ek * (1.0 + (double)factor * (double)m2);
    }
    const float sc = kernel * pref;
    v = make_float2(v.x * sc, v.y * sc);
  }
};

// Block sum of a thread's energy and virial terms, written by thread 0 to e[slot], ev[slot].
__device__ __forceinline__ void block_energy(double energy, double virial, double *e, double *ev, int slot) {
  __shared__ double red[2][32];
  energy = warp_sum(energy);
  virial = warp_sum(virial);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = energy;
    red[1][threadIdx.x >> 5] = virial;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0, total_vir = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      total += red[0][w];
      total_vir += red[1][w];
    }
    e[slot] = total;
    ev[slot] = total_vir;
  }
}

// ------------------------------ x pass: forward FFT, Ewald convolution + energy, inverse
template <bool ENERGY>
__global__ void __launch_bounds__(256) k_fft_x_convolve(const FftTask *__restrict__ tasks,
                                                        const DevSys *__restrict__ sys,
                                                        const FftPlan *__restrict__ plans,
                                                        const float2 *__restrict__ twiddles,
                                                        const float *__restrict__ moduli,
                                                        float2 *__restrict__ half,
                                                        double *__restrict__ e_pme,
                                                        double *__restrict__ e_pme_vir) {
  chain_begin();
  __shared__ float2 bufa[FFT_SMEM], bufb[FFT_SMEM];
  const FftTask t = tasks[blockIdx.x];
  const DevSys &s = sys[t.sys];
  const FftPlan &pl = plans[t.sys];
  const int nx = s.grid[0], ny = s.grid[1], nz = s.grid[2];
  const int kz = t.fixed, y0 = t.first, M = t.count;
  float2 *h = half + s.half_base + (long long)kz * nx * ny + y0;
  const int ld = nx + 1;  // padded lines (bank-conflict-free transpose)
  for (int idx = threadIdx.x; idx < nx * M; idx += blockDim.x) {
    const int x = idx / M, m = idx - x * M;
    bufa[m * ld + x] = h[(long long)x * ny + m];
  }
  float2 *r = fft_lines(bufa, bufb, M, nx, ld, pl.axis[0], twiddles + pl.axis[0].tw_base, false);
  const double weight = (kz == 0 || 2 * kz == nz) ? 1.0 : 2.0;
  const float *modx = moduli + s.moduli_base, *mody = modx + nx, *modz = mody + ny;
  double energy = 0.0, virial = 0.0;
  for (int idx = threadIdx.x; idx < nx * M; idx += blockDim.x) {
    const int m = idx / nx, mx = idx - m * nx;
    const int my = y0 + m;
    const ConvolveLine line(s, my <= ny / 2 ? my : my - ny, kz, mody[my] * modz[kz]);
    line.apply<ENERGY>(r[m * ld + mx], mx <= nx / 2 ? mx : mx - nx, modx[mx], weight, energy, virial);
  }
  float2 *other = (r == bufa) ? bufb : bufa;
  float2 *q = fft_lines(r, other, M, nx, ld, pl.axis[0], twiddles + pl.axis[0].tw_base, true);
  for (int idx = threadIdx.x; idx < nx * M; idx += blockDim.x) {
    const int x = idx / M, m = idx - x * M;
    h[(long long)x * ny + m] = q[m * ld + x];
  }
  if (ENERGY) block_energy(energy, virial, e_pme, e_pme_vir, blockIdx.x);
}

// ------------------------------------------------------------------ two-factor transforms
// The passes below hold a line of N = R1 * R2 points as R1 rows of R2 (pitch R2 made odd, so
// that a thread's row and the threads' columns both fall in different shared-memory banks) and
// transform it in place, one DFT a thread (fft.cuh). Against the Stockham stages they replaced
// (radix 4, one barrier and one trip through shared memory a stage, the lines copied in and out
// in passes of their own) each transform is two steps and one barrier, with the first and last
// step of a pass reading or writing global memory directly. The static inputs (task, twiddles,
// moduli) are read before a kernel waits for its predecessor.
__host__ __device__ inline int odd_pitch(int r2) { return r2 | 1; }

constexpr int FFT_PAIRS = FFT_PAIRS_PER_BLOCK;  // pairs of real lines a z block transforms

// z pass, forward (R2C): FFT_PAIRS pairs of real lines, each pair one complex line. The half
// spectrum is stored plane by plane, half[kz][x * ny + y], so a block's 2 * FFT_PAIRS
// consecutive lines are one 128-byte run of each plane. All of a thread's 2 R1 loads of the
// fixed-point grid are in flight together, and the grid is cleared behind them.
template <int MAXR>
__global__ void __launch_bounds__(256) k_fft_r2c(const FftZTask *__restrict__ tasks,
                                                 const float2 *__restrict__ twiddles,
                                                 unsigned long long *__restrict__ fixed_grid,
                                                 float2 *__restrict__ half) {
  extern __shared__ float2 smem[];
  __shared__ float2 tw[FFT_TWO_MAX];
  const FftZTask t = tasks[blockIdx.x];
  const FftTwo &ax = t.z;
  const int N = ax.n, R1 = ax.r1, R2 = ax.r2, M = t.count, plane = t.plane;
  const int pitch = odd_pitch(R2), ld = (R1 * pitch) | 1;
  for (int k = threadIdx.x; k < N; k += blockDim.x) tw[k] = twiddles[ax.tw_base + k];
  chain_begin();
  unsigned long long *g = fixed_grid + t.grid_base;
  with_radix<MAXR>(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < M * R2; it += blockDim.x) {
      const int p = fast_div(it, ax.r2_div), j = it - p * R2;
      const int l = 2 * (t.first + p);
      const bool two = l + 1 < plane;
      unsigned long long *src = g + (long long)l * N + j;
      unsigned long long a[R], b[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        a[r] = src[r * R2];
        b[r] = two ? src[N + r * R2] : 0ull;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {  // cleared for the next step's spreading
        src[r * R2] = 0ull;
        if (two) src[N + r * R2] = 0ull;
      }
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = make_float2(from_fixed(a[r]), from_fixed(b[r]));
      dft<R, false>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) smem[p * ld + r * pitch + j] = v[r];
    }
  });
  __syncthreads();
  with_radix<MAXR>(R2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < M * R1; it += blockDim.x) {
      const int p = fast_div(it, ax.r1_div), k1 = it - p * R1;
      float2 *line = smem + p * ld + k1 * pitch;
      float2 v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = cmul(line[j], tw[k1 * j]);
      dft<R, false>(v);
#pragma unroll
      for (int j = 0; j < R; ++j) line[j] = v[j];
    }
  });
  __syncthreads();
  float2 *h = half + t.half_base;
  const int nzh = N / 2 + 1;
  const bool wide = (plane & 1) == 0;  // then a pair's two values are 16-byte aligned in every plane
  for (int idx = threadIdx.x; idx < FFT_PAIRS * nzh; idx += blockDim.x) {
    const int p = idx % FFT_PAIRS, k = idx / FFT_PAIRS;
    if (p >= M) continue;
    const int l = 2 * (t.first + p), kc = k == 0 ? 0 : N - k;
    const int q = fast_div(k, ax.r1_div), qc = fast_div(kc, ax.r1_div);
    const float2 z = smem[p * ld + (k - q * R1) * pitch + q];
    const float2 zc = smem[p * ld + (kc - qc * R1) * pitch + qc];
    // A = (Z + conj(Zc))/2, B = -i (Z - conj(Zc))/2
    const float2 a = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
    const float2 b = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
    float2 *out = h + (long long)k * plane + l;
    if (wide) {
      *reinterpret_cast<float4 *>(out) = make_float4(a.x, a.y, b.x, b.y);
    } else {
      out[0] = a;
      if (l + 1 < plane) out[1] = b;
    }
  }
}

// z pass, inverse (C2R), the same shape backwards.
template <int MAXR>
__global__ void __launch_bounds__(256) k_fft_c2r(const FftZTask *__restrict__ tasks,
                                                 const float2 *__restrict__ twiddles,
                                                 const float2 *__restrict__ half, float *__restrict__ real_grid) {
  extern __shared__ float2 smem[];
  __shared__ float2 tw[FFT_TWO_MAX];
  const FftZTask t = tasks[blockIdx.x];
  const FftTwo &ax = t.z;
  const int N = ax.n, R1 = ax.r1, R2 = ax.r2, M = t.count, plane = t.plane;
  const int pitch = odd_pitch(R2), ld = (R1 * pitch) | 1;
  const int nzh = N / 2 + 1;
  for (int k = threadIdx.x; k < N; k += blockDim.x) tw[k] = twiddles[ax.tw_base + k];
  chain_begin();
  const float2 *h = half + t.half_base;
  const bool wide = (plane & 1) == 0;
  with_radix<MAXR>(R2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < FFT_PAIRS * R1; it += blockDim.x) {
      const int p = it % FFT_PAIRS, k1 = it / FFT_PAIRS;
      if (p >= M) continue;
      const int l = 2 * (t.first + p);
      const bool two = l + 1 < plane;
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = k1 + r * R1;
        const bool mirrored = k >= nzh;
        const float2 *in = h + (long long)(mirrored ? N - k : k) * plane + l;
        float2 a, b;
        if (wide) {
          const float4 ab = __ldg(reinterpret_cast<const float4 *>(in));
          a = make_float2(ab.x, ab.y);
          b = make_float2(ab.z, ab.w);
        } else {
          a = __ldg(in);
          b = two ? __ldg(in + 1) : make_float2(0.f, 0.f);
        }
        if (k == 0 || 2 * k == N) a.y = b.y = 0.f;
        if (mirrored) a.y = -a.y, b.y = -b.y;
        v[r] = make_float2(a.x - b.y, a.y + b.x);  // A + iB
      }
      dft<R, true>(v);
#pragma unroll
      for (int j = 0; j < R; ++j) smem[p * ld + k1 * pitch + j] = v[j];
    }
  });
  __syncthreads();
  float *g = real_grid + t.grid_base;
  with_radix<MAXR>(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < M * R2; it += blockDim.x) {
      const int p = fast_div(it, ax.r2_div), j = it - p * R2;
      const int l = 2 * (t.first + p);
      float2 v[R];
#pragma unroll
      for (int k1 = 0; k1 < R; ++k1) {
        const float2 w = tw[k1 * j];
        v[k1] = cmul(smem[p * ld + k1 * pitch + j], make_float2(w.x, -w.y));
      }
      dft<R, true>(v);
      float *out = g + (long long)l * N + j;
#pragma unroll
      for (int r = 0; r < R; ++r) out[r * R2] = v[r].x;
      if (l + 1 < plane)
#pragma unroll
        for (int r = 0; r < R; ++r) out[N + r * R2] = v[r].y;
    }
  });
}

// ----------------- y and x passes of one kz plane fused: forward y, forward x, the Ewald
// convolution (and energy), inverse x, inverse y, by a cluster of `cl` blocks a plane (1 for
// small planes, which a block holds alone). Block r of a cluster owns the x rows
// [r * rows_per, ...) for the y transforms and the columns [r * cols_per, ...) of the
// transformed rows for the x transforms and the convolution. Each line is transformed in place
// (see above) in seven steps:
//   1 y columns-DFT, from global      2 y rows-DFT            (cluster barrier: rows complete)
//   3 x columns-DFT, from the owners' rows (distributed shared memory)
//   4 x rows-DFT, convolution, inverse x rows-DFT, all in registers
//   5 inverse x columns-DFT, into the owners' rows, once every block has read them (step 3)
//                                     (cluster barrier: rows complete)
//   6 inverse y rows-DFT              7 inverse y columns-DFT, to global
// The convolution needs a column's true ky: column c = k1 * R2 + k2 is ky = k1 + R1 * k2.
// `threads` of the plan (not the launch's block size, which other systems of a batch may have
// raised) share the items of each step, so the energy partials' grouping, and with it every bit
// of the energy, depends on the system alone.
struct PlaneTables {
  float2 tw_y[FFT_TWO_MAX], tw_x[FFT_TWO_MAX];
  float mod_x[FFT_TWO_MAX], mod_y[FFT_TWO_MAX];
};

template <bool ENERGY, int MAXR>
__global__ void __launch_bounds__(FFT_PLANE_THREADS)
    k_fft_planes(const FftPlaneTask *__restrict__ tasks, const DevSys *__restrict__ sys, const float2 *__restrict__ twiddles,
                 const float *__restrict__ moduli, float2 *__restrict__ half, int cl, int row_stride,
                 double *__restrict__ e_pme, double *__restrict__ e_pme_vir) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = cl > 1 ? (int)cluster.block_rank() : 0;
  extern __shared__ float2 smem[];
  __shared__ PlaneTables tab;
  const FftPlaneTask t = tasks[blockIdx.x / cl];
  const FftTwo &ay = t.y, &axx = t.x;
  const int nx = axx.n, ny = ay.n, kz = t.kz;
  const int R1y = ay.r1, R2y = ay.r2, R1x = axx.r1, R2x = axx.r2;
  const int pitch = odd_pitch(R2y), ldy = R1y * pitch;
  const int rows_per = t.rows_div.d, cols_per = t.cols_div.d;
  const int x0 = min(nx, rank * rows_per), nr = min(nx, x0 + rows_per) - x0;
  const int c0 = min(ny, rank * cols_per), nc = min(ny, c0 + cols_per) - c0;
  const int nt = t.threads, tid = threadIdx.x < nt ? threadIdx.x : INT_MAX;
  float2 *rows = smem;
  // the columns' own buffer holds point x of local column c at x * cols_per + c; a block that
  // owns the whole plane works on the columns in place
  float2 *cols = cl > 1 ? smem + row_stride : smem;
  const int cstride = cl > 1 ? cols_per : ldy;
  float2 *h = half + t.half_base;  // element (x, y) at h[x * ny + y]
  const float *mod = moduli + t.moduli_base;
  for (int k = threadIdx.x; k < ny; k += blockDim.x) {
    tab.tw_y[k] = twiddles[ay.tw_base + k];
    tab.mod_y[k] = mod[nx + k];
  }
  for (int k = threadIdx.x; k < nx; k += blockDim.x) {
    tab.tw_x[k] = twiddles[axx.tw_base + k];
    tab.mod_x[k] = mod[k];
  }
  const float mod_z = mod[nx + ny + kz];
  chain_begin();
  const DevSys &s = sys[t.sys];
  with_radix<MAXR>(R1y, [&](auto rc) {  // 1
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < nr * R2y; it += nt) {
      const int row = fast_div(it, ay.r2_div), j = it - row * R2y;
      const float2 *in = h + (long long)(x0 + row) * ny + j;
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = in[r * R2y];
      dft<R, false>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) rows[row * ldy + r * pitch + j] = v[r];
    }
  });
  __syncthreads();
  with_radix<MAXR>(R2y, [&](auto rc) {  // 2
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < nr * R1y; it += nt) {
      const int row = fast_div(it, ay.r1_div), k1 = it - row * R1y;
      float2 *line = rows + row * ldy + k1 * pitch;
      float2 v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = cmul(line[j], tab.tw_y[k1 * j]);
      dft<R, false>(v);
#pragma unroll
      for (int j = 0; j < R; ++j) line[j] = v[j];
    }
  });
  if (cl > 1) cluster.sync();
  else __syncthreads();
  with_radix<MAXR>(R1x, [&](auto rc) {  // 3
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < cols_per * R2x; it += nt) {
      const int j = fast_div(it, t.cols_div), c = it - j * cols_per;
      if (c >= nc) continue;  // (the last block of a cluster may own fewer)
      const int k1y = fast_div(c0 + c, ay.r2_div), at = (c0 + c) + (pitch - R2y) * k1y;  // the column in a row
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int x = r * R2x + j;
        const int owner = cl > 1 ? fast_div(x, t.rows_div) : 0;
        const float2 *src = cl > 1 ? cluster.map_shared_rank(rows, owner) : rows;
        v[r] = src[(x - owner * rows_per) * ldy + at];
      }
      dft<R, false>(v);
      float2 *col = cols + (cl > 1 ? c : at);
#pragma unroll
      for (int r = 0; r < R; ++r) col[(r * R2x + j) * cstride] = v[r];
    }
  });
  if (cl > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");  // this block has read the others' rows
  __syncthreads();
  double energy = 0.0, virial = 0.0;
  const double weight = (kz == 0 || 2 * kz == t.nz) ? 1.0 : 2.0;
  with_radix<MAXR>(R2x, [&](auto rc) {  // 4
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < cols_per * R1x; it += nt) {
      const int k1 = fast_div(it, t.cols_div), c = it - k1 * cols_per;
      if (c >= nc) continue;
      const int k1y = fast_div(c0 + c, ay.r2_div), k2y = (c0 + c) - k1y * R2y;
      const int ky = k1y + R1y * k2y;
      float2 *col = cols + (cl > 1 ? c : k1y * pitch + k2y) + (long long)k1 * R2x * cstride;
      float2 v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = cmul(col[j * cstride], tab.tw_x[k1 * j]);
      dft<R, false>(v);
      const ConvolveLine line(s, ky <= ny / 2 ? ky : ky - ny, kz, tab.mod_y[ky] * mod_z);
#pragma unroll
      for (int k2 = 0; k2 < R; ++k2) {
        const int mx = k1 + R1x * k2;
        line.apply<ENERGY>(v[k2], mx <= nx / 2 ? mx : mx - nx, tab.mod_x[mx], weight, energy, virial);
      }
      dft<R, true>(v);
#pragma unroll
      for (int j = 0; j < R; ++j) col[j * cstride] = v[j];
    }
  });
  __syncthreads();
  if (cl > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // every block has read these rows
  with_radix<MAXR>(R1x, [&](auto rc) {  // 5
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < cols_per * R2x; it += nt) {
      const int j = fast_div(it, t.cols_div), c = it - j * cols_per;
      if (c >= nc) continue;  // (the last block of a cluster may own fewer)
      const int k1y = fast_div(c0 + c, ay.r2_div), at = (c0 + c) + (pitch - R2y) * k1y;
      const float2 *col = cols + (cl > 1 ? c : at);
      float2 v[R];
#pragma unroll
      for (int k1 = 0; k1 < R; ++k1) {
        const float2 w = tab.tw_x[k1 * j];
        v[k1] = cmul(col[(k1 * R2x + j) * cstride], make_float2(w.x, -w.y));
      }
      dft<R, true>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int x = r * R2x + j;
        const int owner = cl > 1 ? fast_div(x, t.rows_div) : 0;
        float2 *dst = cl > 1 ? cluster.map_shared_rank(rows, owner) : rows;
        dst[(x - owner * rows_per) * ldy + at] = v[r];
      }
    }
  });
  if (cl > 1) cluster.sync();
  else __syncthreads();
  with_radix<MAXR>(R2y, [&](auto rc) {  // 6
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < nr * R1y; it += nt) {
      const int row = fast_div(it, ay.r1_div), k1 = it - row * R1y;
      float2 *line = rows + row * ldy + k1 * pitch;
      float2 v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = line[j];
      dft<R, true>(v);
#pragma unroll
      for (int j = 0; j < R; ++j) line[j] = v[j];
    }
  });
  __syncthreads();
  with_radix<MAXR>(R1y, [&](auto rc) {  // 7
    constexpr int R = decltype(rc)::value;
    for (int it = tid; it < nr * R2y; it += nt) {
      const int row = fast_div(it, ay.r2_div), j = it - row * R2y;
      float2 v[R];
#pragma unroll
      for (int k1 = 0; k1 < R; ++k1) {
        const float2 w = tab.tw_y[k1 * j];
        v[k1] = cmul(rows[row * ldy + k1 * pitch + j], make_float2(w.x, -w.y));
      }
      dft<R, true>(v);
      float2 *out = h + (long long)(x0 + row) * ny + j;
#pragma unroll
      for (int r = 0; r < R; ++r) out[r * R2y] = v[r];
    }
  });
  if (ENERGY) block_energy(energy, virial, e_pme, e_pme_vir, blockIdx.x);
}
// ------------------------------------------------------------------------- gather
// Force gather with four threads per atom (atoms in cell order, for locality of the grid
// reads): thread q sums the x-planes kx = q, q + 4 (< ORDER), the four partial gradients are
// combined with shuffles, and the first thread adds the force. One thread per atom leaves
// most of the GPU idle at these sizes (23,558 atoms are 185 blocks of 128).
template <int ORDER>
__global__ void k_gather4(const float4 *__restrict__ posq, const int *__restrict__ sorted_orig,
                          const int *__restrict__ sys_of_atom, const DevSys *__restrict__ sys,
                          const float *__restrict__ real_grid, unsigned long long *__restrict__ force,
                          int n_atoms) {
  chain_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = t >> 2, q = t & 3;
  const bool valid = slot < n_atoms;
  const int i = valid ? sorted_orig[slot] : 0;
  const float4 p = valid ? posq[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  float gu = 0.f, gv = 0.f, gw = 0.f;
  const DevSys &s = sys[sys_of_atom[i]];
  if (valid && p.w != 0.f) {
    float w[3][ORDER], dw[3][ORDER];
    int base[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float f = p.x * s.recip[d] + p.y * s.recip[3 + d] + p.z * s.recip[6 + d];
      const float scaled = (f - floorf(f)) * (float)s.grid[d];
      const float fl = floorf(scaled);
      base[d] = (int)fl;
      bspline<ORDER>(scaled - fl, w[d], dw[d]);
    }
    const int nx = s.grid[0], ny = s.grid[1], nz = s.grid[2];
    const float *g = real_grid + s.grid_base;
    int iz[ORDER];
#pragma unroll
    for (int kz = 0; kz < ORDER; ++kz) iz[kz] = wrap_near(base[2] + kz - ORDER + 1, nz);
    // this thread's x-planes: kx = q (and q + 4 for order 5), weights selected without
    // branching so the four threads of an atom run the y and z loops in step
    for (int kx = q; kx < ORDER; kx += 4) {
      float wx = w[0][0], dwx = dw[0][0];
#pragma unroll
      for (int k = 1; k < ORDER; ++k) {
        wx = (kx == k) ? w[0][k] : wx;
        dwx = (kx == k) ? dw[0][k] : dwx;
      }
      const int ix = wrap_near(base[0] + kx - ORDER + 1, nx);
#pragma unroll
      for (int ky = 0; ky < ORDER; ++ky) {
        const int iy = wrap_near(base[1] + ky - ORDER + 1, ny);
        const float *rowp = g + ((long long)ix * ny + iy) * nz;
        const float wxy = wx * w[1][ky], dxy = dwx * w[1][ky], wdy = wx * dw[1][ky];
#pragma unroll
        for (int kz = 0; kz < ORDER; ++kz) {
          const float v = __ldg(rowp + iz[kz]);
          gu = fmaf(dxy * w[2][kz], v, gu);
          gv = fmaf(wdy * w[2][kz], v, gv);
          gw = fmaf(wxy * dw[2][kz], v, gw);
        }
      }
    }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    gu += __shfl_xor_sync(0xffffffffu, gu, o);
    gv += __shfl_xor_sync(0xffffffffu, gv, o);
    gw += __shfl_xor_sync(0xffffffffu, gw, o);
  }
  if (!valid || q != 0 || p.w == 0.f) return;
  // the convolved grid already carries the Coulomb prefactor (and the factor 2)
  const float su = gu * (float)s.grid[0] * p.w, sv = gv * (float)s.grid[1] * p.w, sw = gw * (float)s.grid[2] * p.w;
  add_fixed(force + i, -(su * s.recip[0] + sv * s.recip[1] + sw * s.recip[2]));
  add_fixed(force + n_atoms + i, -(su * s.recip[3] + sv * s.recip[4] + sw * s.recip[5]));
  add_fixed(force + 2 * (long long)n_atoms + i, -(su * s.recip[6] + sv * s.recip[7] + sw * s.recip[8]));
}

static void launch_gather(const LaunchCtx &c, cudaStream_t stream) {
  const int n = c.n_atoms, tb = 128;
  const int blocks = (int)(((long long)n * 4 + tb - 1) / tb);
  if (c.pme_order == 4)
    launch_chained(k_gather4<4>, blocks, tb, 0, stream, c.posq, c.sorted_orig, c.sys_of_atom, c.sys, c.real_grid, c.force, n);
  else
    launch_chained(k_gather4<5>, blocks, tb, 0, stream, c.posq, c.sorted_orig, c.sys_of_atom, c.sys, c.real_grid, c.force, n);
}

// Forward transform of the spread grid to the half spectrum (z and y; x is left to the caller).
static void launch_forward_zy(const LaunchCtx &c, cudaStream_t stream, bool all = false) {
  // The two-factor pass is chained after the spreading like the rest (it reads its tables while the
  // last atomics land: the reciprocal kernels 33.1 -> 30.8 us at 64^3, 20.5 -> 17.9 at 24^3). The
  // generic pass stays a plain launch: chained it was slower at 64^3 (0.067 against 0.049 ms).
  if (c.n_tasks_z2 > 0)
    launch_kernel(c.chain_pme, c.z2_large ? k_fft_r2c<RADIX_ALL> : k_fft_r2c<RADIX_SMALL>, c.n_tasks_z2, c.z2_threads,
                  c.z2_smem * sizeof(float2), stream, c.tasks_z2, c.twiddles, c.fixed_grid, c.half);
  if (c.n_tasks_z > 0)
    k_fft_z_r2c<<<c.n_tasks_z, 256, 0, stream>>>(c.tasks_z, c.sys, c.fft_plans, c.twiddles, c.fixed_grid, c.half);
  const FftTask *ty = all ? c.tasks_y_all : c.tasks_y;
  const int n = all ? c.n_tasks_y_all : c.n_tasks_y;
  if (n > 0) launch_kernel(c.chain_pme, k_fft_y, n, 256, 0, stream, ty, c.sys, c.fft_plans, c.twiddles, c.half, 0);
}

static void launch_inverse_yz(const LaunchCtx &c, cudaStream_t stream, bool all = false) {
  const FftTask *ty = all ? c.tasks_y_all : c.tasks_y;
  const int n = all ? c.n_tasks_y_all : c.n_tasks_y;
  if (n > 0) launch_kernel(c.chain_pme, k_fft_y, n, 256, 0, stream, ty, c.sys, c.fft_plans, c.twiddles, c.half, 1);
  if (c.n_tasks_z2 > 0)
    launch_kernel(c.chain_pme, c.z2_large ? k_fft_c2r<RADIX_ALL> : k_fft_c2r<RADIX_SMALL>, c.n_tasks_z2, c.z2_threads,
                  c.z2_smem * sizeof(float2), stream, c.tasks_z2, c.twiddles, c.half, c.real_grid);
  if (c.n_tasks_z > 0)
    launch_kernel(c.chain_pme, k_fft_z_c2r, c.n_tasks_z, 256, 0, stream, c.tasks_z, c.sys, c.fft_plans, c.twiddles,
                  c.half, c.real_grid);
}

// Planes of at most this many points go to one block each. A block's plane is one serial
// chain, so larger grids run faster shared by a cluster; a batch's small grids fill the GPU with
// one block a plane already (the line between the two was measured with the Stockham passes: one
// block a plane at 64^3 0.071 ms for the reciprocal kernels against 0.056 ms in a cluster, and a
// cluster a plane for 64 grids of 22^3-50^3 0.375 against 0.30 ms).
constexpr long long PLANE_SINGLE_MAX = 52 * 52;

// A block's shared buffers for a plane of a system: its rows, and (in a cluster) its columns.
void fft_plane_buffers(int nx, int ny, int split, int *rows, int *cols) {
  int r1 = 1, r2 = 1;
  fft_two_factors(ny, &r1, &r2);
  *rows = (nx + split - 1) / split * r1 * (r2 | 1);
  *cols = split > 1 ? (ny + split - 1) / split * nx : 0;
}

// Threads that share a plane block's steps: one a DFT of the widest step, within the block limit.
int fft_plane_threads(int nx, int ny, int split) {
  int r1x = 1, r2x = 1, r1y = 1, r2y = 1;
  fft_two_factors(nx, &r1x, &r2x);
  fft_two_factors(ny, &r1y, &r2y);
  const int items = std::max((nx + split - 1) / split * std::max(r1y, r2y), (ny + split - 1) / split * std::max(r1x, r2x));
  // (a cluster's blocks: two rounds when there are more than 256, so that two blocks share an SM)
  const int threads = split > 1 && items > 256 ? (items + 1) / 2 : items;
  return std::min(FFT_PLANE_THREADS, std::max(64, (threads + 31) / 32 * 32));
}

// The rule depends on the system alone, so a system takes the same pass in a batch as alone.
// Planes up to PLANE_SINGLE_MAX points: one block; larger ones a cluster while a block's quarter
// of the rows and of the columns stays within PLANE_QUARTER_MAX points (128 x 128 and a little
// beyond; the largest rows and the largest columns of different systems in one launch still fit
// a block's shared memory together); larger planes and axes without two factors: separate passes.
constexpr int PLANE_QUARTER_MAX = 6400;
static bool plane_axis(int n) {
  int r1, r2, rest = n;
  for (int p : {2, 3, 5})
    while (rest > 0 && rest % p == 0) rest /= p;
  // (an axis that is not 5-smooth is on no grid: the rule answers for its size alone)
  return n >= 1 && n <= FFT_TWO_MAX && (rest != 1 || fft_two_factors(n, &r1, &r2));
}
int fft_plane_split(int nx, int ny) {
  if (!plane_axis(nx) || !plane_axis(ny)) return 0;
  if ((long long)nx * ny <= PLANE_SINGLE_MAX) return 1;
  if (nx < PLANE_CLUSTER || ny < PLANE_CLUSTER) return 0;
  const int rows_per = (nx + PLANE_CLUSTER - 1) / PLANE_CLUSTER, cols_per = (ny + PLANE_CLUSTER - 1) / PLANE_CLUSTER;
  return rows_per * (ny + 1) <= PLANE_QUARTER_MAX && cols_per * (nx + 1) <= PLANE_QUARTER_MAX ? PLANE_CLUSTER : 0;
}

// The largest dynamic shared memory the plane kernels may take, set once per device before any
// launch (and never lowered, so engines with different grids cannot undercut each other).
cudaError_t fft_plane_prepare() {
  const void *fns[4] = {(const void *)k_fft_planes<true, RADIX_SMALL>, (const void *)k_fft_planes<false, RADIX_SMALL>,
                        (const void *)k_fft_planes<true, RADIX_ALL>, (const void *)k_fft_planes<false, RADIX_ALL>};
  for (const void *f : fns) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FFT_PLANE_SMEM_MAX);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

static void launch_planes(const LaunchCtx &c, bool energy, cudaStream_t stream) {
  // partials after the x tasks': the planes' one each, then the clusters' PLANE_CLUSTER each
  double *e = c.e_pme + c.n_tasks_x, *ev = c.e_pme_vir + c.n_tasks_x;
  auto launch = [&](int cl, const FftPlaneTask *tasks, int n, int threads, int rows, int cols) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n * cl);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = ((size_t)rows + cols) * sizeof(float2);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = c.chain_pme ? 2 : 1;
    auto kernel = c.planes_large ? (energy ? k_fft_planes<true, RADIX_ALL> : k_fft_planes<false, RADIX_ALL>)
                                 : (energy ? k_fft_planes<true, RADIX_SMALL> : k_fft_planes<false, RADIX_SMALL>);
    (void)cudaLaunchKernelEx(&cfg, kernel, tasks, (const DevSys *)c.sys, c.twiddles, c.moduli, c.half, cl, rows, e, ev);
  };
  if (c.n_tasks_plane > 0) launch(1, c.tasks_plane, c.n_tasks_plane, c.plane_threads, c.plane_stride, 0);
  e += c.n_tasks_plane;
  ev += c.n_tasks_plane;
  if (c.n_tasks_cluster > 0)
    launch(PLANE_CLUSTER, c.tasks_cluster, c.n_tasks_cluster, c.cluster_threads, c.cluster_rows, c.cluster_cols);
}

int pme_launches(const LaunchCtx &c) {
  if (!c.pme_on) return 0;
  return 2 + 2 * ((c.n_tasks_z > 0 ? 1 : 0) + (c.n_tasks_z2 > 0 ? 1 : 0)) + (c.n_tasks_plane > 0 ? 1 : 0) + (c.n_tasks_cluster > 0 ? 1 : 0) + (c.n_tasks_x > 0 ? 3 : 0);
}

// Everything up to the convolved real grid: spreading, forward transform, convolution (and
// energy), inverse transform.
static void launch_transform_convolve(const LaunchCtx &c, bool energy, cudaStream_t stream) {
  launch_forward_zy(c, stream);
  launch_planes(c, energy, stream);
  if (c.n_tasks_x > 0)
    launch_kernel(c.chain_pme, energy ? k_fft_x_convolve<true> : k_fft_x_convolve<false>, c.n_tasks_x, 256, 0, stream,
                   c.tasks_x, c.sys, c.fft_plans, c.twiddles, c.moduli, c.half, c.e_pme, c.e_pme_vir);
  launch_inverse_yz(c, stream);
}

void launch_pme_grid(const LaunchCtx &c, bool energy, cudaStream_t stream) {
  if (!c.pme_on) return;
  launch_spread_only(c, stream);
  launch_transform_convolve(c, energy, stream);
}

void launch_pme_gather(const LaunchCtx &c, cudaStream_t stream) {
  if (c.pme_on) launch_gather(c, stream);
}

void launch_pme(const LaunchCtx &c, bool energy, cudaStream_t stream) {
  if (!c.pme_on) return;
  launch_spread_only(c, stream);
  launch_transform_convolve(c, energy, stream);
  launch_gather(c, stream);
}

// Debug: forward R2C then C2R of a given real grid (already in real_grid as f32 values
// converted to fixed point by the caller), without the convolution. Used to check the FFT
// against a DFT.
__global__ void k_fft_x_plain(const FftTask *__restrict__ tasks, const DevSys *__restrict__ sys,
                              const FftPlan *__restrict__ plans, const float2 *__restrict__ twiddles,
                              float2 *__restrict__ half, int inverse) {
  __shared__ float2 bufa[FFT_SMEM], bufb[FFT_SMEM];
  const FftTask t = tasks[blockIdx.x];
  const DevSys &s = sys[t.sys];
  const FftPlan &pl = plans[t.sys];
  const int nx = s.grid[0], ny = s.grid[1], M = t.count;
  float2 *h = half + s.half_base + (long long)t.fixed * nx * ny + t.first;
  const int ld = nx + 1;
  for (int idx = threadIdx.x; idx < nx * M; idx += blockDim.x) {
    const int x = idx / M, m = idx - x * M;
    bufa[m * ld + x] = h[(long long)x * ny + m];
  }
  float2 *r = fft_lines(bufa, bufb, M, nx, ld, pl.axis[0], twiddles + pl.axis[0].tw_base, inverse != 0);
  for (int idx = threadIdx.x; idx < nx * M; idx += blockDim.x) {
    const int x = idx / M, m = idx - x * M;
    h[(long long)x * ny + m] = r[m * ld + x];
  }
}

void launch_spread_only(const LaunchCtx &c, cudaStream_t stream) {
  const int n = c.n_atoms;
  const int per_block = c.spread_atoms > 0 ? c.spread_atoms : 8;
  const int blocks = (n + per_block - 1) / per_block;
  if (c.pme_order == 4)
    launch_kernel(c.chain_pme, k_spread<4>, blocks, per_block * 16, 0, stream, c.posq, c.sys_of_atom, c.sys,
                  c.fixed_grid, n);
  else
    launch_kernel(c.chain_pme, k_spread<5>, blocks, per_block * 25, 0, stream, c.posq, c.sys_of_atom, c.sys,
                  c.fixed_grid, n);
}

// (the debug transforms run the separate passes over every system)
void launch_fft_forward(const LaunchCtx &c, cudaStream_t stream) {
  launch_forward_zy(c, stream, true);
  k_fft_x_plain<<<c.n_tasks_x_all, 256, 0, stream>>>(c.tasks_x_all, c.sys, c.fft_plans, c.twiddles, c.half, 0);
}

void launch_fft_inverse(const LaunchCtx &c, cudaStream_t stream) {
  k_fft_x_plain<<<c.n_tasks_x_all, 256, 0, stream>>>(c.tasks_x_all, c.sys, c.fft_plans, c.twiddles, c.half, 1);
  launch_inverse_yz(c, stream, true);
}

}  // namespace rmd
