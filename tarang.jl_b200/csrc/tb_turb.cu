// 2D decaying turbulence in FP32: vorticity q with streamfunction psi and
// velocity u = skew(grad psi), DiagonalIMEX_SBDF2 (examples/
// 2d_decaying_turbulence_gpu.jl; src/core/timesteppers/step_diagonal_imex.jl).
//
// Coefficients q^(kx, ky): rfft along x (kx = 0..Nx/2, Nyquist +Nx/2), fft
// along y in FFT order (ky = 0..Ny/2-1, -Ny/2..-1), unnormalised
// (basis_wavenumbers.jl:68-108).  Stored on the device transposed,
// [kx][ky] with ky fastest, so that the y transforms read whole columns.
//
// One RHS  F = -(u d_x q + v d_y q)  follows the reference's chain:
//   psi^ = -q^/k^2 (0 at k = 0)                  state_utils.jl:1059-1075
//   u^ = -i ky psi^, v^ = i kx psi^, d_x q^ = i kx q^, d_y q^ = i ky q^
//                                                lazy_rhs.jl:1190-1238
//   grid round trip of each factor: the kx = 0 and kx = Nx/2 columns lose
//   their non-Hermitian part in ky (irfft drops Im of DC and Nyquist)
//   3/2 padding in x and y with the even-N Nyquist split X/2 at +-N/2, product
//   on the padded grid, forward transform, fold of the -N/2 images into +N/2
//   and truncation                                nonlinear_padding.jl:182-443
// DiagonalIMEX_SBDF2 (step_diagonal_imex.jl:674-689, constant dt, L^ = nu k^2):
//   first step  q1 = (q0 + dt F0) / (1 + dt L^)
//   then        q_{n+1} = (2 q_n - q_{n-1}/2 + dt (2 F_n - F_{n-1})) / (3/2 + dt L^)
// DiagonalIMEX_RK222 / RK443 (_step_diagonal_imex_rk_impl!,
// step_diagonal_imex.jl:183-296; the full ESDIRK tableau, types.jl:511-620):
//   Y_s = q_n + dt sum_{j<s} (AE_sj F_j - AI_sj L^ Y_j),  Y_s /= 1 + dt AI_ss L^
//   F_s = RHS(Y_s);  q_{n+1} = q_n + dt sum_s (bE_s F_s - bI_s L^ Y_s)
// (a stage RHS whose weights are all zero, the first stage's, is skipped).
//
// Kernels of one right-hand side: k_turb_yinv (groups of kx columns: derived
// fields, projection, y padding, inverse FFT along y, written as rows over
// kx), k_turb_xpass (pairs of padded y rows: packed inverse real FFTs along x,
// products, one packed forward FFT, x truncation), k_turb_yfwd (groups of kx
// columns: forward FFT along y, folds, truncation, and the SBDF update or the
// next RK stage combination).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "tb_fftr.cuh"
#include "tb_internal.h"
#include "tb_plan.h"
#include "tb_turb.h"

using namespace tb;
namespace F = tb::fftg;
namespace Rp = tb::fftr;

struct tb_turb {
  tb_context* ctx = nullptr;
  int Nx = 0, Ny = 0, Mx = 0, My = 0, Kx = 0, Kp = 0;  // Kp: Kx rounded up to whole 32-byte sectors
  double Lx = 0, Ly = 0, nu = 0;
  RPlan rx, ry;            // in-place passes of the Mx and My transforms
  cudaStream_t st = nullptr;
  DevBuf Q[2], Fb;         // q_n / q_{n-1} (roles alternate), F_{n-1} (updated in place); [Kx][Ny] complex64
  DevBuf mix;              // 4 x [My][Kp]: u, v, d_x q, d_y q (and the staging of state copies)
  DevBuf pm;               // [My][Kp]: the products, x truncated
  DevBuf twx, twy, posy;   // twiddles of the Mx and My passes, digit-reversed positions of the My transform
  // DiagonalIMEX RK (rk true): tableau and per-stage states / right-hand sides
  bool rk = false;
  int stages = 0;
  double AE[4][4] = {}, AI[4][4] = {}, bE[4] = {}, bI[4] = {};
  bool f_used[4] = {};
  DevBuf Ys[4], Fs[4];     // Y_s (s >= 1; Y_0 is q_n) and F_s where used
  int cur = 0;             // Q[cur] holds q_n
  long long iteration = 0;
  double graph_dt = -1.0;
  cudaGraphExec_t g[2] = {nullptr, nullptr};  // steady step with q_n in Q[0] / Q[1]

  ~tb_turb() {
    for (auto& e : g)
      if (e) cudaGraphExecDestroy(e);
    if (st) cudaStreamDestroy(st);
  }
};

namespace {

constexpr int kTurbThreads = 256;

struct TurbArgs {
  int Nx, Ny, Mx, My, Kx, Kp;
  float kx0, ky0, nu;
  RPlan rx, ry;
  const float2* twx;
  const float2* twy;
  const unsigned short* posy;  // position of y mode / row i after the dif passes
};

__device__ __forceinline__ float ky_of(int ky, int Ny) { return (float)(ky < Ny / 2 ? ky : ky - Ny); }

// Stage combination of the diagonal IMEX RK step over [kx][ky]:
//   out = (base + sum_t w_t (L^ if isL_t) src_t) / (1 + dgam L^),  L^ = nu k^2.
constexpr int kCombMax = 8;
struct TurbComb {
  const float2* base;
  const float2* src[kCombMax];
  float w[kCombMax];
  int isL[kCombMax];
  int n;
  float dgam;
  float2* out;
};

__device__ __forceinline__ float2 combine_terms(const TurbComb& c, size_t e, float L) {
  float2 acc = c.base[e];
#pragma unroll
  for (int t = 0; t < kCombMax; ++t) {
    if (t < c.n) {
      const float2 v = c.src[t][e];
      const float wt = c.isL[t] ? c.w[t] * L : c.w[t];
      acc = F::mk<float2>(fmaf(wt, v.x, acc.x), fmaf(wt, v.y, acc.y));
    }
  }
  return acc;
}
__device__ __forceinline__ float2 combine_scale(const TurbComb& c, float2 acc, float L) {
  if (c.dgam == 0.f) return acc;
  const float den = 1.0f / (1.0f + c.dgam * L);
  return F::mk<float2>(acc.x * den, acc.y * den);
}

__global__ void __launch_bounds__(256) k_turb_combine(TurbArgs a, TurbComb c) {
  const size_t total = (size_t)a.Kx * a.Ny;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int kx = (int)(e / a.Ny), ky = (int)(e % a.Ny);
    const float kxv = a.kx0 * kx, kyv = a.ky0 * ky_of(ky, a.Ny);
    const float L = a.nu * (kxv * kxv + kyv * kyv);
    c.out[e] = combine_scale(c, combine_terms(c, e, L), L);
  }
}

// Column buffers of the y kernels: entry i of column c at c * ystride + sw(i);
// four extra entries a column put the same entry of neighbouring columns on
// different banks.
__host__ __device__ inline int ystride(int My) { return Rp::rpad<float2>(My) + 4; }

// One factor (blockIdx.y: 0 u, 1 v, 2 d_x q, 3 d_y q) of CW kx columns, with the
// grid round trip's projection, the x Nyquist split and the y padding, inverse
// FFT along y; out: mix[f][y][kx].  The columns of a group share the passes'
// barriers and their rows are stored together (32 bytes at CW = 4), which
// replaces a separate transpose.  At 1024x1024 bound by issue and latency (58 %
// of the issue slots, shared-memory wavefronts 25 % of their peak; most waits
// are for global loads).
template <int CW, int BL>
__global__ void __launch_bounds__(kTurbThreads, BL) k_turb_yinv(TurbArgs a, const float2* __restrict__ q,
                                                               float2* __restrict__ mix) {
  extern __shared__ __align__(16) float2 sm[];
  const int My = a.My, Ny = a.Ny, kx0 = blockIdx.x * CW, f = blockIdx.y;
  const int Ms = ystride(My), hy = Ny / 2;
  float2* tw = sm + CW * Ms;
  for (int t = threadIdx.x; t < a.ry.ntw; t += blockDim.x) tw[t] = a.twy[t];
  for (int t = threadIdx.x; t < CW * Ny; t += blockDim.x) {
    const int c = t / Ny, ky = t - c * Ny, kx = kx0 + c;
    if (kx >= a.Kx) break;
    const float kxv = a.kx0 * kx, kyv = a.ky0 * ky_of(ky, Ny);
    float2 v = q[(size_t)kx * Ny + ky];
    // the kx = 0 / Nyquist columns lose their non-Hermitian part in the grid
    // round trip, before any derivative is taken
    if (kx == 0 || 2 * kx == a.Nx) {
      const float2 w = q[(size_t)kx * Ny + (ky ? Ny - ky : 0)];
      v = F::mk<float2>(0.5f * (v.x + w.x), 0.5f * (v.y - w.y));
    }
    if (f < 2) {  // psi = -q / k^2, 0 at k = 0
      const float k2 = kxv * kxv + kyv * kyv;
      v = k2 > 1e-12f ? F::mk<float2>(-v.x / k2, -v.y / k2) : F::mk<float2>(0.f, 0.f);
    }
    const float d = (f == 0) ? -kyv : (f == 3 ? kyv : kxv);  // u = -i ky psi, v = i kx psi, i kx q, i ky q
    const float xs = (2 * kx == a.Nx) ? 0.5f : 1.0f;         // even-N Nyquist split along x
    v = F::mk<float2>(-(d * v.y) * xs, (d * v.x) * xs);
    float2* col = sm + c * Ms;
    if (ky < hy) {
      col[Rp::sw<float2>(ky)] = v;
    } else if (ky == hy) {
      v = F::scale(v, 0.5f);
      col[Rp::sw<float2>(hy)] = v;
      col[Rp::sw<float2>(My - hy)] = v;
    } else {
      col[Rp::sw<float2>(My - Ny + ky)] = v;
    }
  }
  const int gap = My - Ny - 1;  // y bins hy + 1 .. My - hy - 1 are zero
  for (int t = threadIdx.x; t < gap; t += blockDim.x)
#pragma unroll
    for (int c = 0; c < CW; ++c) sm[c * Ms + Rp::sw<float2>(hy + 1 + t)] = F::mk<float2>(0.f, 0.f);
  __syncthreads();
  for (int s = 0; s < a.ry.np; ++s) {
    Rp::pass_any<true, 1>(sm, CW, Ms, a.ry, s, tw);
    __syncthreads();
  }
  float2* out = mix + (size_t)f * My * a.Kp + kx0;
  for (int t = threadIdx.x; t < CW * My; t += blockDim.x) {
    const int c = t % CW, y = t / CW;
    if (kx0 + c < a.Kx) out[(size_t)y * a.Kp + c] = sm[c * Ms + Rp::sw<float2>(a.posy[y])];
  }
}

// Products u d_x q + v d_y q of two padded y rows (y0, y0 + 1): u + i v and
// d_x q + i d_y q of each row to the padded x grid (four arrays), the products
// of the rows as one complex array forward, bins 0..Nx/2 of both out.  The last
// inverse pass, the product and the first forward pass stay in registers.
template <int R>
__device__ __forceinline__ void xmiddle(float2* __restrict__ A, int Ms, int n) {
  for (int b = threadIdx.x; b < n / R; b += blockDim.x) {
    int at[R];
#pragma unroll
    for (int r = 0; r < R; ++r) at[r] = Rp::sw<float2>(b * R + r);
    float2 u[R], g[R], z[R];
#pragma unroll
    for (int row = 0; row < 2; ++row) {
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = A[(2 * row) * Ms + at[r]];
      Rp::dft<R, 1>(u);
#pragma unroll
      for (int r = 0; r < R; ++r) g[r] = A[(2 * row + 1) * Ms + at[r]];
      Rp::dft<R, 1>(g);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float p = u[r].x * g[r].x + u[r].y * g[r].y;
        if (row)
          z[r].y = p;
        else
          z[r].x = p;
      }
    }
    Rp::dft<R, -1>(z);
#pragma unroll
    for (int r = 0; r < R; ++r) A[at[r]] = z[r];
  }
}

template <int BL>
__global__ void __launch_bounds__(kTurbThreads, BL) k_turb_xpass(TurbArgs a, const float2* __restrict__ mix,
                                                                float2* __restrict__ pm) {
  extern __shared__ __align__(16) float2 sm[];
  const int Mx = a.Mx, hN = a.Nx / 2, y0 = 2 * blockIdx.x;
  const int Ms = Rp::rpad<float2>(Mx);
  float2* tw = sm + 4 * Ms;
  for (int t = threadIdx.x; t < a.rx.ntw; t += blockDim.x) tw[t] = a.twx[t];
  const size_t plane = (size_t)a.My * a.Kp;
  const float2* in = mix + (size_t)y0 * a.Kp;
  for (int k = threadIdx.x; k <= hN; k += blockDim.x) {
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = in[(size_t)(i % 4) * plane + (size_t)(i / 4) * a.Kp + k];
    if (k == 0 || k == hN)  // DC and Nyquist kept real, as the factor's own irfft on Nx points does
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i].y = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // array 2 row + pair: spectrum of first + i second
      const float2 P = v[2 * i], Q = v[2 * i + 1];
      sm[i * Ms + Rp::sw<float2>(k)] = F::mk<float2>(P.x - Q.y, P.y + Q.x);
      if (k > 0) sm[i * Ms + Rp::sw<float2>(Mx - k)] = F::mk<float2>(P.x + Q.y, -P.y + Q.x);
    }
  }
  for (int k = hN + 1 + threadIdx.x; k < Mx - hN; k += blockDim.x)
#pragma unroll
    for (int i = 0; i < 4; ++i) sm[i * Ms + Rp::sw<float2>(k)] = F::mk<float2>(0.f, 0.f);
  __syncthreads();
  const int last = a.rx.np - 1;
  for (int s = 0; s < last; ++s) {
    Rp::pass_any<true, 1>(sm, 4, Ms, a.rx, s, tw);
    __syncthreads();
  }
  switch (a.rx.R[last]) {
    case 8: xmiddle<8>(sm, Ms, Mx); break;
    case 6: xmiddle<6>(sm, Ms, Mx); break;
    case 4: xmiddle<4>(sm, Ms, Mx); break;
    case 3: xmiddle<3>(sm, Ms, Mx); break;
    default: xmiddle<2>(sm, Ms, Mx); break;
  }
  __syncthreads();
  for (int s = last - 1; s >= 0; --s) {
    Rp::pass_any<false, -1>(sm, 1, Ms, a.rx, s, tw);
    __syncthreads();
  }
  float2* out = pm + (size_t)y0 * a.Kp;
  for (int k = threadIdx.x; k <= hN; k += blockDim.x) {
    const float2 c = sm[Rp::sw<float2>(k)], w = sm[Rp::sw<float2>(k ? Mx - k : 0)];
    out[k] = F::mk<float2>(0.5f * (c.x + w.x), 0.5f * (c.y - w.y));
    out[a.Kp + k] = F::mk<float2>(0.5f * (c.y + w.y), -0.5f * (c.x - w.x));
  }
}

// CW kx columns: forward FFT along y, the Nyquist folds and truncation to Ny,
// F = -(...) / (Nx Ny Mx My), then
//   mode 0 SBDF2 / 1 SBDF1: the update; qn: q_n [Kx][Ny], qo: q_{n-1} on entry
//          and q_{n+1} on exit, Fp: F_{n-1} on entry and F_n on exit;
//   mode 2 an RK stage: F_s to Fp (null: no later stage reads it) and the next
//          combination c with the term wF F_s added (the stage's own right-hand
//          side never makes a round trip through memory).
template <int CW>
__global__ void __launch_bounds__(kTurbThreads, 3) k_turb_yfwd(TurbArgs a, const float2* __restrict__ pm,
                                                               const float2* __restrict__ qn, float2* __restrict__ qo,
                                                               float2* __restrict__ Fp, float dt, int mode, TurbComb c,
                                                               float wF) {
  extern __shared__ __align__(16) float2 sm[];
  const int My = a.My, Ny = a.Ny, kx0 = blockIdx.x * CW, hy = Ny / 2;
  const int Ms = ystride(My);
  float2* tw = sm + CW * Ms;
  for (int t = threadIdx.x; t < a.ry.ntw; t += blockDim.x) tw[t] = a.twy[t];
  for (int t = threadIdx.x; t < CW * My; t += blockDim.x) {  // columns past Kx read the row padding
    const int cc = t % CW, y = t / CW;
    sm[cc * Ms + Rp::sw<float2>(y)] = pm[(size_t)y * a.Kp + kx0 + cc];
  }
  __syncthreads();
  for (int s = 0; s < a.ry.np; ++s) {
    Rp::pass_any<true, -1>(sm, CW, Ms, a.ry, s, tw);
    __syncthreads();
  }
  const float sc = -1.0f / ((float)a.Nx * (float)Ny * (float)a.Mx * (float)My);
  for (int t = threadIdx.x; t < CW * Ny; t += blockDim.x) {
    const int cc = t / Ny, ky = t - cc * Ny, kx = kx0 + cc;
    if (kx >= a.Kx) break;
    const bool xnyq = 2 * kx == a.Nx;
    // Q'(y) with the x fold: Q(Nx/2, y) + conj(Q(Nx/2, -y))
    auto qf = [&](int yy) -> float2 {
      float2 v = sm[cc * Ms + Rp::sw<float2>(a.posy[yy])];
      if (xnyq) {
        const float2 w = sm[cc * Ms + Rp::sw<float2>(a.posy[yy ? My - yy : 0])];
        v = F::mk<float2>(v.x + w.x, v.y - w.y);
      }
      return v;
    };
    float2 r = qf(ky <= hy ? ky : My - Ny + ky);
    if (ky == hy) r = F::add(r, qf(My - hy));
    const float2 Fn = F::scale(r, sc);
    const size_t e = (size_t)kx * Ny + ky;
    const float kxv = a.kx0 * kx, kyv = a.ky0 * ky_of(ky, Ny);
    const float L = a.nu * (kxv * kxv + kyv * kyv);
    if (mode == 2) {
      if (Fp) Fp[e] = Fn;
      float2 acc = combine_terms(c, e, L);
      acc = F::mk<float2>(fmaf(wF, Fn.x, acc.x), fmaf(wF, Fn.y, acc.y));
      c.out[e] = combine_scale(c, acc, L);
      continue;
    }
    const float2 q0 = qn[e];
    float2 q1;
    if (mode == 1) {
      const float den = 1.0f / (1.0f + dt * L);
      q1 = F::mk<float2>((q0.x + dt * Fn.x) * den, (q0.y + dt * Fn.y) * den);
    } else {
      const float2 qm = qo[e], Fm = Fp[e];
      const float den = 1.0f / (1.5f + dt * L);
      q1 = F::mk<float2>((2.0f * q0.x - 0.5f * qm.x + dt * (2.0f * Fn.x - Fm.x)) * den,
                         (2.0f * q0.y - 0.5f * qm.y + dt * (2.0f * Fn.y - Fm.y)) * den);
    }
    qo[e] = q1;
    Fp[e] = Fn;
  }
}

// State copies: the device's [kx][ky] FP32 coefficients <-> the caller's layout
// (ky rows of Kx complex128), 32 x 32 tiles.
template <bool OUT>
__global__ void __launch_bounds__(256) k_turb_state(float2* __restrict__ q, double2* __restrict__ pub, int Kx, int Ny) {
  __shared__ float2 tile[32][33];
  const int kx0 = blockIdx.x * 32, ky0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += 8) {
    if (OUT) {
      const int kx = kx0 + i, ky = ky0 + threadIdx.x;
      if (kx < Kx && ky < Ny) tile[i][threadIdx.x] = q[(size_t)kx * Ny + ky];
    } else {
      const int ky = ky0 + i, kx = kx0 + threadIdx.x;
      if (kx < Kx && ky < Ny) {
        const double2 v = pub[(size_t)ky * Kx + kx];
        tile[i][threadIdx.x] = make_float2((float)v.x, (float)v.y);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += 8) {
    if (OUT) {
      const int ky = ky0 + i, kx = kx0 + threadIdx.x;
      if (kx < Kx && ky < Ny) {
        const float2 v = tile[threadIdx.x][i];
        pub[(size_t)ky * Kx + kx] = make_double2(v.x, v.y);
      }
    } else {
      const int kx = kx0 + i, ky = ky0 + threadIdx.x;
      if (kx < Kx && ky < Ny) q[(size_t)kx * Ny + ky] = tile[threadIdx.x][i];
    }
  }
}

size_t y_smem(const tb_turb* T, int cw) { return ((size_t)cw * ystride(T->My) + T->ry.ntw) * sizeof(float2); }
size_t x_smem(const tb_turb* T) { return (4 * (size_t)Rp::rpad<float2>(T->Mx) + T->rx.ntw) * sizeof(float2); }

// kx columns a block: four store and load whole 32-byte sectors, but few
// columns leave SMs idle, so the widest that still gives 1.5 blocks an SM.
int columns_per_block(int Kx, int factors) {
  for (int cw : {4, 2})
    if ((Kx + cw - 1) / cw * factors >= 222) return cw;
  return 1;
}

// Whether a kernel runs its build for four blocks of kTurbThreads an SM (64
// registers, 28 to 72 bytes of spills) instead of three (78): where the grid is
// more than three blocks an SM can hold at once and shared memory has room for
// four. At 1024x1024 the 516 blocks of the inverse y transforms are then one
// wave and not one and a sixth (10 RK443 steps 4452 -> 4115 us; the forward kernel,
// whose blocks all fit at once, has the one build); at 256x256, where a wave
// holds every block, the spills cost 4 %.
bool four_blocks(int blocks, int threads, size_t smem) {
  return (long long)blocks * threads > 3LL * 148 * kTurbThreads && 4 * (smem + 1024) <= 228 * 1024;
}

TurbArgs args_of(const tb_turb* T) {
  TurbArgs a{};
  a.Nx = T->Nx;
  a.Ny = T->Ny;
  a.Mx = T->Mx;
  a.My = T->My;
  a.Kx = T->Kx;
  a.Kp = T->Kp;
  a.kx0 = (float)(2.0 * M_PI / T->Lx);
  a.ky0 = (float)(2.0 * M_PI / T->Ly);
  a.nu = (float)T->nu;
  a.rx = T->rx;
  a.ry = T->ry;
  a.twx = T->twx.as<float2>();
  a.twy = T->twy.as<float2>();
  a.posy = T->posy.as<unsigned short>();
  return a;
}

// The RHS chain on q, ending in k_turb_yfwd with its mode (see there).
void enqueue_rhs(tb_turb* T, const float2* q, float2* qo, float2* Fp, double dt, int mode, const TurbComb& c,
                 double wF) {
  const TurbArgs a = args_of(T);
  float2* mix = T->mix.as<float2>();
  float2* pm = T->pm.as<float2>();
  // about one butterfly of radix 8 a thread
  auto threads = [](int arrays, int n) { return arrays * n <= 1024 ? kTurbThreads / 2 : kTurbThreads; };
  const int ci = columns_per_block(T->Kx, 4), cf = columns_per_block(T->Kx, 1);
  const int bi = (T->Kx + ci - 1) / ci * 4, bx = T->My / 2, ti = threads(ci, T->My), tx = threads(4, T->Mx);
  const bool i4 = four_blocks(bi, ti, y_smem(T, ci)), x4 = four_blocks(bx, tx, x_smem(T));
  auto yinv = ci == 4   ? (i4 ? k_turb_yinv<4, 4> : k_turb_yinv<4, 3>)
              : ci == 2 ? (i4 ? k_turb_yinv<2, 4> : k_turb_yinv<2, 3>)
                        : (i4 ? k_turb_yinv<1, 4> : k_turb_yinv<1, 3>);
  auto xpass = x4 ? k_turb_xpass<4> : k_turb_xpass<3>;
  auto yfwd = cf == 4 ? k_turb_yfwd<4> : cf == 2 ? k_turb_yfwd<2> : k_turb_yfwd<1>;
  yinv<<<dim3(bi / 4, 4), ti, y_smem(T, ci), T->st>>>(a, q, mix);
  xpass<<<bx, tx, x_smem(T), T->st>>>(a, mix, pm);
  yfwd<<<(T->Kx + cf - 1) / cf, threads(cf, T->My), y_smem(T, cf), T->st>>>(a, pm, q, qo, Fp, (float)dt, mode, c,
                                                                            (float)wF);
}

void launch_combine(tb_turb* T, const TurbComb& c) {
  const size_t total = (size_t)T->Kx * T->Ny;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  k_turb_combine<<<blocks, 256, 0, T->st>>>(args_of(T), c);
}

// One DiagonalIMEX RK step from Q[cur] into Q[1 - cur].
void enqueue_rk_step(tb_turb* T, double dt) {
  float2* qn = T->Q[T->cur].as<float2>();
  float2* qo = T->Q[1 - T->cur].as<float2>();
  const float2* Y[4] = {qn, nullptr, nullptr, nullptr};
  auto add = [&](TurbComb& c, const float2* src, double w, int isL) {
    if (c.n >= kCombMax) throw Error{TB_EINVAL, "too many stage terms"};
    c.src[c.n] = src;
    c.w[c.n] = (float)w;
    c.isL[c.n] = isL;
    ++c.n;
  };
  const int s = T->stages;
  // the combination that gives stage i (i = s: q_{n+1}) without the term of its
  // newest right-hand side, whose weight goes to *w
  auto combination = [&](int i, double* w) {
    const double* wE = i < s ? T->AE[i] : T->bE;
    const double* wI = i < s ? T->AI[i] : T->bI;
    TurbComb c{};
    c.base = qn;
    for (int j = 0; j < i; ++j) {
      if (j < i - 1 && std::fabs(wE[j]) > 1e-14) add(c, T->Fs[j].as<float2>(), dt * wE[j], 0);
      if (std::fabs(wI[j]) > 1e-14) add(c, Y[j], -dt * wI[j], 1);
    }
    *w = dt * wE[i - 1];
    c.dgam = i < s && std::fabs(T->AI[i][i]) > 1e-14 ? (float)(dt * T->AI[i][i]) : 0.f;
    c.out = i < s ? T->Ys[i].as<float2>() : qo;
    return c;
  };
  for (int i = 0; i < s; ++i) {
    double w = 0.0;
    if (!T->f_used[i]) {  // no weight anywhere: the next combination stands alone
      launch_combine(T, combination(i + 1, &w));
    } else {
      const TurbComb c = combination(i + 1, &w);
      enqueue_rhs(T, Y[i], nullptr, T->Fs[i].as<float2>(), dt, 2, c, w);  // (null: not kept)
    }
    if (i + 1 < s) Y[i + 1] = T->Ys[i + 1].as<float2>();
  }
}

void enqueue_step(tb_turb* T, double dt, int first) {
  if (T->rk) {
    enqueue_rk_step(T, dt);
    return;
  }
  float2* qn = T->Q[T->cur].as<float2>();
  float2* qo = T->Q[1 - T->cur].as<float2>();
  enqueue_rhs(T, qn, qo, T->Fb.as<float2>(), dt, first, TurbComb{}, 0.0);
}

std::vector<float2> pass_table(const RPlan& p) {
  const std::vector<double> w = rplan_twiddles(p);
  std::vector<float2> t(w.size() / 2);
  for (size_t i = 0; i < t.size(); ++i) t[i] = make_float2((float)w[2 * i], (float)w[2 * i + 1]);
  return t;
}

int padded_len(int n) {
  int m = (int)std::ceil(1.5 * n);
  return (m % 2) ? m + 1 : m;
}

cudaGraphExec_t capture(tb_turb* T, double dt) {
  cudaGraph_t g = nullptr;
  TB_CUDA_TRY(cudaStreamBeginCapture(T->st, cudaStreamCaptureModeThreadLocal));
  enqueue_step(T, dt, 0);
  TB_CUDA_TRY(cudaStreamEndCapture(T->st, &g));
  cudaGraphExec_t ex = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) throw Error{TB_ECUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e)};
  return ex;
}

}  // namespace

size_t tb::turb_estimate_bytes(int Nx, int Ny, int timestepper) {
  const size_t Kx = Nx / 2 + 1, Kp = (Kx + 3) / 4 * 4, My = padded_len(Ny);
  // SBDF2: q_n, q_{n-1}, F_{n-1}; RK: q_n, q_{n+1} and up to 3 stage states
  // and 3 stage right-hand sides (4 stages, the first state and the last RHS not kept)
  const size_t specs = timestepper == TB_SBDF2 ? 3 : (timestepper == TB_RK222 ? 6 : 8);
  return sizeof(float2) * (specs * Kx * Ny + 5 * Kp * My) + (4u << 20);
}

tb_turb* tb::turb_create(tb_context* ctx, const tb_problem_desc& d, const double* q0) {
  TB_REQUIRE(d.program == TB_PROGRAM_TURB2D, TB_EINVAL, "not a turbulence descriptor");
  TB_REQUIRE(d.Nx >= 8 && d.Ny >= 8 && d.Nx % 2 == 0 && d.Ny % 2 == 0, TB_EINVAL, "Nx, Ny must be even and >= 8");
  TB_REQUIRE(d.Nx <= 2048 && d.Ny <= 2048, TB_ENOTSUPPORTED, "Nx, Ny above 2048");
  TB_REQUIRE(d.Lx > 0 && d.Ly > 0 && d.nu >= 0, TB_EINVAL, "bad lengths or viscosity");
  TB_REQUIRE(std::fabs(d.dealias - 1.5) < 1e-12, TB_ENOTSUPPORTED, "only dealias = 3/2 is implemented");
  TB_REQUIRE(q0 != nullptr, TB_EINVAL, "null initial vorticity");
  TB_REQUIRE(d.timestepper == TB_SBDF2 || d.timestepper == TB_RK222 || d.timestepper == TB_RK443, TB_ENOTSUPPORTED,
             "turbulence steps: DiagonalIMEX SBDF2, RK222 or RK443");
  auto T = std::make_unique<tb_turb>();
  if (d.timestepper != TB_SBDF2) {
    const Tableau tb_ = tableau(d.timestepper);
    T->rk = true;
    T->stages = tb_.s;
    for (int i = 0; i < tb_.s; ++i) {
      T->bE[i] = tb_.bE[i];
      T->bI[i] = tb_.bI[i];
      for (int j = 0; j < tb_.s; ++j) {
        T->AE[i][j] = tb_.AE[i][j];
        T->AI[i][j] = tb_.AI[i][j];
      }
    }
    // F_s is computed only where a later stage or the update weighs it
    for (int i = 0; i < tb_.s; ++i) {
      bool used = std::fabs(tb_.bE[i]) > 1e-14;
      for (int k = i + 1; k < tb_.s; ++k) used = used || std::fabs(tb_.AE[k][i]) > 1e-14;
      T->f_used[i] = used;
    }
  }
  T->ctx = ctx;
  T->Nx = d.Nx;
  T->Ny = d.Ny;
  T->Mx = padded_len(d.Nx);
  T->My = padded_len(d.Ny);
  T->Kx = d.Nx / 2 + 1;
  T->Lx = d.Lx;
  T->Ly = d.Ly;
  T->nu = d.nu;
  T->Kp = (T->Kx + 3) / 4 * 4;
  TB_REQUIRE(make_rplan(T->Mx, sizeof(float2), &T->rx, 5) && make_rplan(T->My, sizeof(float2), &T->ry, 2), TB_ENOTSUPPORTED,
             "Nx, Ny must be of the form 2^a 3^b");
  TB_CUDA_TRY(cudaSetDevice(ctx->device));
  TB_CUDA_TRY(create_work_stream(&T->st));
  const size_t spec = (size_t)T->Kx * T->Ny * sizeof(float2);
  for (auto& b : T->Q) b.alloc(spec);
  if (T->rk) {
    for (int i = 1; i < T->stages; ++i) T->Ys[i].alloc(spec);
    // F_i is kept only where a combination after the next one reads it
    for (int i = 0; i < T->stages; ++i) {
      bool later = i + 1 < T->stages && std::fabs(T->bE[i]) > 1e-14;
      for (int k = i + 2; k < T->stages; ++k) later = later || std::fabs(T->AE[k][i]) > 1e-14;
      if (later) T->Fs[i].alloc(spec);
    }
  } else {
    T->Fb.alloc(spec);
  }
  T->mix.alloc(4 * (size_t)T->My * T->Kp * sizeof(float2));
  T->pm.alloc((size_t)T->My * T->Kp * sizeof(float2));
  TB_CUDA_TRY(cudaMemsetAsync(T->pm.p, 0, T->pm.bytes, T->st));  // the row padding stays zero
  upload(T->twx, pass_table(T->rx));
  upload(T->twy, pass_table(T->ry));
  upload(T->posy, rplan_positions(T->ry));
  TB_REQUIRE(x_smem(T.get()) <= 227 * 1024 && y_smem(T.get(), 4) <= 227 * 1024, TB_ENOTSUPPORTED,
             "turbulence grid too large for the shared-memory transforms");
  for (const void* k : {(const void*)k_turb_yinv<1, 3>, (const void*)k_turb_yinv<2, 3>, (const void*)k_turb_yinv<4, 3>,
                        (const void*)k_turb_yinv<1, 4>, (const void*)k_turb_yinv<2, 4>, (const void*)k_turb_yinv<4, 4>,
                        (const void*)k_turb_xpass<3>, (const void*)k_turb_xpass<4>, (const void*)k_turb_yfwd<1>,
                        (const void*)k_turb_yfwd<2>, (const void*)k_turb_yfwd<4>})
    TB_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  turb_set(T.get(), q0);
  return T.release();
}

// Vorticity coefficients from the reference layout (Kx, Ny), x fastest, into
// Q[0] = q_n (device [kx][ky]); the step history restarts.  Everything runs on
// the plan's own (non-blocking) stream, so the next step is ordered after it.
void tb::turb_set(tb_turb* T, const double* q0) {
  const size_t spec = (size_t)T->Kx * T->Ny * sizeof(float2);
  double2* stage = T->mix.as<double2>();  // free between steps
  TB_CUDA_TRY(cudaMemcpyAsync(stage, q0, 2 * spec, cudaMemcpyHostToDevice, T->st));
  k_turb_state<false><<<dim3((T->Kx + 31) / 32, (T->Ny + 31) / 32), dim3(32, 8), 0, T->st>>>(T->Q[0].as<float2>(), stage,
                                                                                            T->Kx, T->Ny);
  TB_CUDA_TRY(cudaGetLastError());
  TB_CUDA_TRY(cudaMemsetAsync(T->Q[1].p, 0, spec, T->st));
  if (T->Fb.p) TB_CUDA_TRY(cudaMemsetAsync(T->Fb.p, 0, spec, T->st));
  TB_CUDA_TRY(cudaStreamSynchronize(T->st));
  T->cur = 0;
  T->iteration = 0;
}

void tb::turb_destroy(tb_turb* T) { delete T; }

cudaStream_t tb::turb_stream(const tb_turb* T) { return T->st; }

void tb::turb_prepare(tb_turb* T, double dt) {
  if (T->graph_dt == dt) return;
  TB_CUDA_TRY(cudaSetDevice(T->ctx->device));
  TB_CUDA_TRY(cudaStreamSynchronize(T->st));
  for (auto& e : T->g)
    if (e) cudaGraphExecDestroy(e), e = nullptr;
  const int keep = T->cur;
  for (int c = 0; c < 2; ++c) {
    T->cur = c;
    T->g[c] = capture(T, dt);
  }
  T->cur = keep;
  T->graph_dt = dt;
}

void tb::turb_launch_steps(tb_turb* T, double dt, int steps) {
  for (int i = 0; i < steps; ++i) {
    if (T->iteration == 0) {
      enqueue_step(T, dt, 1);
    } else {
      turb_prepare(T, dt);
      TB_CUDA_TRY(cudaGraphLaunch(T->g[T->cur], T->st));
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error{TB_ECUDA, std::string("turbulence step: ") + cudaGetErrorString(e)};
    T->cur = 1 - T->cur;
    T->iteration += 1;
  }
}

size_t tb::turb_device_bytes(const tb_turb* T) {
  size_t b = T->Q[0].bytes + T->Q[1].bytes + T->Fb.bytes + T->mix.bytes + T->pm.bytes + T->twx.bytes + T->twy.bytes +
             T->posy.bytes;
  for (int i = 0; i < 4; ++i) b += T->Ys[i].bytes + T->Fs[i].bytes;
  return b;
}

size_t tb::turb_field_doubles(const tb_turb* T) { return 2 * (size_t)T->Kx * T->Ny; }

void tb::turb_fetch(tb_turb* T, double* host) {
  double2* stage = T->mix.as<double2>();  // free between steps
  k_turb_state<true><<<dim3((T->Kx + 31) / 32, (T->Ny + 31) / 32), dim3(32, 8), 0, T->st>>>(T->Q[T->cur].as<float2>(),
                                                                                           stage, T->Kx, T->Ny);
  TB_CUDA_TRY(cudaGetLastError());
  TB_CUDA_TRY(cudaMemcpyAsync(host, stage, (size_t)T->Kx * T->Ny * sizeof(double2), cudaMemcpyDeviceToHost, T->st));
  TB_CUDA_TRY(cudaStreamSynchronize(T->st));
}

extern "C" {

tb_status tb_turb_create(tb_context* ctx, const tb_problem_desc* desc, const double* q0_spec, tb_turb** out) {
  if (!ctx || !desc || !out) return TB_EINVAL;
  *out = nullptr;
  return guarded(ctx, [&] { *out = turb_create(ctx, *desc, q0_spec); });
}

tb_status tb_turb_destroy(tb_turb* T) {
  if (!T) return TB_EINVAL;
  cudaStreamSynchronize(T->st);
  turb_destroy(T);
  return TB_OK;
}

tb_status tb_turb_step(tb_turb* T, double dt, int nsteps) {
  if (!T) return TB_EINVAL;
  return guarded(T->ctx, [&] {
    TB_REQUIRE(dt > 0 && std::isfinite(dt) && nsteps >= 0, TB_EINVAL, "dt must be positive, nsteps >= 0");
    TB_CUDA_TRY(cudaSetDevice(T->ctx->device));
    turb_launch_steps(T, dt, nsteps);
    TB_CUDA_TRY(cudaStreamSynchronize(T->st));
  });
}

tb_status tb_turb_set_vorticity(tb_turb* T, const double* host) {
  if (!T || !host) return TB_EINVAL;
  return guarded(T->ctx, [&] {
    TB_CUDA_TRY(cudaSetDevice(T->ctx->device));
    turb_set(T, host);
  });
}

tb_status tb_turb_get_vorticity(tb_turb* T, double* host) {
  if (!T || !host) return TB_EINVAL;
  return guarded(T->ctx, [&] { turb_fetch(T, host); });
}

}  // extern "C"
