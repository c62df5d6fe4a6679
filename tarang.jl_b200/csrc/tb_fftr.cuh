// In-place mixed-radix FFT passes in shared memory with radices up to 16, for
// batches of equal-length transforms (float2 or double2).
//
// A transform of length n = R_0 R_1 ... R_{p-1} is p passes over one buffer.
// Pass s works on blocks of L_s = n / (R_0 ... R_{s-1}) entries; a butterfly
// reads and writes the same R_s entries, m_s = L_s / R_s apart, so a pass needs
// one barrier and no second buffer.  Decimation in frequency (dif) takes
// natural order to digit-reversed order, decimation in time (dit) the reverse
// over the same radices, so an inverse dif transform, a pointwise product and
// a forward dit transform need no permutation.  The last pass has m = 1: its
// butterflies are runs of R_{p-1} neighbours without twiddles, which lets a
// kernel take the last inverse pass, the product and the first forward pass
// in registers (no shared-memory round trip between them).
//
// Why these radices: the transforms are bound by the instructions, the barrier
// and the shared-memory round trip of each pass (no unit is above 65 % of its
// peak), and all go with the number of passes.
// 1536 points are 3 passes of 12, 16 and 8 here, where radices of at most 8
// take 4.  make_rplan picks the sequence with the fewest shared-memory
// wavefronts (bank conflicts counted), plus a fixed charge per pass.
//
// Divisions by the (runtime) strides are multiplications by ceil(2^32 / d):
// exact for d <= 4096 and items below 2^20 (n <= 3072, at most 64 arrays).
#pragma once

#include <cuda_runtime.h>

#include "tb_chain.cuh"
#include "tb_fft.cuh"
#include "tb_internal.h"

namespace tb {
namespace fftr {

using fftg::add;
using fftg::mk;
using fftg::mul;
using fftg::Real;
using fftg::sub;

// Physical index of entry i: the low bits are XORed with the next ones over
// 128 bytes (8 double2, 16 float2), so unit-stride and stride-R accesses both
// spread over the banks.  Buffers are padded to whole groups (rpad).
template <class C>
__device__ __forceinline__ int sw(int i) {
  return fftg::sidx<C>(i);
}
template <class C>
__host__ __device__ constexpr int rpad(int n) {
  return (n + 15) & ~15;
}

// Products that are rounded on their own: without them the compiler may fuse a
// product into either of two sums, so that two instantiations of a kernel (rows
// a block) would round differently.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

__device__ __forceinline__ int fdiv(int x, unsigned magic) { return magic ? (int)__umulhi((unsigned)x, magic) : x; }

// v * exp(SIGN 2 pi i E / N), N in {6, 9, 12, 16}, 0 <= E < N
template <int N, int E, int SIGN, class C>
__device__ __forceinline__ C mulw(C v) {
  using T = typename Real<C>::type;
  if constexpr (E == 0) {
    return v;
  } else if constexpr (4 * E == N) {
    return SIGN > 0 ? mk<C>(-v.y, v.x) : mk<C>(v.y, -v.x);
  } else if constexpr (2 * E == N) {
    return mk<C>(-v.x, -v.y);
  } else {
    // cos and sin of 2 pi E / N
    constexpr double c[] = {
        // N = 16: E = 1, 2, 3, 4, 6, 9
        0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0, -0.70710678118654752440,
        -0.92387953251128675613,
        // N = 12: E = 1, 2, 4
        0.86602540378443864676, 0.5, -0.5,
        // N = 9: E = 1, 2, 4
        0.76604444311897803520, 0.17364817766693034885, -0.93969262078590838405,
        // N = 6: E = 1, 2
        0.5, -0.5};
    constexpr double s[] = {
        0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0, 0.70710678118654752440,
        -0.38268343236508977173,
        0.5, 0.86602540378443864676, 0.86602540378443864676,
        0.64278760968653932632, 0.98480775301220805937, 0.34202014332566873304,
        0.86602540378443864676, 0.86602540378443864676};
    constexpr int i = N == 16  ? (E == 1 ? 0 : E == 2 ? 1 : E == 3 ? 2 : E == 4 ? 3 : E == 6 ? 4 : E == 9 ? 5 : -1)
                      : N == 12 ? (E == 1 ? 6 : E == 2 ? 7 : E == 4 ? 8 : -1)
                      : N == 9  ? (E == 1 ? 9 : E == 2 ? 10 : E == 4 ? 11 : -1)
                                : (E == 1 ? 12 : E == 2 ? 13 : -1);
    static_assert(i >= 0, "twiddle not listed");
    constexpr T cc = (T)c[i], ss = (T)(SIGN > 0 ? s[i] : -s[i]);
    return mk<C>(v.x * cc - v.y * ss, v.x * ss + v.y * cc);
  }
}

template <int R, int SIGN, class C>
__device__ __forceinline__ void dft(C (&v)[R]);

// R1 R2 points as R2 transforms of length R1, twiddles, R1 transforms of R2
template <int R1, int R2, int SIGN, class C, int K1, int N2>
__device__ __forceinline__ void dft_twiddle(C (&y)[R1 * R2]) {
  if constexpr (K1 < R1) {
    y[K1 * R2 + N2] = mulw<R1 * R2, K1 * N2, SIGN>(y[K1 * R2 + N2]);
    if constexpr (N2 + 1 < R2)
      dft_twiddle<R1, R2, SIGN, C, K1, N2 + 1>(y);
    else
      dft_twiddle<R1, R2, SIGN, C, K1 + 1, 1>(y);
  }
}
template <int R1, int R2, int SIGN, class C>
__device__ __forceinline__ void dft_split(C (&x)[R1 * R2]) {
  C y[R1 * R2];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) {
    C a[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) a[n1] = x[R2 * n1 + n2];
    dft<R1, SIGN>(a);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) y[k1 * R2 + n2] = a[k1];
  }
  dft_twiddle<R1, R2, SIGN, C, 1, 1>(y);
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) {
    C b[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) b[n2] = y[k1 * R2 + n2];
    dft<R2, SIGN>(b);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) x[k1 + R1 * k2] = b[k2];
  }
}

// In-register DFT of length R (2, 3, 4, 6, 8, 9, 12, 16), natural order,
// exponent SIGN, unnormalised.
template <int R, int SIGN, class C>
__device__ __forceinline__ void dft(C (&v)[R]) {
  if constexpr (R == 2 || R == 3 || R == 4 || R == 8)
    fftg::dft_small<R>(v, SIGN);
  else if constexpr (R == 6)
    dft_split<2, 3, SIGN>(v);
  else if constexpr (R == 9)
    dft_split<3, 3, SIGN>(v);
  else if constexpr (R == 12)
    dft_split<4, 3, SIGN>(v);
  else
    dft_split<4, 4, SIGN>(v);
}

// v_r *= w^r, r < R, with w = w1; above radix 8 the powers are built from w1
// and w4 = w1^4 (both from the table), which keeps their error at that of at
// most three table entries a factor.
template <int R, class C>
__device__ __forceinline__ void powers(C (&v)[R], C w1, C w4) {
  if constexpr (R >= 2) v[1] = mul(v[1], w1);
  if constexpr (R >= 3) {
    const C w2 = mul(w1, w1);
    v[2] = mul(v[2], w2);
    if constexpr (R >= 4) {
      const C w3 = mul(w1, w2);
      v[3] = mul(v[3], w3);
      if constexpr (R >= 6) {
        if constexpr (R <= 8) w4 = mul(w2, w2);
        v[4] = mul(v[4], w4);
        v[5] = mul(v[5], mul(w1, w4));
        if constexpr (R >= 8) {
          v[6] = mul(v[6], mul(w2, w4));
          v[7] = mul(v[7], mul(w3, w4));
        }
        if constexpr (R >= 9) {
          const C w8 = mul(w4, w4);
          v[8] = mul(v[8], w8);
          if constexpr (R >= 12) {
            v[9] = mul(v[9], mul(w1, w8));
            v[10] = mul(v[10], mul(w2, w8));
            v[11] = mul(v[11], mul(w3, w8));
          }
          if constexpr (R >= 16) {
            const C w12 = mul(w4, w8);
            v[12] = mul(v[12], w12);
            v[13] = mul(v[13], mul(w1, w12));
            v[14] = mul(v[14], mul(w2, w12));
            v[15] = mul(v[15], mul(w3, w12));
          }
        }
      }
    }
  }
}

// One pass of radix R over NA arrays Ms apart (m > 1 or the last pass, m = 1).
// Twiddle table of the pass: exp(-2 pi i j / L) for j < m, then, above radix
// 8, exp(-2 pi i 4 j / L).
template <int R, bool DIF, int SIGN, class C>
__device__ __forceinline__ void pass(C* __restrict__ buf, int NA, int Ms, const RPlan& p, int s,
                                     const C* __restrict__ tw) {
  const int m = p.m[s], nb = p.n / R, total = NA * nb;
  const C* t = tw + p.tw[s];
  for (int item = threadIdx.x; item < total; item += blockDim.x) {
    const int arr = fdiv(item, p.db[s]), b = item - arr * nb;
    const int block = fdiv(b, p.dm[s]), j = b - block * m;
    C* x = buf + (size_t)arr * Ms;
    const int base = block * m * R + j;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = x[sw<C>(base + r * m)];
    C w1 = mk<C>(1, 0), w4 = mk<C>(1, 0);
    if (m > 1) {
      w1 = t[j];
      if constexpr (R > 8) w4 = t[m + j];
      if constexpr (SIGN > 0) {
        w1.y = -w1.y;
        w4.y = -w4.y;
      }
    }
    if constexpr (DIF) {
      dft<R, SIGN>(v);
      if (m > 1) powers<R>(v, w1, w4);
    } else {
      if (m > 1) powers<R>(v, w1, w4);
      dft<R, SIGN>(v);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) x[sw<C>(base + r * m)] = v[r];
  }
}

template <bool DIF, int SIGN, class C>
__device__ __forceinline__ void pass_any(C* buf, int NA, int Ms, const RPlan& p, int s, const C* tw) {
  switch (p.R[s]) {
    case 16: pass<16, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    case 12: pass<12, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    case 9: pass<9, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    case 8: pass<8, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    case 6: pass<6, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    case 4: pass<4, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    case 3: pass<3, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
    default: pass<2, DIF, SIGN>(buf, NA, Ms, p, s, tw); break;
  }
}

// Row products -(u . grad f), f = b, u_x, u_z, on the padded grid, per grid row
// z (and stacked instance y): the velocity spectrum and the three gradient
// spectra from one read of the six half-plane inputs, dif passes over the four
// arrays, the last inverse pass with the products and the first forward pass
// in registers, dit passes over the two product arrays, truncation.
//
// Bound by the latency of the passes (1024x256 FP64: 16 warps an SM, a third of
// the issue slots and of the shared-memory peak; barriers and loads first among
// the waits).  Against the radix-8 form
// of the same transforms (4 + 4 passes and a product sweep between them) the
// 1536-point row makes 36 instead of 60 shared-memory accesses an entry.
// Args: XProdArgs-like (ev, ov, ed, od, out, iptw, rp, Nx, Nk, M, Nz, k0, ld,
// instances).
template <int R, class C>
__device__ __forceinline__ void middle(C* __restrict__ A, int Ms, int n) {
  using T = typename Real<C>::type;
  for (int b = threadIdx.x; b < n / R; b += blockDim.x) {
    int at[R];
#pragma unroll
    for (int r = 0; r < R; ++r) at[r] = sw<C>(b * R + r);
    C u[R], g[R], z[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = A[at[r]];
    dft<R, 1>(u);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const C* x = A + (size_t)(1 + f) * Ms;
#pragma unroll
      for (int r = 0; r < R; ++r) g[r] = x[at[r]];
      dft<R, 1>(g);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const T q = -(u[r].x * g[r].x + u[r].y * g[r].y);
        if (f == 1)
          z[r].y = q;
        else
          z[r] = mk<C>(q, (T)0);
      }
      if (f > 0) {  // (b + i u_x) into array 0, u_z into array 1 (both read above by this thread only)
        dft<R, -1>(z);
        C* o = A + (size_t)(f - 1) * Ms;
#pragma unroll
        for (int r = 0; r < R; ++r) o[at[r]] = z[r];
      }
    }
  }
}

template <int NT, int CTAS, class C, class Args>
__global__ void __launch_bounds__(NT, CTAS) k_xprod_r(Args a) {
  using T = typename Real<C>::type;
  extern __shared__ __align__(16) unsigned char xr_raw[];
  const int M = a.M, Nk = a.Nk, hN = a.Nx / 2;
  const int Ms = rpad<C>(M);
  C* A = reinterpret_cast<C*>(xr_raw);
  C* tw = A + 4 * Ms;
  for (int t = threadIdx.x; t < a.rp.ntw; t += NT) tw[t] = a.iptw[t];
  grid_wait();
  const int z = blockIdx.x, zm = a.Nz - 1 - z;
  const bool lower = z <= zm;
  const size_t ld = a.ld > 0 ? (size_t)a.ld : (size_t)Nk, col0 = (size_t)blockIdx.y * Nk;
  const size_t rr = (size_t)(lower ? z : zm) * ld + col0;
  auto put2 = [&](C* dst, int q, C P, C Q) {  // spectrum of P + i Q (half spectra) on M points
    dst[sw<C>(q)] = mk<C>(P.x - Q.y, P.y + Q.x);
    if (q > 0) dst[sw<C>(M - q)] = mk<C>(P.x + Q.y, -P.y + Q.x);
  };
  // The Nyquist bin (only its real part enters, split in half) is read ahead of
  // the loop by the last thread: N/2 bins are a whole number of rounds at the
  // power-of-two lengths, and one more bin would cost a round's memory latency.
  const bool nyq = threadIdx.x == NT - 1;
  T gn[3], dn[3];
  if (nyq) {
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const T e = a.ev[f][rr + hN].x, o = a.ov[f][rr + hN].x;
      const T ed = a.ed[f][rr + hN].x, od = a.od[f][rr + hN].x;
      gn[f] = (T)0.5 * (lower ? e + o : e - o);
      dn[f] = (T)0.5 * (lower ? ed + od : od - ed);
    }
  }
  for (int q = threadIdx.x; q < hN; q += NT) {
    C g[3], d[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const C e = a.ev[f][rr + q], o = a.ov[f][rr + q];
      const C ed = a.ed[f][rr + q], od = a.od[f][rr + q];
      g[f] = lower ? add(e, o) : sub(e, o);
      d[f] = lower ? add(ed, od) : sub(od, ed);
    }
    if (q == 0) g[1].y = g[2].y = d[0].y = d[1].y = d[2].y = (T)0;  // DC kept real
    put2(A, q, g[1], g[2]);
    const T kk = a.k0 * (T)q;
#pragma unroll
    for (int f = 0; f < 3; ++f) put2(A + (size_t)(1 + f) * Ms, q, mk<C>(-kk * g[f].y, kk * g[f].x), d[f]);  // i k g
  }
  if (nyq) {
    put2(A, hN, mk<C>(gn[1], 0), mk<C>(gn[2], 0));
#pragma unroll
    for (int f = 0; f < 3; ++f) put2(A + (size_t)(1 + f) * Ms, hN, mk<C>(0, 0), mk<C>(dn[f], 0));
  }
  for (int k = hN + 1 + threadIdx.x; k < M - hN; k += NT)  // bins N/2 < k < M - N/2 are zero
#pragma unroll
    for (int arr = 0; arr < 4; ++arr) A[(size_t)arr * Ms + sw<C>(k)] = mk<C>(0, 0);
  __syncthreads();
  const int last = a.rp.np - 1;
  for (int s = 0; s < last; ++s) {
    pass_any<true, 1>(A, 4, Ms, a.rp, s, tw);
    __syncthreads();
  }
  switch (a.rp.R[last]) {
    case 8: middle<8>(A, Ms, M); break;
    case 6: middle<6>(A, Ms, M); break;
    case 4: middle<4>(A, Ms, M); break;
    case 3: middle<3>(A, Ms, M); break;
    default: middle<2>(A, Ms, M); break;
  }
  __syncthreads();
  for (int s = last - 1; s >= 0; --s) {
    pass_any<false, -1>(A, 2, Ms, a.rp, s, tw);
    __syncthreads();
  }
  const T sc = T(1) / ((T)M * (T)a.Nx);
  const size_t ro = (size_t)z * ld + col0;
  for (int k = threadIdx.x; k < Nk; k += NT) {
    const C c = A[sw<C>(k)], cm = A[sw<C>(k ? M - k : 0)], c2 = A[(size_t)Ms + sw<C>(k)];
    // first: (c + conj(cm))/2, second: (c - conj(cm))/(2i); the -N/2 image folds onto N/2
    const bool edge = k == 0 || k == hN;
    const T h = k == hN ? (T)2 * sc : sc;
    a.out[0][ro + k] = mk<C>(h * (T)0.5 * (c.x + cm.x), edge ? (T)0 : h * (T)0.5 * (c.y - cm.y));
    a.out[1][ro + k] = mk<C>(h * (T)0.5 * (c.y + cm.y), edge ? (T)0 : h * (T)-0.5 * (c.x - cm.x));
    a.out[2][ro + k] = mk<C>(h * c2.x, edge ? (T)0 : h * c2.y);
  }
}

template <class C>
inline size_t xprod_r_smem_bytes(int M, int ntw) {
  return (4 * (size_t)rpad<C>(M) + (size_t)ntw) * sizeof(C);
}

// 256 threads while two CTAs share an SM (128 threads measured 1 to 2 us slower
// from 384 points on and no faster below), else one CTA of 512.
template <class C, class Args>
inline void launch_xprod_r_t(const Args& a, cudaStream_t st) {
  const size_t smem = xprod_r_smem_bytes<C>(a.M, a.rp.ntw);
  const dim3 grid(a.Nz, a.instances > 0 ? a.instances : 1);
  if (2 * smem <= 227 * 1024)
    launch_chained(k_xprod_r<256, 2, C, Args>, grid, 256, smem, st, a);
  else
    launch_chained(k_xprod_r<512, 1, C, Args>, grid, 512, smem, st, a);
}

template <class C, class Args>
inline cudaError_t xprod_r_set_limits(int bytes) {
  cudaError_t e = cudaFuncSetAttribute(k_xprod_r<256, 2, C, Args>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_xprod_r<512, 1, C, Args>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace fftr
}  // namespace tb
