// |V3|^2 of 3-band cells with the class sums taken axis by axis.
//
// Replaces calculate_w3_ibz_split_sq + matrix_elt_simplified
// (THERMACOND/sub.f90:1050-1233, 5888-6011) and cal_eiqr2 (sub.f90:6015) for
// small cells.  ald_v3_pair.cu forms, for every pair (q1, q2),
//     A[l1][j0 be][k0 ga] = sum_{c in group (j0,k0)} P_c(q2) H[c][be ga][l1],
// one term per phase class c (79 for the argon crystal of the benchmark suite).
// The phase of a class is a product over the mesh axes,
//     P_c(m) = w_0^(m_0 n_c0) w_1^(m_1 n_c1) w_2^(m_2 n_c2) * sign_c,
// so the sum over classes is a separable discrete Fourier sum.  It is taken
// in three steps:
//   1. v3_plane_kernel, per row and m_0: H2[s2] = sum over the classes that
//      share (j0, k0, n_c1, n_c2) ("slot 2");
//   2. same kernel, per m_1: H3[s3] = sum over the slots 2 that share
//      (j0, k0, n_c2) ("slot 3"); stored per row and line (m_0, m_1);
//   3. v3_line3_kernel, per q2: A = sum over the slots 3.
// Steps 1 and 2 are done once per line of N_2 mesh points; step 3 has 7 terms
// instead of 79.  The mode products with e(q2), e(q3) and |V|^2 (const33/den)^2
// follow in the same thread, so nothing but e, H3 and the result crosses the
// memory system.
//
// Measured on B200 (argon, stage times).  FP64 26^3, all 1001 rows: 30.3 ms
// with one sum over the classes per pair (ald_v3_pair.cu), 4.8 here.  Mixed
// 32^3, 1768 rows: 10.6 ms with the class sums as split-FP16 tcgen05 MMAs,
// 8.0 here, and the linewidths' error against 64 bits falls from 8.5e-7 to
// 3.2e-8.  The line kernel is bound by issue and latency (with the Gaussian
// delta, FP32: issue slots 62 % busy, 128 registers, 16 warps per SM; FP64:
// FP64 pipe 34 %, 168 registers, 12 warps).
//
// Steps 1 and 2 are in FP64 in both precisions; ALD_MIXED rounds H3 to FP32
// and runs step 3 and the mode products in FP32, as the pair kernel runs its
// class sums.  Sums are reordered against the reference: agreement to
// rounding.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "ald_internal.h"

namespace ald {

namespace {

template <class T>
struct Cx;
template <>
struct Cx<double> {
  using t = double2;
};
template <>
struct Cx<float> {
  using t = float2;
};

template <class C>
__device__ __forceinline__ void cmac(C& acc, const C& a, const C& b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
template <class C>
__device__ __forceinline__ C cvt(const double2& v);
template <>
__device__ __forceinline__ double2 cvt<double2>(const double2& v) {
  return v;
}
template <>
__device__ __forceinline__ float2 cvt<float2>(const double2& v) {
  return make_float2((float)v.x, (float)v.y);
}

__device__ __forceinline__ void decompose(const Geometry& g, int n, int* m) {
  m[0] = n / (g.nc[1] * g.nc[2]);
  m[1] = (n / g.nc[2]) % g.nc[1];
  m[2] = n % g.nc[2];
}
// mesh index of q3 = -q1-q2, wrapped by compares: -m1 - m2 + nc/2 lies in (-2 nc, nc)
__device__ __forceinline__ int idx_q3(const Geometry& g, const int* m1, const int* m2) {
  int m3[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int n = g.nc[a];
    int v = -m1[a] - m2[a] + (g.shifted ? n / 2 : 0);
    v += v < 0 ? n : 0;
    v += v < 0 ? n : 0;
    m3[a] = v;
  }
  return m3[2] + g.nc[2] * (m3[1] + g.nc[1] * m3[0]);
}

// Per mesh mode: 1/sqrt|lambda| -- (const33/den)^2 with den = sqrt(8 sqrt|l1
// l2 l3|) is const33^2/8 times three of them -- and the eigenvectors in the
// kernel's precision.
template <class T>
struct LineModes {
  const double* t;
  const typename Cx<T>::t* e;
};
// what the Gaussian delta needs (GAUSS 1); R1, R2 of the chunk's rows
struct LineGauss {
  const double* freq;
  const double* dist;
  double gc1, gc2, fnorm;  // 1/(2 sigma^2), 1/(sqrt(2 pi) sigma), (2 pi)^2/nkc
  float fc1, fc2;
  double* R1;
  double* R2;
};
__global__ void v3_line_modes_kernel(const double* __restrict__ w2, const double2* __restrict__ ev, int n, double* t,
                                     float2* e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) t[i] = 1.0 / sqrt(fabs(w2[i]));
  if (e)
    for (int k = i; k < 3 * n; k += gridDim.x * blockDim.x) e[k] = make_float2((float)ev[k].x, (float)ev[k].y);
}

// Steps 1 and 2.  A CTA takes one row and one m_0; H2 of all 9 b components
// (be ga, l1) stays in shared memory while m_1 runs.  About a sixth of the line kernel's time (argon 26^3, 299 rows: 0.22
// of 1.23 ms); bound by the phase and H2 loads.
constexpr int kPlaneThreads = 256, kPlaneM = 4;
template <class C, int COMPS>
__global__ void __launch_bounds__(kPlaneThreads) v3_plane_kernel(V3Args a, V3LineTables t, C* __restrict__ H3) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* H2 = reinterpret_cast<double2*>(smraw);  // [slot 2][component]
  const int m0 = blockIdx.x, row = blockIdx.y;
  const int N0 = a.geo.nc[0], N1 = a.geo.nc[1], ns3 = t.ns3;
  const double2* H = static_cast<const double2*>(a.hbuf) + (size_t)row * a.ncls * COMPS;
  const double2* ph0 = reinterpret_cast<const double2*>(t.ph0) + (size_t)m0 * a.ncls;
  const double2* ph1 = reinterpret_cast<const double2*>(t.ph1);
  for (int e = threadIdx.x; e < t.ns2 * COMPS; e += kPlaneThreads) {
    const int s = e / COMPS, k = e - s * COMPS;
    double2 acc = make_double2(0.0, 0.0);
    for (int c = t.s2_off[s]; c < t.s2_off[s + 1]; ++c) cmac(acc, ph0[c], H[(size_t)t.cls[c] * COMPS + k]);
    H2[s * COMPS + k] = acc;
  }
  __syncthreads();
  // a thread takes kPlaneM values of m_1 and the components k, k + COMPS/3, k + 2 COMPS/3:
  // 4 phases and 3 sums loaded for 12 products
  C* out = H3 + ((size_t)row * N0 + m0) * N1 * ns3 * COMPS;
  constexpr int K3 = COMPS / 3;
  const int nm = (N1 + kPlaneM - 1) / kPlaneM;
  for (int e = threadIdx.x; e < nm * ns3 * K3; e += kPlaneThreads) {
    const int ms = e / K3, k = e - ms * K3, mb = ms / ns3, s = ms - mb * ns3;
    const double2* p[kPlaneM];
    double2 acc[kPlaneM][3];
#pragma unroll
    for (int i = 0; i < kPlaneM; ++i) {
      p[i] = ph1 + (size_t)min(mb * kPlaneM + i, N1 - 1) * t.ns2;
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[i][j] = make_double2(0.0, 0.0);
    }
    for (int c = t.s3_off[s]; c < t.s3_off[s + 1]; ++c) {
      double2 h[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) h[j] = H2[c * COMPS + k + K3 * j];
#pragma unroll
      for (int i = 0; i < kPlaneM; ++i) {
        const double2 ph = p[i][c];
#pragma unroll
        for (int j = 0; j < 3; ++j) cmac(acc[i][j], ph, h[j]);
      }
    }
#pragma unroll
    for (int i = 0; i < kPlaneM; ++i) {
      if (mb * kPlaneM + i >= N1) continue;
      C* o = out + ((size_t)(mb * kPlaneM + i) * ns3 + s) * COMPS;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int kj = k + K3 * j;  // [be ga][l1]; 3 bands: to [l1][be ga]
        o[COMPS == 27 ? kj % 3 * 9 + kj / 3 : kj] = cvt<C>(acc[i][j]);
      }
    }
  }
}

// Step 3.  Thread = q2; the nine class sums of one band l1 at a time stay in
// registers.
//   GAUSS 0: |V3|^2 goes to the chunk (a.v3sq or a.v3sq_f32) in its layout;
//   GAUSS 1: it is weighted where it stands by the Gaussian delta and the
//     Bose factors of both processes (delta_point_kernel's, ald_tetra.cu) and
//     summed over l3; R1 at w = q2 and R2 at w = -q2 (whose q3 = q1 - w is the
//     same point) are staged in shared memory and leave as contiguous runs.
constexpr int kQT = 128, kSP = 30;  // q2 per CTA; slot pitch: [l1][9 padded to 10]
template <class T, int GAUSS>
__global__ void __launch_bounds__(kQT, sizeof(T) == 4 ? (GAUSS ? 4 : 5) : 3)
    v3_line3_kernel(V3Args a, V3LineTables t, const typename Cx<T>::t* __restrict__ H3, LineModes<T> md, int npmax,
                    LineGauss d) {
  using C = typename Cx<T>::t;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sh = reinterpret_cast<C*>(smraw);
  C* sp = sh + npmax * t.ns3 * kSP;
  __shared__ double s_r[GAUSS ? 2 : 1][GAUSS ? kQT * 9 : 1];
  __shared__ int s_neg[GAUSS ? kQT : 1];
  const Geometry& g = a.geo;
  const int N2 = g.nc[2], row = blockIdx.y, base = blockIdx.x * kQT, ns3 = t.ns3, tid = threadIdx.x;
  const int nq = min(kQT, g.nkc - base), p0 = base / N2, np = (base + nq - 1) / N2 - p0 + 1;
  // the H3 lines the CTA's points touch, and the phases of axis 2 with an odd
  // pitch (no bank conflicts when lanes walk m_2)
  {
    const C* src = H3 + ((size_t)row * g.nc[0] * g.nc[1] + p0) * ns3 * 27;
    for (int e = tid; e < np * ns3 * 27; e += kQT) sh[e / 9 * 10 + e % 9] = src[e];
    const double2* ph2 = reinterpret_cast<const double2*>(t.ph2);
    for (int e = tid; e < N2 * ns3; e += kQT) sp[e / ns3 * (ns3 | 1) + e % ns3] = cvt<C>(ph2[e]);
  }
  __syncthreads();
  const int q2 = base + tid;
  if (tid < nq) {
    const int q1 = a.mapinv[a.n1_first + row];
    int m1[3], m2[3];
    decompose(g, q1, m1);
    decompose(g, q2, m2);
    const int q3 = idx_q3(g, m1, m2);
    C e2[9], e3[9];  // [l][i]
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      e2[i] = md.e[(size_t)q2 * 9 + i];
      e3[i] = md.e[(size_t)q3 * 9 + i];
    }
    const double* t1 = md.t + (size_t)q1 * 3;
    double t2[3], t3[3];
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      t2[l] = md.t[(size_t)q2 * 3 + l];
      t3[l] = md.t[(size_t)q3 * 3 + l];
    }
    const double c33 = a.const33 * a.const33 / 8;
    // den = 0 (or a scale that overflows) can only come with the largest factors
    const bool chk = !(c33 * fmax(fmax(t1[0], t1[1]), t1[2]) * fmax(fmax(t2[0], t2[1]), t2[2]) *
                           fmax(fmax(t3[0], t3[1]), t3[2]) < 1.0 / 0.0);
    // Gaussian: omega and n at w = q2 and w = -q2 (band l2) and at q1 + q2 (band l3)
    double w2a[3], w2b[3], w3[3], n3[3];
    int wn = 0;
    unsigned zero = 0;  // bits 0..2: band l2 of process 1, 2, band l3 left out (the zone-centre test)
    if constexpr (GAUSS) {
      const int h[3] = {g.nc[0] / 2, g.nc[1] / 2, g.nc[2] / 2};
      int mn[3], mp[3];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        mn[x] = m2[x] == 0 ? 0 : g.nc[x] - m2[x];
        int v = m1[x] + m2[x] - (g.shifted ? h[x] : 0);
        v += v < 0 ? g.nc[x] : 0;
        mp[x] = v >= g.nc[x] ? v - g.nc[x] : v;
      }
      wn = mn[2] + g.nc[2] * (mn[1] + g.nc[1] * mn[0]);
      const int qp = mp[2] + g.nc[2] * (mp[1] + g.nc[1] * mp[0]);
      zero = (unsigned)(m2[0] == h[0] && m2[1] == h[1] && m2[2] == h[2]) |
             (unsigned)(mn[0] == h[0] && mn[1] == h[1] && mn[2] == h[2]) << 1 |
             (unsigned)(mp[0] == h[0] && mp[1] == h[1] && mp[2] == h[2]) << 2;
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        w2a[l] = d.freq[(size_t)q2 * 3 + l];
        w2b[l] = d.freq[(size_t)wn * 3 + l];
        w3[l] = d.freq[(size_t)qp * 3 + l];
        n3[l] = d.dist[(size_t)qp * 3 + l] + 1;
      }
    }
    const C* hl = sh + (q2 / N2 - p0) * ns3 * kSP;
    const C* pl = sp + m2[2] * (ns3 | 1);
    const size_t nk = g.nkc;
    // layout 1: [row][l2][l3][l1][q2]; 0: [row][q2][l1][l2][l3]
    const size_t o = a.v3_layout == 1 ? (size_t)row * 27 * nk + q2 : ((size_t)row * nk + q2) * 27;
    const int s1 = a.v3_layout == 1 ? (int)nk : 9, s23 = a.v3_layout == 1 ? 3 * (int)nk : 1;
#pragma unroll 1
    for (int l1 = 0; l1 < 3; ++l1) {
      C A[9];
#pragma unroll
      for (int j = 0; j < 9; ++j) A[j] = C{0, 0};
      for (int s = 0; s < ns3; ++s) {
        const C p = pl[s];
        const C* h = hl + s * kSP + l1 * 10;
        if constexpr (sizeof(T) == 4) {  // two complex values per load
#pragma unroll
          for (int j = 0; j < 5; ++j) {
            const float4 x = reinterpret_cast<const float4*>(h)[j];
            cmac(A[2 * j], p, C{x.x, x.y});
            if (j < 4) cmac(A[2 * j + 1], p, C{x.z, x.w});
          }
        } else {
#pragma unroll
          for (int j = 0; j < 9; ++j) cmac(A[j], p, h[j]);
        }
      }
      const double sc1 = c33 * t1[l1];
      const size_t ol = o + (size_t)l1 * s1;
      const double om1 = GAUSS ? d.freq[(size_t)q1 * 3 + l1] : 0.0;
#pragma unroll
      for (int l2 = 0; l2 < 3; ++l2) {
        C Tv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Tv[c] = C{0, 0};
#pragma unroll
          for (int i = 0; i < 3; ++i) cmac(Tv[c], A[i * 3 + c], e2[l2 * 3 + i]);
        }
        const double sc12 = sc1 * t2[l2];
        double r1 = 0.0, r2 = 0.0;
        const double xa = GAUSS ? om1 + w2a[l2] : 0.0, xb = GAUSS ? om1 - w2b[l2] : 0.0;
#pragma unroll
        for (int l3 = 0; l3 < 3; ++l3) {
          C v = C{0, 0};
#pragma unroll
          for (int c = 0; c < 3; ++c) cmac(v, Tv[c], e3[l3 * 3 + c]);
          const double sc = sc12 * t3[l3];
          double r = (double)fma(v.x, v.x, v.y * v.y) * sc;
          if (chk && !(sc < 1.0 / 0.0)) {
            r = 0.0;
            atomicOr(a.err, 2);  // matrix_elt_simplified: den = 0
          }
          if constexpr (GAUSS == 0) {
            const size_t oi = ol + (size_t)((l2 * 3 + l3) * s23);
            if (a.v3sq_f32) a.v3sq_f32[oi] = (float)r;
            else a.v3sq[oi] = r;
          } else {
            r = zero & 4 ? 0.0 : r * n3[l3];
            const double x1 = xa - w3[l3], x2 = xb - w3[l3];
            if constexpr (sizeof(T) == 4) {  // FP32 exp, underflows beyond 104
              const float f1 = (float)x1, f2 = (float)x2, a1 = f1 * f1 * d.fc1, a2 = f2 * f2 * d.fc1;
              if (a1 < 104.0f) r1 += (double)(expf(-a1) * d.fc2) * r;
              if (a2 < 104.0f) r2 += (double)(expf(-a2) * d.fc2) * r;
            } else {  // beyond 746
              const double a1 = x1 * x1 * d.gc1, a2 = x2 * x2 * d.gc1;
              if (a1 < 746.0) r1 = fma(exp(-a1) * d.gc2, r, r1);
              if (a2 < 746.0) r2 = fma(exp(-a2) * d.gc2, r, r2);
            }
          }
        }
        if constexpr (GAUSS) {
          const double n1f = d.dist[(size_t)q1 * 3 + l1] * d.fnorm;
          s_r[0][tid * 9 + l1 * 3 + l2] = zero & 1 ? 0.0 : r1 * (n1f * d.dist[(size_t)q2 * 3 + l2]);
          s_r[1][tid * 9 + l1 * 3 + l2] = zero & 2 ? 0.0 : r2 * (n1f * (d.dist[(size_t)wn * 3 + l2] + 1));
        }
      }
    }
    if constexpr (GAUSS) s_neg[tid] = wn;
  }
  if constexpr (GAUSS) {
    __syncthreads();
    const size_t rb = (size_t)row * g.nkc * 9;
    for (int e = tid; e < nq * 9; e += kQT) {
      d.R1[rb + (size_t)base * 9 + e] = s_r[0][e];
      d.R2[rb + (size_t)s_neg[e / 9] * 9 + e % 9] = s_r[1][e];
    }
  }
}

// lines (m_0, m_1) that kQT consecutive mesh points can touch
int lines_touched(const Geometry& g) { return std::min((kQT + g.nc[2] - 2) / g.nc[2] + 1, g.nc[0] * g.nc[1]); }
template <class T>
size_t line_smem(const Geometry& g, int ns3) {
  return ((size_t)lines_touched(g) * ns3 * kSP + (size_t)g.nc[2] * (ns3 | 1)) * sizeof(typename Cx<T>::t);
}
// the work buffer: 1/sqrt|lambda| and the FP32 eigenvectors of the mesh, then H3
size_t line_align(size_t x) { return (x + 255) / 256 * 256; }
size_t line_t_bytes(const Geometry& g) { return line_align((size_t)g.nkc * g.b * sizeof(double)); }
size_t line_e_bytes(const Geometry& g) { return line_align((size_t)g.nkc * g.b * g.b * sizeof(float2)); }

template <class C, int COMPS>
cudaError_t launch_plane_t(const V3Args& a, const V3LineTables& t, void* lines, cudaStream_t s) {
  const size_t smem = (size_t)t.ns2 * COMPS * sizeof(double2);
  const cudaError_t e = raise_smem_limit((const void*)v3_plane_kernel<C, COMPS>, smem);
  if (e != cudaSuccess) return e;
  v3_plane_kernel<C, COMPS><<<dim3(a.geo.nc[0], a.nrows), kPlaneThreads, smem, s>>>(a, t, static_cast<C*>(lines));
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_line_t(const V3Args& a, const V3LineTables& t, void* work, const LineGauss* d, cudaStream_t s) {
  using C = typename Cx<T>::t;
  const Geometry& g = a.geo;
  char* w = static_cast<char*>(work);
  double* ts = reinterpret_cast<double*>(w);
  float2* ef = sizeof(T) == 4 ? reinterpret_cast<float2*>(w + line_t_bytes(g)) : nullptr;
  C* H3 = reinterpret_cast<C*>(w + line_t_bytes(g) + line_e_bytes(g));
  const double2* ev = reinterpret_cast<const double2*>(a.evec);
  v3_line_modes_kernel<<<(g.nkc * 3 + 255) / 256, 256, 0, s>>>(a.w2, ev, g.nkc * 3, ts, ef);
  cudaError_t e = launch_v3_rows_f64(a, s);
  if (e != cudaSuccess) return e;
  e = launch_v3_lines(a, t, H3, sizeof(T) == 4 ? ALD_MIXED : ALD_FP64, s);
  if (e != cudaSuccess) return e;
  const size_t smem = line_smem<T>(g, t.ns3);
  LineModes<T> md;
  md.t = ts;
  if constexpr (sizeof(T) == 4) md.e = ef;
  else md.e = ev;
  const dim3 grid((g.nkc + kQT - 1) / kQT, a.nrows);
  if (d) {
    e = raise_smem_limit((const void*)v3_line3_kernel<T, 1>, smem);
    if (e != cudaSuccess) return e;
    v3_line3_kernel<T, 1><<<grid, kQT, smem, s>>>(a, t, H3, md, lines_touched(g), *d);
  } else {
    e = raise_smem_limit((const void*)v3_line3_kernel<T, 0>, smem);
    if (e != cudaSuccess) return e;
    v3_line3_kernel<T, 0><<<grid, kQT, smem, s>>>(a, t, H3, md, lines_touched(g), LineGauss());
  }
  return cudaGetLastError();
}

}  // namespace

bool v3_lines_supported(const Geometry& g, const V3LineTables& t) {
  return (g.b == 3 || g.b == 6) && t.ns2 >= 1 && (size_t)t.ns2 * 9 * g.b * sizeof(double2) <= 200 * 1024;
}

cudaError_t launch_v3_lines(const V3Args& a, const V3LineTables& t, void* lines, int precision, cudaStream_t s) {
  if (!v3_lines_supported(a.geo, t)) return cudaErrorInvalidValue;
  if (precision == ALD_FP64)
    return a.geo.b == 3 ? launch_plane_t<double2, 27>(a, t, lines, s) : launch_plane_t<double2, 54>(a, t, lines, s);
  return a.geo.b == 3 ? launch_plane_t<float2, 27>(a, t, lines, s) : launch_plane_t<float2, 54>(a, t, lines, s);
}

bool v3_line_supported(const Geometry& g, const V3LineTables& t, int precision) {
  if (g.b != 3 || !v3_lines_supported(g, t)) return false;
  return (precision == ALD_FP64 ? line_smem<double>(g, t.ns3) : line_smem<float>(g, t.ns3)) <= 200 * 1024;
}

size_t v3_line_row_bytes(const Geometry& g, const V3LineTables& t, int precision) {
  const size_t cplx = precision == ALD_FP64 ? sizeof(double2) : sizeof(float2);
  return (size_t)g.nc[0] * g.nc[1] * t.ns3 * 9 * g.b * cplx;
}

size_t v3_line_work_bytes(const Geometry& g, const V3LineTables& t, int nrows, int precision) {
  return line_t_bytes(g) + line_e_bytes(g) + nrows * v3_line_row_bytes(g, t, precision);
}

cudaError_t launch_v3_line(const V3Args& a, const V3LineTables& t, void* work, int precision, cudaStream_t s) {
  if (!v3_line_supported(a.geo, t, precision)) return cudaErrorInvalidValue;
  return precision == ALD_FP64 ? launch_line_t<double>(a, t, work, nullptr, s)
                               : launch_line_t<float>(a, t, work, nullptr, s);
}

cudaError_t launch_v3_line_gauss(const V3Args& a, const V3LineTables& t, void* work, int precision,
                                 const CombineArgs& ca, cudaStream_t s) {
  if (!v3_line_supported(a.geo, t, precision) || !ca.gauss || ca.R1p || ca.R2p || ca.P1s || ca.P2s || ca.P1 ||
      ca.P2)
    return cudaErrorInvalidValue;
  LineGauss d;
  d.freq = ca.freq;
  d.dist = ca.dist;
  d.gc1 = 0.5 / (ca.sigma * ca.sigma);
  d.gc2 = 1.0 / (std::sqrt(2 * PhysConst::pi) * ca.sigma);
  d.fc1 = (float)d.gc1;
  d.fc2 = (float)d.gc2;
  d.fnorm = (2 * PhysConst::pi) * (2 * PhysConst::pi) / a.geo.nkc;
  d.R1 = ca.R1;
  d.R2 = ca.R2;
  return precision == ALD_FP64 ? launch_line_t<double>(a, t, work, &d, s) : launch_line_t<float>(a, t, work, &d, s);
}

}  // namespace ald
