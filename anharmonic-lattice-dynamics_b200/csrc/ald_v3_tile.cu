// |V3|^2 for cells of 9 bands and up whose pairs fit shared memory: the class
// sums and both eigenvector mode products of a pair without leaving the SM.
//
// Replaces calculate_w3_ibz_split_sq + matrix_elt_simplified
// (THERMACOND/sub.f90:1050-1233, 5888-6011) and cal_eiqr2 (sub.f90:6015).
// With the phase classes of ald_v3_pair.cu, and one band l1 at a time, a pair
// (q1, q2) is three b x b x b products of complex matrices:
//   A[jb][kc]  = sum_{c in group (j0,k0)} P_c(q2) H[l1][c][be ga]
//   T[l2][kc]  = sum_jb e2[l2][jb] A[jb][kc]
//   V[l2][l3]  = sum_kc T[l2][kc] e3[l3][kc]
// A CTA takes one IBZ row and QT consecutive q2, keeps e(q2), e(q3) and the
// phases of its points in shared memory and walks l1 in steps of LG: QT LG
// matrices at a time, each with a TM x TM register tile per thread, T written
// over A.  Every H value that it loads serves QT pairs.  Nothing but H, the
// eigenvectors and |V3|^2 crosses L2, where the batched GEMMs of
// ald_v3_dense.cu and ald_v3_dense_tc.cu send T1 and T2 through memory (16 b^3
// bytes and more per pair) and pad b to 64 or 128.
//
// T = double for ALD_FP64, float (FP32 accumulation) for ALD_MIXED.  The sums
// of an element run in the same order whatever QT, LG and TM are, so a row
// formed alone has the same bits as in a chunk.  Sums are reordered against
// the reference: agreement to rounding.
//
// Bound by issue and latency (24 bands FP32: issue slots 56 % busy, FMA pipe
// 39 %, 17 warps per SM; 12 bands FP64: FP64 pipe 37 %, 14 warps).  Of the FP32 work at
// 24 bands the class sums are a sixth of the products.
#include <cuda_runtime.h>

#include <algorithm>

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
__device__ __forceinline__ int phase_index(const int* pc, const int* m, int L, int L32) {
  if (L32) {  // the sum fits in 32 bits: a 32-bit remainder
    const unsigned t = (unsigned)(m[0] * pc[0] + m[1] * pc[1] + m[2] * pc[2] + pc[3]);
    return (int)(t % (unsigned)L);
  }
  long long t = (long long)m[0] * pc[0] + (long long)m[1] * pc[1] + (long long)m[2] * pc[2] + pc[3];
  return (int)(t % L);
}

// H[row][c][l1][be ga] (ald_v3_pair.cu's row stage; here the be ga of several
// l1 of one class are one run)
template <class C>
__global__ void v3_tile_row_kernel(V3Args a, C* __restrict__ Hout) {
  const Geometry& g = a.geo;
  const int b = g.b, row = blockIdx.y, n = a.ncls * 9 * b;
  const int q1 = a.mapinv[a.n1_first + row];
  int m1[3];
  decompose(g, q1, m1);
  C* H = Hout + (size_t)row * n;
  const double2* roots = reinterpret_cast<const double2*>(a.roots);
  const double2* e1 = reinterpret_cast<const double2*>(a.evec) + (size_t)q1 * b * b;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int bg = e % 9, l1 = e / 9 % b, c = e / (9 * b);
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int s = a.cls_trip_off[c]; s < a.cls_trip_off[c + 1]; ++s) {
      const int t = a.cls_trip[s], i0 = a.cls_trip_i0[s], k = a.cls_trip_k[s];
      const int ph = phase_index(a.phase_coef + 4 * k, m1, g.L, g.L32);
      const double2 r = roots[ph == 0 ? 0 : g.L - ph];  // exp(-i q1.R_k)
      double2 x = make_double2(0.0, 0.0);
      for (int al = 0; al < 3; ++al) {
        const double w = a.fc3w[27 * (size_t)t + al * 9 + bg];
        const double2 v = e1[l1 * b + 3 * i0 + al];
        x.x = fma(w, v.x, x.x);
        x.y = fma(w, v.y, x.y);
      }
      cmac(acc, r, x);
    }
    H[e] = cvt<C>(acc);
  }
}

// 1/sqrt|lambda| of every mesh mode: (const33/den)^2 with den = sqrt(8 sqrt|l1
// l2 l3|) is const33^2/8 times three of them
__global__ void v3_tile_modes_kernel(const double* __restrict__ w2, double* __restrict__ t, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) t[i] = 1.0 / sqrt(fabs(w2[i]));
}

// the pair's shape: QT q2 and LG bands l1 at a time, nb = ceil(b / TM) tiles
// per side, matrices of b rows of pitch bp = nb TM, mp complex apart (4 more
// than a multiple of the banks, so that the matrices of a warp do not collide)
struct TileShape {
  int qt, lg, tm, nb, bp, mp, nt;
  size_t smem;
};

// The TM rows (or columns) of thread t among nb: t, t + nb, ...; in FP32 with
// TM = 4 in neighbouring pairs.  The threads of a warp then read consecutive
// 16-byte words, where blocks of TM neighbours would fall on the same banks.
template <class C, int TM>
__device__ __forceinline__ int tile_at(int t, int i, int nb) {
  if constexpr (sizeof(C) == 8 && TM == 4) return (i & 1) + 2 * t + (i >> 1) * 2 * nb;
  else return i * nb + t;
}
template <int TM, class C>
__device__ __forceinline__ void load_row(const C* p, int t, int nb, C* v) {
  if constexpr (sizeof(C) == 8 && TM == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p + 2 * t);
    const float4 y = *reinterpret_cast<const float4*>(p + 2 * nb + 2 * t);
    v[0] = C{x.x, x.y};
    v[1] = C{x.z, x.w};
    v[2] = C{y.x, y.y};
    v[3] = C{y.z, y.w};
  } else {
#pragma unroll
    for (int i = 0; i < TM; ++i) v[i] = p[i * nb + t];
  }
}
// the phases of QT points: QT consecutive values
template <int QT, class C>
__device__ __forceinline__ void load_phases(const C* p, C* v) {
  if constexpr (sizeof(C) == 8 && QT % 2 == 0) {
#pragma unroll
    for (int i = 0; i < QT / 2; ++i) {
      const float4 x = reinterpret_cast<const float4*>(p)[i];
      v[2 * i] = C{x.x, x.y};
      v[2 * i + 1] = C{x.z, x.w};
    }
  } else {
#pragma unroll
    for (int i = 0; i < QT; ++i) v[i] = p[i];
  }
}

// acc[r][c] = sum_k X[k][row r of ty] Y[k][column c of tx], rows of pitch bp
template <int TM, class C>
__device__ __forceinline__ void tile_product(const C* X, const C* Y, int ty, int tx, int nb, int b, int bp,
                                             C (&acc)[TM][TM]) {
#pragma unroll
  for (int r = 0; r < TM; ++r)
#pragma unroll
    for (int c = 0; c < TM; ++c) acc[r][c] = C{0, 0};
#pragma unroll 2
  for (int k = 0; k < b; ++k) {
    C x[TM], y[TM];
    load_row<TM>(X + k * bp, ty, nb, x);
    load_row<TM>(Y + k * bp, tx, nb, y);
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
      for (int c = 0; c < TM; ++c) cmac(acc[r][c], x[r], y[c]);
  }
}

// two CTAs per SM: one's class sums and barriers under the other's products
template <class T>
constexpr int kTileThreads = sizeof(T) == 4 ? 320 : 256;
template <class T, int TM, int QT>
__global__ void __launch_bounds__(kTileThreads<T>, 2)
    v3_tile_kernel(V3Args a, TileShape sh, const typename Cx<T>::t* __restrict__ Hall,
                   const double* __restrict__ ts, int nk1) {
  using C = typename Cx<T>::t;
  extern __shared__ __align__(16) unsigned char smraw[];
  const Geometry& g = a.geo;
  const int b = g.b, b2 = b * b, bp = sh.bp, mp = sh.mp, nb = sh.nb, LG = sh.lg, tid = threadIdx.x, nt = sh.nt;
  const int row = blockIdx.y, base = blockIdx.x * QT, nq = min(QT, g.nkc - base);
  C* E2 = reinterpret_cast<C*>(smraw);  // [q][jb][l2]
  C* E3 = E2 + QT * mp;                 // [q][kc][l3]
  C* A = E3 + QT * mp;                  // [q][l][jb][kc], then T as [kc][l2]; then |V|^2
  C* P = A + QT * LG * mp;              // [class][q]
  // per group: its classes (first, end) and its place in A
  ushort4* grps = reinterpret_cast<ushort4*>(P + QT * a.ncls);
  __shared__ int s_q3[QT];
  const int q1 = a.mapinv[a.n1_first + row];
  // zero the padded columns once: no later write touches them but with zeros
  for (int i = tid; i < (2 + LG) * QT * mp; i += nt) E2[i] = C{0, 0};
  if (tid < QT) {
    int m1[3], m2[3];
    decompose(g, q1, m1);
    decompose(g, min(base + tid, g.nkc - 1), m2);
    s_q3[tid] = idx_q3(g, m1, m2);
  }
  __syncthreads();
  const double2* ev = reinterpret_cast<const double2*>(a.evec);
  for (int i = tid; i < QT * b2; i += nt) {  // e[l][i] -> [i][l]; the last tile repeats the last point
    const int q = i / b2, e = i - q * b2, l = e / b, k = e - l * b;
    E2[q * mp + k * bp + l] = cvt<C>(ev[(size_t)min(base + q, g.nkc - 1) * b2 + e]);
    E3[q * mp + k * bp + l] = cvt<C>(ev[(size_t)s_q3[q] * b2 + e]);
  }
  const double2* roots = reinterpret_cast<const double2*>(a.roots);
  for (int i = tid; i < QT * a.ncls; i += nt) {
    const int c = i / QT, q = i - c * QT;
    int m2[3];
    decompose(g, min(base + q, g.nkc - 1), m2);
    P[i] = cvt<C>(roots[phase_index(a.cls_pc + 4 * c, m2, g.L, g.L32)]);
  }
  for (int e = tid; e < g.nat0 * g.nat0; e += nt) {
    const int j0 = e / g.nat0, k0 = e - j0 * g.nat0;
    grps[e] = make_ushort4((unsigned short)a.cls_grp_off[e], (unsigned short)a.cls_grp_off[e + 1],
                           (unsigned short)(3 * j0 * bp + 3 * k0), 0);
  }
  // this thread's matrix (q, l) and tile
  const int grp = tid / (nb * nb), t = tid - grp * nb * nb, ty = t / nb, tx = t - ty * nb;
  const int q = grp / LG, l = grp - q * LG;
  const int q2 = base + q;
  const double c33 = a.const33 * a.const33 / 8;
  const C* H = Hall + (size_t)row * a.ncls * 9 * b;
  C* Ag = A + grp * mp;
  const double* t2 = ts + (size_t)min(q2, g.nkc - 1) * b;
  const double* t3 = ts + (size_t)s_q3[q] * b;
  for (int l0 = 0; l0 < nk1; l0 += LG) {
    const int nl = min(LG, nk1 - l0);
    __syncthreads();  // operands staged; the previous step's A free
    // element (group, l, be ga), be ga fastest: a warp reads runs of H and one
    // or two groups' phases
    for (int e = tid; e < nl * b2; e += nt) {
      const int gr = e / (9 * nl), lb = e - gr * 9 * nl, el = lb / 9, bg = lb - el * 9, be = bg / 3;
      const ushort4 d = grps[gr];
      const C* h = H + l0 * 9 + lb;
      C acc[QT];
#pragma unroll
      for (int k = 0; k < QT; ++k) acc[k] = C{0, 0};
#pragma unroll 4
      for (int c = d.x; c < d.y; ++c) {
        const C hv = h[(size_t)(c * 9 * b)];
        C p[QT];
        load_phases<QT>(P + c * QT, p);
#pragma unroll
        for (int k = 0; k < QT; ++k) cmac(acc[k], p[k], hv);
      }
      C* out = A + el * mp + d.z + be * bp + bg - 3 * be;
#pragma unroll
      for (int k = 0; k < QT; ++k) out[k * LG * mp] = acc[k];
    }
    __syncthreads();
    C acc[TM][TM];
    tile_product<TM>(E2 + q * mp, Ag, ty, tx, nb, b, bp, acc);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < TM; ++c) {
      const int kc = tile_at<C, TM>(tx, c, nb);
      if (kc < b)
#pragma unroll
        for (int r = 0; r < TM; ++r) Ag[kc * bp + tile_at<C, TM>(ty, r, nb)] = acc[r][c];
    }
    __syncthreads();
    tile_product<TM>(Ag, E3 + q * mp, ty, tx, nb, b, bp, acc);
    __syncthreads();
    // |V|^2 (FP32: the square in FP32, the mode factors in FP64): layout 0
    // straight out ([row][q2][l1][l2][l3], runs of l3); layout 1
    // ([row][l2][l3][l1][q2]) through shared memory as [l][l2 l3][q]
    const size_t nk = g.nkc, b3 = (size_t)b2 * b;
    double* Sd = reinterpret_cast<double*>(A);
    float* Sf = reinterpret_cast<float*>(A);
    const bool f32 = a.v3sq_f32 != nullptr, slices = a.v3_layout == 1;
    if (q < nq && l < nl) {
      const double sc1 = c33 * ts[(size_t)q1 * b + l0 + l];
      double t3c[TM];
#pragma unroll
      for (int c = 0; c < TM; ++c) {
        const int l3 = tile_at<C, TM>(tx, c, nb);
        t3c[c] = l3 < b ? t3[l3] : 0.0;
      }
      const size_t row0 = ((size_t)row * nk + q2) * b3 + (size_t)(l0 + l) * b2;
#pragma unroll
      for (int r = 0; r < TM; ++r) {
        const int l2 = tile_at<C, TM>(ty, r, nb);
        if (l2 >= b) continue;
        const double sc12 = sc1 * t2[l2];
        const int so = (l * b + l2) * b * QT + q;
#pragma unroll
        for (int c = 0; c < TM; ++c) {
          const int l3 = tile_at<C, TM>(tx, c, nb);
          if (l3 >= b) continue;
          const double sc = sc12 * t3c[c];
          double v = 0.0;
          if (sc < 1.0 / 0.0) v = (double)fma(acc[r][c].x, acc[r][c].x, acc[r][c].y * acc[r][c].y) * sc;
          else atomicOr(a.err, 2);  // matrix_elt_simplified: den = 0
          if (slices) {
            if (f32) Sf[so + l3 * QT] = (float)v;
            else Sd[so + l3 * QT] = v;
          } else if (f32) {
            a.v3sq_f32[row0 + l2 * b + l3] = (float)v;
          } else {
            a.v3sq[row0 + l2 * b + l3] = v;
          }
        }
      }
    }
    if (slices) {
      __syncthreads();
      const int k = tid % QT;  // nt is a multiple of QT
      if (k < nq)
        for (int el = 0; el < nl; ++el) {
          const size_t o0 = (size_t)row * nk * b3 + (size_t)(l0 + el) * nk + base + k, st = (size_t)b * nk;
          for (int x = tid / QT; x < b2; x += nt / QT) {
            if (f32) a.v3sq_f32[o0 + x * st] = Sf[(el * b2 + x) * QT + k];
            else a.v3sq[o0 + x * st] = Sd[(el * b2 + x) * QT + k];
          }
        }
      if (bp > b) {  // the staging went over the padded columns of A
        __syncthreads();
        for (int i = tid; i < QT * LG * mp; i += nt) A[i] = C{0, 0};
      }
    }
  }
}

template <class T>
bool tile_shape(const Geometry& g, int ncls, TileShape& s) {
  constexpr size_t cb = sizeof(typename Cx<T>::t);
  const int b = g.b;
  if (ncls > 65535 || b > 88) return false;  // 16-bit class numbers and offsets in the group table
  s.tm = b % 4 == 0 || b > 24 ? 4 : 3;
  s.nb = (b + s.tm - 1) / s.tm;
  s.bp = s.nb * s.tm;
  s.mp = b * s.bp + 4;
  // Two CTAs per SM, in FP32 with two points each: cells that miss it were
  // measured slower than the batched GEMMs (48 bands, 4x8x8 mesh: FP64 229 ms
  // against 138, mixed 55 against 51), those that make it faster (36 bands,
  // 4x6x6: 13.0 against 24.6 and 8.3 against 9.0; 24 bands, 4x8x8: 6.3 against
  // 21.7 and 3.6 against 9.2; 12 bands, 12^3: 6.9 against 25.7 and 5.3 against 21.4)
  const size_t limit = 113 * 1024;
  for (int qt : {4, 2, 1}) {
    if (sizeof(T) == 4 && qt == 1) continue;
    if (qt * s.nb * s.nb > kTileThreads<T>) continue;
    for (int lmax = std::min(b, kTileThreads<T> / (qt * s.nb * s.nb)); lmax >= 1; --lmax) {
      const int steps = (b + lmax - 1) / lmax, lg = (b + steps - 1) / steps;  // steps of equal width
      const size_t sm =
          ((size_t)(2 + lg) * qt * s.mp + (size_t)qt * ncls) * cb + (size_t)g.nat0 * g.nat0 * sizeof(ushort4);
      if (sm > limit) continue;
      s.qt = qt;
      s.lg = lg;
      s.nt = qt * lg * s.nb * s.nb;
      s.smem = sm;
      if (s.nt >= 128) return true;
      break;
    }
  }
  return false;
}

size_t tile_align(size_t x) { return (x + 255) / 256 * 256; }

template <class T, int TM, int QT>
cudaError_t launch_tile_q(const V3Args& a, const TileShape& sh, const typename Cx<T>::t* H, const double* ts, int nk1,
                          cudaStream_t s) {
  cudaError_t e = raise_smem_limit((const void*)v3_tile_kernel<T, TM, QT>, sh.smem);
  if (e != cudaSuccess) return e;
  v3_tile_kernel<T, TM, QT><<<dim3((a.geo.nkc + QT - 1) / QT, a.nrows), sh.nt, sh.smem, s>>>(a, sh, H, ts, nk1);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_tile_t(const V3Args& a, void* work, int l1_keep, cudaStream_t s) {
  using C = typename Cx<T>::t;
  const Geometry& g = a.geo;
  TileShape sh;
  if (!tile_shape<T>(g, a.ncls, sh)) return cudaErrorInvalidValue;
  double* ts = static_cast<double*>(work);
  C* H = reinterpret_cast<C*>(static_cast<char*>(work) + tile_align((size_t)g.nkc * g.b * sizeof(double)));
  v3_tile_modes_kernel<<<(g.nkc * g.b + 255) / 256, 256, 0, s>>>(a.w2, ts, g.nkc * g.b);
  v3_tile_row_kernel<C><<<dim3((a.ncls * 9 * g.b + 255) / 256, a.nrows), 256, 0, s>>>(a, H);
  const int nk1 = l1_keep > 0 && l1_keep < g.b ? l1_keep : g.b;
  if (sh.tm == 4)
    return sh.qt == 4   ? launch_tile_q<T, 4, 4>(a, sh, H, ts, nk1, s)
           : sh.qt == 2 ? launch_tile_q<T, 4, 2>(a, sh, H, ts, nk1, s)
                        : launch_tile_q<T, 4, 1>(a, sh, H, ts, nk1, s);
  return sh.qt == 4   ? launch_tile_q<T, 3, 4>(a, sh, H, ts, nk1, s)
         : sh.qt == 2 ? launch_tile_q<T, 3, 2>(a, sh, H, ts, nk1, s)
                      : launch_tile_q<T, 3, 1>(a, sh, H, ts, nk1, s);
}

}  // namespace

bool v3_tile_supported(const Geometry& g, int ncls, int precision) {
  if (g.b < 9 || (precision != ALD_FP64 && precision != ALD_MIXED)) return false;
  TileShape s;
  return precision == ALD_FP64 ? tile_shape<double>(g, ncls, s) : tile_shape<float>(g, ncls, s);
}

cudaError_t launch_v3_rows_by_class_f32(const V3Args& a, cudaStream_t s) {
  v3_tile_row_kernel<float2><<<dim3((a.ncls * 9 * a.geo.b + 255) / 256, a.nrows), 256, 0, s>>>(
      a, static_cast<float2*>(a.hbuf));
  return cudaGetLastError();
}

size_t v3_tile_work_bytes(const Geometry& g, int ncls, int nrows, int precision) {
  const size_t cplx = precision == ALD_FP64 ? sizeof(double2) : sizeof(float2);
  return tile_align((size_t)g.nkc * g.b * sizeof(double)) + (size_t)nrows * ncls * 9 * g.b * cplx;
}

cudaError_t launch_v3_tile(const V3Args& a, void* work, int precision, cudaStream_t s, int l1_keep) {
  if (!v3_tile_supported(a.geo, a.ncls, precision) || a.v3_layout > 1) return cudaErrorInvalidValue;
  return precision == ALD_FP64 ? launch_tile_t<double>(a, work, l1_keep, s) : launch_tile_t<float>(a, work, l1_keep, s);
}

}  // namespace ald
