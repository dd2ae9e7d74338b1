// Three-phonon self-energy at arbitrary q on the device (THERMACOND job=2).
//
//   function_self_w3  THERMACOND/rest.f90:4012-4124  (Lorentzian, four terms, real + imaginary)
//   function_self_w4  THERMACOND/rest.f90:4126-4240  (Gaussian, three terms, imaginary only)
//   matrix_elt_full   THERMACOND/rest.f90:3664-3719
//   check_inside_bz   THERMACOND/extratools.f90:325-341, get_direct_components :561-592
//
// For a path point q, a mode la with target frequency omega and every mesh
// point k2 (k3 = -q - k2), the reference sums over l2, l3
//   |w33(q la, k2 l2, k3 l3)|^2 * self(omega, om2, om3)
// into the normal or umklapp part by check_inside_bz(k3).  Here one CTA owns
// a path point and a tile of consecutive k2; for each (q, k2) pair:
//   1. the phases exp(i (k2.R_j + k3.R_k)) per FC3 atom triple, from the
//      per-atom dot products (sum(v*w) order, no fused multiply-add);
//   2. the Fourier sum Phi[a,b,c] = sum_triples W[a,b,c] P (b^3 complex);
//   3. three mode products with e(q) (every la), e(k2), e(k3), no conjugation;
//   4. per (la, l2, l3): den, the v3_threshold cut, |w33|^2 and self, whose
//      parts are rounded to REAL(4) because CMPLX(x, y) without KIND is
//      default COMPLEX in the reference;
//   5. per-la sums over (l2, l3) and the CTA's pairs in a fixed order, as
//      per-CTA partials; self_final_kernel adds them in tile order and applies
//      the /nkc * pi of the reference.
// The eigenpairs at k3 come from the phonon kernel run on the list of k3
// points (ndisp = 1).  Compiled with -fmad=false: the arithmetic of the
// self terms follows the reference's operation order.
#include <cuda_runtime.h>

#include <algorithm>

#include "ald_internal.h"

namespace ald {

namespace {

constexpr int kSelfBlock = 256;

__device__ __forceinline__ double nbe_self(double w, double t, int m, int& bad) {  // nbe, extratools.f90:257
  if (t <= 0 || w <= 0) {
    bad = 1;
    return 0.0;
  }
  double z = w / t;
  if (m == 0) {
    if (z > 60) return 0.0;
    if (z < (double)0.0010f) return 1 / (z * (1 + z / 2 * (1 + z / 3)));
    return 1 / (exp(z) - 1);
  }
  return 1 / z;
}

__device__ __forceinline__ double dot_a(const double* v, const double* w) {  // sum(v*w)
  return __dadd_rn(__dadd_rn(__dmul_rn(v[0], w[0]), __dmul_rn(v[1], w[1])), __dmul_rn(v[2], w[2]));
}

__device__ __forceinline__ void cmac(double2& acc, const double2 e, const double2 f) {
  acc.x += e.x * f.x - e.y * f.y;
  acc.y += e.x * f.y + e.y * f.x;
}

__global__ void k3_points_kernel(int np, int nkc, const double* qp, const double* kpc, double* k3) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= (size_t)np * nkc) return;
  const int p = (int)(i / nkc), k = (int)(i % nkc);
  for (int c = 0; c < 3; ++c) k3[3 * i + c] = -qp[3 * p + c] - kpc[3 * k + c];
}

// Shared memory (double2): the point's e1 (b*b) and mode values (b: omq, omega),
// then for each pair e2, e3 (b*b each), phi, tmp (b^3 each), P (ntrip), the
// dot products k2.R and k3.R (natoms) and the modes' values (3b).
__host__ __device__ inline size_t self_point_elems(int b) { return (size_t)b * b + b; }
__host__ __device__ inline size_t self_pair_elems(int b, int ntrip, int natoms) {
  return 2 * (size_t)b * b + 2 * (size_t)b * b * b + ntrip + natoms + 3 * b;
}

// A group of nt threads takes PP pairs of one path point.  Bound by the FP64
// arithmetic of the self terms (divisions), then by the Fourier sum: the
// frequencies and occupations are formed once per mode of a pair instead of
// once per (la, l2, l3), a weight or a coefficient of e(q) read serves the PP
// pairs, and what a pair no longer needs holds its next result, so that four
// pairs' work shares a CTA of 256 threads with three resident.
template <int PP>
__global__ void __launch_bounds__(kSelfBlock) self_kernel(SelfArgs a, int nt) {
  extern __shared__ double2 sm[];
  const int b = a.b, b2 = b * b, b3 = b2 * b, nkc = a.nkc;
  const int grp = threadIdx.x / nt, lt = threadIdx.x % nt, ng = kSelfBlock / nt;
  const int p = blockIdx.y;
  const size_t per_pair = self_pair_elems(b, a.ntrip, a.natoms);
  double2* e1 = sm;
  double* omq = reinterpret_cast<double*>(sm + b2);  // omq [b], omega [b]
  double2* base = sm + self_point_elems(b) + (size_t)grp * PP * per_pair;
  const int kfirst = (blockIdx.x * ng + grp) * PP;  // pair u: k2 = kfirst + u; past the mesh: the last k2, discarded
  // where a pair's parts lie
  const size_t oe3 = b2, ophi = 2 * (size_t)b2, otmp = ophi + b3, oP = otmp + b3, od = oP + a.ntrip,
               om = od + a.natoms;  // om: om2 [b], nb2 [b], om3 [b], nb3 [b], then ints: bad2 [b], bad3 [b], inside
  const double2* evq = reinterpret_cast<const double2*>(a.evq) + (size_t)p * b2;
  const double2* ev2 = reinterpret_cast<const double2*>(a.ev2);
  const double2* ev3 = reinterpret_cast<const double2*>(a.ev3);
  const double cn = a.cnst, eta = a.eta, pi = a.pi;
  const double q[3] = {a.qp[3 * p], a.qp[3 * p + 1], a.qp[3 * p + 2]};
  for (int e = threadIdx.x; e < b2; e += blockDim.x) e1[e] = evq[e];
  for (int l = threadIdx.x; l < b; l += blockDim.x) {
    omq[l] = sqrt(fabs(a.wq[(size_t)p * b + l])) * cn;
    omq[b + l] = a.omega[(size_t)p * b + l];
  }
  for (int e = lt; e < PP * b2; e += nt) {
    const int u = e / b2, r = e - u * b2, k2 = min(kfirst + u, nkc - 1);
    base[u * per_pair + r] = ev2[(size_t)k2 * b2 + r];
    base[u * per_pair + oe3 + r] = ev3[((size_t)p * nkc + k2) * b2 + r];
  }
  for (int e = lt; e < PP * a.natoms; e += nt) {
    const int u = e / a.natoms, j = e - u * a.natoms, k2 = min(kfirst + u, nkc - 1);
    double kk2[3], k3[3];
    for (int c = 0; c < 3; ++c) {
      kk2[c] = a.kpc[3 * k2 + c];
      k3[c] = -q[c] - kk2[c];
    }
    double* d23 = reinterpret_cast<double*>(base + u * per_pair + od);
    d23[j] = dot_a(kk2, a.rr + 3 * j);
    d23[a.natoms + j] = dot_a(k3, a.rr + 3 * j);
  }
  for (int e = lt; e < PP * 2 * b; e += nt) {
    const int u = e / (2 * b), h = (e - u * 2 * b) / b, l = e % b, k2 = min(kfirst + u, nkc - 1);
    double* md = reinterpret_cast<double*>(base + u * per_pair + om);
    const double w = h ? a.w3[((size_t)p * nkc + k2) * b + l] : a.w2[(size_t)k2 * b + l];
    const double o = sqrt(fabs(w)) * cn;
    int bad = 0;
    md[2 * h * b + l] = o;
    md[2 * h * b + b + l] = nbe_self(o, a.temp, a.classical, bad);
    reinterpret_cast<int*>(md + 4 * b)[h * b + l] = bad;
  }
  for (int u = lt; u < PP; u += nt) {  // check_inside_bz of k3
    const int k2 = min(kfirst + u, nkc - 1);
    double q2[3];
    for (int c = 0; c < 3; ++c) q2[c] = (-q[c] - a.kpc[3 * k2 + c]) + a.ghalf[c];
    int inside = 1;
    for (int r = 0; r < 3; ++r) {
      const double x = dot_a(q2, a.gd + 3 * r) + 5e-10;
      if (x < 0 || x >= 1) inside = 0;
    }
    reinterpret_cast<int*>(reinterpret_cast<double*>(base + u * per_pair + om) + 4 * b)[2 * b] = inside;
  }
  __syncthreads();
  for (int e = lt; e < PP * a.ntrip; e += nt) {
    const int u = e / a.ntrip, t = e - u * a.ntrip;
    const double* d23 = reinterpret_cast<const double*>(base + u * per_pair + od);
    double sn, cs;
    sincos(__dadd_rn(d23[a.trip_j[t]], d23[a.natoms + a.trip_k[t]]), &sn, &cs);
    base[u * per_pair + oP + t] = make_double2(cs, sn);
  }
  __syncthreads();
  // Fourier sum: channel (a,b,c) = (3*i0+al, 3*j0+be, 3*k0+ga)
  const int nat0 = a.nat0;
  for (int o = lt; o < b3; o += nt) {
    const int ca = o / b2, cb = (o / b) % b, cc = o % b;
    const int blk = ((ca / 3) * nat0 + cb / 3) * nat0 + cc / 3;
    const int comp = (ca % 3) * 9 + (cb % 3) * 3 + (cc % 3);
    double2 acc[PP];
#pragma unroll
    for (int u = 0; u < PP; ++u) acc[u] = make_double2(0.0, 0.0);
    const int t1 = a.blk_off[blk + 1];
#pragma unroll 2
    for (int t = a.blk_off[blk]; t < t1; ++t) {
      const double w = __ldg(a.fc3w + 27 * (size_t)t + comp);
#pragma unroll
      for (int u = 0; u < PP; ++u) {
        const double2 ph = base[u * per_pair + oP + t];
        acc[u].x += w * ph.x;
        acc[u].y += w * ph.y;
      }
    }
#pragma unroll
    for (int u = 0; u < PP; ++u) base[u * per_pair + ophi + o] = acc[u];
  }
  __syncthreads();
  // tmp[la][b][c] = sum_a e1[la][a] phi[a][b][c]
  for (int o = lt; o < b3; o += nt) {
    const int l1 = o / b2, bc = o % b2;
    double2 acc[PP];
#pragma unroll
    for (int u = 0; u < PP; ++u) acc[u] = make_double2(0.0, 0.0);
    for (int k = 0; k < b; ++k) {
      const double2 e = e1[l1 * b + k];
#pragma unroll
      for (int u = 0; u < PP; ++u) cmac(acc[u], e, base[u * per_pair + ophi + k * b2 + bc]);
    }
#pragma unroll
    for (int u = 0; u < PP; ++u) base[u * per_pair + otmp + o] = acc[u];
  }
  __syncthreads();
  // phi[la][l2][c] = sum_b e2[l2][b] tmp[la][b][c]
  for (int o = lt; o < b3; o += nt) {
    const int l1 = o / b2, l2 = (o / b) % b, c = o % b;
    double2 acc[PP];
#pragma unroll
    for (int u = 0; u < PP; ++u) acc[u] = make_double2(0.0, 0.0);
    for (int k = 0; k < b; ++k)
#pragma unroll
      for (int u = 0; u < PP; ++u)
        cmac(acc[u], base[u * per_pair + l2 * b + k], base[u * per_pair + otmp + l1 * b2 + k * b + c]);
#pragma unroll
    for (int u = 0; u < PP; ++u) base[u * per_pair + ophi + o] = acc[u];
  }
  __syncthreads();
  // the third product and the self terms: tmp[la][l2][l3]
  for (int e = lt; e < PP * b3; e += nt) {
    const int u = e / b3, o = e - u * b3, l1 = o / b2, l2 = (o / b) % b, l3 = o % b;
    double2* pr = base + u * per_pair;
    const double* md = reinterpret_cast<const double*>(pr + om);
    const int* bad = reinterpret_cast<const int*>(md + 4 * b);
    double2 acc = make_double2(0.0, 0.0);
    for (int k = 0; k < b; ++k) cmac(acc, pr[oe3 + l3 * b + k], pr[ophi + l1 * b2 + l2 * b + k]);
    double2 con = make_double2(0.0, 0.0);
    const double om2 = md[l2], om3 = md[2 * b + l3], omega = omq[b + l1];
    const double den = sqrt(8 * omq[l1] * om2 * om3 / (cn * cn * cn));
    const bool live = kfirst + u < nkc;
    if (den == 0.0) {
      if (live) atomicOr(a.err, 2);
    } else if (live) {
      const double re = acc.x / den * a.const33, im = acc.y / den * a.const33;
      const double term = __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
      // |w33| < v3_threshold, by the squares unless they are within rounding of each other
      const double lim = a.v3thr * a.v3thr;
      const bool below = term < lim * (1 - 1e-12) ? true : term > lim * (1 + 1e-12) ? false : hypot(re, im) < a.v3thr;
      if (!below) {
        if (bad[l2] | bad[b + l3]) atomicOr(a.err, 1);
        const double nb2 = md[b + l2], nb3 = md[3 * b + l3];
        double ires = 0, rres = 0, arg;
        if (!a.gauss) {
          arg = (omega - om3) - om2;
          if (fabs(arg) < a.etacut) {
            ires = (nb3 + nb2 + 1) * (eta / (arg * arg + eta * eta) / pi);
            rres = (nb3 + nb2 + 1) * arg / (arg * arg + eta * eta);
          }
          arg = (omega + om3) + om2;
          if (fabs(arg) < a.etacut) {
            ires = ires - (nb3 + nb2 + 1) * (eta / (arg * arg + eta * eta) / pi);
            rres = rres - (nb3 + nb2 + 1) * arg / (arg * arg + eta * eta);
          }
          arg = (omega - om3) + om2;
          if (fabs(arg) < a.etacut) {
            ires = ires + (nb2 - nb3) * (eta / (arg * arg + eta * eta) / pi);
            rres = rres + (nb2 - nb3) * arg / (arg * arg + eta * eta);
          }
          arg = (omega - om2) + om3;
          if (fabs(arg) < a.etacut) {
            ires = ires + (nb3 - nb2) * (eta / (arg * arg + eta * eta) / pi);
            rres = rres + (nb3 - nb2) * arg / (arg * arg + eta * eta);
          }
        } else {
          const double g0 = sqrt(2 * pi);
          arg = (omega - om3) - om2;
          if (fabs(arg) < a.etacut) ires = (nb3 + nb2 + 1) * (exp(-arg * arg / 2.0 / eta / eta) / g0 / eta);
          arg = (omega - om3) + om2;
          if (fabs(arg) < a.etacut) ires = ires + (nb2 - nb3) * (exp(-arg * arg / 2.0 / eta / eta) / g0 / eta);
          arg = (omega - om2) + om3;
          if (fabs(arg) < a.etacut) ires = ires + (nb3 - nb2) * (exp(-arg * arg / 2.0 / eta / eta) / g0 / eta);
        }
        const double sre = (double)__double2float_rn(rres), sim = (double)__double2float_rn(ires * pi);
        con = make_double2(term * sre, term * sim);
      }
    }
    pr[otmp + o] = con;
  }
  __syncthreads();
  // per-la sums over (l2, l3), four lanes to a sum; then over the CTA's pairs
  // in their order, into the normal or the umklapp part
  for (int r0 = 0; r0 < PP * 2 * b; r0 += nt / 4) {
    const int r = r0 + lt / 4, u = min(r, PP * 2 * b - 1) / (2 * b), h = r % (2 * b);
    const double* con = reinterpret_cast<const double*>(base + u * per_pair + otmp + (h / 2) * b2);
    double s = 0;
    for (int v = lt & 3; v < b2; v += 4) s += con[2 * v + (h & 1)];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (r < PP * 2 * b && (lt & 3) == 0) reinterpret_cast<double*>(base + u * per_pair)[h] = s;  // over e2
  }
  __syncthreads();
  for (int r = threadIdx.x; r < 4 * b; r += blockDim.x) {
    const int l1 = r / 4, part = r % 4;
    double s = 0;
    for (int u = 0; u < ng * PP; ++u) {
      const double2* pr = sm + self_point_elems(b) + u * per_pair;
      const int inside = reinterpret_cast<const int*>(reinterpret_cast<const double*>(pr + om) + 4 * b)[2 * b];
      if (inside == (part < 2)) s += reinterpret_cast<const double*>(pr)[2 * l1 + (part & 1)];
    }
    a.part[((size_t)p * gridDim.x + blockIdx.x) * 4 * b + r] = s;
  }
}

// a CTA per path point: its threads take (slice of the tiles, value), the
// slices are added in their order
__global__ void __launch_bounds__(kSelfBlock) self_final_kernel(int b, int nblk, int nkc, double pi,
                                                                const double* part, double* out) {
  __shared__ double red[kSelfBlock];
  const int p = blockIdx.x, w = 4 * b, nsl = kSelfBlock / w, r = threadIdx.x % w, sl = threadIdx.x / w;
  double s = 0;
  if (sl < nsl)
#pragma unroll 8
    for (int k = sl; k < nblk; k += nsl) s += part[((size_t)p * nblk + k) * w + r];
  red[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < w) {
    for (int k = 1; k < nsl; ++k) s += red[k * w + r];
    out[(size_t)p * w + r] = s / (double)nkc * pi;  // nself/nkc*pi, uself/nkc*pi
  }
}

// threads to a group, pairs to a group; returns the shared memory
size_t self_shape(const SelfArgs& a, int* nt_out, int* pp_out) {
  const int b3 = a.b * a.b * a.b;
  int nt = 32;
  while (nt < b3 && nt < kSelfBlock) nt *= 2;
  const size_t pair = self_pair_elems(a.b, a.ntrip, a.natoms) * sizeof(double2);
  const size_t point = self_point_elems(a.b) * sizeof(double2);
  int pp = 4;  // as many as leave three CTAs to an SM, then two; else one pair at a time
  auto bytes = [&] { return point + (size_t)(kSelfBlock / nt) * pp * pair; };
  while (pp > 1 && bytes() > 75 * 1024) pp /= 2;
  while (nt < kSelfBlock && bytes() > 113 * 1024) nt *= 2;
  *nt_out = nt;
  *pp_out = pp;
  return bytes();
}

}  // namespace

size_t self_partial_doubles(const SelfArgs& a) {
  int nt, pp;
  self_shape(a, &nt, &pp);
  const int ppb = kSelfBlock / nt * pp;
  return (size_t)a.np * ((a.nkc + ppb - 1) / ppb) * 4 * a.b;
}

cudaError_t launch_k3_points(int np, int nkc, const double* qp, const double* kpc, double* k3, cudaStream_t s) {
  const size_t n = (size_t)np * nkc;
  k3_points_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(np, nkc, qp, kpc, k3);
  return cudaGetLastError();
}

cudaError_t launch_self(const SelfArgs& a, double* out, cudaStream_t s) {
  int nt, pp;
  const size_t sm = self_shape(a, &nt, &pp);
  if (sm > 200 * 1024) return cudaErrorInvalidValue;
  auto kern = pp == 4 ? self_kernel<4> : pp == 2 ? self_kernel<2> : self_kernel<1>;
  if (sm > 48 * 1024) {
    cudaError_t e = raise_smem_limit((const void*)kern, sm);
    if (e != cudaSuccess) return e;
  }
  const int ppb = kSelfBlock / nt * pp, nblk = (a.nkc + ppb - 1) / ppb;
  kern<<<dim3(nblk, a.np), kSelfBlock, sm, s>>>(a, nt);
  self_final_kernel<<<a.np, kSelfBlock, 0, s>>>(a.b, nblk, a.nkc, a.pi, a.part, out);
  return cudaGetLastError();
}

}  // namespace ald
