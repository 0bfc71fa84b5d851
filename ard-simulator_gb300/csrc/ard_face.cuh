// Fused 2D transforms of the face layers (sm_103a): both transforms of a pair
// of layers in one kernel, in quadrants.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "ard_device.cuh"
#include "ard_kernels.cuh"

namespace ard {

constexpr int kFaceThreads = 256;

// Half length of a transform, its padded form, and the row pitch of staged
// operands: 4 mod 8 elements, so that consecutive rows start in distinct
// 16-byte bank groups.
__host__ __device__ inline int face_half(int n) { return (n + 1) >> 1; }
__host__ __device__ inline int face_half4(int n) { return (face_half(n) + 3) & ~3; }
__host__ __device__ inline int face_pitch(int n) {
  const int n4 = face_half4(n);
  return n4 + ((n4 & 7) ? 0 : 4);
}

// Parity-split transform tables of extent n, for one basis (C or Ci):
//   Hr[p][m][j] = basis(2 m + p, j)   rows: transform index of parity p
//   Hf[p][j][m] = basis(2 m + p, j)   the transposes
// for j < half, rows of pitch half4, zeros where 2 m + p >= n and in the
// padding.  Stored as Hr(C), Hf(C), Hr(Ci), Hf(Ci).
__host__ __device__ inline long long face_table_elems(int n) { return 2LL * face_half(n) * face_half4(n); }
enum { kFaceHr = 0, kFaceHf = 1, kFaceC = 0, kFaceCi = 2 };

// Shared memory of a launch, in elements (maxima over its jobs).
struct FaceSmem {
  int f;   // quadrants of the layers, then (inverse) of the results
  int a;   // table along V
  int b;   // table along U, the job's columns
  int t;   // between the two products
};

// What a block makes of job J (entry `half` of its pair, Face2DJob::split).
struct FaceShape {
  int no;        // outputs (even / odd combination of the layer pair)
  int o0;        // first of them
  int npu, pu0;  // parities along U
  int c0, nc;    // columns of each quadrant
};
__host__ __device__ inline FaceShape face_shape(const Face2DJob& J, int half, bool inverse) {
  FaceShape s;
  s.no = J.which == 0 ? 2 : 1;
  s.o0 = J.which == 2 ? 1 : 0;
  s.npu = 2;
  s.pu0 = 0;
  s.c0 = J.u0 >> 1;
  s.nc = (J.ub + 1) >> 1;
  if (J.split && !inverse) {        // one parity each
    s.npu = 1;
    s.pu0 = half;
  } else if (J.split) {             // half of the columns each
    const int first = (((s.nc + 1) >> 1) + 3) & ~3;
    if (half) {
      s.c0 += first;
      s.nc = s.nc > first ? s.nc - first : 0;
    } else {
      s.nc = s.nc < first ? s.nc : first;
    }
  }
  return s;
}
inline FaceSmem face_smem(const Face2DJob& J, int half, bool inverse) {
  const FaceShape s = face_shape(J, half, inverse);
  const int hv = face_half(J.V), nc4 = (s.nc + 3) & ~3, units = s.no * 2 * s.npu;
  FaceSmem m;
  m.f = units * hv * face_pitch(J.U);
  if (inverse) m.f = std::max(m.f, units * hv * nc4);
  m.a = 2 * hv * face_pitch(J.V);
  m.b = s.npu * face_half4(J.U) * nc4;
  m.t = units * face_half4(J.V) * nc4;
  return m;
}

// Division by a value of the job: i / d = umulhi(i + 1, floor((2^32 - 1) / d)),
// exact for 0 <= i, (i + 1) d <= 2^32.  The kernel's loops split their flat
// index by such values all the time; with the compiler's division that was
// half of its instructions.
struct FaceDiv {
  unsigned m;
  int d;
  __device__ __forceinline__ explicit FaceDiv(int v) : m(0xffffffffu / (unsigned)v), d(v) {}
  __device__ __forceinline__ int split(int i, int& rem) const {
    const int q = (int)__umulhi((unsigned)i + 1u, m);
    rem = i - q * d;
    return q;
  }
};

// One half-size product per unit: W[u][r][c] = sum_k L[u][r][k] R[u][k][c] for
// r < rows, c < 4 nq, k < K (a multiple of 4; operands are zero past their
// extent), from the last k down if REV.  A thread owns MR rows x 4 columns; its
// rows are rg apart, so the rows that a warp loads together are consecutive.
template <typename T, bool REV, int MR, typename LOf, typename ROf, typename Out>
__device__ __forceinline__ void face_product(int units, int rows, int K, const FaceDiv& nq, int lp, int rp, LOf l_of,
                                             ROf r_of, Out out) {
  const FaceDiv rg((rows + MR - 1) / MR);
  for (int tile = threadIdx.x; tile < units * rg.d * nq.d; tile += kFaceThreads) {
    int ct, rt;
    const int u = rg.split(nq.split(tile, ct), rt);
    const T* L = l_of(u) + rt * lp;
    const T* Rr = r_of(u) + 4 * ct;
    int lo[MR];
#pragma unroll
    for (int i = 0; i < MR; ++i) lo[i] = (rt + i * rg.d < rows ? i * rg.d : 0) * lp;
    Pair<T> acc[MR][2];
#pragma unroll
    for (int i = 0; i < MR; ++i) acc[i][0] = acc[i][1] = {0, 0};
#pragma unroll 2
    for (int k = REV ? K - 4 : 0; REV ? k >= 0 : k < K; k += REV ? -4 : 4) {
      T l[MR][4];
      Pair<T> r[4][2];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) load4(Rr + (k + kk) * rp, r[kk]);
#pragma unroll
      for (int i = 0; i < MR; ++i) load4(L + lo[i] + k, l[i]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int kk = REV ? 3 - q : q;
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
          for (int c = 0; c < 2; ++c) acc[i][c] = fma2(dup2(l[i][kk]), r[kk][c], acc[i][c]);
      }
    }
#pragma unroll
    for (int i = 0; i < MR; ++i)
      if (rt + i * rg.d < rows) {
        const T v[4] = {acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y};
        out(u, rt + i * rg.d, 4 * ct, v);
      }
  }
}

// Four elements p[0..3] with p[e] read where e < n (zeros past them); `vec`: p
// is aligned for one 128-bit load.
template <typename T>
__device__ __forceinline__ void load_quad(const T* p, int n, bool vec, T (&v)[4]) {
  if (vec && n >= 4) {
    load4(p, v);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = e < n ? p[e] : (T)0;
  }
}

// One block per job (pair entry) of the list: the 2D transforms
//   out0 = scale A (X0 + X1) B,   out1 = scale A (X0 - X1) B
// of a pair of V x U layers (row pitch ld), for a slab of output columns.
//
// The bases satisfy basis(k, n - 1 - j) = (-1)^k basis(k, j), so a transform of
// length n is two of half the length, on the even / odd parts of the input
// (INV false: sums over j) or giving the even / odd parts of the output (INV
// true: sums over k).  Along both axes that makes four quadrants (pv, pu) per
// output, each a chain of two half-size products T = F B, O = A T: half the
// arithmetic of the full products, and quadrants are independent until the
// inverse's last butterfly.
//   INV false: F[pv][pu] = the layer folded along both axes, O = out[2 o + pv][2 c + pu]
//   INV true:  F[pv][pu][i][j] = the layer at (2 i + pv, 2 j + pu); the four O at (o, c)
//              combine to out at (o | V - 1 - o, c | U - 1 - c)
// A job takes 16 columns c of each quadrant and one or both outputs; the
// entries of a split job take one parity pu each (INV false) or half of the
// columns each (INV true).
//
// The inverse adds its modes from the highest down (REV).  Its even and odd
// parts hold the sum and the difference of a cell and its mirror cell, so a quiet
// cell opposite a loud one gets the rounding of the loud one's sums, where a
// full-length sum rounds by its own size; with the low modes, the largest, added
// last, the sums are small until their last terms.  FP32 against FP64, 64 random
// scenes, recorders over 1200 steps, full-length products / half-length from the
// low modes up / from the high ones down: geometric mean 3.14e-6 / 3.11e-6 /
// 3.00e-6, worst (a scene that grows) 7.7e-5 / 1.5e-4 / 7.3e-5.  The order costs
// no time; sums in blocks of four modes gained nothing more (+4 % in batches).
//
// Small launches (one room) are bound by the chain load - product - product -
// store of one block, large ones (batches) by the barriers between those phases
// with two blocks per SM (issue 37 %).  Layers go through registers once (folded
// or sorted by parity on the way), tables by cp.async underneath; indexes are
// split by multiplication (FaceDiv) and the products run on packed FP32 pairs.
// GB300, both directions of a step, against full-length products with rows split
// over a cluster: one 100^3 room 25 -> 17 us, the L-shaped room of 1.9 M cells
// 51 -> 38 us, 128 scenes 714 -> 435 us (485 us with compiled divisions, 449 us
// with scalar products); FP64 (0.24 M cells) 213 -> 129 us.
template <typename T, bool INV>
__global__ void __launch_bounds__(kFaceThreads, 2) face_kernel(T* __restrict__ buf, const Face2DJob* __restrict__ jobs,
                                                               int entries, FaceSmem sm) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const Fs = reinterpret_cast<T*>(smem_raw);
  T* const As = Fs + sm.f;
  T* const Bs = As + sm.a;
  T* const Ts = Bs + sm.b;
  const int tid = threadIdx.x;
  bool waited = false;   // jobs and tables are constants: loaded while the predecessor drains
  for (int it = blockIdx.x; it < entries; it += gridDim.x) {
    const Face2DJob J = jobs[it];
    const FaceShape s = face_shape(J, it & 1, INV);
    if (J.V == 0 || s.nc <= 0) continue;
    const int V = J.V, U = J.U, ld = J.ld;
    const int hv = face_half(V), hu = face_half(U), hv4 = face_half4(V), hu4 = face_half4(U);
    const int fp = face_pitch(U), ap = face_pitch(V);
    const int nq = (s.nc + 3) >> 2, ncp = 4 * nq;
    const int npu = s.npu, units = s.no * 2 * npu;   // unit = (out 2 + pv) npu + pu
    const int su = npu - 1;                          // npu is 1 or 2: u / npu = u >> su, u % npu = u & su
    const FaceDiv dq(nq);
    __syncthreads();   // the previous job is done with shared memory
    // ---- tables (zero-padded rows, always 16-byte aligned) ----
    const FaceDiv dv(hv4 >> 2), du(hu4);
    for (int i = tid; i < 2 * hv * dv.d; i += kFaceThreads) {
      int q;
      const int row = dv.split(i, q);
      cp_async4(As + row * ap + 4 * q, buf + J.tabA + (long long)row * hv4 + 4 * q, true);
    }
    for (int i = tid; i < npu * hu4 * nq; i += kFaceThreads) {
      int c, j;
      const int p = du.split(dq.split(i, c), j);
      const bool ok = j < hu && s.c0 + 4 * c < hu4;
      cp_async4(Bs + (p * hu4 + j) * ncp + 4 * c,
                buf + J.tabB + (ok ? ((long long)(s.pu0 + p) * hu + j) * hu4 + s.c0 + 4 * c : 0), ok);
    }
    cp_async_commit();
    for (int i = tid; i < (hv4 - hv) * ncp; i += kFaceThreads)   // rows past the half length read as zero
      for (int u = 0; u < units; ++u) Ts[(u * hv4 + hv) * ncp + i] = (T)0;
    if (!waited) {
      grid_dependency_wait();
      waited = true;
    }
    // ---- the layers, combined and folded (or sorted by parity) ----
    const T* X[2] = {buf + J.in0, buf + J.in1};
    const bool al = ((J.in0 | J.in1 | ld) & 3) == 0;
    if constexpr (!INV) {
      const bool alr = al && (U & 3) == 0;
      const FaceDiv dqu(hu4 >> 2);
      for (int i = tid; i < hv * dqu.d; i += kFaceThreads) {
        int q;
        const int r = dqu.split(i, q), r2 = V - 1 - r;
        const int n = min(4, hu - 4 * q);
        T d[2][2][4], m[2][2][4];   // [layer][row r, row r2]: direct, mirrored along U
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const T* p = X[x] + (long long)(y ? r2 : r) * ld;
            load_quad(p + 4 * q, n, al, d[x][y]);
            if (alr && n >= 4) {
              T v[4];
              load4(p + U - 4 - 4 * q, v);
#pragma unroll
              for (int e = 0; e < 4; ++e) m[x][y][e] = v[3 - e];
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) m[x][y][e] = e < n ? p[U - 1 - 4 * q - e] : (T)0;
            }
          }
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          if (o < s.o0 || o >= s.o0 + s.no) continue;
          T e0[2][4], e1[2][4];   // [row]: even, odd part along U
#pragma unroll
          for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const bool mid = 2 * (4 * q + e) + 1 == U;
              const T a = o ? d[0][y][e] - d[1][y][e] : d[0][y][e] + d[1][y][e];
              const T b = o ? m[0][y][e] - m[1][y][e] : m[0][y][e] + m[1][y][e];
              e0[y][e] = mid ? a : a + b;
              e1[y][e] = mid ? (T)0 : a - b;
            }
          const bool midr = r == r2;
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            if (p < s.pu0 || p >= s.pu0 + npu) continue;
            T fe[4], fo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const T a = p ? e1[0][e] : e0[0][e], b = p ? e1[1][e] : e0[1][e];
              fe[e] = midr ? a : a + b;
              fo[e] = midr ? (T)0 : a - b;
            }
            T* f = Fs + ((o - s.o0) * 2 * npu + p - s.pu0) * hv * fp + r * fp + 4 * q;
            store4(f, fe);
            store4(f + npu * hv * fp, fo);
          }
        }
      }
    } else {
      // quads of two half-columns: rows kv (zeros past V), columns 4 q .. 4 q + 3
      const FaceDiv dq2(hu4 >> 1);
      for (int i = tid; i < 2 * hv * dq2.d; i += kFaceThreads) {
        int q;
        const int kv = dq2.split(i, q);
        const int n = kv < V ? U - 4 * q : 0;
        T x0[4], x1[4];
        load_quad(X[0] + (long long)kv * ld + 4 * q, n, al, x0);
        load_quad(X[1] + (long long)kv * ld + 4 * q, n, al, x1);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          if (o < s.o0 || o >= s.o0 + s.no) continue;
          T wv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) wv[e] = o ? x0[e] - x1[e] : x0[e] + x1[e];
          T* f = Fs + (((o - s.o0) * 2 + (kv & 1)) * 2) * hv * fp + (kv >> 1) * fp + 2 * q;
          f[0] = wv[0];
          f[1] = wv[2];
          f[hv * fp] = wv[1];
          f[hv * fp + 1] = wv[3];
        }
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    // ---- T = F B ----
    auto f_of = [&](int u) { return Fs + u * hv * fp; };
    auto b_of = [&](int u) { return Bs + (u & su) * hu4 * ncp; };
    auto to_t = [&](int u, int r, int c, const T (&v)[4]) { store4(Ts + (u * hv4 + r) * ncp + c, v); };
    const bool wide = units * ((hv + 3) >> 2) * nq >= kFaceThreads / 2;
    if (wide) face_product<T, INV, 4>(units, hv, hu4, dq, fp, ncp, f_of, b_of, to_t);
    else      face_product<T, INV, 2>(units, hv, hu4, dq, fp, ncp, f_of, b_of, to_t);
    __syncthreads();
    if (it + (int)gridDim.x >= entries) grid_launch_dependents();
    // ---- O = A T ----
    const T scale = (T)J.scale;
    auto a_of = [&](int u) { return As + (u >> su & 1) * hv * ap; };
    auto t_of = [&](int u) { return Ts + u * hv4 * ncp; };
    if constexpr (!INV) {
      auto to_out = [&](int u, int r, int c, const T (&v)[4]) {
        const int pu = s.pu0 + (u & su), pv = u >> su & 1, o = s.o0 + (u >> su >> 1);
        const int kv = 2 * r + pv, ku = 2 * (s.c0 + c) + pu;
        if (kv >= V) return;
        T* p = buf + (o ? J.out1 : J.out0) + (long long)kv * ld + ku;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c + e < s.nc && ku + 2 * e < U) p[2 * e] = v[e] * scale;
      };
      if (wide) face_product<T, INV, 4>(units, hv, hv4, dq, ap, ncp, a_of, t_of, to_out);
      else      face_product<T, INV, 2>(units, hv, hv4, dq, ap, ncp, a_of, t_of, to_out);
    } else {
      auto to_o = [&](int u, int r, int c, const T (&v)[4]) { store4(Fs + (u * hv + r) * ncp + c, v); };
      if (wide) face_product<T, INV, 4>(units, hv, hv4, dq, ap, ncp, a_of, t_of, to_o);
      else      face_product<T, INV, 2>(units, hv, hv4, dq, ap, ncp, a_of, t_of, to_o);
      __syncthreads();
      // ---- the quadrants' butterfly ----
      const FaceDiv dc(ncp), dr(hv);
      for (int i = tid; i < s.no * hv * ncp; i += kFaceThreads) {
        int c, r;
        const int o = dr.split(dc.split(i, c), r);
        const int u = s.c0 + c, u2 = U - 1 - u, r2 = V - 1 - r;
        if (c >= s.nc || u >= hu) continue;
        const T* q = Fs + (o * 4 * hv + r) * ncp + c;   // units (pv, pu) = 0 .. 3, hv rows apart
        const T ee = q[0], eo = q[hv * ncp], oe = q[2 * hv * ncp], oo = q[3 * hv * ncp];
        T* p = buf + (s.o0 + o ? J.out1 : J.out0);
        const T a = ee + oe, b = eo + oo, d = ee - oe, f = eo - oo;
        p[(long long)r * ld + u] = (a + b) * scale;
        if (u2 != u) p[(long long)r * ld + u2] = (a - b) * scale;
        if (r2 != r) {
          p[(long long)r2 * ld + u] = (d + f) * scale;
          if (u2 != u) p[(long long)r2 * ld + u2] = (d - f) * scale;
        }
      }
    }
  }
  if (!waited) grid_dependency_wait();   // no job: still not done before the predecessor
}

// Launch over a list of 2 n entries, at most max_ctas blocks.
template <typename T, bool INV>
inline cudaError_t launch_face(long long n, int max_ctas, size_t smem, cudaStream_t s, T* buf, const Face2DJob* jobs,
                               const FaceSmem& sm) {
  if (n <= 0) return cudaSuccess;
  const long long b = std::max(1LL, std::min(2 * n, (long long)max_ctas));
  return launch_dep(face_kernel<T, INV>, b, kFaceThreads, smem, s, buf, jobs, (int)(2 * n), sm);
}

// The parity-split tables of extent n at `off`, from the extent's cosine table
// at `cos` (C, Ci: n x n each).
template <typename T>
__global__ void face_table_kernel(T* buf, long long off, long long cos, int n) {
  const int h = face_half(n), h4 = face_half4(n);
  const long long S = face_table_elems(n), nn = (long long)n * n;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < S; i += (long long)gridDim.x * blockDim.x) {
    const int col = (int)(i % h4), row = (int)(i / h4 % h), p = (int)(i / ((long long)h4 * h));
    for (int b = 0; b < 2; ++b) {   // C, Ci
      auto basis = [&](int m, int j) -> T {
        const int k = 2 * m + p;
        return k < n && j < h ? buf[cos + b * nn + (long long)k * n + j] : (T)0;
      };
      buf[off + 2 * b * S + i] = basis(row, col);       // Hr[p][row = m][col = j]
      buf[off + (2 * b + 1) * S + i] = basis(col, row); // Hf[p][row = j][col = m]
    }
  }
}

}  // namespace ard
