// Modal update of the air partitions (sm_103a): expansion of the face
// transforms into the force modes, the recurrence, and the contraction of the
// new modes onto the face rows, in one pass over the modes.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "ard_async.cuh"
#include "ard_device.cuh"
#include "ard_kernels.cuh"

namespace ard {

template <typename T>
struct ModalArgs {
  T* buf;
  const DctDev* dct;
  const ModalTile* tiles;
  int ntiles;
  const PointDev* srcs;
  const PointDev* recs;
  const float* series;      // [n_sources][max_steps]
  long long max_steps;
  const long long* tcount;  // steps completed before the current launch sequence
  int tstep;                // step offset inside the sequence (adjoint: counted backwards)
  int par;
  const T* resid;           // adjoint: recorder residuals [steps][n_rec_total]
  int n_rec_total;
  const CUtensorMap* maps;  // kModalMaps per air partition (build_tensor_maps)
  int* err;                 // set to 1 when a bounded wait runs out
};

// Tensor maps of an air partition: {tabA, tabB, M[0], M[1]} as one [4][d][h][wp]
// tensor (the four arrays lie one array size apart in the pool), PY as
// [6][d][wp]; for the adjoint {tabA, tabB} and {AM[0], AM[1]}.
constexpr int kModalMaps = 4;
enum { kMapForward = 0, kMapPY = 1, kMapTables = 2, kMapAdjoint = 3 };

// Shared memory in elements of T.  Stage: the tile's plane of tabA, tabB and
// the two modal levels, [32 ky][32 kx] each, and PY [6][32 kx], filled by two
// TMA boxes; a ring of kModalStages planes runs ahead across the block's tiles.
constexpr int kModalPlane = kModalTX * kModalTY;
constexpr int kModalStageElems = 4 * kModalPlane + 6 * kModalTX;
constexpr int kModalStages = 2;
constexpr int kModalRySlot = kModalWarps * 6 * kModalTX;   // [warps][ky parity][n][32 kx]
constexpr int kModalRxPitch = 8;                           // 8 lanes' partials per (q, row)
constexpr int kModalRxSlot = 6 * kModalTY * kModalRxPitch;
constexpr int kModalPt = kModalTX + kModalTY;              // a point's kx weights, ky weights
constexpr int kModalSmemElems = kModalStages * kModalStageElems + 2 * kModalRySlot + 2 * kModalRxSlot +
                                2 * kMaxPointsPerPart * kModalPt + kModalWarps * kMaxPointsPerPart;
template <typename T>
constexpr size_t modal_smem_bytes() {
  return (size_t)kModalSmemElems * sizeof(T) + 128;   // + alignment of the TMA boxes
}

// One block (4 warps) per tile of 32 kx x 32 ky x nkz planes of one kz parity;
// a thread owns 4 consecutive kx of two ky rows (y and y + 4) and walks the
// planes.  Per mode it reads M(t-1), M(t-2) and the two tables and writes
// M(t), expands the face transforms into the force mode F, and contracts M(t)
// onto the face rows: along kz in registers (partial per kz tile), along ky
// over the thread's rows, one shuffle fold and shared memory (partial per ky
// tile), along kx through shared memory (partial per kx tile).  A tile holds
// planes of one parity only, because the even / odd parts of the Z layers
// then need half the registers.
//
// The pass is bound by HBM for large partitions (20 bytes per mode) and by the
// plane-to-plane chain of one block (about 0.9 us) for small ones.  Both want
// the loads off the threads (two TMA boxes per plane, issued by warp 0 while
// the others finish the previous plane's sums) and two rows per thread, so
// that the ky sums, the Y layers and the loop are paid for once per two rows
// and two independent chains cover each other's latency.  GB300, per launch,
// against one row per thread, cp.async and 256-thread blocks before: 187.5 M
// cells in 24 partitions with 16 sources and recorders 1.67 -> 0.75 ms (5.0
// TB/s of the 20 bytes), 48.7 M cells in 128 scenes 604 -> 375 us, 12.4 M
// cells 120 -> 72 us, 1 M cells 18 -> 13 us.  A third stage takes L1 from the
// other loads (187.5 M cells 737 against 746 us, 128 scenes 378 against 375,
// rooms equal).  Points cost a launch of
// their partition 10-20 %; two are handled together to overlap their chains.
// REF selects the reference's arithmetic.
//
// ADJ runs the transposed step of the adjoint, backwards in time, on the
// adjoint modal levels mu: mu(t) = alpha mu(t+1) - a mu(t+2) + G(t), where
// alpha and -a are the forward recurrence's coefficients of M(t-1) and M(t-2)
// and G is the expansion of the adjoint face transforms with the REDFT01
// weights plus the recorder residuals injected with the recorder basis.  The
// contraction then runs on beta mu(t) (beta: the forward coefficient of the
// force mode F) with the REDFT10 weights onto the face rows and onto the
// source cells (source-series gradient partials).
template <typename T, bool REF, bool ADJ = false>
__global__ void __launch_bounds__(kModalThreads, modal_blocks_per_sm<T>()) modal_kernel(ModalArgs<T> a) {
  constexpr int TX = kModalTX, TY = kModalTY, R = 2;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const stage = reinterpret_cast<T*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  T* const ry_s = stage + kModalStages * kModalStageElems;
  T* const rx_s = ry_s + 2 * kModalRySlot;
  T* const pts = rx_s + 2 * kModalRxSlot;                   // [8 injected, 8 read out][kModalPt]
  T* const red = pts + 2 * kMaxPointsPerPart * kModalPt;    // [warps][kMaxPointsPerPart]
  __shared__ uint64_t full[kModalStages];
  __shared__ volatile int s_abort;
  __shared__ ModalTile s_it;   // thread 0's tile being loaded (kept out of the registers)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int s = 0; s < kModalStages; ++s) mbar_init(&full[s], 1);
    mbar_init_fence();
    s_abort = 0;
  }
  T* __restrict__ buf = a.buf;

  // thread 0's issue cursor over the block's (tile, plane) sequence
  int itile = blockIdx.x, ipl = 0, ist = 0;
  if (tid == 0 && itile < a.ntiles) s_it = a.tiles[itile];
  auto issue_next = [&]() {
    while (itile < a.ntiles && ipl == s_it.nkz) {
      itile += gridDim.x;
      ipl = 0;
      if (itile < a.ntiles) s_it = a.tiles[itile];
    }
    if (itile >= a.ntiles) return;
    const int x = s_it.kx0, y = s_it.ky0, kz = s_it.kz0 + 2 * ipl;
    const CUtensorMap* mp = a.maps + (long long)kModalMaps * s_it.part;
    T* st = stage + ist * kModalStageElems;
    uint64_t* bar = &full[ist];
    mbar_arrive_expect_tx(bar, (uint32_t)(kModalStageElems * sizeof(T)));
    if constexpr (ADJ) {
      tma_load_4d(st, mp + kMapTables, x, y, kz, 0, bar);
      tma_load_4d(st + 2 * kModalPlane, mp + kMapAdjoint, x, y, kz, 0, bar);
    } else {
      tma_load_4d(st, mp + kMapForward, x, y, kz, 0, bar);
    }
    tma_load_3d(st + 4 * kModalPlane, mp + kMapPY, x, kz, 0, bar);
    ist = ist + 1 == kModalStages ? 0 : ist + 1;
    ++ipl;
  };
  // Nothing that an earlier kernel writes is read before this point of the
  // block's first tile: its descriptors and basis rows are loaded while the
  // predecessor drains.
  long long t = 0;
  bool waited = false;
  auto wait_predecessor = [&]() {
    grid_dependency_wait();
    __syncthreads();   // the barriers are initialised
    t = ADJ ? (*a.tcount - a.tstep) : (*a.tcount + a.tstep);
    if (tid == 0)
      for (int s = 0; s < kModalStages; ++s) issue_next();
    waited = true;
  };

  const int li = lane & 7, yrow = lane >> 3;
  const int rs = warp * 8 + yrow;     // the thread's ky rows in the tile: rs and rs + 4 (same parity)
  const int kl0 = 4 * li;
  int sg = 0;                         // stage and phase of the plane being computed
  uint32_t phase = 0;
  int slot = 0;                       // contraction slot, alternating per plane
  bool stop = false;
  for (int tile_id = blockIdx.x; tile_id < a.ntiles && !stop; tile_id += gridDim.x) {
    const ModalTile tl = a.tiles[tile_id];
    const DctDev& D = a.dct[tl.part];
    const int w = D.w, h = D.h, d = D.d, wp = D.wp;
    const int kx0 = tl.kx0 + kl0, ky = tl.ky0 + rs;
    const int zpar = tl.kz0 & 1, nkz = tl.nkz;
    const bool colok = kx0 < wp;
    bool rowok[R];
#pragma unroll
    for (int r = 0; r < R; ++r) rowok[r] = ky + 4 * r < h;
    // FP64 is bound by its arithmetic: warps without rows in the partition skip
    // it and only keep the barriers (in FP32 the branch costs more than it saves)
    constexpr bool kSkip = sizeof(T) == 8;
    const int nact = kSkip ? min(kModalWarps, (h - tl.ky0 + 7) / 8) : kModalWarps;
    const int ninj = ADJ ? D.nrec : D.nsrc, nout = ADJ ? D.nsrc : D.nrec;
    const long long planeX = (long long)d * h, planeY = (long long)d * wp, planeZ = (long long)h * wp;
    const T* Cw = buf + D.cw;
    const T* Ch = buf + D.ch;
    const T* Cd = buf + D.cd;
    // basis rows: cx[n] as (even, odd) kx pairs, cy[n]; the REDFT01 halving of
    // the k = 0 rows sits in the contraction (forward) or the expansion (adjoint)
    bool act[4];
    Pair<T> cx[3][2];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      act[e] = kx0 + e < w;
      const T* c = Cw + (long long)min(kx0 + e, w - 1) * w;
#pragma unroll
      for (int n = 0; n < 3; ++n) (e & 1 ? cx[n][e >> 1].y : cx[n][e >> 1].x) = c[n];
    }
    T cy[R][3];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int n = 0; n < 3; ++n) cy[r][n] = rowok[r] ? Ch[(long long)(ky + 4 * r) * h + n] : (T)0;
    if (!waited) wait_predecessor();
    const T* zsrc = Cd + min(lane, 2);   // per plane: lanes 0-2 the basis row Cd[kz][0..2], lanes 8.. / 16.. the points'
    if (ninj + nout > 0) {
      // injected points (sources; adjoint: recorders) and read-out points
      // (recorders; adjoint: sources): their kx and ky weights in shared
      // memory (zeros for absent points), their kz weights
      // read by one lane each
      const T* Cwi = Cw + (long long)w * w;
      const T* Chi = Ch + (long long)h * h;
      const T* Cdi = Cd + (long long)d * d;
      const PointDev* injp = ADJ ? a.recs + D.rec0 : a.srcs + D.src0;
      const PointDev* outp = ADJ ? a.srcs + D.src0 : a.recs + D.rec0;
      if (lane >= 8 && lane - 8 < min(ninj, 8)) zsrc = (ADJ ? Cdi : Cd) + injp[lane - 8].z;
      if (lane >= 16 && lane - 16 < min(nout, 8)) zsrc = (ADJ ? Cd : Cdi) + outp[lane - 16].z;
      for (int i = tid; i < 2 * kMaxPointsPerPart * kModalPt; i += kModalThreads) {
        const int p = i / kModalPt, k = i % kModalPt;
        const bool inj = p < kMaxPointsPerPart;
        const int idx = inj ? p : p - kMaxPointsPerPart, cnt = inj ? ninj : nout;
        T v = 0;
        if (idx < cnt) {
          const PointDev q = inj ? injp[idx] : outp[idx];
          const bool ci = inj == ADJ;   // REDFT01 weights: recorders (read out forward, injected by the adjoint)
          if (k >= TX) {
            const int y = tl.ky0 + k - TX;
            if (y < h) v = (ci ? Chi : Ch)[(long long)y * h + q.y];
          } else {
            const int x = tl.kx0 + k;
            if (x < w) {
              v = (ci ? Cwi : Cw)[(long long)x * w + q.x];
              if (inj) {
                if constexpr (ADJ) v *= (T)D.si * a.resid[t * a.n_rec_total + q.slot];
                else v *= (T)D.sf * (T)(t < a.max_steps ? a.series[(long long)q.slot * a.max_steps + t] : 0.0f);
              }
            }
          }
        }
        pts[i] = v;
      }
      __syncthreads();
    }

    Pair<T> pz[R][3][2], rz[R][3][2];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        pz[r][n][0] = pz[r][n][1] = rz[r][n][0] = rz[r][n][1] = {0, 0};
        if (colok && rowok[r]) load4(buf + D.PZ + (zpar * 3 + n) * planeZ + (long long)(ky + 4 * r) * wp + kx0, pz[r][n]);
      }
    const T wx0 = kx0 == 0 ? (T)0.5 : (T)1, wy = ky == 0 ? (T)0.5 : (T)1;
    T racc[kMaxPointsPerPart];
#pragma unroll
    for (int r = 0; r < kMaxPointsPerPart; ++r) racc[r] = 0;
    const T damping = (T)D.damping;
    T* mout = buf + (ADJ ? D.AM[a.par] : D.M[a.par]) + (long long)tl.kz0 * planeZ + (long long)ky * wp + kx0;
    // per plane, lane q < 6 of a row holds PX[q][kz][ky] (q = parity 3 + n) of both rows, one plane ahead
    const T* pxp = buf + D.PX + (long long)min(li, 5) * planeX + (long long)tl.kz0 * h + (rowok[0] ? ky : 0);
    const int px4 = rowok[1] ? 4 : 0;
    zsrc += (long long)tl.kz0 * d;
    // sums of a plane: warps 1-3, two of the six RY rows (parity, n) and two of the six RX rows (q) each
    const int task = 2 * (warp - 1);
    const bool yw = warp > 0 && tl.kx0 + lane < wp, xw = warp > 0 && tl.ky0 + lane < h;
    T* yd = buf + D.RY + ((long long)tl.by * 6 + max(task, 0)) * planeY + (long long)tl.kz0 * wp + tl.kx0 + lane;
    T* xd = buf + D.RX + ((long long)tl.bx * 6 + max(task, 0)) * planeX + (long long)tl.kz0 * h + tl.ky0 + lane;
    T pxn[R] = {0, 0}, zvn = 0;   // the next plane's values
    if (nkz > 0) {
      pxn[0] = pxp[0];
      pxn[1] = pxp[px4];
      zvn = *zsrc;
    }
    for (int ip = 0; ip < nkz; ++ip) {
      const T pxv[R] = {pxn[0], pxn[1]}, zv = zvn;
      pxp += 2LL * h;
      zsrc += 2LL * d;
      if (ip + 1 < nkz) {
        pxn[0] = pxp[0];
        pxn[1] = pxp[px4];
        zvn = *zsrc;
      }
      const bool kz0th = tl.kz0 + ip == 0;   // plane kz = kz0 + 2 ip is 0
      if (!kSkip || warp < nact) {
        mbar_wait_bounded(&full[sg], phase, &s_abort);
        const T* sb = stage + sg * kModalStageElems;
        const T* st = sb + rs * TX + kl0;
        T cz[3];
        Pair<T> py[3][2], F[R][2], M[R][2];
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          cz[n] = __shfl_sync(kAll, zv, n);
          load4(sb + 4 * kModalPlane + ((yrow & 1) * 3 + n) * TX + kl0, py[n]);
        }
        // ---- expansion ----
#pragma unroll
        for (int r = 0; r < R; ++r) {
          Pair<T> fx[2], fy[2], fz[2];
#pragma unroll
          for (int n = 0; n < 3; ++n) {
            const Pair<T> px = {__shfl_sync(kAll, pxv[r], (lane & 24) + n), __shfl_sync(kAll, pxv[r], (lane & 24) + 3 + n)};
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              fx[g] = n == 0 ? mul2(cx[n][g], px) : fma2(cx[n][g], px, fx[g]);
              if constexpr (kSkip && !ADJ) {   // FP64: one running sum, the fewest operations
                fx[g] = fma2(dup2(cy[r][n]), py[n][g], fx[g]);
                fx[g] = fma2(dup2(cz[n]), pz[r][n][g], fx[g]);
              } else {
                fy[g] = n == 0 ? mul2(dup2(cy[r][n]), py[n][g]) : fma2(dup2(cy[r][n]), py[n][g], fy[g]);
                fz[g] = n == 0 ? mul2(dup2(cz[n]), pz[r][n][g]) : fma2(dup2(cz[n]), pz[r][n][g], fz[g]);
              }
            }
          }
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if constexpr (ADJ) {
              if (g == 0) fx[0].x *= wx0;
              if (r == 0) fy[g] = mul2(dup2(wy), fy[g]);
              F[r][g] = add2(fx[g], fma2(dup2(kz0th ? (T)0.5 : (T)1), fz[g], fy[g]));
            } else {
              F[r][g] = kSkip ? fx[g] : add2(add2(fx[g], fy[g]), fz[g]);
            }
          }
        }
#pragma unroll 1
        for (int s0 = 0; s0 < ninj; s0 += 2) {
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const T* c = pts + (s0 + s) * kModalPt;
            const T zs = __shfl_sync(kAll, zv, 8 + s0 + s);
            Pair<T> cw[2];
            load4(c + kl0, cw);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const T coef = c[TX + rs + 4 * r] * zs;
              F[r][0] = fma2(dup2(coef), cw[0], F[r][0]);
              F[r][1] = fma2(dup2(coef), cw[1], F[r][1]);
            }
          }
        }
        // ---- recurrence ----
#pragma unroll
        for (int r = 0; r < R; ++r) {
          Pair<T> m[2], mp[2], ta[2], tb[2];
          load4(st + 4 * r * TX, ta);
          load4(st + 4 * r * TX + kModalPlane, tb);
          load4(st + 4 * r * TX + (2 + (a.par ^ 1)) * kModalPlane, m);    // M(t-1) (adjoint: mu(t+1))
          load4(st + 4 * r * TX + (2 + a.par) * kModalPlane, mp);         // M(t-2) (adjoint: mu(t+2))
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if constexpr (REF) {   // dct_partition.cpp:68: a (2 M cwt - M_prev + (2 F / w2) (1 - cwt))
              auto one = [&](T m1, T m2, T c, T w2, T f) -> T {
                if constexpr (ADJ) return damping * ((T)2 * m1 * c - m2) + f;
                else return damping * ((T)2 * m1 * c - m2 + ((T)2 * f / (w2 != (T)0 ? w2 : (T)1)) * ((T)1 - c));
              };
              M[r][g].x = one(m[g].x, mp[g].x, ta[g].x, tb[g].x, F[r][g].x);
              M[r][g].y = one(m[g].y, mp[g].y, ta[g].y, tb[g].y, F[r][g].y);
            } else {               // the same recurrence with ta = 1 - cwt, tb = 2 (1 - cwt) / w2
              Pair<T> v = kSkip ? fma2(dup2((T)2), m[g], Pair<T>{-mp[g].x, -mp[g].y})
                                : fma2(dup2((T)-1), mp[g], add2(m[g], m[g]));
              v = fma2(mul2(dup2((T)-2), ta[g]), m[g], v);
              if constexpr (ADJ) M[r][g] = fma2(dup2(damping), v, F[r][g]);
              else M[r][g] = mul2(dup2(damping), fma2(tb[g], F[r][g], v));
            }
            M[r][g].x = act[2 * g] && rowok[r] ? M[r][g].x : (T)0;
            M[r][g].y = act[2 * g + 1] && rowok[r] ? M[r][g].y : (T)0;
          }
          if (colok && rowok[r]) store4(mout + 4LL * r * wp, M[r]);
          if constexpr (ADJ) {   // contracted: beta mu(t), the adjoint of the force mode
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              if constexpr (REF) {
                M[r][g].x *= damping * ((T)2 / (tb[g].x != (T)0 ? tb[g].x : (T)1)) * ((T)1 - ta[g].x);
                M[r][g].y *= damping * ((T)2 / (tb[g].y != (T)0 ? tb[g].y : (T)1)) * ((T)1 - ta[g].y);
              } else {
                M[r][g] = mul2(M[r][g], mul2(dup2(damping), tb[g]));
              }
            }
          }
        }
        mout += 2 * planeZ;
        // ---- read-out points, two at a time ----
        auto read_out = [&](auto first) {
          constexpr int s0 = decltype(first)::value;
#pragma unroll
          for (int s = s0; s < s0 + 2; ++s) {
            const T* c = pts + (kMaxPointsPerPart + s) * kModalPt;
            const T zs = __shfl_sync(kAll, zv, 16 + s);
            Pair<T> cw[2];
            load4(c + kl0, cw);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const Pair<T> v = fma2(cw[1], M[r][1], mul2(cw[0], M[r][0]));
              racc[s] += (c[TX + rs + 4 * r] * zs) * (v.x + v.y);
            }
          }
        };
        if (nout > 0) read_out(std::integral_constant<int, 0>{});
        if (nout > 2) read_out(std::integral_constant<int, 2>{});
        if (nout > 4) read_out(std::integral_constant<int, 4>{});
        if (nout > 6) read_out(std::integral_constant<int, 6>{});
        // ---- contraction: kz in registers, ky over the rows and by one fold, kx as 8 partials per row ----
        {
          const T wz = (!ADJ && kz0th) ? (T)0.5 : (T)1;
          T* rys = ry_s + slot * kModalRySlot + (warp * 6 + (yrow & 1) * 3) * TX + kl0;
          T* rxs = rx_s + slot * kModalRxSlot + rs * kModalRxPitch;
          Pair<T> my[2], mx[R];
          my[0] = M[0][0];
          my[1] = M[0][1];
          if (!ADJ && (!kSkip || tl.ky0 == 0)) {
            my[0] = mul2(dup2(wy), my[0]);
            my[1] = mul2(dup2(wy), my[1]);
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            mx[r] = M[r][0];
            if (!ADJ && (!kSkip || tl.kx0 == 0)) mx[r].x *= wx0;
          }
#pragma unroll
          for (int n = 0; n < 3; ++n) {
            const T czw = wz * cz[n];
            Pair<T> ry[2];
#pragma unroll
            for (int g = 0; g < 2; ++g) {
#pragma unroll
              for (int r = 0; r < R; ++r) rz[r][n][g] = fma2(dup2(czw), M[r][g], rz[r][n][g]);
              ry[g] = fma2(dup2(cy[1][n]), M[1][g], mul2(dup2(cy[0][n]), my[g]));
              ry[g] = add2(ry[g], Pair<T>{__shfl_xor_sync(kAll, ry[g].x, 16), __shfl_xor_sync(kAll, ry[g].y, 16)});
            }
            if (yrow < 2) store4(rys + n * TX, ry);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const Pair<T> v = fma2(cx[n][1], M[r][1], mul2(cx[n][0], mx[r]));   // (even, odd) kx
              // the two 16-byte halves of rows 4-7 (mod 8) are swapped, so that eight rows' reads hit all banks
              rxs[(n * TY + 4 * r) * kModalRxPitch + (li ^ (4 * r))] = v.x;
              rxs[((3 + n) * TY + 4 * r) * kModalRxPitch + (li ^ (4 * r))] = v.y;
            }
          }
        }
      }
      __syncthreads();   // partials written; stage sg read by every thread
      if (s_abort) {
        stop = true;
        break;
      }
      if (tid == 0) issue_next();
      if (yw) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const T* p = ry_s + slot * kModalRySlot + (task + k) * TX + lane;
          T v = p[0];
#pragma unroll
          for (int q = 1; q < kModalWarps; ++q)
            if (!kSkip || q < nact) v += p[q * 6 * TX];
          yd[k * planeY] = v;
        }
      }
      yd += 2LL * wp;
      if (xw) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          T p0[4], p1[4];
          const T* p = rx_s + slot * kModalRxSlot + ((task + k) * TY + lane) * kModalRxPitch;
          load4(p + (lane & 4), p0);
          load4(p + (~lane & 4), p1);
          xd[k * planeX] = ((p0[0] + p0[1]) + (p0[2] + p0[3])) + ((p1[0] + p1[1]) + (p1[2] + p1[3]));
        }
      }
      xd += 2LL * h;
      slot ^= 1;
      if (++sg == kModalStages) {
        sg = 0;
        phase ^= 1;
      }
    }
    if (stop) break;
    if (tile_id + (int)gridDim.x >= a.ntiles) grid_launch_dependents();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (colok && rowok[r]) {
#pragma unroll
        for (int n = 0; n < 3; ++n)
          store4(buf + D.RZ + ((long long)tl.bz * 6 + zpar * 3 + n) * planeZ + (long long)(ky + 4 * r) * wp + kx0, rz[r][n]);
      }
    if (nout > 0) {
#pragma unroll
      for (int r = 0; r < kMaxPointsPerPart; ++r)
        if (r < nout) {
          const T s = warp_sum(racc[r]);
          if (lane == 0) red[warp * kMaxPointsPerPart + r] = s;
        }
      __syncthreads();
      if (tid < nout) {
        T s = 0;
        for (int k = 0; k < kModalWarps; ++k) s += red[k * kMaxPointsPerPart + tid];
        buf[(ADJ ? D.srcpart : D.recpart) + (long long)tl.local * nout + tid] = s;
      }
    }
    if (ninj + nout > 0) __syncthreads();   // the points' weights and sums are read before the next tile writes its own
  }
  if (!waited) grid_dependency_wait();   // no tile: still not done before the predecessor
  if (s_abort) {
    // a wait ran out: report it, and give loads still in flight time to land
    // (bounded) before the block's shared memory is released
    if (tid == 0) {
      atomicExch(a.err, 1);
      const long long t0 = clock64();
      while (clock64() - t0 < 20000000LL) {
      }
    }
    __syncthreads();
  }
}

}  // namespace ard
