// Update kernel of the split stage with the conserved state staged by the
// Tensor Memory Accelerator (sm_100a).
//
// k_update waits on memory (8.7 of 14 warp cycles per issued instruction at
// 24 warps per SM): per point it reads 14 variables x (six faces, the state,
// the state at the step's start), and the registers of the temperature and
// transport evaluation that follow leave room for few of these loads in
// flight.  Here the two conserved states, more than half of the bytes, arrive
// by cp.async.bulk.tensor: one 4D box (UX x UY points of one plane, every
// variable) per state, requested for plane k + 1 as soon as the new state of
// plane k is in registers, so that the copies run beside the Newton, the
// transport and the stores of plane k and take no registers.  The faces are
// read while the box is on its way, all before the first is used.  60 KB per
// CTA at 9 species (57 of them the boxes), two CTAs of 128 registers per SM.
// The autotuner times it against k_update: FP32 takes it (128^3: 0.308 to 0.314
// against 0.346 ms per stage; the channel's steady step, which reads one state
// and has a time step per point, 0.054 against 0.061).  FP64, whose faces and
// states together spill here, would not (97 x 85 x 71: 0.286 against 0.248 ms)
// and is not timed with it.
//
// Waits are bounded as in the face kernel: a CTA whose box does not arrive
// sets kStatusTmaTimeout, waits (bounded) for its copies and leaves.
#pragma once
#include "stage_tma.cuh"

namespace ccb {

template <typename T, int NS>
struct UpdateTmaLayout {
  static constexpr int NV = 5 + SpecCount<NS>::kArr;
  static constexpr size_t kBox = sizeof(double) * NV * 256;  // one state of a tile's plane
  // alignment slack + barrier + both states + records
  static constexpr size_t kBytes = 128 + 128 + 2 * kBox + StageSmem<T, NS>::kRecBytes;
};

// Tiles of UX x (256 / UX) points; maps_in and maps_n: per block, the boxes of
// a.Qin and a.Qn (read when a.a != 0).
template <typename T, int NS, int UX>
__global__ void __launch_bounds__(256, 2)
    k_update_tma(const StageArgs<T> a, const CUtensorMap *__restrict__ maps_in, const CUtensorMap *__restrict__ maps_n,
                 const __grid_constant__ ChemParams C) {
  using L = UpdateTmaLayout<T, NS>;
  constexpr int A = SpecCount<NS>::kArr;
  constexpr int NV = L::NV;
  const int ns = SpecCount<NS>::n(C);
  const int nv = 5 + ns;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char *smem_raw = smem_dyn + ((128u - (smem_u32(smem_dyn) & 127u)) & 127u);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw);
  double *sQ = reinterpret_cast<double *>(smem_raw + 128);  // [nv][256]
  double *sQn = sQ + NV * 256;
  double *sRecD = sQn + NV * 256;
  T *sRec = reinterpret_cast<T *>(reinterpret_cast<unsigned char *>(sRecD) +
                                  (sizeof(T) == sizeof(double) ? 0 : StageSmem<T, NS>::kRecD));
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * UX + tx;
  const Tile t = a.tiles[blockIdx.x];
  const BlockInfo B = a.blocks[t.blk];
  const bool use_n = a.a != 0.0;
  const CUtensorMap *map_in = maps_in + t.blk, *map_n = maps_n + t.blk;
  const unsigned box_bytes = (unsigned)(sizeof(double) * nv * 256);
  // request the states of plane k (thread 0): tensor coordinates i0 + g, j0 + g, k + g
  auto issue = [&](int k) {
#ifdef CC_BOUNDS_CHECK
    const bool ok = ((t.i0 + B.g) * (int)sizeof(double)) % 16 == 0 && k + B.g >= 0 && k + B.g < B.nz;
    CCB_CHECK(C, ok);
    if (!ok) return;
#endif
    mbar_arrive_expect_tx(bar, use_n ? 2 * box_bytes : box_bytes);
    tma_load_plane(sQ, map_in, t.i0 + B.g, t.j0 + B.g, k + B.g, bar);
    if (use_n) tma_load_plane(sQn, map_n, t.i0 + B.g, t.j0 + B.g, k + B.g, bar);
  };
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(map_in))
                 : "memory");
    if (use_n)
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(map_n))
                   : "memory");
    issue(t.k0);
  }
  for (int e = tid, nrec = ns * kRecRanges * kRecLen; e < nrec; e += 256) {
    sRecD[e] = param_rec<double>(C)[e];
    if (sizeof(T) != sizeof(double)) sRec[e] = param_rec<T>(C)[e];
  }
  __syncthreads();

  const int i = t.i0 + tx, j = t.j0 + ty;
  const bool act = (i < B.mx) && (j < B.my);
  const int N = (int)a.N, sj = B.nx, sk = B.nx * B.ny;
  const bool three_d = B.mz > 1;
  const T *__restrict__ P = a.P;
  const T *__restrict__ Fx = a.faces;
  const T *__restrict__ Fy = a.faces + face_base(1, nv, (int)sizeof(T), N);
  const T *__restrict__ Fz = a.faces + face_base(2, nv, (int)sizeof(T), N);
  unsigned flags = 0, phase = 0;
  double dt_min = 1e300;
  const int col = (int)B.base + (act ? i + sj * j : 0);
  const double dt_global = a.local_dt ? 0.0 : *a.dt;
  bool aborted = false;
  for (int k = t.k0; k < t.k1; ++k) {
    const int p = CCB_IDX(C, col + sk * k, N);
    T acc[NV];
    double dtj = 0.0, t_warm = 0.0, gcl[3] = {0.0, 0.0, 0.0};
    bool want_dt = false;
    if (act) {
      if (a.gcl)
#pragma unroll
        for (int c = 0; c < 3; ++c) gcl[c] = a.gcl[c * N + p];
      const double jac = (double)geo_jac(a.G, N, p);
      t_warm = (double)P[5 * N + p];
      // dq = -(sum over directions of F(+1/2) - F(-1/2)), the fused kernel's order
      if (a.dq_direct) {  // dq differenced by the face kernel (k_faces_dq)
#pragma unroll
        for (int l = 0; l < NV; ++l)
          if (l < nv) acc[l] = -Fx[l * N + p];
      } else {
        // the minus-side faces (checked in bounds-checked builds)
        const int px = CCB_IDX(C, p - 1, N), py = CCB_IDX(C, p - sj, N), pz = CCB_IDX(C, three_d ? p - sk : p, N);
        // kBatch groups are loaded before the first is used (registers are
        // free here), so that a plane waits for memory once or twice
        constexpr int W = kFaceGroup<T>, kGroups = kFaceGroups<T, NV>, kBatch = sizeof(T) == 4 ? 4 : 7;
#pragma unroll
        for (int g0 = 0; g0 < kGroups; g0 += kBatch) {
          T x0[kBatch][W], x1[kBatch][W], y0[kBatch][W], y1[kBatch][W], z0[kBatch][W], z1[kBatch][W];
#pragma unroll
          for (int b = 0; b < kBatch; ++b) {
            const int g = g0 + b;
            if (g >= kGroups || W * g >= nv) continue;
            load_faces(Fx, N, nv, g, p, x1[b]), load_faces(Fx, N, nv, g, px, x0[b]);
            load_faces(Fy, N, nv, g, p, y1[b]), load_faces(Fy, N, nv, g, py, y0[b]);
            load_faces(Fz, N, nv, g, p, z1[b]), load_faces(Fz, N, nv, g, pz, z0[b]);
          }
#pragma unroll
          for (int b = 0; b < kBatch; ++b)
#pragma unroll
            for (int m = 0; m < W; ++m) {
              const int l = W * (g0 + b) + m;
              if (l >= NV || l >= nv) continue;
              acc[l] = x1[b][m] - x0[b][m];
              acc[l] += y1[b][m] - y0[b][m];
              acc[l] += z1[b][m] - z0[b][m];
            }
        }
      }
      double dt = dt_global;
      if (a.local_dt) {
        T Y[A];
#pragma unroll
        for (int l = 0; l < A; ++l)
          if (l < ns) Y[l] = P[(6 + l) * N + p];
        T gam, c;
        gamma_and_c<T, NS>(C, sRec, P[5 * N + p], Y, gam, c);
        dt = local_time_step<T>(C, a.G, N, p, (double)P[p], (double)P[N + p], (double)P[2 * N + p],
                                (double)P[3 * N + p], (double)c, (double)gam, (double)a.Pr[p], three_d);
      }
      dtj = dt / jac;
      // whether this point's step enters the next global time step
      want_dt = a.dt_next && !((a.skip_dt[p >> 5] >> (p & 31)) & 1u);
    }
    const bool late = !mbar_wait_bounded(bar, phase, C.max_spins);
    if (__syncthreads_or(late)) {
      if (tid == 0) atomicOr(a.status, kStatusTmaTimeout);
      aborted = true;
      break;
    }
    phase ^= 1u;
    double q[NV];
    if (act) {
#pragma unroll
      for (int l = 0; l < NV; ++l)
        if (l < nv)
          q[l] = stage_value<T>(C, a, l, -(double)acc[l], gcl[l >= 1 && l <= 3 ? l - 1 : 0], dtj, three_d,
                                sQ[l * 256 + tid], use_n ? sQn[l * 256 + tid] : 0.0);
    }
    __syncthreads();  // the boxes are read
    if (k + 1 < t.k1 && tid == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(k + 1);
    }
    if (act) point_finish<T, NS>(C, sRec, sRecD, a, p, N, q, t_warm, three_d, want_dt, flags, dt_min);
  }
  if (aborted) {
    // let this CTA's copies in flight land before it leaves (bounded)
    if (tid == 0) {
      long long spins = 0;
      while (!mbar_try_wait(bar, phase) && ++spins < kMaxSpins) {
      }
    }
    __syncthreads();
    return;
  }
  if (a.dt_next) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dt_min = fmin(dt_min, __shfl_xor_sync(0xffffffffu, dt_min, o));
    if ((tid & 31) == 0) atomic_min_pos_double(a.dt_next, dt_min);
  }
  const unsigned any = __reduce_or_sync(0xffffffffu, flags);
  if (any && (tid & 31) == 0) atomicOr(a.status, any);
}

}  // namespace ccb
