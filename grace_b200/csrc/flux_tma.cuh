// Face fluxes from shared-memory tiles staged by TMA (tuned mode).
//
// Same arithmetic as getflux<dir> + mhd_fluxes<dir> (grmhd.hh:551-970) on the
// tuned face ranges; what changes is where the stencil comes from.  One CTA
// takes W x R faces of one block: W consecutive faces (x) across the warp
// lanes, R rows of them along the "row" axis, one index along the third.
// Thread 0 issues two 5-D TMA loads (cp.async.bulk.tensor, no multicast)
// into shared memory: the 10 reconstructed aux variables (RHO .. ENTROPY,
// aux variables 0..9) and the 10 metric variables (GXX .. BETAZ, state
// variables 7..16) of every cell the tile's stencils touch, the full x
// extent of the block (boxes start at x = 0, so every copy is 16-byte
// aligned).  Rows past the end of the block are zero-filled by the copy and
// feed only idle threads.  All threads wait on one mbarrier (bounded), then
// each reconstructs its face from shared memory: a cell read by six faces
// comes from DRAM once per tile.
#pragma once
#include <cuda.h>

#include "stage_kernels.cuh"

namespace grb {

// Tile geometry of one direction (host-computed).
struct FluxTile {
  int lo[3], n[3];  // face box of the tuned range
  int R;            // face rows per CTA
  int BY, BZ;       // box extent along y and z (cells)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void tma_load5(uint32_t dst, const CUtensorMap* tm, int c0, int c1, int c2, int c3,
                                          int c4, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      :
      : "r"(dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(mbar)
      : "memory");
}
// Bounded wait for phase `parity` of an mbarrier; false after `limit` tries.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, int limit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The r-th reconstructed variable: its aux index, its place in the primitives.
__host__ __device__ constexpr int tile_var(int r) {
  return r < 4 ? GRB_RHO + r : r == 4 ? GRB_YE : r == 5 ? GRB_TEMP : r == 6 ? GRB_ENTROPY : GRB_BX + r - 7;
}
__host__ __device__ constexpr int tile_prim(int r) {
  return r == 0 ? GRB_P_RHO : r < 4 ? GRB_P_ZX + r - 1 : r == 4 ? GRB_P_YE : r == 5 ? GRB_P_TEMP : r == 6 ? GRB_P_ENT : GRB_P_BX + r - 7;
}

// getflux<dir> on a staged stencil after the reconstruction (pl, pr).  M:
// metric tile at stencil cell 0 (the cell three before the face) of variable
// 0; vs: variable stride; st: stencil stride (cells along dir).
template <int dir>
__device__ __forceinline__ void getflux_states(const DevParams& P, bool rusanov, const double* M, int vs, int st,
                                               double bface, double* pl, double* pr, double f[7], double vb[4]) {
  double gm[10];
#pragma unroll
  for (int a = 0; a < 10; ++a) {
    const double* p = M + a * vs;
    gm[a] = face4(p[st], p[2 * st], p[3 * st], p[4 * st]);
  }
  const Met m = make_met<true>(gm, gm + 7, gm[6]);
  const double bn = bface * m.isqrtg;
  pl[GRB_P_BX + dir] = bn;
  pr[GRB_P_BX + dir] = bn;
  eos_PT_f(P.eos, pl);
  eos_PT_f(P.eos, pr);
  mhd_fluxes_f<dir>(P, rusanov, pl, pr, m, f, vb);
}
// Both with the reconstruction; A: aux tile at stencil cell 0.
template <int dir>
__device__ __forceinline__ void getflux_tile(const DevParams& P, int recon, bool rusanov, const double* A,
                                             const double* M, int vs, int st, double bface, double f[7],
                                             double vb[4]) {
  const double alpl = M[(GRB_ALP - GRB_GXX) * vs + 2 * st];
  const double alpr = M[(GRB_ALP - GRB_GXX) * vs + 3 * st];
  double pl[13], pr[13];
  const bool donor = (alpl <= P.alp_ex || alpr <= P.alp_ex);
  // WENO-Z's nine reconstructions without a branch between them, the other
  // kinds apart: the code that runs is then one stretch, which instruction
  // fetch (17 % of the issue slots) pays for.  64 blocks of 16^3: y and z
  // faces 51 us a launch with the kind tested per variable, 45 us so.
  if (recon == GRB_RECON_WENOZ) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      if (r == 7 + dir) continue;  // the face's own normal field
      const double* p = A + tile_var(r) * vs;
      double u[6];
#pragma unroll
      for (int o = 0; o < 6; ++o) u[o] = p[o * st];
      weno_z_face(u, pl[tile_prim(r)], pr[tile_prim(r)]);
    }
  } else {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      if (r == 7 + dir) continue;
      const double* p = A + tile_var(r) * vs;
      double u[6];
#pragma unroll
      for (int o = 0; o < 6; ++o) u[o] = p[o * st];
      recon6_fast(recon, u, pl[tile_prim(r)], pr[tile_prim(r)]);
    }
  }
  if (donor) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      if (r == 7 + dir) continue;
      pl[tile_prim(r)] = A[tile_var(r) * vs + 2 * st];
      pr[tile_prim(r)] = A[tile_var(r) * vs + 3 * st];
    }
  }
  getflux_states<dir>(P, rusanov, M, vs, st, bface, pl, pr, f, vb);
}

constexpr int kTmaWaitLimit = 1 << 22;

// Shared memory of one CTA: aux tile and metric tile, each
// [10 vars][BZ][BY][NX] doubles, the metric tile starting on a 128-byte
// boundary, then the mbarrier and one more word (the persistent form's
// current tile).
__host__ __device__ inline int flux_tile_doubles(const Geo& G, const FluxTile& T) {
  return (10 * T.BY * T.BZ * G.NX + 15) / 16 * 16;
}
__host__ __device__ inline size_t flux_tile_smem(const Geo& G, const FluxTile& T) {
  return 2 * sizeof(double) * (size_t)flux_tile_doubles(G, T) + 16;
}

// The x faces of a staged tile.  A thread takes one cell: WENO-Z's states on
// its two faces share their weights (weno_z_cell), and the left state of its
// lower face comes from the lane below.  A row's n + 1 cells (the one below
// the first face included) follow each other over the lanes, consecutive
// warps overlapping by one cell, whose face the lower warp computes: 31 of 32
// lanes and n of n + 1 cells have a face.  Along y and z the neighbour sits
// in another warp, and passing the states through shared memory costs the
// gain again, so those reconstruct per face.
__device__ __forceinline__ void flux_tile_face_x(const DevParams& P, const Geo& G, const FluxTile& T,
                                                 const double* sa, const double* sm, int vs, int oy, int oz,
                                                 int64_t q, const double* __restrict__ bface, const StageBufs& B) {
  const int lane = threadIdx.x & 31, W = T.n[0] + 1;
  const int c = (threadIdx.x >> 5) * 31 + lane;
  int r = c / W, x = c - r * W;
  bool face = lane > 0 && x > 0 && r < T.R && oy + r < T.lo[1] + T.n[1];
  if (r >= T.R) { r = 0; x = 1; }
  const int i = T.lo[0] - 1 + x;
  const int base = r * G.NX + i - 3;  // stencil cell 0 of face i
  const double* A = sa + base;
  double pl[13], pr[13];
  if (P.recon == GRB_RECON_WENOZ) {
#pragma unroll
    for (int v = 0; v < 10; ++v) {
      if (v == 7) continue;  // the face's own normal field
      const double* p = A + tile_var(v) * vs + 1;
      const double u[5] = {p[0], p[1], p[2], p[3], p[4]};
      double hi;
      weno_z_cell(u, pr[tile_prim(v)], hi);
      pl[tile_prim(v)] = __shfl_up_sync(0xffffffffu, hi, 1);
    }
    if (!face) return;
    if (sm[base + (GRB_ALP - GRB_GXX) * vs + 2] <= P.alp_ex || sm[base + (GRB_ALP - GRB_GXX) * vs + 3] <= P.alp_ex) {
#pragma unroll
      for (int v = 0; v < 10; ++v) {
        if (v == 7) continue;
        pl[tile_prim(v)] = A[tile_var(v) * vs + 2];
        pr[tile_prim(v)] = A[tile_var(v) * vs + 3];
      }
    }
  } else {
    if (!face) return;
    const bool donor = sm[base + (GRB_ALP - GRB_GXX) * vs + 2] <= P.alp_ex ||
                       sm[base + (GRB_ALP - GRB_GXX) * vs + 3] <= P.alp_ex;
#pragma unroll
    for (int v = 0; v < 10; ++v) {
      if (v == 7) continue;
      const double* p = A + tile_var(v) * vs;
      const double u[6] = {p[0], p[1], p[2], p[3], p[4], p[5]};
      double ul, ur;
      recon6_fast(P.recon, u, ul, ur);
      pl[tile_prim(v)] = donor ? u[2] : ul;
      pr[tile_prim(v)] = donor ? u[3] : ur;
    }
  }
  double f[7], vb[4];
  const int j = oy + r, k = oz;
  getflux_states<0>(P, P.riemann == GRB_RIEMANN_LLF, sm + base, vs, 1, __ldg(bface + bxi(G, i, j, k, q)), pl, pr, f, vb);
  store_face(G, B, P.emf, 0, i, j, k, q, f, vb);
}

// The face of this thread in a staged tile (box origin oy, oz of block q):
// lanes along x, rows along the tile's row axis; threads past the tile's
// faces do nothing.
template <int dir>
__device__ __forceinline__ void flux_tile_face(const DevParams& P, const Geo& G, const FluxTile& T,
                                               const double* sa, const double* sm, int vs, int oy, int oz,
                                               int64_t q, const double* __restrict__ bface, const StageBufs& B) {
  if (dir == 0) {
    flux_tile_face_x(P, G, T, sa, sm, vs, oy, oz, q, bface, B);
    return;
  }
  const int W = T.n[0];
  const int w = threadIdx.x % W, r = threadIdx.x / W;
  if (r >= T.R) return;
  const int i = T.lo[0] + w;
  int j, k;
  if (dir == 1) {
    j = oy + 3 + r; k = oz;
    if (j >= T.lo[1] + T.n[1]) return;
  } else {
    j = oy; k = oz + 3 + r;
    if (k >= T.lo[2] + T.n[2]) return;
  }
  const int base = r * G.NX + i, st = G.NX;
  const int64_t bi = dir == 1 ? byi(G, i, j, k, q) : bzi(G, i, j, k, q);
  double f[7], vb[4];
  getflux_tile<dir>(P, P.recon, P.riemann == GRB_RIEMANN_LLF, sa + base, sm + base, vs, st, __ldg(bface + bi), f, vb);
  store_face(G, B, P.emf, dir, i, j, k, q, f, vb);
}

// grid: (ceil(n_row / R), n_other, nq); NT threads (128 or 256); W = n[0]
// <= NT; R = NT / W rows, for dir 0 (31 NT / 32 + 1) / (W + 1) (a 256-thread
// tile re-reads the 5-row stencil halo of the y and z directions over twice
// as many rows).
//   dir 0: lanes i (cells), rows j, other k; box rows j (BY = R, BZ = 1)
//   dir 1: lanes i, rows j (faces), other k; box rows j - 3 .. (BY = R + 5)
//   dir 2: lanes i, rows k (faces), other j; box rows k - 3 .. (BZ = R + 5)
template <int dir>
__device__ __forceinline__ void flux_tma_tile(const DevParams& P, const Geo& G, const FluxTile& T,
                                              const CUtensorMap* tm_aux, const CUtensorMap* tm_met,
                                              const double* __restrict__ bface, const StageBufs& B, int tile,
                                              int other, int64_t q) {
  extern __shared__ __align__(128) unsigned char sm_raw[];
  const int vs = T.BY * T.BZ * G.NX;  // variable stride in the tile
  const int td = flux_tile_doubles(G, T);
  double* sa = reinterpret_cast<double*>(sm_raw);
  double* sm = sa + td;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + td);
  // box origin in cells (x always 0)
  int oy, oz;
  if (dir == 0) { oy = T.lo[1] + tile * T.R; oz = T.lo[2] + other; }
  else if (dir == 1) { oy = T.lo[1] + tile * T.R - 3; oz = T.lo[2] + other; }
  else { oy = T.lo[1] + other; oz = T.lo[2] + tile * T.R - 3; }
  const uint32_t mb = smem_u32(mbar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  // both destinations start on 128-byte boundaries (checked: no copy is
  // issued otherwise, and the wait below then gives up)
  const bool aligned = ((smem_u32(sa) | smem_u32(sm)) & 127u) == 0;
  if (threadIdx.x == 0 && aligned) {
    const uint32_t bytes = (uint32_t)(2 * 10 * vs * sizeof(double));
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
    tma_load5(smem_u32(sa), tm_aux, 0, oy, oz, 0, (int)q, mb);
    tma_load5(smem_u32(sm), tm_met, 0, oy, oz, GRB_GXX, (int)q, mb);
  }
  if (!aligned) {
    if (threadIdx.x == 0) atomicOr(B.flags, GRB_FLAG_WAIT_TIMEOUT);
    return;
  }
  if (!mbar_wait(mb, 0, kTmaWaitLimit)) {
    if (threadIdx.x == 0) atomicOr(B.flags, GRB_FLAG_WAIT_TIMEOUT);
    return;
  }
  flux_tile_face<dir>(P, G, T, sa, sm, vs, oy, oz, q, bface, B);
}
template <int dir, int MINB, int NT = 128>
__global__ void __launch_bounds__(NT, MINB) k_flux_tma(DevParams P, Geo G, FluxTile T,
                                                      const __grid_constant__ CUtensorMap tm_aux,
                                                      const __grid_constant__ CUtensorMap tm_met,
                                                      const double* __restrict__ bface, StageBufs B) {
  flux_tma_tile<dir>(P, G, T, &tm_aux, &tm_met, bface, B, blockIdx.x, blockIdx.y, blockIdx.z);
}

// The three directions in one launch: blockIdx.x runs over the tiles of x,
// then y, then z (first[d] the first of direction d, ntx[d] its tiles along
// the row axis).  For small grids, where a direction on its own leaves most
// SMs idle in its first or last wave.
struct FluxTma3 {
  FluxTile T[3];
  int ntx[3], first[3];
  const double* bf[3];
  CUtensorMap aux[3], met[3];
};
template <int MINB, int NT>
__global__ void __launch_bounds__(NT, MINB) k_flux_tma3(DevParams P, Geo G, const __grid_constant__ FluxTma3 A,
                                                       StageBufs B) {
  const int x = blockIdx.x;
  if (x < A.first[1]) {
    flux_tma_tile<0>(P, G, A.T[0], &A.aux[0], &A.met[0], A.bf[0], B, x % A.ntx[0], x / A.ntx[0], blockIdx.z);
  } else if (x < A.first[2]) {
    const int t = x - A.first[1];
    flux_tma_tile<1>(P, G, A.T[1], &A.aux[1], &A.met[1], A.bf[1], B, t % A.ntx[1], t / A.ntx[1], blockIdx.z);
  } else {
    const int t = x - A.first[2];
    flux_tma_tile<2>(P, G, A.T[2], &A.aux[2], &A.met[2], A.bf[2], B, t % A.ntx[2], t / A.ntx[2], blockIdx.z);
  }
}

// The same as a persistent launch (tuned candidate): one wave of CTAs, each
// taking tiles, numbered tile row fastest, then the other index, then the
// block, from the device work queue *queue (zeroed before the launch) until
// they run out; per tile the same two TMA loads into the same shared
// memory, the mbarrier's phase alternating from tile to tile.  Every thread
// reaches every barrier; a wait that gives up sets the flag and ends the
// CTA.  ntx, nother: tiles along the row axis, indices along the third.
template <int dir, int MINB, int NT = 128>
__global__ void __launch_bounds__(NT, MINB) k_flux_tma_queue(DevParams P, Geo G, FluxTile T,
                                                            const __grid_constant__ CUtensorMap tm_aux,
                                                            const __grid_constant__ CUtensorMap tm_met,
                                                            const double* __restrict__ bface, StageBufs B,
                                                            unsigned long long* __restrict__ queue, int ntx,
                                                            int nother) {
  extern __shared__ __align__(128) unsigned char sm_raw[];
  const int vs = T.BY * T.BZ * G.NX;
  const int td = flux_tile_doubles(G, T);
  double* sa = reinterpret_cast<double*>(sm_raw);
  double* sm = sa + td;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + td);
  // the tile taken from the queue, in the second word after the mbarrier
  unsigned long long& item = *reinterpret_cast<unsigned long long*>(mbar + 1);
  const uint32_t mb = smem_u32(mbar);
  // both destinations start on 128-byte boundaries (the same for every
  // thread, so the CTA leaves as a whole otherwise)
  if (((smem_u32(sa) | smem_u32(sm)) & 127u) != 0) {
    if (threadIdx.x == 0) atomicOr(B.flags, GRB_FLAG_WAIT_TIMEOUT);
    return;
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  const unsigned long long ntiles = (unsigned long long)ntx * (unsigned long long)nother * (unsigned long long)G.nq;
  const uint32_t bytes = (uint32_t)(2 * 10 * vs * sizeof(double));
  uint32_t parity = 0;
  for (;;) {
    // every thread is done with the previous tile's shared memory here
    __syncthreads();
    if (threadIdx.x == 0) item = atomicAdd(queue, 1ull);
    __syncthreads();
    const unsigned long long t = item;
    if (t >= ntiles) break;
    const int tile = (int)(t % (unsigned long long)ntx);
    const unsigned long long rest = t / (unsigned long long)ntx;
    const int other = (int)(rest % (unsigned long long)nother);
    const int64_t q = (int64_t)(rest / (unsigned long long)nother);
    int oy, oz;
    if (dir == 0) { oy = T.lo[1] + tile * T.R; oz = T.lo[2] + other; }
    else if (dir == 1) { oy = T.lo[1] + tile * T.R - 3; oz = T.lo[2] + other; }
    else { oy = T.lo[1] + other; oz = T.lo[2] + tile * T.R - 3; }
    if (threadIdx.x == 0) {
      // the async proxy overwrites what the generic proxy just read
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
      tma_load5(smem_u32(sa), &tm_aux, 0, oy, oz, 0, (int)q, mb);
      tma_load5(smem_u32(sm), &tm_met, 0, oy, oz, GRB_GXX, (int)q, mb);
    }
    const bool ok = mbar_wait(mb, parity, kTmaWaitLimit);
    parity ^= 1u;
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) atomicOr(B.flags, GRB_FLAG_WAIT_TIMEOUT);
      return;
    }
    flux_tile_face<dir>(P, G, T, sa, sm, vs, oy, oz, q, bface, B);
  }
}

}  // namespace grb
