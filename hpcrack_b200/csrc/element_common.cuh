// Shared by the element-operator kernels (element_kernels.cu, mech_tile.cu): launch arguments, the
// epilogue of one finished node, launch set-up.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "internal.h"

namespace hpc {

struct StripGeo {
  int tx, ty, tz;            // strips per axis
  int wy, cz;                // element rows (2..kWY) and output planes per strip
  long long nstrips;
};


template <typename T>
struct MechKT {
  LevelGeo g;
  StripGeo sg;
  const T* fields[6];  // staged: u0,u1,u2 then K,G,d (finest) or Ke,Ge (coarse)
  T* out;
  const int8_t* choice;
  double small_k;
  T* fu;
  T* r_out;
  int set_fnorm;
  const T* invM;
  const T* gpm;  // finest level, precomputed Gauss-point moduli: K - 2G/3 at [g * n + e], G at [(8 + g) * n + e]
  RedTarget red;
  double* err;   // tensor-core kernel / TMA staging: set to 1 when a bounded wait ran out (the context's, host memory)
  // PCG direction formed while the planes are staged (mech_tile.cu): p = r M^-1 + beta p_old, beta =
  // red.scal[s_rz] / red.scal[s_rz_prev] (p = r M^-1 if dir_first), written to p_new; fields[0..2] hold p_old
  const T* dir_r;
  const T* dir_m;
  T* p_new;
  int dir_first, s_rz, s_rz_prev;
  alignas(64) CUtensorMap rmap, mmap;  // dir_r, dir_m as {px, ny, nz, 3}
  alignas(64) CUtensorMap tmap;  // TMA staging: the staged vector as {px, ny, nz, 3}
  alignas(64) CUtensorMap gmap;  // TMA staging: the Gauss-point moduli as {px, ny, nz, 16} (finest applies)
};
using MechK = MechKT<double>;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// What a kernel does with the finished operator row tot of node (x, ey, kk), by epilogue; own_p is the
// applied vector at the node (EPI_PCG); pre_f and pre_m are f and (where k.invM is set) M^-1 at the node
// (EPI_RESIDUAL), or pre_f what out holds there and pre_m M^-1 (EPI_FAS); bc
// the node's Dirichlet flags (those three and EPI_REACTION).
template <typename T, int EPI>
__device__ __forceinline__ void node_epilogue(const MechKT<T>& k, int x, int ey, int kk, const T (&tot)[3],
                                              const T (&own_p)[3], const T (&pre_f)[3], const T (&pre_m)[3],
                                              const BcFlags& bc, double& red0, double& red1, double& red2) {
  const long long n = (long long)x + (long long)ey * k.g.px + (long long)kk * k.g.plane;
  const long long N = k.g.n;
  if (EPI == EPI_PLAIN) {
#pragma unroll
    for (int m = 0; m < 3; ++m) k.out[n + m * N] = tot[m];
  } else if (EPI == EPI_RESIDUAL) {
    const bool fix[3] = {bc.c0, bc.c1, bc.c2};
    // a slab's ghost planes keep the sums as they are (a select: ghost values may be anything)
    const bool own = owned_plane(k.g, kk);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      T fv = pre_f[m];
      if (k.set_fnorm && fix[m]) {
        fv = tot[m];
        k.fu[n + m * N] = fv;
      }
      if (k.red.slot[0] >= 0) {  // sums nobody reads are skipped
        const double s0 = fma((double)fv, (double)fv, red0);
        red0 = own ? s0 : red0;
      }
      const T rv = fix[m] ? T(0) : fv - tot[m];
      k.out[n + m * N] = rv;
      if (k.invM) {
        const double s1 = fma((double)rv, (double)(rv * pre_m[m]), red1);
        red1 = own ? s1 : red1;
      }
      if (k.red.slot[2] >= 0) {
        const double s2 = fma((double)rv, (double)rv, red2);
        red2 = own ? s2 : red2;
      }
    }
  } else if (EPI == EPI_PCG) {  // w = K p, (p, w)
    const bool own = owned_plane(k.g, kk);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      k.out[n + m * N] = tot[m];
      const double s0 = fma((double)own_p[m], (double)tot[m], red0);
      red0 = own ? s0 : red0;
    }
  } else if (EPI == EPI_FAS) {
    // the second half of coarsen_fu: out holds the full weighting of the fine residual.  With r_out that is
    // also the first residual of the coarse smoother, f - K u for the injected u
    const bool fix[3] = {bc.c0, bc.c1, bc.c2};
    const bool own = owned_plane(k.g, kk);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      k.out[n + m * N] = tot[m] + pre_f[m];
      if (k.r_out) {
        const T rv = fix[m] ? T(0) : pre_f[m];
        k.r_out[n + m * N] = rv;
        const double s1 = fma((double)rv, (double)(rv * pre_m[m]), red1);
        red1 = own ? s1 : red1;
      }
    }
  } else if (EPI == EPI_REACTION) {
    // Dirichlet_force_u (boundary_conditions.cpp:69-111)
    if (bc.c0) k.out[n] = tot[0];
    if (bc.c1) k.out[n + N] = tot[1];
    if (bc.c2) k.out[n + 2 * N] = tot[2];
  }
}

// Opt-in of a kernel's dynamic shared memory (max_smem) and its resident blocks per SM at `smem` bytes and
// `threads` threads, looked up on first use so that later launches - also those inside a stream
// capture - only enqueue work.
int kernel_cfg(const void* kern, size_t max_smem, size_t smem, int threads, int* per_sm);
int num_sms();
// A level's vector (components n apart) or moduli array (ncomp planes n apart) as a TMA tensor
// {px, ny, nz, ncomp}, x fastest, with the given box.
template <typename T>
int encode_tensor(const LevelGeo& g, const T* src, int ncomp, int bx, int by, int bz, CUtensorMap* map);
constexpr int kTileX = 16;    // element columns of a tile in x
constexpr int kMinTileY = 4;  // the fewest element rows of a tile
// Element rows of a tile for a level of ny node rows: `full` of them, or by halves down to `least` where that computes
// at most three quarters of the rows (a tile of ty finishes ty - 1 node rows and computes ty whatever it finishes).
// For the phase field; the displacement tiles are halved for boxes of one tile only (run_tile_h).  Boxes thin in y paid
// for whole tiles.  1025 x 3 x 1025 nodes: phase-field operator call 289 us, now 102; two cycles of the displacement
// solve in FP64 12.9 ms, now 10.0, in the precision form 13.5, now 10.4.  1025 x 17 x 513: operator 367 us, now 271.
int tile_rows(int ny, int full, int least);
// The row a thread of a tile of TY rows works on.  A warp's two half-warps work 4 rows apart (2 in the lowest tile):
// with the staged row pitch that spreads an FP32 warp over all 32 banks.
template <int TY>
__device__ __forceinline__ int tile_row(int warp, int lane) {
  constexpr int H = TY < 8 ? TY / 2 : 4;
  return warp % H + H * (lane >> 4) + 2 * H * (warp / H);
}
// Tiles of a level, `ty` element rows high, and their z chunks (tz) for `slots` resident blocks; at most cap
// blocks where one chunk allows it.
StripGeo tile_geo(const LevelGeo& g, int ty, long long slots, long long cap);
// Whether a tile kernel leaves its sums to launch_combine.  A block that counts itself in holds its place on the SM
// about 1.7 us longer, which nothing hides where blocks are many and march few planes: 1025 x 1025 x 3 nodes, four
// iterations of pcg_d 1067 us, 1008 with a combining kernel; two cycles of the FP64 displacement solve 8.38 and 7.93 ms.
// From nine blocks a place on; a grid that size runs for at least ten times the second launch.
inline bool combine_apart(const StripGeo& sg, long long slots) { return sg.nstrips > 8 * slots; }
// Tile kernels (mech_tile.cu): the mechanical operator with precomputed Gauss-point moduli (finest level,
// k.gpm set) or element-constant moduli (coarse levels).
template <typename T>
int launch_mech_tile(hpc_ctx* c, MechKT<T>& k, bool finest, int epi);  // EPI_PCG with k.p_new: fused direction

}  // namespace hpc
