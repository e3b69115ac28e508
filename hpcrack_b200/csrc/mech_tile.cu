// Mechanical operator on column tiles: the finest level with the Gauss-point moduli of the running
// solve, the coarse levels with element-constant moduli, FP64 and FP32, with the fused epilogues of
// element_common.cuh.
//
// A block owns a tile of kTX x TY element columns (one thread each) and marches it up z over a chunk of
// output planes; it finishes the (kTX - 1) x (TY - 1) inner node columns.  Marching lets a thread keep,
// per node plane, what both element layers that touch the plane need:
//   * forward: the in-plane part of the gradients (the x- and y-derivatives interpolated to the 2x2
//     in-plane Gauss coordinates, and the interpolated values) is formed once per plane, not once per
//     element, from 4 nodes per component;
//   * adjoint: the stresses of the layers below and above a plane are added in that in-plane form, and
//     taken back to the 4 nodes once per plane.
// That is about 365 floating-point operations per element against 600 for element-by-element sum
// factorisation, and half the node assembly.  x-neighbours are combined with a shuffle inside a row of
// 16 lanes, y-neighbours through a shared-memory row exchange, one block barrier per layer.
// Node planes and moduli arrive up to three layers ahead in shared-memory stages (tensor copies by one
// thread, completion on the stage's mbarrier, or per-thread cp.async); the carried parts stay in
// registers, two layers per loop turn so that they swap roles instead of being moved.
//
// The smoothers' applies form the PCG direction on the way (DIR): r, M^-1 and the old direction are staged
// instead of the new one, each thread forms its share of a plane one layer before it is needed, and the
// tile that owns a node writes the new direction (into the other of two arrays: neighbours still read the
// old one).  That replaces a pass of 96 (48) bytes a node and its launch: an iteration's apply and
// direction take 842 us on 257^3 in FP64 against 656 + 250, 513 us in FP32 against 401 + 125, and one
// launch less where launches count; increments -1 to -5 %.  A plane is formed in units of 16 bytes, one
// (FP32) or two (FP64) a thread; single nodes took 4 rounds of loads, masks and stores.
//
// The residual's f and M^-1 are staged the same way, and the Dirichlet flags read ahead.  As loads of each
// thread from global memory they came due at the end of the layer they were issued in, which is shorter than
// DRAM's latency under load: 935 us a residual on 257^3 in FP64, 591 in FP32, now 866 and 557.  Both changes: increments of
// 257^3 1300 -> 1268 ms (FAS, crack), 358 -> 349 (precision form), 257x129x65 154 -> 149, 129^3 18.8 -> 18.55.
//
// What bounds it: FP64, the FP64 pipe (66 % of its cycles on 193^3; two warps per scheduler cannot hide
// all dependent latencies); FP32, instruction issue (80 % of the slots).  Per launch on B200, with the
// element-by-element strip kernel it replaced in brackets: 257^3 FP64 656 us (1043), FP32 401 us (759);
// 129^3 109 (196), 68 (151); 65^3 28 (63), 21 (53); 33^3 16 (25), 15 (23).  At 176 (88) bytes a node the
// 257^3 applies move 4.6 (3.7) TB/s.
// Coarse levels with equal spacing work in sum/difference modes (ModeState): fewer operations, fewer registers, 3
// blocks per SM in FP64.  What bounds a level of 33^3 to 65^3 is the march itself, 6 to 10 dependent layers.
// Every node is written once, by the tile that owns it, with the same arithmetic wherever tile and
// chunk boundaries fall: no atomics, deterministic, independent of the chunk height except for the
// order of the reductions.
#include <algorithm>
#include <type_traits>

#include "element_common.cuh"

namespace hpc {

// Tiles of a level and the z chunks they are marched in: a chunk of cz planes costs its block cz + 1 layers
// and a pipeline start of about two layers' time, and blocks run in waves of `slots`; the number of
// chunks that minimises waves x (cz + 3) wins.
StripGeo tile_geo(const LevelGeo& g, int ty, long long slots, long long cap) {
  StripGeo s;
  s.wy = ty;
  s.tx = (g.nx + kTileX - 2) / (kTileX - 1);
  s.ty = (g.ny + ty - 2) / (ty - 1);
  const long long tiles = (long long)s.tx * s.ty;
  long long best = -1;
  for (int n = 1; n <= g.nz && (n == 1 || tiles * n <= cap); ++n) {
    const int cz = (g.nz + n - 1) / n;
    const long long cost = ((tiles * n + slots - 1) / slots) * (cz + 3);
    if (best < 0 || cost < best) {
      best = cost;
      s.cz = cz;
      s.tz = n;
    }
  }
  s.nstrips = tiles * s.tz;
  return s;
}

int tile_rows(int ny, int full, int least) {
  const auto computed = [ny](int ty) { return (ny + ty - 2) / (ty - 1) * ty; };
  int best = full;
  for (int ty = full / 2; ty >= least; ty /= 2)
    if (4 * computed(ty) <= 3 * computed(best)) best = ty;
  return best;
}

// One chunk's blocks are a plane's tiles, however many (1025 x 865 nodes: 8556); tile_geo cuts into more chunks only
// while the grid fits, and the persistent grids of the strip and vector kernels are smaller.
size_t partials_doubles(int nx, int ny) {
  const size_t tx = (size_t)(nx + kTileX - 2) / (kTileX - 1), ty = (size_t)(ny + kMinTileY - 2) / (kMinTileY - 1);
  return 3 * std::max<size_t>(8192, tx * ty);
}

namespace {

constexpr int kTX = kTileX;  // element columns of a tile in x: a half-warp, 128 B (64 B) of FP64 (FP32) per row
constexpr unsigned kTileWaitPolls = 1u << 24;  // far above any copy's latency; then the kernel reports

// Columns staged per row: the 17 nodes of a tile plus the offset to the copy's 16-byte aligned start.
template <typename T> struct TileVec;
template <> struct TileVec<double> { using type = double2; };
template <> struct TileVec<float> { using type = float4; };
template <typename T> struct TileRow;
template <> struct TileRow<double> { static constexpr int BX = 18; };
template <> struct TileRow<float> { static constexpr int BX = 20; };

// Shared memory of a block: [0, 128) the stages' mbarriers; the stages' node planes and (finest) moduli
// layers; the y exchange.
// EX: a stage also holds two more planes: r and M^-1 the direction is formed from, or the residual's f and M^-1.
template <typename T, bool GPM, int TY, int NS, bool EX>
struct TileSmem {
  static constexpr int BX = TileRow<T>::BX, NT = kTX * TY, XP = 20;  // XP: exchange row pitch (bank spread)
  static constexpr size_t up(size_t b) { return (b + 127) / 128 * 128; }
  static constexpr size_t plane = up(sizeof(T) * 3 * (TY + 1) * BX), node = plane * (EX ? 3 : 1), mod = GPM ? up(sizeof(T) * 16 * TY * BX) : 0;
  static constexpr size_t o_node = 128, o_mod = o_node + NS * node, o_exch = o_mod + NS * mod;
  static constexpr size_t total = o_exch + sizeof(T) * 2 * 3 * TY * XP;
  static constexpr size_t bytes = total + 128;  // + alignment of the dynamic base
};

// What a thread carries from one element layer to the next: of the node plane between them the in-plane
// forward parts (ex, dy, iy; see plane_forward), the lower layer's adjoint parts (aex, ady, and its
// stresses sz acting through d/dz), and the thread's own node value.
template <typename T>
struct PlaneState {
  T ex[3][2], dy[3][2], iy[3][4], aex[3][2], ady[3][2], sz[3][4], own[3];
  T f[3], im[3];  // residual: f and M^-1 at the thread's own node
};

// The same where moduli are element-constant and the spacing is equal (the coarse levels): in the
// sum/difference modes of mech_modes a plane's part is its 4 nodes (v) and its in-plane modes x, y and xy (h) on
// the way in, and the lower layer's share of the modes (acc) on the way out.  About 160 operations an element
// instead of 365: a PCG apply of 129^3 takes 67 us in FP32 (96), of 65^3 16.5 (21.5).
template <typename T>
struct ModeState {
  T v[3][4], h[3][3], acc[3][4], own[3], f[3], im[3];
};

// In-plane modes x, y, xy of a component's 4 nodes v[a + 2b].  Differences are taken before sums, here and along
// z (see haar).
template <typename T>
__device__ __forceinline__ void plane_modes(const T (&v)[4], T (&h)[3]) {
  const T d0 = v[1] - v[0], d1 = v[3] - v[2];
  h[0] = d0 + d1;
  h[1] = (v[2] - v[0]) + (v[3] - v[1]);
  h[2] = d1 - d0;
}
// The transpose, with the constant mode h[0].
template <typename T>
__device__ __forceinline__ void plane_modes_adjoint(const T (&h)[4], T (&f)[4]) {
  const T a0 = h[0] - h[2], a1 = h[0] + h[2], b0 = h[1] - h[3], b1 = h[1] + h[3];
  f[0] = a0 - b0;
  f[1] = a0 + b0;
  f[2] = a1 - b1;
  f[3] = a1 + b1;
}

// In-plane part of one node plane, per component: ex[p] = d/dx at in-plane Gauss row p, dy[q] = d/dy at
// Gauss column q, iy[q + 2p] = value.  v[a + 2b] = node (a, b).
template <typename T>
__device__ __forceinline__ void plane_forward(const T (&v)[4], const T (&t)[2], T (&ex)[2], T (&dy)[2], T (&iy)[4]) {
  const T d0 = v[1] - v[0], d1 = v[3] - v[2], dd = d1 - d0;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const T i0 = fma(t[q], d0, v[0]), i1 = fma(t[q], d1, v[2]);
    dy[q] = i1 - i0;
    iy[q] = fma(t[0], dy[q], i0);
    iy[q + 2] = fma(t[1], dy[q], i0);
    ex[q] = fma(t[q], dd, d0);
  }
}
// Exact transpose of plane_forward.
template <typename T>
__device__ __forceinline__ void plane_adjoint(const T (&ex)[2], const T (&dy)[2], const T (&iy)[4], const T (&t)[2],
                                              T (&f)[4]) {
  T d1 = fma(t[1], ex[1], t[0] * ex[0]);
  T d0 = ex[0] + ex[1] - d1;
  T i0[2], i1[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    i1[q] = fma(t[1], iy[q + 2], fma(t[0], iy[q], dy[q]));
    i0[q] = iy[q] + iy[q + 2] - i1[q];
  }
  d0 = fma(t[1], i0[1], fma(t[0], i0[0], d0));
  d1 = fma(t[1], i1[1], fma(t[0], i1[0], d1));
  f[1] = d0;
  f[0] = i0[0] + i0[1] - d0;
  f[3] = d1;
  f[2] = i1[0] + i1[1] - d1;
}

template <typename T, bool GPM, int EPI, bool ISO, bool TMA, int TY, int MINB, int NS, bool DIR>
__global__ void __launch_bounds__(kTX* TY, MINB) mech_tile_kernel(const __grid_constant__ MechKT<T> k) {
  constexpr bool RES = EPI == EPI_RESIDUAL, EX = DIR || RES, MODES = !GPM && ISO;
  using State = typename std::conditional<MODES, ModeState<T>, PlaneState<T>>::type;
  using S = TileSmem<T, GPM, TY, NS, EX>;
  constexpr int BX = S::BX, NT = S::NT, NY = TY + 1;
  extern __shared__ __align__(128) unsigned char tile_smem[];
  unsigned char* base = tile_smem + ((128u - (smem_u32(tile_smem) & 127u)) & 127u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base);
  T* exch = reinterpret_cast<T*>(base + S::o_exch);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & (kTX - 1);
  const int row = tile_row<TY>(warp, lane);
  constexpr int A16 = 16 / (int)sizeof(T);  // columns per 16 bytes: a tensor copy's x start is a multiple
  const SFt<T> s = make_sf<T>(k.g);
  const T wg = ISO ? T(k.g.wg) * (s.ih[0] * s.ih[0]) : T(k.g.wg);
  double red0 = 0.0, red1 = 0.0, red2 = 0.0;
  int bad = 0;

  if constexpr (TMA) {
    if (tid == 0) {
#pragma unroll
      for (int i = 0; i < NS; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + i)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
  }
  // tiles fastest: the blocks resident together work the same planes of neighbouring tiles, so that the
  // cache lines and DRAM pages a tile's rows share with its neighbours are fetched once
  const int tiles = k.sg.tx * k.sg.ty, chunks = (int)gridDim.x / tiles;
  const int tile = (int)(blockIdx.x % (unsigned)tiles), chunk = (int)(blockIdx.x / (unsigned)tiles);
  const int z0 = (int)((long long)k.g.nz * chunk / chunks), zend = (int)((long long)k.g.nz * (chunk + 1) / chunks) - 1;
  const int x0 = (tile % k.sg.tx) * (kTX - 1), y0 = (tile / k.sg.tx) * (TY - 1);
  const int x = x0 - 1 + tx, y = y0 - 1 + row;
  const int nl = zend - z0 + 2;  // element layers z0 - 1 .. zend; plane j of the stream is z0 - 1 + j
  const int xs = x0 - 1 >= 0 ? (x0 - 1) / A16 * A16 : -A16;
  const int off = (x0 - 1) - xs;
  const bool xy_elem = x >= 0 && x <= k.g.nx - 2 && y >= 0 && y <= k.g.ny - 2;
  const bool out_node = tx >= 1 && row >= 1 && x < k.g.nx && y < k.g.ny;
  constexpr bool BC = EPI != EPI_PCG && EPI != EPI_PLAIN;  // Dirichlet flags wanted
  const uint8_t fx = BC && out_node ? k.g.bx[x] : 0, fy = BC && out_node ? k.g.by[y] : 0;

  auto node_slot = [&](int j) {
    return reinterpret_cast<T*>(base + S::o_node + (size_t)((unsigned)j % NS) * S::node);
  };
  auto mod_slot = [&](int j) {
    return reinterpret_cast<T*>(base + S::o_mod + (size_t)((unsigned)j % NS) * S::mod);
  };
  // Stage j: node plane j and (finest) the moduli of element layer j - 1, the one below the plane.
  auto issue = [&](int j) {
    if (j <= nl) {
      const int kk = z0 - 1 + j;
      if constexpr (TMA) {
        if (tid == 0) {
          const uint32_t bar = smem_u32(bars + (unsigned)j % NS);
          const bool mods = GPM && j >= 1;
          const bool old = !DIR || !k.dir_first, minv = EX && k.dir_m;
          const int planes = (old ? 1 : 0) + (EX ? 1 : 0) + (minv ? 1 : 0);
          const int bytes = (int)sizeof(T) * BX * (3 * NY * planes + (mods ? 16 * TY : 0));
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
          auto copy = [&](const CUtensorMap* map, T* dst) {
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
                "%4, %5}], [%6];" ::"r"(smem_u32(dst)),
                "l"(map), "r"(xs), "r"(y0 - 1), "r"(kk), "r"(0), "r"(bar)
                : "memory");
          };
          if (old) copy(&k.tmap, node_slot(j));
          if constexpr (EX) {
            copy(&k.rmap, node_slot(j) + S::plane / sizeof(T));
            if (minv) copy(&k.mmap, node_slot(j) + 2 * (S::plane / sizeof(T)));
          }
          if (mods)
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                "%3, %4, %5}], [%6];" ::"r"(smem_u32(mod_slot(j))),
                "l"(&k.gmap), "r"(xs), "r"(y0 - 1), "r"(kk - 1), "r"(0), "r"(bar)
                : "memory");
        }
      } else {
        // the same boxes in 16-byte units: whole units of the pitch, padding included, zeros outside (three FAS cycles of
        // 193^3 in FP64: 25.7 ms; one value a copy 33.0)
        constexpr int U = BX / A16;
        auto unit = [&](const T* src, T* dst, int u, int gy, int z) {
          const int gx = xs + u * A16;
          const bool ok = gx >= 0 && gx < k.g.px && gy >= 0 && gy < k.g.ny && z >= 0 && z < k.g.nz;
          src += ok ? (long long)gx + (long long)gy * k.g.px + (long long)z * k.g.plane : 0;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst + u * A16)), "l"(src),
                       "r"(ok ? 16 : 0)
                       : "memory");
        };
        for (int f = 0; f < (EX ? 3 : 1); ++f) {
          if ((f == 0 && DIR && k.dir_first) || (f == 2 && !k.dir_m)) continue;
          T* dst = node_slot(j) + f * (S::plane / sizeof(T));
          for (int q = tid; q < 3 * NY * U; q += NT) {
            const int r = q / U, m = r / NY;
            unit(f == 0 ? k.fields[m] : (f == 1 ? k.dir_r : k.dir_m) + m * k.g.n, dst + r * BX, q % U, y0 - 1 + r % NY, kk);
          }
        }
        if (GPM && j >= 1) {
          for (int q = tid; q < 16 * TY * U; q += NT) {
            const int r = q / U;
            unit(k.gpm + (r / TY) * k.g.n, mod_slot(j) + r * BX, q % U, y0 - 1 + r % TY, kk - 1);
          }
        }
      }
    }
    if constexpr (!TMA) asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // Stage j has landed, for every thread: this thread's wait; without tensor copies the others' too.  A
  // wait that runs out returns false: the block then stops and reports.
  auto wait = [&](int j) -> bool {
    if constexpr (TMA) {
            const uint32_t bar = smem_u32(bars + (unsigned)j % NS), parity = ((unsigned)j / NS) & 1u;
      for (unsigned i = 0; i < kTileWaitPolls; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, "
            "p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
      }
      return false;
    } else {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(DIR ? NS - 2 : NS - 1) : "memory");
      __syncthreads();
      return true;
    }
  };
  // DIR: the direction at this thread's share of a staged plane, 16 bytes at a time, in place of p_old (0 beyond
  // the grid's last column, where p_old's padding may hold anything)
  using V = typename TileVec<T>::type;
  constexpr int CN = 3 * NY * BX / A16, CT = DIR ? (CN + NT - 1) / NT : 1;  // 16-byte units of a plane
  static_assert(BX % A16 == 0, "a unit stays in its row");
  int c_in[CT];  // the unit's columns inside the grid
  T beta = T(0);
  auto form_direction = [&](int j) {
    if constexpr (DIR) {
      V* p = reinterpret_cast<V*>(node_slot(j));
      const V *r = p + S::plane / sizeof(V), *m = r + S::plane / sizeof(V);
#pragma unroll
      for (int t = 0; t < CT; ++t) {
        const int q = tid + t * NT;
        if (CN % NT != 0 && q >= CN) continue;
        const V rv = r[q], mv = m[q];
        V pv{};
        if (!k.dir_first) pv = p[q];
        T *pe = reinterpret_cast<T*>(&pv);
        const T *re = reinterpret_cast<const T*>(&rv), *me = reinterpret_cast<const T*>(&mv);
#pragma unroll
        for (int e = 0; e < A16; ++e) {
          const T z = re[e] * me[e];
          const T v = k.dir_first ? z : fma(beta, pe[e], z);
          pe[e] = e < c_in[t] ? v : T(0);
        }
        p[q] = pv;
      }
      if (TMA) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the next copy overwrites this plane
    }
  };
  // coarse levels: the element's moduli one layer ahead in registers
  T lam_n = T(0), G_n = T(0);
  auto coarse_mod = [&](int kk) {
    lam_n = G_n = T(0);
    if (!GPM && xy_elem && kk >= 0 && kk <= k.g.nz - 2) {
      const long long e = (long long)x + (long long)y * k.g.px + (long long)kk * k.g.plane;
      const T K = k.fields[3][e] * wg;
      G_n = k.fields[4][e] * wg;
      lam_n = fma(T(-2.0 / 3.0), G_n, K);
    }
  };

  // One element layer li: state a of the node plane below it -> state b of the plane above; the plane
  // below is finished.  False when a wait ran out.
  auto layer = [&](int li, const State& a, State& b) -> bool {
    const int kk = z0 - 1 + li;
    const T lam_c = lam_n, G_c = G_n;
    if (!GPM) coarse_mod(kk + 1);
    const uint8_t fz = BC && out_node && kk >= z0 ? k.g.bz[kk] : 0;
    // FAS: what out holds at this plane's node, in flight under the arithmetic
    T pre_f[3], pre_m[3];
    if (EPI == EPI_FAS && out_node && kk >= z0) {
      const long long n = (long long)x + (long long)y * k.g.px + (long long)kk * k.g.plane;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        pre_f[m] = k.out[n + m * k.g.n];
        pre_m[m] = k.invM ? k.invM[n + m * k.g.n] : T(0);
      }
    }
    if constexpr (RES) {  // staged with this plane, read when it was the upper one
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        pre_f[m] = a.f[m];
        pre_m[m] = a.im[m];
      }
    }
    if (!DIR && !wait(li + 1)) bad = 1;
    T X0[3];
    T* ex_w = exch + (size_t)(li & 1) * 3 * TY * S::XP + row * S::XP + tx;
    const T* nd = node_slot(li + 1) + row * BX + off + tx;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      b.own[m] = nd[m * NY * BX];
      if constexpr (RES) {
        b.f[m] = nd[S::plane / sizeof(T) + m * NY * BX];
        b.im[m] = k.dir_m ? nd[2 * (S::plane / sizeof(T)) + m * NY * BX] : T(0);
      }
    }
    auto combine = [&](int m, const T(&f)[4]) {  // x-neighbours by shuffle, y-neighbours by exchange
      X0[m] = f[0] + __shfl_up_sync(kFull, f[1], 1, kTX);
      ex_w[m * TY * S::XP] = f[2] + __shfl_up_sync(kFull, f[3], 1, kTX);
    };
    if constexpr (MODES) {
      T M[3][8];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        b.v[m][0] = b.own[m];
        b.v[m][1] = nd[m * NY * BX + 1];
        b.v[m][2] = nd[m * NY * BX + BX];
        b.v[m][3] = nd[m * NY * BX + BX + 1];
        plane_modes(b.v[m], b.h[m]);
        M[m][4] = ((b.v[m][0] - a.v[m][0]) + (b.v[m][1] - a.v[m][1])) + ((b.v[m][2] - a.v[m][2]) + (b.v[m][3] - a.v[m][3]));
#pragma unroll
        for (int q = 1; q < 4; ++q) {
          M[m][q] = a.h[m][q - 1] + b.h[m][q - 1];
          M[m][4 + q] = b.h[m][q - 1] - a.h[m][q - 1];
        }
      }
      mech_modes(M, lam_c, G_c);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        T lo[4], f[4];
        lo[0] = a.acc[m][0] - M[m][4];
        b.acc[m][0] = M[m][4];
#pragma unroll
        for (int q = 1; q < 4; ++q) {
          lo[q] = a.acc[m][q] + (M[m][q] - M[m][4 + q]);
          b.acc[m][q] = M[m][q] + M[m][4 + q];
        }
        plane_modes_adjoint(lo, f);
        combine(m, f);
      }
    } else {
      // ---- upper node plane: in-plane parts; d/dz between the planes
      T gz[3][4];
      {
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const T v[4] = {b.own[m], nd[m * NY * BX + 1], nd[m * NY * BX + BX], nd[m * NY * BX + BX + 1]};
          plane_forward(v, s.t, b.ex[m], b.dy[m], b.iy[m]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            gz[m][q] = b.iy[m][q] - a.iy[m][q];
            if (!ISO) gz[m][q] *= s.ih[2];
          }
        }
      }
      // ---- stresses of the layer by Gauss level r; lo: the lower plane's adjoint with the layer below
      T lo_ex[3][2], lo_dy[3][2];
      const T* mod = mod_slot(li + 1) + row * BX + off + tx;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        T gx[3][2], gy[3][2], sx[3][2], sy[3][2];
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            gx[m][q] = fma(s.t[r], b.ex[m][q] - a.ex[m][q], a.ex[m][q]);
            gy[m][q] = fma(s.t[r], b.dy[m][q] - a.dy[m][q], a.dy[m][q]);
            if (!ISO) {
              gx[m][q] *= s.ih[0];
              gy[m][q] *= s.ih[1];
            }
          }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int i = q + 2 * p;
            const T lam = GPM ? mod[(i + 4 * r) * TY * BX] : lam_c, G = GPM ? mod[(8 + i + 4 * r) * TY * BX] : G_c;
            const T exx = gx[0][p], eyy = gy[1][q], ezz = gz[2][i];
            const T lt = lam * (exx + eyy + ezz), G2 = G + G;
            const T sxy = G * (gx[1][p] + gy[0][q]), sxz = G * (gx[2][p] + gz[0][i]), syz = G * (gy[2][q] + gz[1][i]);
            const T sxx = fma(G2, exx, lt), syy = fma(G2, eyy, lt), szz = fma(G2, ezz, lt);
            sx[0][p] = q ? sx[0][p] + sxx : sxx;
            sx[1][p] = q ? sx[1][p] + sxy : sxy;
            sx[2][p] = q ? sx[2][p] + sxz : sxz;
            sy[0][q] = p ? sy[0][q] + sxy : sxy;
            sy[1][q] = p ? sy[1][q] + syy : syy;
            sy[2][q] = p ? sy[2][q] + syz : syz;
            b.sz[0][i] = r ? b.sz[0][i] + sxz : sxz;
            b.sz[1][i] = r ? b.sz[1][i] + syz : syz;
            b.sz[2][i] = r ? b.sz[2][i] + szz : szz;
          }
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (!ISO) {
              sx[m][q] *= s.ih[0];
              sy[m][q] *= s.ih[1];
            }
            // 1 - t[r] = t[1 - r]
            lo_ex[m][q] = fma(s.t[1 - r], sx[m][q], r ? lo_ex[m][q] : a.aex[m][q]);
            lo_dy[m][q] = fma(s.t[1 - r], sy[m][q], r ? lo_dy[m][q] : a.ady[m][q]);
            b.aex[m][q] = r ? fma(s.t[1], sx[m][q], b.aex[m][q]) : s.t[0] * sx[m][q];
            b.ady[m][q] = r ? fma(s.t[1], sy[m][q], b.ady[m][q]) : s.t[0] * sy[m][q];
          }
      }
      // ---- lower plane finished: back to its nodes
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        T iy[4], f[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (!ISO) b.sz[m][q] *= s.ih[2];
          iy[q] = a.sz[m][q] - b.sz[m][q];
        }
        plane_adjoint(lo_ex[m], lo_dy[m], iy, s.t, f);
        combine(m, f);
      }
    }
    if (DIR && li + 2 <= nl) {  // the next layer's upper plane: the barrier publishes it
      if (!wait(li + 2)) bad = 1;
      form_direction(li + 2);
    }
    bad = __syncthreads_or(bad);
    if (bad) return false;
    issue(li + 1 + NS);  // into the stage every thread has just read
    if (kk >= z0 && out_node) {
      T tot[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) tot[m] = X0[m] + ex_w[m * TY * S::XP - S::XP];
      node_epilogue<T, EPI>(k, x, y, kk, tot, a.own, pre_f, pre_m, bc_flags_of(fx, fy, fz), red0, red1, red2);
      if constexpr (DIR) {
        const long long n = (long long)x + (long long)y * k.g.px + (long long)kk * k.g.plane;
#pragma unroll
        for (int m = 0; m < 3; ++m) k.p_new[n + m * k.g.n] = a.own[m];
      }
    }
    return true;
  };

#pragma unroll
  for (int j = 0; j < NS; ++j) issue(j);
  if constexpr (DIR) {  // under the first copies
    if (!k.dir_first) beta = (T)(k.red.scal[k.s_rz] / k.red.scal[k.s_rz_prev]);
#pragma unroll
    for (int t = 0; t < CT; ++t) c_in[t] = k.g.nx - (xs + (tid + t * NT) % (BX / A16) * A16);
  }
  coarse_mod(z0 - 1);
  State a, b;
  if constexpr (DIR) {
    if (TMA && !wait(0)) bad = 1;
    if (!wait(1)) bad = 1;  // cp.async: planes 0 and 1
    form_direction(0);
    form_direction(1);
    __syncthreads();
  } else if (!wait(0)) {
    bad = 1;
  }
  {
    const T* nd = node_slot(0) + row * BX + off + tx;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const T v[4] = {nd[m * NY * BX], nd[m * NY * BX + 1], nd[m * NY * BX + BX], nd[m * NY * BX + BX + 1]};
      a.own[m] = v[0];
      if constexpr (MODES) {
        plane_modes(v, a.h[m]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a.v[m][q] = v[q];
          a.acc[m][q] = T(0);
        }
      } else {
        plane_forward(v, s.t, a.ex[m], a.dy[m], a.iy[m]);
#pragma unroll
        for (int q = 0; q < 4; ++q) a.sz[m][q] = T(0);
#pragma unroll
        for (int q = 0; q < 2; ++q) a.aex[m][q] = a.ady[m][q] = T(0);
      }
    }
  }
  bad = __syncthreads_or(bad);
  if (!bad) issue(NS);
  // two layers per turn: the two states swap roles instead of being copied
  for (int li = 0; !bad;) {
    if (!layer(li, a, b) || ++li == nl) break;
    if (!layer(li, b, a) || ++li == nl) break;
  }
  if constexpr (!TMA) asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (TMA && bad && tid == 0 && k.err) *k.err = 1.0;
  if (EPI == EPI_RESIDUAL || EPI == EPI_PCG || (EPI == EPI_FAS && k.red.slot[1] >= 0)) {
    double v[3] = {red0, red1, red2};
    grid_reduce<3, RED_SUM, true>(v, k.red);
  }
}

// Tile height, resident blocks the registers are budgeted for, and staged layers.  FP64: 8 rows, 2 blocks of
// 128 threads (a layer's state and arithmetic take 230-250 registers); 16 rows in one block leave nothing
// to run across the layer barrier (257^3 apply 822 us against 737 us), a third block needs the carried
// state in shared memory, whose traffic then binds (815 us).  FP32: 16 rows, 2 blocks of 256 threads (125
// registers); with 8 rows the tiles overlap more (410 against 401 us).  Two stages instead of three cost
// FP64 7 % (703 against 656 us): a layer's arithmetic is too short to cover the copies.
// In modes (coarse levels) FP64 needs 160 registers, so a third block fits: 65^3 FAS increments 5.67 ms against 5.75
// with 2; in FP32 a third block spills: 97^3 precision form 98.9 ms against 98.2 with 2.
// LOW: half the rows and twice the blocks an SM, for levels of few node rows (run_tile_h).
template <typename T, bool MODES, bool LOW> struct TileShape {
  static constexpr bool F64 = sizeof(T) == 8;
  static constexpr int FULL = F64 ? 8 : 16, TY = LOW ? FULL / 2 : FULL, MINB = (F64 && MODES ? 3 : 2) * (LOW ? 2 : 1), NS = 3;
  static_assert(TY >= kMinTileY, "partials_doubles");
};

template <typename T, bool GPM, int EPI, bool ISO, bool TMA, bool DIR, bool LOW>
int run_tile(hpc_ctx* c, MechKT<T>& k, int cls) {
  using Shape = TileShape<T, !GPM && ISO, LOW>;
  constexpr int TY = Shape::TY, NS = Shape::NS;
  constexpr bool EX = DIR || EPI == EPI_RESIDUAL;
  using S = TileSmem<T, GPM, TY, NS, EX>;
  if (EPI == EPI_RESIDUAL) {
    k.dir_r = k.fu;
    k.dir_m = k.invM;
  }
  auto kern = mech_tile_kernel<T, GPM, EPI, ISO, TMA, TY, Shape::MINB, NS, DIR>;
  int per_sm = 1, rc;
  if ((rc = kernel_cfg((const void*)kern, S::bytes, S::bytes, kTX * TY, &per_sm))) return rc;
  k.sg = tile_geo(k.g, TY, (long long)num_sms() * per_sm, (long long)c->partials_cap / 3);
  if ((size_t)k.sg.nstrips * 3 > c->partials_cap) return cuda_fail(cudaErrorInvalidValue, "partials buffer");
  if constexpr (TMA) {
    if ((rc = encode_tensor<T>(k.g, k.fields[0], 3, S::BX, TY + 1, 1, &k.tmap))) return rc;
    if (EX && ((rc = encode_tensor<T>(k.g, k.dir_r, 3, S::BX, TY + 1, 1, &k.rmap)) ||
               (k.dir_m && (rc = encode_tensor<T>(k.g, k.dir_m, 3, S::BX, TY + 1, 1, &k.mmap)))))
      return rc;
    if (GPM && (rc = encode_tensor<T>(k.g, k.gpm, 16, S::BX, TY, 1, &k.gmap))) return rc;
  }
  const bool apart = (k.red.slot[0] >= 0 || k.red.slot[1] >= 0 || k.red.slot[2] >= 0) &&
                     combine_apart(k.sg, (long long)num_sms() * per_sm);
  if (apart) k.red.counter = nullptr;
  timing_begin(c, cls);
  kern<<<(unsigned)k.sg.nstrips, kTX * TY, S::bytes, c->stream>>>(k);
  if (apart) launch_combine(c, k.red, (int)k.sg.nstrips, kTX * TY);
  timing_end(c, cls);
  HPC_CHECK_LAUNCH(c);
  return HPC_OK;
}

// Half the rows where one such tile holds the whole box.  More boxes (17 rows: 24 computed instead of 32) gain 3 to 8 %
// in single solves of 513 x 17 x 1025 nodes, but cost a batch of six small specimens 0.5 %.
template <typename T, bool GPM, int EPI, bool ISO, bool TMA, bool DIR>
int run_tile_h(hpc_ctx* c, MechKT<T>& k, int cls) {
  if (k.g.ny < TileShape<T, !GPM && ISO, true>::TY) return run_tile<T, GPM, EPI, ISO, TMA, DIR, true>(c, k, cls);
  return run_tile<T, GPM, EPI, ISO, TMA, DIR, false>(c, k, cls);
}
template <typename T, bool GPM, int EPI, bool DIR = false>
int run_tile_e(hpc_ctx* c, MechKT<T>& k, int cls) {
  const bool iso = k.g.hx == k.g.hy && k.g.hy == k.g.hz;
  if (c->tma_stage)
    return iso ? run_tile_h<T, GPM, EPI, true, true, DIR>(c, k, cls) : run_tile_h<T, GPM, EPI, false, true, DIR>(c, k, cls);
  return iso ? run_tile_h<T, GPM, EPI, true, false, DIR>(c, k, cls) : run_tile_h<T, GPM, EPI, false, false, DIR>(c, k, cls);
}

}  // namespace

// What the drivers ask for: reactions on the finest level, the plain operator (hpc_internal_force) on coarse levels,
// both in FP64 only.
template <typename T>
int launch_mech_tile(hpc_ctx* c, MechKT<T>& k, bool finest, int epi) {
  constexpr bool F64 = sizeof(T) == 8;
  if (finest) {
    const int pcg = F64 ? HPC_KC_MECH_PCG_FINEST : HPC_KC_MECH32_PCG_FINEST;
    switch (epi) {
      case EPI_RESIDUAL: return run_tile_e<T, true, EPI_RESIDUAL>(c, k, HPC_KC_NONE);
      case EPI_PCG: return k.p_new ? run_tile_e<T, true, EPI_PCG, true>(c, k, pcg) : run_tile_e<T, true, EPI_PCG>(c, k, pcg);
      case EPI_REACTION:
        if constexpr (F64) return run_tile_e<T, true, EPI_REACTION>(c, k, HPC_KC_NONE);
    }
    return HPC_ERR_ARG;
  }
  switch (epi) {
    case EPI_RESIDUAL: return run_tile_e<T, false, EPI_RESIDUAL>(c, k, HPC_KC_NONE);
    case EPI_PCG:
      return k.p_new ? run_tile_e<T, false, EPI_PCG, true>(c, k, HPC_KC_NONE) : run_tile_e<T, false, EPI_PCG>(c, k, HPC_KC_NONE);
    case EPI_FAS: return run_tile_e<T, false, EPI_FAS>(c, k, HPC_KC_NONE);
    case EPI_PLAIN:
      if constexpr (F64) return run_tile_e<T, false, EPI_PLAIN>(c, k, HPC_KC_NONE);
  }
  return HPC_ERR_ARG;
}
template int launch_mech_tile<double>(hpc_ctx*, MechKT<double>&, bool, int);
template int launch_mech_tile<float>(hpc_ctx*, MechKT<float>&, bool, int);

}  // namespace hpc
