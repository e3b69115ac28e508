// Smoothers of small levels in one thread-block cluster: pcg_u (mechanical_pcg.cpp:223-330) with all of
// its iterations - Dirichlet values, residual, direction, K p, dots, updates - in one launch, the
// level's vectors in the cluster's shared memory.  The V-cycle calls the coarsest solve once per cycle
// with 50 iterations (mechanical_multigrid.cpp:29-32) and the next levels' smoothers with a few; as
// separate kernels an iteration costs three dependent launches and their reduction tails.
//
// The level is cut into slabs of node planes along its longest axis, one slab per block of the cluster.
// A block computes every element layer that touches its planes (the layers between two slabs are
// computed by both), so an iteration exchanges only two things: the dot-product partials, written by
// every warp to every block, and the preconditioned residual of the slabs' boundary planes, from which
// a neighbour forms its ghost copy of the direction.  They travel as asynchronous stores into the
// receiver's shared memory that its mbarrier counts, two exchanges per iteration: (p, w), and (r, M^-1 r)
// with the boundary planes.  A buffer is written again only after every warp has read it: a block sends
// the next (p, w) when it has every warp's (r, M^-1 r), which a warp sends after reading its (p, w).
//
// Element forces are computed element-parallel into shared memory and gathered per node in a fixed order
// (layer below, layer above): no atomics, the sums are the same for every number of blocks; the
// partials are added in rank and warp order.  The rounding differs from the
// tile kernels' only in the order of the same sums.
//
// What bounds it: the serial chain of an iteration (about 2.4 us on 9^3: a third the element arithmetic and
// gather, a third the two sums with their quotients, the rest the direction, the updates and the
// exchanges).  50 iterations on 9^3: 121 us, against 388 us in one thread block, and 194 us with cluster
// barriers and release fences instead of counted stores; 4 iterations on 17^3 take 33 us against about
// 90 us in separate kernels.  Increments: 33^3 FAS 6.3 -> 5.1 ms, 65^3 precision form (3) 98 -> 74 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "device_common.cuh"
#include "internal.h"

namespace hpc {
namespace {

constexpr int kBlocks = 16;  // cluster size (non-portable)
constexpr size_t kMaxSmem = 220 * 1024;

// How a level is laid over the cluster.
struct ClusterPlan {
  int axis;            // planes are cut along this axis (0 x, 1 y, 2 z)
  int planes, n1, n2;  // extent along it; the other two axes, n1 the lower-numbered one
  int active;          // blocks that hold planes
  int lp;              // element layers a block computes at most
  int shape;           // block shape (kShapes)
  int threads, slots;  // threads a block; own nodes and elements a thread at most
  size_t smem;
};

// Block shapes, smallest first: a level takes the first that holds a block's share.  Own nodes and elements
// are unrolled over `slots` (the nodes' vectors live in registers): a coarsest level that needs one slot
// does not run through the code of more, which a few iterations would mostly spend fetching.
constexpr int kShapes[][2] = {{128, 1}, {256, 2}, {512, 2}};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);

// Components of the field, and coefficients an element keeps: lam and G, or the phase field's mass and
// gradient weights at its 8 Gauss points.
template <bool PF> struct FieldShape { static constexpr int NC = PF ? 1 : 3, NM = PF ? 16 : 2; };

// The level's longest axis is cut; false where a block's share exceeds the register slots or shared memory.
template <typename T, bool PF>
bool cluster_plan(const LevelGeo& g, ClusterPlan* p) {
  const int n[3] = {g.nx, g.ny, g.nz};
  if (n[0] < 2 || n[1] < 2 || n[2] < 2) return false;
  p->axis = 2;
  for (int a = 1; a >= 0; --a)
    if (n[a] > n[p->axis]) p->axis = a;
  p->planes = n[p->axis];
  p->n1 = p->axis == 0 ? n[1] : n[0];
  p->n2 = p->axis == 2 ? n[1] : n[2];
  p->active = std::min(kBlocks, p->planes);
  const size_t PN = (size_t)p->n1 * p->n2, EN = (size_t)(p->n1 - 1) * (p->n2 - 1);
  const size_t np = (size_t)(p->planes + p->active - 1) / p->active;
  p->lp = (int)np + 1;
  constexpr int NC = FieldShape<PF>::NC, NM = FieldShape<PF>::NM;
  const size_t vals = 2 * NC * PN + NC * (np + 2) * PN + (NM + 8 * NC) * (np + 1) * EN;
  for (p->shape = 0; p->shape < kNumShapes; ++p->shape) {
    const auto& sh = kShapes[p->shape];
    p->threads = sh[0];
    p->slots = sh[1];
    p->smem = sizeof(double) * 4 * kBlocks * (sh[0] / 32) + sizeof(T) * vals + 32;
    const size_t most = (size_t)sh[0] * sh[1];
    if (np * PN <= most && (np + 1) * EN <= most) return p->smem <= kMaxSmem;
  }
  return false;
}

// u, fu, ru in IO; the arithmetic and the material in T.
template <typename T, typename IO>
struct ClusterArgs {
  LevelGeo g;
  ClusterPlan p;
  IO* u;
  const IO* fu;
  IO* ru;
  const T* invM;
  const T* Ke;  // element moduli; phase field: nodal gc and element H
  const T* Ge;
  T Ut;  // top value of u_z; phase field: the length scale lc
  int nb;
  double* scal;
  int r_given;  // ru holds the first residual: no apply for it
  int s_rnorm, s_fnorm;  // |r|^2 of the first residual, |f|^2 (phase field); -1: not wanted
  double* err;  // the context's: set to 1 when a bounded wait ran out
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// A value into another block's shared memory, counted by the mbarrier beside it (no fence, no cluster
// barrier: the receiver waits for the bytes).
__device__ __forceinline__ void put(uint32_t addr, uint32_t bar, double v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void put(uint32_t addr, uint32_t bar, float v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void expect(uint32_t bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
constexpr unsigned kClusterPolls = 1u << 22;  // far above any exchange's latency; then the kernel reports
// The phase of `bar` with this parity has completed; false when the wait ran out.
__device__ __forceinline__ bool arrived(uint32_t bar, uint32_t parity) {
  for (unsigned i = 0; i < kClusterPolls; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, "
        "1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T, typename IO, bool PF, bool ISO, int kThreads, int kSlots>
__global__ void __launch_bounds__(kThreads, 1) cluster_pcg_kernel(const __grid_constant__ ClusterArgs<T, IO> A) {
  constexpr int kWarpsC = kThreads / 32, NC = FieldShape<PF>::NC, NM = FieldShape<PF>::NM;
  extern __shared__ __align__(16) unsigned char csm[];
  const LevelGeo& g = A.g;
  const ClusterPlan& P = A.p;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)blockIdx.x;
  const int PN = P.n1 * P.n2, E1 = P.n1 - 1, EN = E1 * (P.n2 - 1);
  // own planes [a, b), element layers [la, lb); local plane 0 of the direction is plane a - 1
  const bool active = rank < P.active;
  const int a = active ? (int)((long long)P.planes * rank / P.active) : 0;
  const int b = active ? (int)((long long)P.planes * (rank + 1) / P.active) : 0;
  const int np = b - a, la = max(a - 1, 0), lb = active ? min(b, P.planes - 1) : la;
  const int NO = np * PN, NE = (lb - la) * EN;     // own nodes, elements computed
  // mbarriers of the two exchanges of an iteration, then what they bring
  const uint32_t barA = smem_addr(csm), barB = barA + 8;
  double* partA = reinterpret_cast<double*>(csm + 16);  // (p, w) partials of every warp of the cluster
  double* partB = partA + kBlocks * kWarpsC;       // (r, M^-1 r)
  double* partN = partB + kBlocks * kWarpsC;       // |r|^2 of the first residual, then |f|^2
  // M^-1 r of planes a - 1 and b, from the neighbours (ahead of what depends on a block's own np: every
  // block has it at the same address)
  T* zh = reinterpret_cast<T*>(partN + 2 * kBlocks * kWarpsC);
  const int SP = (np + 2) * PN;
  T* sp = zh + 2 * NC * PN;  // direction, component stride SP
  T* sc = sp + NC * SP;         // element coefficients [i][element]
  T* sf = sc + NM * P.lp * EN;  // element forces [m*8+n][element]
  const int FS = P.lp * EN;
  const SFt<T> s = make_sf<T>(g);
  const T wg = ISO ? T(g.wg) * (s.ih[0] * s.ih[0]) : T(g.wg);
  // local offsets of a step in x, y, z (nodes)
  const int sx = P.axis == 0 ? PN : 1, sy = P.axis == 0 ? 1 : (P.axis == 1 ? PN : P.n1), sz = P.axis == 2 ? PN : P.n1;
  auto coords = [&](int plane, int i1, int i2, int& i, int& j, int& k) {
    if (P.axis == 0) {
      i = plane, j = i1, k = i2;
    } else if (P.axis == 1) {
      i = i1, j = plane, k = i2;
    } else {
      i = i1, j = i2, k = plane;
    }
  };
  auto node = [&](int pl, int in) {
    int i, j, k;
    coords(pl, in % P.n1, in / P.n1, i, j, k);
    return nidx(g, i, j, k);
  };
  auto node_fix = [&](int pl, int in, bool& top) -> unsigned {
    int i, j, k;
    coords(pl, in % P.n1, in / P.n1, i, j, k);
    const BcFlags bc = bc_flags(g, i, j, k);
    top = bc.top;
    return (bc.c0 ? 1u : 0u) | (bc.c1 ? 2u : 0u) | (bc.c2 ? 4u : 0u);
  };

  // ---- load: the direction buffer takes u with its Dirichlet values (Dirichlet_BD), ghost planes included
  for (int q = tid; q < SP; q += kThreads) {
    const int pl = a - 1 + q / PN, in = q % PN;
    const bool inside = active && pl >= 0 && pl < P.planes;
    bool top = false;
    const unsigned fx = !PF && inside ? node_fix(pl, in, top) : 0u;
    const long long n = inside ? node(pl, in) : 0;
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      T uv = inside ? (T)A.u[n + m * g.n] : T(0);
      if ((fx >> m) & 1u) uv = (m == 2 && top) ? A.Ut : T(0);
      sp[m * SP + q] = uv;
    }
  }
  // elements q = tid + t kThreads: where element q's corner 0 sits in the direction buffer
  int corner0[kSlots];
#pragma unroll
  for (int t = 0; t < kSlots; ++t) {
    const int q = tid + t * kThreads;
    corner0[t] = 0;
    if (q < NE) {
      const int l = la + q / EN, e = q % EN;
      int i, j, k;
      coords(l, e % E1, e / E1, i, j, k);
      const long long n = nidx(g, i, j, k);
      if constexpr (PF) {
        double gcn[8], gcg[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) gcn[c] = A.Ke[nidx(g, i + (c & 1), j + ((c >> 1) & 1), k + (c >> 2))];
        gp_material(gcn, s, gcg);
        const double H2 = 2.0 * A.Ge[n], inv_lc = 1.0 / A.Ut;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          sc[c * FS + q] = g.wg * fma(gcg[c], inv_lc, H2);
          sc[(8 + c) * FS + q] = wg * (gcg[c] * A.Ut);
        }
      } else {
        const T G = A.Ge[n] * wg;
        sc[q] = ISO ? fma(T(-2.0 / 3.0), G, A.Ke[n] * wg) : A.Ke[n] * wg;
        sc[FS + q] = G;
      }
      corner0[t] = (l - (a - 1)) * PN + (e / E1) * P.n1 + e % E1;
    }
  }
  // own nodes q = tid + t kThreads: vectors in registers; the Dirichlet rows (bits 0-2), which corners of
  // the node have an element (bits 8 + d + 2 d1 + 4 d2, d along the axis), and its corner-0 element's slot
  T u[kSlots][NC], r[kSlots][NC], mi[kSlots][NC], w[kSlots][NC];
  unsigned info[kSlots];
  int eslot[kSlots];
#pragma unroll
  for (int t = 0; t < kSlots; ++t) {
    const int q = tid + t * kThreads;
    info[t] = 0;
    eslot[t] = 0;
    if (q < NO) {
      const int pl = a + q / PN, in = q % PN, i1 = in % P.n1, i2 = in / P.n1;
      const long long n = node(pl, in);
      bool top = false;
      info[t] = PF ? 0u : node_fix(pl, in, top);
      eslot[t] = (pl - la) * EN + i2 * E1 + i1;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int d = c & 1, d1 = (c >> 1) & 1, d2 = c >> 2;
        if (pl - d >= 0 && pl - d < P.planes - 1 && i1 - d1 >= 0 && i1 - d1 < E1 && i2 - d2 >= 0 && i2 - d2 < P.n2 - 1)
          info[t] |= 256u << c;
      }
#pragma unroll
      for (int m = 0; m < NC; ++m) {
        u[t][m] = (T)A.u[n + m * g.n];
        if ((info[t] >> m) & 1u) u[t][m] = (m == 2 && top) ? A.Ut : T(0);
        mi[t][m] = A.invM[n + m * g.n];
      }
    }
  }
  // element corner (d along the axis, d1, d2) -> corner number in x, y, z
  const int cd = P.axis == 0 ? 1 : (P.axis == 1 ? 2 : 4), c1 = P.axis == 0 ? 2 : 1, c2 = P.axis == 2 ? 2 : 4;
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barA) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barB) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster_sync();  // every block of the cluster has started and its barriers exist: it may be written to
  // bytes an exchange brings to this block: a partial of every warp; with (r, M^-1 r) also the ghost planes
  constexpr int kPartBytes = kBlocks * kWarpsC * (int)sizeof(double);
  const int zbytes = active ? ((rank > 0) + (rank + 1 < P.active)) * NC * PN * (int)sizeof(T) : 0;
  bool ok = true;
  uint32_t phA = 0, phB = 0;
  auto receive = [&](uint32_t bar, uint32_t& phase) {  // after a wait that ran out none is tried again
    if (ok && !arrived(bar, phase)) ok = false;
    phase ^= 1u;
  };

  // K v of the own nodes into w, v in the direction buffer
  auto apply = [&]() {
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      const int q = tid + t * kThreads;
      if (q >= NE) break;
      const T* v = sp + corner0[t];
      T f[NC][8];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int o = (n & 1) * sx + ((n >> 1) & 1) * sy + (n >> 2) * sz;
#pragma unroll
        for (int m = 0; m < NC; ++m) f[m][n] = v[m * SP + o];
      }
      if constexpr (PF) {
        double xv[8], aw[8], bw[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          xv[c] = f[0][c];
          aw[c] = sc[c * FS + q];
          bw[c] = sc[(8 + c) * FS + q];
        }
        pf_element<ISO>(xv, aw, bw, s, f[0]);
      } else if constexpr (ISO) {
        mech_element_const(f, sc[q], sc[FS + q]);
      } else {
        T uu[3][8], Kw[8], Gw[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          Kw[n] = sc[q];
          Gw[n] = sc[FS + q];
#pragma unroll
          for (int m = 0; m < 3; ++m) uu[m][n] = f[m][n];
        }
        mech_element<false>(uu, Kw, Gw, s, f);
      }
#pragma unroll
      for (int m = 0; m < NC; ++m)
#pragma unroll
        for (int n = 0; n < 8; ++n) sf[(m * 8 + n) * FS + q] = f[m][n];
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      if (tid + t * kThreads >= NO) continue;
      T acc[NC] = {};
#pragma unroll
      for (int d = 1; d >= 0; --d)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int d1 = c & 1, d2 = c >> 1;
          if (info[t] & (256u << (d + 2 * d1 + 4 * d2))) {
            const T* fe = sf + (d * cd + d1 * c1 + d2 * c2) * FS + eslot[t] - (d * EN + d2 * E1 + d1);
#pragma unroll
            for (int m = 0; m < NC; ++m) acc[m] += fe[m * 8 * FS];
          }
        }
#pragma unroll
      for (int m = 0; m < NC; ++m) w[t][m] = acc[m];
    }
  };
  // this warp's partial to every block of the cluster
  auto share = [&](double* part, uint32_t bar, double v) {
    v = warp_sum(v);
    if (lane < kBlocks) put(remote(smem_addr(part + rank * kWarpsC + warp), lane), remote(bar, lane), v);
  };
  // the cluster's sum, the same bits in every thread (rank and warp order, then the shuffle tree)
  auto total = [&](const double* part) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < kBlocks * kWarpsC / 32; ++q) v += part[q * 32 + lane];
    return warp_sum(v);
  };
  // M^-1 r of an own node on a boundary plane to the neighbour's ghost copy
  auto share_z = [&](int q, int m, T z) {
    if (q < PN && rank > 0) put(remote(smem_addr(zh + (NC + m) * PN + q), rank - 1), remote(barB, rank - 1), z);
    if (q >= NO - PN && rank + 1 < P.active)
      put(remote(smem_addr(zh + m * PN + q - (NO - PN)), rank + 1), remote(barB, rank + 1), z);
  };

  // ---- initial residual r = f - K u, zero on Dirichlet rows
  if (tid == 0) expect(barB, (PF ? 3 : 2) * kPartBytes + zbytes);
  if (!A.r_given) apply();
  double rz = 0.0, rn = 0.0, ff = 0.0;
#pragma unroll
  for (int t = 0; t < kSlots; ++t) {
    const int q = tid + t * kThreads;
    if (q >= NO) continue;
    const long long n = node(a + q / PN, q % PN);
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const T fv = A.r_given ? (T)A.ru[n + m * g.n] : (T)A.fu[n + m * g.n];
      const T rv = (info[t] >> m) & 1u ? T(0) : (A.r_given ? fv : fv - w[t][m]), z = rv * mi[t][m];
      if (PF) ff = fma((double)fv, (double)fv, ff);
      r[t][m] = rv;
      rz = fma((double)rv, (double)z, rz);
      rn = fma((double)rv, (double)rv, rn);
      share_z(q, m, z);
    }
  }
  share(partB, barB, rz);
  share(partN, barB, rn);
  if (PF) share(partN + kBlocks * kWarpsC, barB, ff);
  receive(barB, phB);
  rz = total(partB);
  if (rank == 0 && warp == 0 && A.s_rnorm >= 0) {
    rn = total(partN);
    if (lane == 0) A.scal[A.s_rnorm] = rn;
    if (PF) {
      ff = total(partN + kBlocks * kWarpsC);
      if (lane == 0) A.scal[A.s_fnorm] = ff;
    }
  }

  double rz_prev = 1.0;
  for (int it = 0; it < A.nb; ++it) {
    // direction p = M^-1 r + beta p; on the ghost planes from the neighbours' M^-1 r (planes outside the
    // level stay zero)
    const T beta = it == 0 ? T(0) : (T)(rz / rz_prev);
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      const int q = tid + t * kThreads;
      if (q >= NO) continue;
#pragma unroll
      for (int m = 0; m < NC; ++m) {
        const T z = r[t][m] * mi[t][m];
        T* p = sp + m * SP + PN + q;
        *p = it == 0 ? z : fma(beta, *p, z);
      }
    }
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      if (side ? b >= P.planes : a == 0) continue;
      for (int in = tid; in < PN; in += kThreads)
#pragma unroll
        for (int m = 0; m < NC; ++m) {
          T* p = sp + m * SP + (side ? SP - PN : 0) + in;
          const T z = zh[(side * NC + m) * PN + in];
          *p = it == 0 ? z : fma(beta, *p, z);
        }
    }
    if (tid == 0) expect(barA, kPartBytes);
    __syncthreads();
    apply();
    double pw = 0.0;
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      const int q = tid + t * kThreads;
      if (q >= NO) continue;
#pragma unroll
      for (int m = 0; m < NC; ++m) pw = fma((double)sp[m * SP + PN + q], (double)w[t][m], pw);
    }
    share(partA, barA, pw);
    const bool more = it + 1 < A.nb;
    if (more && tid == 0) expect(barB, kPartBytes + zbytes);
    receive(barA, phA);
    const T alpha = (T)(rz / total(partA));
    double rz_new = 0.0;
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      const int q = tid + t * kThreads;
      if (q >= NO) continue;
#pragma unroll
      for (int m = 0; m < NC; ++m) {
        u[t][m] = fma(sp[m * SP + PN + q], alpha, u[t][m]);
        const T rv = (info[t] >> m) & 1u ? T(0) : fma(-w[t][m], alpha, r[t][m]), z = rv * mi[t][m];
        r[t][m] = rv;
        rz_new = fma((double)rv, (double)z, rz_new);
        if (more) share_z(q, m, z);
      }
    }
    if (more) {
      share(partB, barB, rz_new);
      receive(barB, phB);
      rz_prev = rz;
      rz = total(partB);
    }
  }

  // ---- write u and the last residual back
#pragma unroll
  for (int t = 0; t < kSlots; ++t) {
    const int q = tid + t * kThreads;
    if (q >= NO) continue;
    const long long n = node(a + q / PN, q % PN);
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      A.u[n + m * g.n] = (IO)u[t][m];
      A.ru[n + m * g.n] = (IO)r[t][m];
    }
  }
  if (!ok && lane == 0) *A.err = 1.0;
  cluster_sync();  // no block ends while another may still write to it
}

template <typename T, typename IO>
using ClusterKernel = void (*)(const ClusterArgs<T, IO>);
template <typename T, typename IO, bool PF, bool ISO>
ClusterKernel<T, IO> shape_kernel(int threads) {
  if (threads == 128) return cluster_pcg_kernel<T, IO, PF, ISO, 128, 1>;
  if (threads == 256) return cluster_pcg_kernel<T, IO, PF, ISO, 256, 2>;
  return cluster_pcg_kernel<T, IO, PF, ISO, 512, 2>;
}

cudaLaunchConfig_t cluster_config(int threads, size_t smem, cudaStream_t stream, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kBlocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = kBlocks;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

template <bool PF, typename T, typename IO>
int launch_cluster(hpc_ctx* c, ClusterArgs<T, IO>& a) {
  if (!cluster_plan<T, PF>(a.g, &a.p)) return HPC_ERR_ARG;
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = cluster_config(a.p.threads, a.p.smem, c->stream, &at);
  const bool iso = a.g.hx == a.g.hy && a.g.hy == a.g.hz;
  HPC_CUDA(cudaLaunchKernelEx(
      &cfg, iso ? shape_kernel<T, IO, PF, true>(a.p.threads) : shape_kernel<T, IO, PF, false>(a.p.threads), a));
  HPC_CHECK_LAUNCH(c);
  return HPC_OK;
}

// Sets the kernels' attributes; false where the device refuses one.
template <typename T, typename IO, bool PF>
bool prepare(int shape) {
  for (ClusterKernel<T, IO> k : {shape_kernel<T, IO, PF, true>(kShapes[shape][0]), shape_kernel<T, IO, PF, false>(kShapes[shape][0])})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      return false;
  return true;
}
// Whether a whole cluster of a shape can be resident with all the shared memory a level may ask for.  The kernels of a
// shape have the same threads and registers for one such block an SM: one answers for all.
bool resident(int shape) {
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = cluster_config(kShapes[shape][0], kMaxSmem, nullptr, &at);
  int n = 0;
  return cudaOccupancyMaxActiveClusters(&n, (const void*)shape_kernel<double, double, false, true>(kShapes[shape][0]),
                                        &cfg) == cudaSuccess && n > 0;
}

}  // namespace

// A level is smoothed in a cluster where its share fits a block and the device can hold such a cluster; a device
// that offers fewer SMs side by side (a partitioned GPU) runs the per-iteration kernels.
template <bool PF>
static bool fits(const hpc_ctx* c, const LevelGeo& g) {
  ClusterPlan p;
  return cluster_plan<double, PF>(g, &p) && ((c->cluster_shapes >> p.shape) & 1u);
}
bool cluster_pcg_fits_geo(const hpc_ctx* c, const LevelGeo& g) { return fits<false>(c, g); }
bool cluster_pcg_fits(const hpc_ctx* c, int level) {
  if (level == c->maxlevel) return false;  // the finest level's material is nodal, not element-constant
  return cluster_pcg_fits_geo(c, c->L[level]);
}

// The block shapes a cluster can be resident with on a device (a bit each); asked once per device, by hpc_create.
unsigned cluster_pcg_shapes(int device) {
  static std::mutex mu;
  static std::map<int, unsigned> known;
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(device);
  if (it != known.end()) return it->second;
  unsigned shapes = 0;
  for (int s = 0; s < kNumShapes; ++s)
    if (prepare<double, double, false>(s) && prepare<double, float, false>(s) && prepare<float, float, false>(s) &&
        prepare<double, double, true>(s) && resident(s))
      shapes |= 1u << s;
    else
      cudaGetLastError();  // a refusal is an answer
  return known[device] = shapes;
}

int launch_cluster_pcg_on(hpc_ctx* c, const LevelGeo& g, double* u, const double* fu, double* ru, const double* invM,
                          const double* Ke, const double* Ge, double Ut, int nb) {
  const int r_given = 0;
  ClusterArgs<double, double> a{g, {}, u, fu, ru, invM, Ke, Ge, Ut, nb, c->scal, r_given, S_RNORM, -1, c->err};
  return launch_cluster<false>(c, a);
}

int launch_cluster_pcg(hpc_ctx* c, int level, double Ut, int nb, bool r_given) {
  const LevelFields& F = c->F[level];
  ClusterArgs<double, double> a{c->L[level], {}, F.u, F.fu, F.ru, F.preMu, F.Ke, F.Ge, Ut, nb, c->scal, r_given, S_RNORM, -1,
                                c->err};
  return launch_cluster<false>(c, a);
}

int launch_cluster_pcg_f32(hpc_ctx* c, int level, int nb, bool r_given) {
  const LevelF32& F = c->F32[level];
  ClusterArgs<float, float> a{c->L[level], {}, F.u, F.fu, F.ru, F.invM, F.Ke, F.Ge, 0.f, nb, c->scal, r_given, -1, -1, c->err};
  return launch_cluster<false>(c, a);
}

int launch_cluster_pcg_mixed(hpc_ctx* c, int level, int nb, bool r_given) {
  const LevelFields& F = c->F[level];
  const LevelF32& G = c->F32[level];
  ClusterArgs<double, float> a{c->L[level], {}, G.u, G.fu, G.ru, F.preMu, F.Ke, F.Ge, 0.0, nb, c->scal, r_given, S_RNORM, -1, c->err};
  return launch_cluster<false>(c, a);
}

bool cluster_pcg_d_fits(const hpc_ctx* c, int level) { return fits<true>(c, c->L[level]); }

// pcg_d (phase_field_pcg.cpp:133-214) of a small level.
int launch_cluster_pcg_d(hpc_ctx* c, int level, double lc, int nb) {
  const LevelFields& F = c->F[level];
  ClusterArgs<double, double> a{c->L[level], {}, F.d, F.fd, F.R, F.preMd, F.gc, F.H, lc, nb, c->scal, 0, S_RNORM, S_FDNORM,
                                c->err};
  return launch_cluster<true>(c, a);
}

}  // namespace hpc
