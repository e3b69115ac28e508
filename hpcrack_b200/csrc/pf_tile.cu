// Phase-field operator A_d on column tiles marched in z (every level), with the residual, PCG, FAS and
// plain epilogues: the scheme of mech_tile.cu for one scalar field whose coefficients come from the nodal
// toughness gc and the element history H.
//
// Per node plane a thread keeps the in-plane parts of x (derivatives and values at the 2x2 in-plane Gauss
// coordinates), the interpolated gc, and the adjoint of the layer below: about 190 operations an element
// against about 330 element by element.  Planes of x and gc arrive up to three layers ahead in
// shared-memory stages (tensor copies, or per-thread cp.async).
//
// What bounds it: the FP64 pipe on the large levels, the layers' serial chain on the small ones.  Per
// launch, with the strip kernel it replaced in brackets: 257^3 437 us (591), 129^3 69 (115), 65^3 19 (43),
// 33^3 13 (21).  16 x 16 columns, two blocks of 256 threads an SM (124 registers); on levels of few node rows 8 or 4
// element rows and as many threads an SM (tile_rows).
#include <algorithm>

#include "element_common.cuh"

namespace hpc {
namespace {

constexpr int kTX = kTileX, kStages = 3, kBX = 18, kXP = 20;
constexpr unsigned kPfWaitPolls = 1u << 24;  // far above any copy's latency; then the kernel reports
// A tile of TY rows: threads, staged rows, shared memory, resident blocks the registers are budgeted for.
template <int TY> struct PfShape {
  static constexpr int NT = kTX * TY, NY = TY + 1, MINB = 32 / TY;
  static constexpr size_t plane = (sizeof(double) * NY * kBX + 127) / 128 * 128;
  static constexpr size_t o_exch = 128 + kStages * 2 * plane, bytes = o_exch + sizeof(double) * 2 * TY * kXP + 128;
  static_assert(TY >= kMinTileY, "partials_doubles");
};

struct PfTileK {
  LevelGeo g;
  int tx, ty;  // tiles per axis
  const double *x, *gc, *H;
  double* out;
  double lc;
  const double* fd;
  const double* invM;
  RedTarget red;
  double* err;
  alignas(64) CUtensorMap xmap;
  alignas(64) CUtensorMap cmap;
};

// In-plane values of a nodal plane at the 2x2 Gauss coordinates, iy[q + 2p].
__device__ __forceinline__ void plane_values(const double (&v)[4], const double (&t)[2], double (&iy)[4]) {
  const double d0 = v[1] - v[0], d1 = v[3] - v[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double i0 = fma(t[q], d0, v[0]), i1 = fma(t[q], d1, v[2]), dy = i1 - i0;
    iy[q] = fma(t[0], dy, i0);
    iy[q + 2] = fma(t[1], dy, i0);
  }
}

struct PfState {
  double ex[2], dy[2], iy[4], gc[4], aex[2], ady[2], aiy[4], own;
  bool zero;  // a node of the plane's quad has gc == 0 (gauss_point_MP's zero rule)
};

template <int EPI, bool ISO, bool TMA, int TY>
__global__ void __launch_bounds__(kTX* TY, PfShape<TY>::MINB) pf_tile_kernel(const __grid_constant__ PfTileK k) {
  using S = PfShape<TY>;
  constexpr int NT = S::NT, NY = S::NY;
  extern __shared__ __align__(128) unsigned char pf_smem[];
  unsigned char* base = pf_smem + ((128u - (smem_u32(pf_smem) & 127u)) & 127u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base);
  double* exch = reinterpret_cast<double*>(base + S::o_exch);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & (kTX - 1);
  const int row = tile_row<TY>(warp, lane);
  const SF s = make_sf(k.g);
  // ISO: only the gradient term carries 1/h^2 (see sf_forward); the mass term keeps wg
  const double wgb = (ISO ? k.g.wg * (s.ih[0] * s.ih[0]) : k.g.wg) * k.lc, wga = k.g.wg / k.lc, wgh = 2.0 * k.g.wg;
  double red0 = 0.0, red1 = 0.0, red2 = 0.0;
  int bad = 0;
  if constexpr (TMA) {
    if (tid == 0) {
#pragma unroll
      for (int i = 0; i < kStages; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + i)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
  }
  const int tiles = k.tx * k.ty, chunks = (int)gridDim.x / tiles;
  const int tile = (int)(blockIdx.x % (unsigned)tiles), chunk = (int)(blockIdx.x / (unsigned)tiles);
  const int z0 = (int)((long long)k.g.nz * chunk / chunks), zend = (int)((long long)k.g.nz * (chunk + 1) / chunks) - 1;
  const int x0 = (tile % k.tx) * (kTX - 1), y0 = (tile / k.tx) * (TY - 1);
  const int x = x0 - 1 + tx, y = y0 - 1 + row;
  const int nl = zend - z0 + 2;  // element layers z0 - 1 .. zend; plane j of the stream is z0 - 1 + j
  const int xs = x0 - 1 >= 0 ? (x0 - 1) / 2 * 2 : -2, off = (x0 - 1) - xs;  // a copy starts on 16 bytes
  const bool xy_elem = x >= 0 && x <= k.g.nx - 2 && y >= 0 && y <= k.g.ny - 2;
  const bool out_node = tx >= 1 && row >= 1 && x < k.g.nx && y < k.g.ny;

  auto slot = [&](int j, int f) {
    return reinterpret_cast<double*>(base + 128 + (size_t)(((unsigned)j % kStages) * 2 + f) * S::plane);
  };
  auto issue = [&](int j) {
    if (j <= nl) {
      const int kk = z0 - 1 + j;
      if constexpr (TMA) {
        if (tid == 0) {
          const uint32_t bar = smem_u32(bars + (unsigned)j % kStages);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"((int)sizeof(double) * 2 * NY * kBX)
                       : "memory");
#pragma unroll
          for (int f = 0; f < 2; ++f)
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
                "%4, %5}], [%6];" ::"r"(smem_u32(slot(j, f))),
                "l"(f ? &k.cmap : &k.xmap), "r"(xs), "r"(y0 - 1), "r"(kk), "r"(0), "r"(bar)
                : "memory");
        }
      } else {
        constexpr int U = kBX / 2;  // 16-byte units of a row: whole ones, padding included, zeros outside the grid
        for (int q = tid; q < 2 * NY * U; q += NT) {
          const int u = q % U, r = q / U, ry = r % NY, f = r / NY;
          const int gx = xs + 2 * u, gy = y0 - 1 + ry;
          const bool ok = gx >= 0 && gx < k.g.px && gy >= 0 && gy < k.g.ny && kk >= 0 && kk < k.g.nz;
          const double* src = (f ? k.gc : k.x) + (ok ? nidx(k.g, gx, gy, kk) : 0);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(slot(j, f) + ry * kBX + 2 * u)),
                       "l"(src), "r"(ok ? 16 : 0)
                       : "memory");
        }
      }
    }
    if constexpr (!TMA) asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto wait = [&](int j) -> bool {
    if constexpr (TMA) {
      const uint32_t bar = smem_u32(bars + (unsigned)j % kStages), parity = ((unsigned)j / kStages) & 1u;
      for (unsigned i = 0; i < kPfWaitPolls; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
      }
      return false;
    } else {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 1) : "memory");
      __syncthreads();
      return true;
    }
  };
  // in-plane parts of stream plane j
  auto load_plane = [&](int j, PfState& b) {
    const double* n = slot(j, 0) + row * kBX + off + tx;
    const double* c = slot(j, 1) + row * kBX + off + tx;
    const double v[4] = {n[0], n[1], n[kBX], n[kBX + 1]}, g[4] = {c[0], c[1], c[kBX], c[kBX + 1]};
    const double d0 = v[1] - v[0], d1 = v[3] - v[2], dd = d1 - d0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double i0 = fma(s.t[q], d0, v[0]), i1 = fma(s.t[q], d1, v[2]);
      b.dy[q] = i1 - i0;
      b.iy[q] = fma(s.t[0], b.dy[q], i0);
      b.iy[q + 2] = fma(s.t[1], b.dy[q], i0);
      b.ex[q] = fma(s.t[q], dd, d0);
    }
    plane_values(g, s.t, b.gc);
    b.zero = bits_zero(g[0]) || bits_zero(g[1]) || bits_zero(g[2]) || bits_zero(g[3]);
    b.own = v[0];
  };
  double h_n = 0.0;  // 2 wg H of the next layer's element, one layer ahead
  auto history = [&](int kk) {
    h_n = xy_elem && kk >= 0 && kk <= k.g.nz - 2 ? wgh * k.H[nidx(k.g, x, y, kk)] : 0.0;
  };

  auto layer = [&](int li, const PfState& a, PfState& b) -> bool {
    const int kk = z0 - 1 + li;
    const double h = h_n;
    history(kk + 1);
    double pre_f = 0.0, pre_m = 0.0;
    if ((EPI == EPI_RESIDUAL || EPI == EPI_FAS) && out_node && kk >= z0) {
      const long long n = nidx(k.g, x, y, kk);
      pre_f = EPI == EPI_FAS ? k.out[n] : k.fd[n];
      if (EPI == EPI_RESIDUAL && k.invM) pre_m = k.invM[n];
    }
    if (!wait(li + 1)) bad = 1;
    load_plane(li + 1, b);
    const bool valid = xy_elem && kk >= 0 && kk <= k.g.nz - 2;
    const bool gzero = a.zero || b.zero;
    double gz[4], sz[4], lo_ex[2], lo_dy[2], lo_iy[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) gz[i] = b.iy[i] - a.iy[i];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      double gx[2], gy[2], sx[2], sy[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        gx[q] = fma(s.t[r], b.ex[q] - a.ex[q], a.ex[q]);
        gy[q] = fma(s.t[r], b.dy[q] - a.dy[q], a.dy[q]);
      }
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = q + 2 * p;
          const double gi = fma(s.t[r], b.gc[i] - a.gc[i], a.gc[i]);
          const double gc = gzero || !valid ? 0.0 : gi;
          const double aw = fma(gc, wga, h), bw = gc * wgb;
          const double sv = aw * fma(s.t[r], gz[i], a.iy[i]);
          const double bz = ISO ? gz[i] : gz[i] * (s.ih[2] * s.ih[2]);
          sx[p] = q ? fma(bw, gx[p], sx[p]) : bw * gx[p];
          sy[q] = p ? fma(bw, gy[q], sy[q]) : bw * gy[q];
          sz[i] = r ? fma(bw, bz, sz[i]) : bw * bz;
          // values: 1 - t[r] = t[1 - r]
          lo_iy[i] = fma(s.t[1 - r], sv, r ? lo_iy[i] : a.aiy[i]);
          b.aiy[i] = r ? fma(s.t[1], sv, b.aiy[i]) : s.t[0] * sv;
        }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (!ISO) {
          sx[q] *= s.ih[0] * s.ih[0];
          sy[q] *= s.ih[1] * s.ih[1];
        }
        lo_ex[q] = fma(s.t[1 - r], sx[q], r ? lo_ex[q] : a.aex[q]);
        lo_dy[q] = fma(s.t[1 - r], sy[q], r ? lo_dy[q] : a.ady[q]);
        b.aex[q] = r ? fma(s.t[1], sx[q], b.aex[q]) : s.t[0] * sx[q];
        b.ady[q] = r ? fma(s.t[1], sy[q], b.ady[q]) : s.t[0] * sy[q];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      lo_iy[i] -= sz[i];
      b.aiy[i] += sz[i];
    }
    // lower plane finished: back to its nodes (the transpose of load_plane)
    double f[4];
    {
      double d1 = fma(s.t[1], lo_ex[1], s.t[0] * lo_ex[0]), d0 = lo_ex[0] + lo_ex[1] - d1, i0[2], i1[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        i1[q] = fma(s.t[1], lo_iy[q + 2], fma(s.t[0], lo_iy[q], lo_dy[q]));
        i0[q] = lo_iy[q] + lo_iy[q + 2] - i1[q];
      }
      d0 = fma(s.t[1], i0[1], fma(s.t[0], i0[0], d0));
      d1 = fma(s.t[1], i1[1], fma(s.t[0], i1[0], d1));
      f[1] = d0;
      f[0] = i0[0] + i0[1] - d0;
      f[3] = d1;
      f[2] = i1[0] + i1[1] - d1;
    }
    const double X0 = f[0] + __shfl_up_sync(kFull, f[1], 1, kTX);
    double* ex_w = exch + (size_t)(li & 1) * TY * kXP + row * kXP + tx;
    *ex_w = f[2] + __shfl_up_sync(kFull, f[3], 1, kTX);
    bad = __syncthreads_or(bad);
    if (bad) return false;
    issue(li + 1 + kStages);  // into the stage every thread has just read
    if (kk >= z0 && out_node) {
      const double tot = X0 + ex_w[-kXP];
      const long long n = nidx(k.g, x, y, kk);
      const bool own = owned_plane(k.g, kk);  // a slab's ghost planes add nothing to the sums
      if (EPI == EPI_PLAIN) {
        k.out[n] = tot;
      } else if (EPI == EPI_RESIDUAL) {
        const double rv = pre_f - tot;
        k.out[n] = rv;
        const double s0 = fma(pre_f, pre_f, red0), s1 = fma(rv, rv, red1), s2 = fma(rv, rv * pre_m, red2);
        red0 = own ? s0 : red0;
        red1 = own ? s1 : red1;
        red2 = own ? s2 : red2;
      } else if (EPI == EPI_PCG) {
        k.out[n] = tot;
        const double s0 = fma(a.own, tot, red0);
        red0 = own ? s0 : red0;
      } else if (EPI == EPI_FAS) {
        k.out[n] = tot + pre_f;  // out holds the full weighting of the fine residual
      }
    }
    return true;
  };

#pragma unroll
  for (int j = 0; j < kStages; ++j) issue(j);
  history(z0 - 1);
  PfState a, b;
  if (!wait(0)) bad = 1;
  load_plane(0, a);
#pragma unroll
  for (int i = 0; i < 4; ++i) a.aiy[i] = 0.0;
  a.aex[0] = a.aex[1] = a.ady[0] = a.ady[1] = 0.0;
  bad = __syncthreads_or(bad);
  if (!bad) issue(kStages);
  for (int li = 0; !bad;) {
    if (!layer(li, a, b) || ++li == nl) break;
    if (!layer(li, b, a) || ++li == nl) break;
  }
  if constexpr (!TMA) asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (TMA && bad && tid == 0 && k.err) *k.err = 1.0;
  if (EPI == EPI_RESIDUAL || EPI == EPI_PCG) {
    double v[3] = {red0, red1, red2};
    grid_reduce<3, RED_SUM, true>(v, k.red);
  }
}

template <int EPI, bool ISO, bool TMA, int TY>
int run_pf(hpc_ctx* c, PfTileK& k, int cls) {
  using S = PfShape<TY>;
  auto kern = pf_tile_kernel<EPI, ISO, TMA, TY>;
  int per_sm = 1, rc;
  if ((rc = kernel_cfg((const void*)kern, S::bytes, S::bytes, S::NT, &per_sm))) return rc;
  const StripGeo sg = tile_geo(k.g, TY, (long long)num_sms() * per_sm, (long long)c->partials_cap / 3);
  if ((size_t)sg.nstrips * 3 > c->partials_cap) return cuda_fail(cudaErrorInvalidValue, "partials buffer");
  k.tx = sg.tx;
  k.ty = sg.ty;
  if constexpr (TMA) {
    if ((rc = encode_tensor<double>(k.g, k.x, 1, kBX, S::NY, 1, &k.xmap))) return rc;
    if ((rc = encode_tensor<double>(k.g, k.gc, 1, kBX, S::NY, 1, &k.cmap))) return rc;
  }
  const bool apart = (k.red.slot[0] >= 0 || k.red.slot[1] >= 0 || k.red.slot[2] >= 0) &&
                     combine_apart(sg, (long long)num_sms() * per_sm);
  if (apart) k.red.counter = nullptr;
  timing_begin(c, cls);
  kern<<<(unsigned)sg.nstrips, S::NT, S::bytes, c->stream>>>(k);
  if (apart) launch_combine(c, k.red, (int)sg.nstrips, S::NT);
  timing_end(c, cls);
  HPC_CHECK_LAUNCH(c);
  return HPC_OK;
}

template <int EPI, bool ISO, bool TMA>
int run_pf_h(hpc_ctx* c, PfTileK& k, int cls) {
  switch (tile_rows(k.g.ny, 16, 4)) {
    case 4: return run_pf<EPI, ISO, TMA, 4>(c, k, cls);
    case 8: return run_pf<EPI, ISO, TMA, 8>(c, k, cls);
    default: return run_pf<EPI, ISO, TMA, 16>(c, k, cls);
  }
}

template <int EPI>
int run_pf_e(hpc_ctx* c, PfTileK& k, int cls) {
  const bool iso = k.g.hx == k.g.hy && k.g.hy == k.g.hz;
  if (c->tma_stage) return iso ? run_pf_h<EPI, true, true>(c, k, cls) : run_pf_h<EPI, false, true>(c, k, cls);
  return iso ? run_pf_h<EPI, true, false>(c, k, cls) : run_pf_h<EPI, false, false>(c, k, cls);
}

}  // namespace

int launch_pf(hpc_ctx* c, const PfCall& p) {
  PfTileK k{};
  k.g = c->L[p.level];
  k.x = p.src;
  k.gc = c->F[p.level].gc;
  k.H = c->F[p.level].H;
  k.out = p.out;
  k.lc = p.lc;
  k.fd = p.fd;
  k.invM = p.invM;
  k.red = make_red(c, p.s_out0, p.s_out1, p.s_out2);
  k.err = c->err;
  switch (p.epi) {
    case EPI_PLAIN: return run_pf_e<EPI_PLAIN>(c, k, HPC_KC_NONE);
    case EPI_RESIDUAL: return run_pf_e<EPI_RESIDUAL>(c, k, HPC_KC_NONE);
    case EPI_PCG: return run_pf_e<EPI_PCG>(c, k, p.level == c->maxlevel ? HPC_KC_PF_PCG_FINEST : HPC_KC_NONE);
    case EPI_FAS: return run_pf_e<EPI_FAS>(c, k, HPC_KC_NONE);
  }
  return HPC_ERR_ARG;
}

}  // namespace hpc
