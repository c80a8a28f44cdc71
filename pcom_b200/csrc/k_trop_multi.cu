// k_trop_multi.cu -- the barotropic subcycle of int_trop (mod_int.f90:153-296)
// of one FP64 domain with more tiles than SMs: a persistent cooperative
// launch, one CTA per SM, that walks its share of the tiles in every substep
// and meets the others at a grid barrier between substeps.
//
// Per tile the four stages of trop_stages.cuh run on the tile's region, one
// point per thread.  A point's coefficients do not stay on the chip from one
// substep to the next (about 220 bytes per point), so what bounds this kernel
// is their way to the SM: read where a stage needs them, every stage waited
// for L2 or HBM (13.4 ms for the 1440 x 640 domain's 120 substeps).  Instead
//  - k_ms_prep packs them once per step into planes of 16-byte pairs, with
//    the reference's neighbour shifts and the stages' factors applied, on a
//    grid of its own with two wrapped columns at each end, so that any tile's
//    region is a box;
//  - one thread brings the next tile's box of all planes and of the state
//    (the masks travel with ch) with two tensor loads while the current tile
//    is computed; the threads take their point's values into registers at the
//    start of a tile, which frees the box for the next one.  (cp.async by
//    every thread for its own point: 9.0 ms; its issue alone took 2,600-3,700
//    cycles of a tile's 7,500);
//  - the tiles are walked forwards and backwards in turn, so that a substep
//    starts with what the last one left in L2;
//  - tiles without sea are not walked: land keeps its state, so only their
//    sums are formed, once at the end.  int_trop of a 720 x 320 globe with
//    28 % of such tiles: 2.12 -> 1.77 ms, of 611 x 253: 1.69 -> 1.37 ms; a
//    domain with none pays nothing.
// Floor of a 1440 x 640 substep: 270 MB from HBM or L2 (40 us at 6.5 TB/s) and
// ~38 us of stages; measured 61 (7.28 ms for the 120).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cuda/atomic>

#include "pcom_dev.cuh"
#include "pcom_kernels.h"
#include "trop_stages.cuh"

namespace {

// planes of coefficient pairs; the last is the first substep's viscosity
enum { M_PRH, M_RPRH, M_SAM, M_UT, M_BX, M_BY, M_GX, M_GY, M_GH, M_VS0, M_COUNT };
// the state's planes: (ub, vb) and (ch, masks: 1 lev_u >= 1, 2 lev_t >= 1)
enum { M_UV, M_CH, M_STATE };

PD unsigned saddr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
PD void mb_init(unsigned m, unsigned n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(m), "r"(n)); }
PD void mb_expect(unsigned m, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(m), "r"(bytes) : "memory");
}
// bounded wait for a phase: ~seconds at most (a load that never lands)
PD bool mb_wait(unsigned m, unsigned parity) {
  for (int it = 0; it < (1 << 22); ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(m), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
PD void box_load(unsigned dst, const CUtensorMap *map, int x, int y, unsigned m) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(0), "r"(m)
      : "memory");
}
PD void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned m) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(m)
               : "memory");
}
// orders generic-proxy accesses to global memory and the tensor loads' (async
// proxy) of the same locations
PD void fence_proxy() { asm volatile("fence.proxy.async;" ::: "memory"); }

// packs the step's coefficients, the state the first substep starts from, the
// accumulators, and every tile row's and column's metric vectors
__global__ void k_ms_prep(const __grid_constant__ Dev P, MultiTrop M, int TX, int TY, int ntx, int nty) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;  // column of the packed grid
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int G = P.glo_ni, nj = P.nj, W = TX + 4, H = TY + 4;
  auto ring_i = [&](int r) { r %= G; if (r < 0) r += G; return r + 2; };
  const int nx = gridDim.x * blockDim.x, all = nx * gridDim.y * blockDim.y;
  const int t = (blockIdx.y * blockDim.y + threadIdx.y) * nx + x;
  for (int v = t; v < ntx * kXVecs * W; v += all) {
    const int l = v % W, n = v / W % kXVecs, tx = v / (W * kXVecs);
    M.xm[v] = trop_xvec(P, n, ring_i(tx * TX - 2 + l));
  }
  for (int v = t; v < nty * kYVecs * H; v += all) {
    const int l = v % H, n = v / H % kYVecs, ty = v / (H * kYVecs);
    M.ym[v] = trop_yvec(P, n, min(max(ty * TY - 1 + l, 1), nj));
  }
  if (x >= M.pitch || j > nj) return;
  const long long q = I2(P, ring_i(x - 2), j), pq = x + (long long)M.pitch * (j - 1), pn = (long long)M.pitch * nj;
  const bool nrow = j <= P.njm;
  const int lu = P.lev_u[q], lt = P.lev_t[q];
  auto put = [&](int f, double a, double b) { M.cf[f * pn + pq] = make_double2(a, b); };
  put(M_PRH, 0.5 * P.prh_u[q], P.prh_t[q]);
  put(M_RPRH, P.rprh_t[q], P.rwt[q]);
  put(M_SAM, (double)(lu >= 1) * P.am[q], P.cor[q]);
  put(M_UT, P.ut[q], P.vt[q]);
  put(M_BX, P.bphi[0][q], nrow ? P.bphi[1][q + P.ni] : 0.0);
  put(M_BY, P.bphi[2][q], P.bphi[3][q + 1]);
  put(M_GX, 0.5 * P.bgra[0][q], nrow ? 0.5 * P.bgra[1][q + P.ni] : 0.0);
  put(M_GY, 0.5 * P.bgra[2][q], 0.5 * P.bgra[3][q + 1]);
  put(M_GH, 2.0 * P.graphihx[q], 2.0 * P.graphihy[q]);
  const double2 uv = make_double2(P.ubp[q], P.vbp[q]);
  const double2 ch = make_double2(P.chp[q], (double)((lu >= 1) + 2 * (lt >= 1)));
  M.st[0][M_UV * pn + pq] = uv;
  M.st[0][M_CH * pn + pq] = ch;
  if (lu < 1 && lt < 1) {
    // land keeps its state (its viscosity is sam1 = 0 times a difference);
    // tiles without sea, which the substeps skip, are read as neighbours
    M.st[1][M_UV * pn + pq] = uv;
    M.st[1][M_CH * pn + pq] = ch;
    put(M_VS0, 0.0, 0.0);
  }
  if (x >= 2 && x < G + 2) {
    P.tr_acc[1][q] = P.chc[q];
    M.acc[q] = make_double2(P.ubc[q], P.vbc[q]);
  }
}

template <int TX, int TY>
__host__ __device__ constexpr int ms_threads() { return ((TX + 4) * (TY + 4) + 31) / 32 * 32; }
// shared memory: the boxes (128-byte aligned), the region's fields, two sets
// of metric vectors
template <int TX, int TY>
__host__ __device__ constexpr int ms_boxes() { return ((M_COUNT + M_STATE) * (TX + 4) * (TY + 4) * 16 + 127) / 128 * 128; }
template <int TX, int TY>
__host__ __device__ constexpr int ms_fields() { return (X_COUNT * (TX + 4) * (TY + 4) + 2 * x_pad(TX + 4) + 32 + 15) / 16 * 16; }
template <int TX, int TY>
__host__ __device__ constexpr int ms_vecs() { return (kXVecs * (TX + 4) + kYVecs * (TY + 4) + 15) / 16 * 16; }
template <int TX, int TY>
__host__ __device__ constexpr int ms_smem() {
  return 128 + ms_boxes<TX, TY>() + (ms_fields<TX, TY>() + 2 * ms_vecs<TX, TY>()) * 8;
}

}  // namespace

template <int TX, int TY>
__global__ void __launch_bounds__((ms_threads<TX, TY>()), 1)
    k_trop_multi(const __grid_constant__ Dev P, const __grid_constant__ MultiTrop M, int ntx, int ntiles,
                 int nwet, unsigned long long *cnt, const __grid_constant__ CUtensorMap cmap,
                 const __grid_constant__ CUtensorMap smap0, const __grid_constant__ CUtensorMap smap1) {
  constexpr int W = TX + 4, H = TY + 4, RS = W * H, NV = ms_vecs<TX, TY>();
  static_assert(RS % 4 == 0, "the state's box starts on 128 bytes");
  static_assert((kXVecs * W * 8) % 16 == 0 && (kYVecs * H * 8) % 16 == 0, "bulk copies of whole 16 bytes");
  extern __shared__ __align__(128) unsigned char raw[];
  __shared__ __align__(8) unsigned long long mbar[2];  // coefficients and metrics; state
  __shared__ int s_stop;
  unsigned char *const base = raw + ((128 - (saddr(raw) & 127)) & 127);
  const double2 *const cbox = reinterpret_cast<const double2 *>(base);
  const double2 *const sbox = cbox + M_COUNT * RS;
  double *const fields = reinterpret_cast<double *>(base + ms_boxes<TX, TY>());
  double *const fs = fields + x_pad(W), *const vec = fields + ms_fields<TX, TY>();
  const int tid = threadIdx.x, nj = P.nj, G = P.glo_ni, nstep = P.nstep;
  const long long pn = (long long)M.pitch * nj;
  const double a = P.c.a, ra = P.ra, bt = (double)P.bt, gamma_b = P.c.gamma_b;
  const int p = tid;
  const int ly = min(p / W, H - 1), lx = p - ly * W < W ? p - ly * W : 0;
  const bool inR = p < RS;
  const int pr = inR ? p : 0;  // this thread's point in the boxes
  const unsigned mc = saddr(&mbar[0]), ms = saddr(&mbar[1]);
  if (tid == 0) {
    mb_init(mc, 1);
    mb_init(ms, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // (one thread) a tile's coefficients and metric vectors (into set b), and its state
  auto fetch_c = [&](int tx, int ty, int b) {
    mb_expect(mc, (unsigned)((M_COUNT * RS * 2 + kXVecs * W + kYVecs * H) * 8));
    box_load(saddr(cbox), &cmap, 2 * tx * TX, ty * TY - 2, mc);
    bulk_load(saddr(vec + b * NV), M.xm + (long long)tx * kXVecs * W, kXVecs * W * 8, mc);
    bulk_load(saddr(vec + b * NV + kXVecs * W), M.ym + (long long)ty * kYVecs * H, kYVecs * H * 8, mc);
  };
  auto fetch_s = [&](int tx, int ty, int d) {
    mb_expect(ms, (unsigned)(M_STATE * RS * 16));
    box_load(saddr(sbox), d ? &smap1 : &smap0, 2 * tx * TX, ty * TY - 2, ms);
  };
  // tiles with sea of this CTA (all of them have one, unless there is none)
  const int mine = (nwet - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  unsigned ph = 0;  // parity of both barriers' current phase
  int b = 0;
  int next = M.tiles[blockIdx.x], tx = next % ntx, ty = next / ntx;
  if (tid == 0 && mine > 0) {
    fetch_c(tx, ty, 0);
    fetch_s(tx, ty, 0);
  }
  // averages of a point (mod_int.f90:276-288) from the sums with ch's first
  // half (am1)
  auto finish = [&](int i, long long q, double am1, double am2, double2 auv) {
    const double ub = auv.x / (nstep + 1), vb = auv.y / (nstep + 1);
    const double mch = am1 / (nstep / 2 + 1), mch2 = am2 / (nstep + 1);
    st2(P.ubc, P, i, q, ub);
    st2(P.vbc, P, i, q, vb);
    st2(P.ubp, P, i, q, ub);
    st2(P.vbp, P, i, q, vb);
    st2(P.mch, P, i, q, mch);
    st2(P.mch2, P, i, q, mch2);
    st2(P.chc, P, i, q, mch2);
    st2(P.chp, P, i, q, mch2);
    st2(P.acch, P, i, q, P.acch[q] + mch2);
  };
  bool ok = true, through = mine == 0;
  for (int nt = 1; nt <= nstep && mine > 0; ++nt) {
    const int d = nt & 1;
    for (int m = 0; m < mine; ++m, b ^= 1, ph ^= 1) {
      const int r0 = tx * TX, j0 = ty * TY + 1;
      const int tw = min(TX, G - r0), th = min(TY, nj - j0 + 1);
      const int j = j0 - 2 + ly;
      const bool active = inR && j >= 1 && j <= nj && lx < tw + 4 && ly < th + 4;
      const bool nrow = j <= P.njm;
      const bool inS2 = active && lx < tw + 3 && ly < th + 3;
      const bool inS6 = active && lx >= 1 && lx < tw + 2 && ly >= 1 && ly < th + 2;
      const bool inS8 = active && lx >= 2 && lx < tw + 2 && ly >= 2 && ly < th + 2;
      // (an interior column's ring index is r0 - 2 + lx, so its i is r0 + lx)
      const long long q = inS8 ? I2(P, r0 + lx, j) : 0;
      // the tile after this one; past the last, the next substep's first.
      // Substeps walk the CTA's tiles 0, 1, .. and .., 1, 0 in turn
      const bool more = m + 1 < mine;
      next = M.tiles[(int)blockIdx.x + (more ? (d ? m + 1 : mine - 2 - m) : (d ? mine - 1 : 0)) * (int)gridDim.x];
      ok = mb_wait(mc, ph) && mb_wait(ms, ph);
      TropCoef K;
      double2 w;
      w = cbox[M_PRH * RS + pr]; K.prh_uh = w.x; K.prh_t = w.y;
      w = cbox[M_RPRH * RS + pr]; K.rprh_t = w.x; K.rden = w.y;
      w = cbox[M_SAM * RS + pr]; K.sam1 = w.x; K.cor = w.y;
      w = cbox[M_UT * RS + pr]; K.ut = w.x; K.vt = w.y;
      w = cbox[M_BX * RS + pr]; K.bxn = w.x; K.bxs = w.y;
      w = cbox[M_BY * RS + pr]; K.bye = w.x; K.byw = w.y;
      w = cbox[M_GX * RS + pr]; K.gxn = w.x; K.gxs = w.y;
      w = cbox[M_GY * RS + pr]; K.gye = w.x; K.gyw = w.y;
      w = cbox[M_GH * RS + pr]; K.ghx = w.x; K.ghy = w.y;
      w = cbox[M_VS0 * RS + pr];
      double vs0u = w.x, vs0v = w.y;
      TropState s{};
      w = sbox[M_UV * RS + pr]; s.u0 = w.x; s.v0 = w.y;
      w = sbox[M_CH * RS + pr]; s.c0 = w.x;
      const double flag = w.y;
      const int fl = active ? (int)flag : 0;
      K.sea_u = fl & 1;
      K.sea_t = fl & 2;
      const TropPoint<false> T{fs + p, vec + b * NV + lx, vec + b * NV + kXVecs * W + ly, W, RS, W, H, 1, inR, nrow, j >= 2,
                               inS2 && K.sea_u && nrow, inS6 && K.sea_u && nrow, K.sea_u && !nrow};
      if (inR) { T.S(X_CH, 0) = s.c0; T.S(X_UB, 0) = s.u0; T.S(X_VB, 0) = s.v0; }
      if (__syncthreads_or(!ok)) {
        ok = false;
        break;
      }
      // the next tile's loads, in flight behind this tile's stages; of the
      // next substep's first tile all but what other CTAs still write (its
      // state, and the viscosity that the first substep sets)
      if (more || nt < nstep) {
        tx = next % ntx;
        ty = next / ntx;
        if (tid == 0) {
          if (more || nt > 1) fetch_c(tx, ty, b ^ 1);
          if (more) fetch_s(tx, ty, 1 - d);
        }
      }
      double am2 = 0.0;
      double2 auv = make_double2(0.0, 0.0);
      double land = s.c0;
      if (nt == 1 && active) {
        int r = (r0 - 2 + lx) % G;
        if (r < 0) r += G;
        land = P.chc[I2(P, r + 2, j)];
      }
      if (inS8) {
        am2 = P.tr_acc[1][q];
        auv = M.acc[q];
      }
      trop_s2(T, K, s);
      __syncthreads();
      trop_s4(T, K, s, bt, gamma_b, land, nt == 1, vs0u, vs0v);
      __syncthreads();
      trop_s6(T, K, s, bt, a, ra);
      __syncthreads();
      if (inS8) {
        const int i = r0 + lx;
        const double chn = trop_s8(T, K, s, bt);
        am2 = am2 + chn;
        auv.x = auv.x + s.ubc;
        auv.y = auv.y + s.vbc;
        // (mch and mch2 have the same terms up to half the substeps)
        if (nt == nstep / 2) P.tr_acc[0][q] = am2;
        if (nt < nstep) {
          // the packed grid's column is i; its two wrapped columns at each end
          const long long pq = i + (long long)M.pitch * (j - 1);
          auto put = [&](long long o) {
            M.st[d][M_UV * pn + o] = make_double2(s.ubc, s.vbc);
            M.st[d][M_CH * pn + o] = make_double2(chn, flag);
            if (nt == 1) M.cf[M_VS0 * pn + o] = make_double2(vs0u, vs0v);
          };
          put(pq);
          if (i < 4) put(pq + G);
          if (i >= G) put(pq - G);
          P.tr_acc[1][q] = am2;
          M.acc[q] = auv;
        } else {
          finish(i, q, P.tr_acc[0][q], am2, auv);
        }
      }
    }
    if (nt == nstep) through = ok;
    if (!ok || nt == nstep) break;
    // grid barrier: release-ordered arrival, bounded acquire wait, outcome
    // through shared memory; the state crosses from this CTA's stores to the
    // other CTAs' tensor loads
    fence_proxy();
    __syncthreads();
    if (tid == 0) {
      cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> c(*cnt);
      c.fetch_add(1ULL, cuda::memory_order_release);
      s_stop = wait_count(cnt, (unsigned long long)nt * gridDim.x, P.err, P.wait_ns, P.err_step) ? 0 : 1;
      if (!s_stop) {
        fence_proxy();
        if (nt == 1) fetch_c(tx, ty, b);
        fetch_s(tx, ty, d);
      }
    }
    __syncthreads();
    if (s_stop) {
      // the coefficients fetched ahead have landed before the CTA exits
      if (nt > 1) mb_wait(mc, ph);
      break;
    }
  }
  // tiles without sea: their state is the same after every substep; only the
  // sums are formed (their neighbours read them last behind the barriers)
  for (int n = nwet + (int)blockIdx.x; through && n < ntiles; n += (int)gridDim.x) {
    const int r0 = M.tiles[n] % ntx * TX, j0 = M.tiles[n] / ntx * TY + 1;
    const int tw = min(TX, G - r0), th = min(TY, nj - j0 + 1);
    if (tid >= tw * th) continue;
    const int i = r0 + 2 + tid % tw;
    const long long q = I2(P, i, j0 + tid / tw);
    const double c = P.chp[q], u = P.ubp[q], v = P.vbp[q];
    double am1 = 0.0, am2 = P.chc[q];
    double2 auv = make_double2(P.ubc[q], P.vbc[q]);
    for (int nt = 1; nt <= nstep; ++nt) {
      am2 = am2 + c;
      auv.x = auv.x + u;
      auv.y = auv.y + v;
      if (nt == nstep / 2) am1 = am2;
    }
    finish(i, q, am1, am2, auv);
  }
  if (!ok && tid == 0) give_up(P.err, P.err_step);
}

namespace {
struct MultiForm {
  const void *fn;
  int smem, nth;
};
MultiForm multi_form(int TX, int TY) {
#define PCOM_MULTI_SHAPE(x, y) \
  if (TX == (x) && TY == (y)) return {(const void *)k_trop_multi<(x), (y)>, ms_smem<(x), (y)>(), ms_threads<(x), (y)>()};
  PCOM_MULTI_SHAPES(PCOM_MULTI_SHAPE)
#undef PCOM_MULTI_SHAPE
  return {nullptr, 0, 0};
}

// cuTensorMapEncodeTiled through the runtime's driver entry-point table (the
// library links no libcuda)
PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)f;
  }();
  return fn;
}
// planes of pitch x nj pairs of doubles; box: W x H pairs of every plane
bool pair_map(CUtensorMap *tm, const double2 *p, int pitch, int nj, int planes, int W, int H) {
  auto enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)pitch * 2, (cuuint64_t)nj, (cuuint64_t)planes};
  const cuuint64_t strides[2] = {(cuuint64_t)pitch * 16, (cuuint64_t)pitch * 16 * nj};
  const cuuint32_t box[3] = {(cuuint32_t)(2 * W), (cuuint32_t)H, (cuuint32_t)planes};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double2 *>(p), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
size_t xm_doubles(int glo_ni, int TX) { return (size_t)((glo_ni + TX - 1) / TX) * kXVecs * (TX + 4); }
size_t ym_doubles(int nj, int TY) { return (size_t)((nj + TY - 1) / TY) * kYVecs * (TY + 4); }
}  // namespace

size_t trop_multi_state_bytes(int glo_ni, int nj) {
  const size_t pn = (size_t)(glo_ni + 4) * nj, n2 = (size_t)(glo_ni + 2) * nj;
  return (2 * M_STATE * pn + n2) * sizeof(double2);
}

size_t trop_multi_scratch_bytes(int glo_ni, int nj) {
  const size_t pn = (size_t)(glo_ni + 4) * nj;
  size_t by_shape = 0;  // metric vectors and tile list
#define PCOM_MULTI_SHAPE(x, y)                                                                                   \
  by_shape = std::max(by_shape, (xm_doubles(glo_ni, (x)) + ym_doubles(nj, (y))) * sizeof(double) +               \
                                    (size_t)((glo_ni + (x) - 1) / (x)) * ((nj + (y) - 1) / (y)) * sizeof(int));
  PCOM_MULTI_SHAPES(PCOM_MULTI_SHAPE)
#undef PCOM_MULTI_SHAPE
  return M_COUNT * pn * sizeof(double2) + by_shape;
}

void trop_multi_bind(MultiTrop &M, void *state, void *scratch, int glo_ni, int nj, int TX, int TY) {
  const size_t pn = (size_t)(glo_ni + 4) * nj;
  M.pitch = glo_ni + 4;
  M.st[0] = (double2 *)state;  // every part starts on 16 bytes
  M.st[1] = M.st[0] + M_STATE * pn;
  M.acc = M.st[1] + M_STATE * pn;
  M.cf = (double2 *)scratch;
  M.xm = (double *)(M.cf + M_COUNT * pn);
  M.ym = M.xm + xm_doubles(glo_ni, TX);
  M.tiles = (int *)(M.ym + ym_doubles(nj, TY));
}

int trop_multi_max_blocks(int TX, int TY) {
  int dev = 0, nsm = 0, per = 0;
  const MultiForm f = multi_form(TX, TY);
  if (!f.fn) return 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaFuncSetAttribute(f.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, f.smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f.fn, f.nth, f.smem) != cudaSuccess) return 0;
  return per * nsm;
}

cudaError_t launch_trop_multi(const Dev &P, const MultiTrop &M, int TX, int TY, int nblocks, unsigned long long *cnt,
                              cudaStream_t s) {
  const MultiForm f = multi_form(TX, TY);
  if (!f.fn) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(f.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, f.smem);
  if (e != cudaSuccess) return e;
  int ntx = (P.glo_ni + TX - 1) / TX;
  const int nty = (P.nj + TY - 1) / TY;
  int ntiles = ntx * nty, nwet = M.nwet;
  k_ms_prep<<<dim3((M.pitch + 31) / 32, (P.nj + 7) / 8), dim3(32, 8), 0, s>>>(P, M, TX, TY, ntx, nty);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  CUtensorMap cm, s0, s1;
  if (!pair_map(&cm, M.cf, M.pitch, P.nj, M_COUNT, TX + 4, TY + 4) ||
      !pair_map(&s0, M.st[0], M.pitch, P.nj, M_STATE, TX + 4, TY + 4) ||
      !pair_map(&s1, M.st[1], M.pitch, P.nj, M_STATE, TX + 4, TY + 4))
    return cudaErrorInvalidValue;
  // the barrier counter starts from zero in every launch
  e = cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  void *args[] = {(void *)&P, (void *)&M, (void *)&ntx, (void *)&ntiles, (void *)&nwet, (void *)&cnt, (void *)&cm, (void *)&s0, (void *)&s1};
  return cudaLaunchCooperativeKernel(f.fn, dim3(nblocks), dim3(f.nth), args, f.smem, s);
}
