// k_trop_mixed.cu -- the barotropic subcycle of int_trop (mod_int.f90:153-296)
// for the mixed-precision path: the resident kernel of k_trop.cu (one tile
// per CTA, one region point per thread, coefficients in registers, and the
// same messages between neighbouring tiles, ub and vb packed in one word)
// with FP32 arithmetic wherever it does not decide
// the bottom pressure:
//
//   FP64: ch, the predictor ch, their 4-point means, every difference of
//         them (the bottom-pressure gradient), ter(ch) x bgraphi + graphih
//         (two large terms that nearly cancel), the ch update, and the
//         ch / mch / mch2 / ub / vb accumulators;
//   FP32: ub, vb and the volume fluxes, divergence, viscosity, Coriolis
//         adjustment, sqrt(ter(ch)), divisions (by FP32 reciprocals).
//
// The 2-D buffers it shares with the FP64 path stay FP64 in memory.
#include <cuda/atomic>

#include "pcom_dev.cuh"
#include "pcom_kernels.h"

namespace {

constexpr int kThreads = 640, kSide = kThreads / 5;  // threads; longest side of a region

enum { D_CH, D_PRED, D_COUNT };                                         // FP64 region fields
enum { F_UB, F_VB, F_S1, F_X2, F_A1U, F_A1V, F_A2U, F_A2V, F_COUNT };  // FP32 region fields
// entries before the first and after the last region field (k_trop_fast: the
// stages run without branches and may read past the region)
__host__ __device__ constexpr int pad(int W) { return W + 1; }
constexpr int kVx = 8, kVy = 19;  // FP32 metric vectors over lx and ly

// (ub, vb) as the 64-bit value of one message
__device__ __forceinline__ double pack_uv(float u, float v) {
  return __hiloint2double(__float_as_int(v), __float_as_int(u));
}
__device__ __forceinline__ void unpack_uv(double w, float &u, float &v) {
  u = __int_as_float(__double2loint(w));
  v = __int_as_float(__double2hiint(w));
}

}  // namespace

// CTX, CTY > 0: compiled for one tile shape (constant region strides);
// CTX = CTY = 0: any shape, laid out as in k_trop_fast (19 warps in rows of 32
// points for 360 x 162: 339 -> 323 us; 211 x 99: 248 -> 233)
template <int CTX = 0, int CTY = 0>
__global__ void __launch_bounds__(kThreads, 1)
    k_trop_mixed(const __grid_constant__ Dev P, int TX, int TY, int ntx, unsigned long long seq) {
  constexpr bool FREE = CTX == 0;
  if (!FREE) { TX = CTX; TY = CTY; }
  extern __shared__ double smd[];
  const int nj = P.nj, njm = P.njm, ni = P.ni, G = P.glo_ni;
  const float ra = (float)P.ra, bt = (float)P.bt, gamma_b = (float)P.c.gamma_b;
  const int nstep = P.nstep;
  const int tid = threadIdx.x;
  const int tx = blockIdx.x % ntx, ty = blockIdx.x / ntx;
  const int R0 = tx * TX, J0 = ty * TY + 1;
  const int tw = min(TX, G - R0), th = min(TY, nj - J0 + 1);
  const int rr0 = R0 - 2, jj0 = J0 - 2;
  auto ring_i = [&](int r) { r %= G; if (r < 0) r += G; return r + 2; };

  // (the layout of k_trop_fast)
  const int W = (FREE ? tw : TX) + 4, H = (FREE ? th : TY) + 4, N = W * H;
  const int RS = FREE ? kThreads : N, margin = FREE ? pad(kSide) : pad(W);
  const int XS = FREE ? 1 : W, XC = FREE ? kVx + 1 : 1, YS = FREE ? 1 : H, YR = FREE ? kVy : 1;
  double *const ds = smd + margin;
  float *const fs = reinterpret_cast<float *>(ds + D_COUNT * RS + margin + 32) + margin;
  float *vx = fs + F_COUNT * RS + margin + 32, *vy = vx + (FREE ? XC : kVx) * W;
  for (int l = tid; l < W; l += blockDim.x) {
    const int i = ring_i(rr0 + l);
    for (int g = 1; g <= 4; ++g) {
      vx[l * XC + (g - 1) * XS] = (float)ld(P.dxx1d[g], i - 1);
      vx[l * XC + (4 + g - 1) * XS] = (float)ld(P.rdxx1d[g], i - 1);
    }
  }
  for (int l = tid; l < H; l += blockDim.x) {
    const int j = min(max(jj0 + l, 1), nj);
    float *const v = vy + l * YR;
    for (int g = 1; g <= 4; ++g) {
      v[(g - 1) * YS] = (float)ld(P.dxy1d[g], j - 1);
      v[(4 + g - 1) * YS] = (float)ld(P.rdxy1d[g], j - 1);
      v[(8 + g - 1) * YS] = (float)ld(P.rh1d[g], j - 1);
    }
    v[12 * YS] = (float)ld(P.arh1d[1], j - 1);
    v[13 * YS] = (float)ld(P.rarh1d[1], j - 1);
    v[14 * YS] = (float)ld(P.arh1d[2], j - 1);
    v[15 * YS] = (float)ld(P.rarh1d[2], j - 1);
    v[16 * YS] = (float)ld(P.rrh1d[4], j - 1);
    v[17 * YS] = (float)ld(P.aarh3, j - 1);
    v[18 * YS] = (float)ld(P.raarh3, j - 1);
  }

  const int p = tid;
  const int ly = min(p / W, H - 1), lx = p - ly * W < W ? p - ly * W : 0;
  const int j = jj0 + ly;
  const bool inR = p < N;
  const bool active = inR && j >= 1 && j <= nj;
  const int i = active ? ring_i(rr0 + lx) : 2;
  const long long q = active ? I2(P, i, j) : 0;
  const bool nrow = j <= njm, srow = j >= 2;
  const bool inS2 = active && lx < tw + 3 && ly < th + 3;
  const bool inS4 = active && lx >= 1 && lx < tw + 3 && ly >= 1 && ly < th + 3;
  const bool inS6 = active && lx >= 1 && lx < tw + 2 && ly >= 1 && ly < th + 2;
  const bool inS8 = active && lx >= 2 && lx < tw + 2 && ly >= 2 && ly < th + 2;
  const bool border = inS8 && (lx < 4 || lx >= tw || ly < 4 || ly >= th);  // as in k_trop_fast
  const bool ring = active && !inS8 && lx < tw + 4 && ly < th + 4;
  const int levu = active ? __ldg(P.lev_u + q) : 0, levt = active ? __ldg(P.lev_t + q) : 0;
  const float seau = (float)(levu >= 1), mskt1 = (float)(levt >= 1);
  const float prh_u = active ? (float)ld(P.prh_u, q) : 1.f;
  const float rprh_t = active ? (float)ld(P.rprh_t, q) : 1.f;
  const float rden = active ? (float)ld(P.rwt, q) : 1.f;
  // where sqrt(ter()) is 1 (land, points that need none) or 0 (row nj)
  const bool s2sea = inS2 && levu > 0 && nrow, s2zero = levu > 0 && !nrow, s6sea = inS6 && levu > 0 && nrow;
  float sam1 = 0, bxn = 0, bxs = 0, bye = 0, byw = 0, cor = 0, ut = 0, vt = 0;
  double gxn = 0, gxs = 0, gye = 0, gyw = 0, ghx = 0, ghy = 0;
  if (inS6) {
    sam1 = seau * (float)ld(P.am, q);
    bxn = (float)ld(P.bphi[0], q); bye = (float)ld(P.bphi[2], q); byw = (float)ld(P.bphi[3], q + 1);
    gxn = ld(P.bgra[0], q); gye = ld(P.bgra[2], q); gyw = ld(P.bgra[3], q + 1);
    if (nrow) { bxs = (float)ld(P.bphi[1], q + ni); gxs = ld(P.bgra[1], q + ni); }
    ghx = ld(P.graphihx, q); ghy = ld(P.graphihy, q);
    cor = (float)ld(P.cor, q); ut = (float)ld(P.ut, q); vt = (float)ld(P.vt, q);
  }
  float vs0u = 0.f, vs0v = 0.f;
  double acc_m = 0, acc_m2 = 0, acc_u = 0, acc_v = 0;
  if (inS8) {
    acc_m = P.chc[q]; acc_m2 = acc_m;
    acc_u = P.ubc[q]; acc_v = P.vbc[q];
  }
  const double land_ch0 = inS4 ? P.chc[q] : 0.0;
  // ch, ub, vb at this thread's point, as staged for the current substep
  double c0 = 0.0;
  float u0 = 0.f, v0 = 0.f;
  if (active && (inS8 || ring)) {
    c0 = __ldcg(P.chp + q);
    if (inS2) { u0 = (float)__ldcg(P.ubp + q); v0 = (float)__ldcg(P.vbp + q); }
  }
  double *const fd = ds + p;
  float *const ff = fs + p;
#define SD(F, o) fd[(F) * RS + (o)]
#define SF(F, o) ff[(F) * RS + (o)]
  vx += lx * XC;
  vy += ly * YR;
#define RDXX(g) vx[(4 + (g) - 1) * XS]
#define RDXY(g) vy[(4 + (g) - 1) * YS]
#define RH(g) vy[(8 + (g) - 1) * YS]
  if (inR) { SD(D_CH, 0) = c0; SF(F_UB, 0) = u0; SF(F_VB, 0) = v0; }
  __syncthreads();

  // the stages of k_trop_fast, straight through for every thread.  Which
  // products fuse with a sum is written out (_rn intrinsics) wherever two
  // roundings are possible, so that the results do not depend on how the
  // stages are arranged: sums of the neighbours' quantities, the divergence,
  // the viscosity and its change are of rounded terms, the rest is fused
  for (int nt = 1; nt <= nstep; ++nt) {
    ulonglong2 *const out = P.xch + (long long)(nt & 1) * 3 * P.n2 + q;
    // S2: fluxes prh_u sqrt(ter(ch)) (ub, vb rh3); the viscosity's differences
    float s1, x2, a1u, a1v, a2u, a2v;
    {
      const double w = (c0 + SD(D_CH, W) + SD(D_CH, 1) + SD(D_CH, W + 1)) * 0.25;
      float sch = sqrtf(s2sea ? (float)w : 1.f);
      if (s2zero) sch = 0.f;
      const float ps = prh_u * sch;
      s1 = __fmul_rn(ps, u0);
      x2 = __fmul_rn(ps * v0, RH(3));
      const float rdx4 = RDXX(4), rrh4 = vy[16 * YS];
      a1u = __fmul_rn((u0 - SF(F_UB, -1)) * rdx4, rrh4);
      a1v = __fmul_rn((v0 - SF(F_VB, -1)) * rdx4, rrh4);
      const float rdy2 = RDXY(2), rh2 = RH(2);
      a2u = __fmul_rn((u0 - SF(F_UB, -W)) * rdy2, rh2);
      a2v = __fmul_rn((v0 - SF(F_VB, -W)) * rdy2, rh2);
      if (!srow) a2u = a2v = 0.f;
      if (inR) {
        SF(F_S1, 0) = s1;
        SF(F_X2, 0) = x2;
        SF(F_A1U, 0) = a1u;
        SF(F_A1V, 0) = a1v;
        SF(F_A2U, 0) = a2u;
        SF(F_A2V, 0) = a2v;
      }
    }
    __syncthreads();
    // S4: predictor ch; the viscosity
    double pred;
    float dvu, dvv;
    {
      float tEc = 0.5f * (SF(F_S1, -W) + s1), tEw = 0.5f * (SF(F_S1, -W - 1) + SF(F_S1, -1));
      const float tNc = 0.5f * (SF(F_X2, -1) + x2), tNs = 0.5f * (SF(F_X2, -W - 1) + SF(F_X2, -W));
      if (!srow) tEc = tEw = 0.f;
      const float A = __fmul_rn(tEc - tEw, RDXX(1));
      float B = __fmul_rn(tNc - tNs, RDXY(1));
      if (!srow) B = 0.f;
      const float div = __fadd_rn(A, B) * vy[13 * YS];
      pred = c0 - (double)(div * bt * gamma_b * rprh_t);
      if (levt <= 0) pred = nt == 1 ? land_ch0 : c0;
      const float rdx3 = RDXX(3), rdy3 = RDXY(3), raarh = vy[18 * YS];
      const float L1u = __fmul_rn(SF(F_A1U, 1) - a1u, rdx3), L1v = __fmul_rn(SF(F_A1V, 1) - a1v, rdx3);
      float L2u = __fmul_rn(SF(F_A2U, W) - a2u, rdy3), L2v = __fmul_rn(SF(F_A2V, W) - a2v, rdy3);
      if (!nrow) L2u = L2v = 0.f;
      const float vsu = __fmul_rn(sam1, __fadd_rn(L1u, L2u) * raarh);
      const float vsv = __fmul_rn(sam1, __fadd_rn(L1v, L2v) * raarh);
      if (nt == 1) { vs0u = vsu; vs0v = vsv; }
      dvu = __fsub_rn(vsu, vs0u);
      dvv = __fsub_rn(vsv, vs0v);
      if (inR) SD(D_PRED, 0) = pred;
    }
    __syncthreads();
    // S6: sqrt(ter(pred)), pred's gradients and means, corrector velocity
    float ubc, vbc;
    {
      const double pe = SD(D_PRED, 1), pn = SD(D_PRED, W), pne = SD(D_PRED, W + 1);
      const double w = (pred + pn + pe + pne) * 0.25;
      float sch = sqrtf(s6sea ? (float)w : 1.f);
      if (s2zero) sch = 0.f;
      const float rdx2 = RDXX(2), rdy4 = RDXY(4);
      const float gx0 = (float)(pe - pred) * rdx2 * vy[15 * YS], gx1 = (float)(pne - pn) * rdx2 * vy[15 * YS + YR];
      const float gy0 = (float)(pn - pred) * rdy4 * ra, gy1 = (float)(pne - pe) * rdy4 * ra;
      const double ce0 = 0.5 * (pred + pe), ce1 = 0.5 * (pn + pne), cn0 = 0.5 * (pred + pn), cn1 = 0.5 * (pe + pne);
      float gi1 = 0.5f * __fmaf_rn(gx0, bxn, __fmul_rn(gx1, bxs)), gi2 = 0.5f * __fmaf_rn(gy0, bye, __fmul_rn(gy1, byw));
      double cg1 = 0.5 * __fma_rn(ce0, gxn, __dmul_rn(ce1, gxs)), cg2 = 0.5 * __fma_rn(cn0, gye, __dmul_rn(cn1, gyw));
      if (!nrow) { gi1 = gi2 = 0.f; cg1 = cg2 = 0.0; }
      const float f1 = (float)((double)gi1 + cg1 + ghx) * seau, f2 = (float)((double)gi2 + cg2 + ghy) * seau;  // pg / sch
      const float hc = 0.5f * cor, cb = hc * bt;
      float p1 = seau * __fmaf_rn(hc, v0, __fmaf_rn(-f1, sch, dvu + ut));
      float p2 = seau * __fmaf_rn(-hc, u0, __fmaf_rn(-f2, sch, dvv + vt));
      const float w1 = __fmaf_rn(p1, bt, u0), w2 = __fmaf_rn(p2, bt, v0);
      const float u1 = 0.5f * __fmaf_rn(__fmaf_rn(cb, w2, w1), rden, u0);
      const float v1 = 0.5f * __fmaf_rn(__fmaf_rn(-cb, w1, w2), rden, v0);
      p1 = seau * __fmaf_rn(cor, v1, __fmaf_rn(-f1, sch, dvu) + ut);
      p2 = seau * __fmaf_rn(-cor, u1, __fmaf_rn(-f2, sch, dvv) + vt);
      ubc = __fmaf_rn(p1, bt, u0);
      vbc = __fmaf_rn(p2, bt, v0);
      if (border && nt < nstep) xch_put(out + P.n2, pack_uv(ubc, vbc), seq + nt);
      const float ps = prh_u * sch;
      s1 = __fmul_rn(ps, ubc);
      x2 = __fmul_rn(ps * vbc, RH(3));
      if (inR) {
        SF(F_S1, 0) = s1;
        SF(F_X2, 0) = x2;
      }
    }
    __syncthreads();
    // S8: corrector ch, send, accumulate
    if (inS8) {
      float tEc = 0.5f * (SF(F_S1, -W) + s1), tEw = 0.5f * (SF(F_S1, -W - 1) + SF(F_S1, -1));
      const float tNc = 0.5f * (SF(F_X2, -1) + x2), tNs = 0.5f * (SF(F_X2, -W - 1) + SF(F_X2, -W));
      if (!srow) tEc = tEw = 0.f;
      const float A = __fmul_rn(tEc - tEw, RDXX(1));
      float B = __fmul_rn(tNc - tNs, RDXY(1));
      if (!srow) B = 0.f;
      const float div = __fadd_rn(A, B) * vy[13 * YS];
      c0 = c0 - (double)(mskt1 * div * bt * rprh_t);
      if (border && nt < nstep) xch_put(out, c0, seq + nt);
      u0 = ubc; v0 = vbc;
      SD(D_CH, 0) = c0;
      SF(F_UB, 0) = u0;
      SF(F_VB, 0) = v0;
      if (nt <= nstep / 2) acc_m = acc_m + c0;
      acc_m2 = acc_m2 + c0;
      acc_u = acc_u + (double)ubc;
      acc_v = acc_v + (double)vbc;
    }
    if (nt == nstep) break;
    // the ring's state of this substep from the tiles around, as in k_trop_fast
    __syncwarp();
    int fail = 0;
    if (ring) {
      const ulonglong2 *const in[2] = {out, inS2 ? out + P.n2 : out};
      double v[2] = {0.0, 0.0};
      fail = !xch_wait(in, seq + nt, v, P.err, P.wait_ns, P.err_step);
      c0 = v[0];
      unpack_uv(v[1], u0, v0);
      SD(D_CH, 0) = c0;
      SF(F_UB, 0) = u0;
      SF(F_VB, 0) = v0;
    }
    if (__syncthreads_or(fail)) return;
  }
#undef SD
#undef SF
#undef RDXX
#undef RDXY
#undef RH
  if (inS8) {
    const double ub = acc_u / (nstep + 1), vb = acc_v / (nstep + 1);
    const double mch = acc_m / (nstep / 2 + 1), mch2 = acc_m2 / (nstep + 1);
    st2(P.ubc, P, i, q, ub);
    st2(P.vbc, P, i, q, vb);
    st2(P.ubp, P, i, q, ub);
    st2(P.vbp, P, i, q, vb);
    st2(P.mch, P, i, q, mch);
    st2(P.mch2, P, i, q, mch2);
    st2(P.chc, P, i, q, mch2);
    st2(P.chp, P, i, q, mch2);
    st2(P.acch, P, i, q, P.acch[q] + mch2);
  }
}

namespace {
// the fixed-shape form for a tile shape where one is compiled, the general
// one otherwise
const void *mixed_kernel(int TX, int TY) {
#define PCOM_MIXED_SHAPE(x, y) \
  if (TX == (x) && TY == (y)) return (const void *)k_trop_mixed<(x), (y)>;
  PCOM_TROP_SMALL(PCOM_MIXED_SHAPE)
#undef PCOM_MIXED_SHAPE
  return (const void *)k_trop_mixed<>;
}
}  // namespace

size_t trop_mixed_smem_bytes(int TX, int TY) {
  bool free = true;
#define PCOM_MIXED_SHAPE(x, y) \
  if (TX == (x) && TY == (y)) free = false;
  PCOM_TROP_SMALL(PCOM_MIXED_SHAPE)
#undef PCOM_MIXED_SHAPE
  const int W = TX + 4, H = TY + 4;
  const size_t rs = free ? kThreads : (size_t)W * H, margin = 2 * (size_t)pad(free ? kSide : W) + 32;
  return (D_COUNT * rs + margin) * sizeof(double) +
         (F_COUNT * rs + margin + (kVx + free) * W + kVy * (H + 1)) * sizeof(float);
}

int trop_mixed_max_blocks(int TX, int TY) {
  int dev = 0, nsm = 0, per = 0;
  if ((TX + 4) * (TY + 4) > kThreads) return 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = trop_mixed_smem_bytes(TX, TY);
  const void *fn = mixed_kernel(TX, TY);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  const int nthreads = ((TX + 4) * (TY + 4) + 31) / 32 * 32;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, nthreads, smem) != cudaSuccess) return 0;
  return per * nsm;
}

cudaError_t launch_trop_mixed(const Dev &P, int TX, int TY, unsigned long long seq, cudaStream_t s) {
  const int ntx = (P.glo_ni + TX - 1) / TX, nty = (P.nj + TY - 1) / TY;
  const size_t smem = trop_mixed_smem_bytes(TX, TY);
  const void *fn = mixed_kernel(TX, TY);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int nthreads = ((TX + 4) * (TY + 4) + 31) / 32 * 32;
  void *args[] = {(void *)&P, (void *)&TX, (void *)&TY, (void *)&ntx, (void *)&seq};
  return cudaLaunchCooperativeKernel(fn, dim3(ntx * nty), dim3(nthreads), args, smem, s);
}
