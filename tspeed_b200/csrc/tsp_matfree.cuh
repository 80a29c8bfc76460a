// Matrix-free leap-frog step (FP64) on the FP64 tensor cores (internal header
// of tspeed_b200).
//
// The action of B on u^k is computed from the factorised reference-element
// tables and per-element geometry and materials instead of stored blocks. Same
// terms as the assembled operator (Matrices_imp.hpp:22-215 with I <- I + I^T
// and B = pen N^2 S + I + A), evaluated at quadrature points:
//   volume   y^m += |detJ| sum_ab K^{ab} (sum_n alpha^{mn}_ab x^n)
//   face l   with J^n(k) = u_e^n(k) - u_nb^n(Q-1-k) (jump at edge point k),
//            T_e^m(k) = L/2 sum_{n,a} beta^{nm}_a(e) g_e^n_a(k) (half the
//            face's traction of u_e), T_nb^m the neighbour's own:
//     y^m_i += sum_k w_k b_i(k) [pen N^2 sum_n c_mn J^n - (T_e^m - T_nb^m)]
//            + sum_k w_k sum_a g^a_i(k) [-L/2 sum_n beta^{mn}_a(e) J^n]
//
// Every product is one reference table times a matrix whose columns are
// elements, so a warp advances a tile of eight elements with mma.sync
// m8n8k4.f64 (exact FP64 products, FP64 accumulation): the table fragment is
// the A operand, stored in fragment order in shared memory, and the tile's two
// displacement components are two B operands that share it. Measured, us per
// step with one warp per element on the CUDA cores (neighbours' traces
// recomputed, tables read element by element) / now: 160,000 triangles N = 6
// 1146 / 249; 40,000 triangles N = 4 153 / 32, N = 8 579 / 169; 6,734 triangles
// N = 3 24.9 / 7.5. Bound: the FP64 tensor rate (478 MMAs per tile at N = 6:
// 132 us for 160,000 triangles; the pipe is busy half of the time) and the
// latency of a tile's loads, of which
// two rounds are left: what a tile starts with (face records, neighbours,
// inverse masses) is copied to shared memory a tile ahead (N = 6 262 without),
// every edge value is requested at once. Twelve warps per SM: sixteen spill at
// N = 6 (285 us); coefficients requested a tile ahead, or edge values in flight
// during the volume term, spill too (272 to 318 us).
//
// The face values are the step's only coupling between elements: every
// element keeps u and T at its 3Q edge points (four values each) beside its
// coefficients. The step reads its own and its neighbours' values of u^k and
// writes those of u^{k+1} from the coefficients it has just computed, so no
// trace is computed twice; k_matfree_traces computes them from coefficients
// where a run starts, resumes, or a single product is asked for.
//
// Fragments (lane = 4 g + t): A[row g][k t], B[k t][column g], C[row g][columns
// 2t, 2t + 1]. B operands that other lanes produce pass through shared memory
// as rows of eight elements, row k's halves exchanged where k & 2, which keeps
// both the fragment loads and the C-order stores free of bank conflicts.
#pragma once

#include <stdint.h>

#include "tsp_kernels.cuh"
#include "tsp_tcgen05.cuh"

namespace tsp {

struct MatFreeParams {
  const double* tables;  // fragment-ordered volume, lift and trace tables (MFCfg)
  const double* alpha;   // [ne][10] |detJ| alpha: (00: 00 01 11) (11: 00 01 11) (01: 00 01 10 11)
  // [ne][3][12]: pen N^2 (c00, c01, c11), 4 * neighbour + its face (a whole
  // number's bits, -1 on the boundary), L/2 beta^{mn}_a [m][n][a]
  const double* face;
  const double* din;     // [ne][3Q][4] u^0, u^1, T^0, T^1 of u^k at the edge points
  double* dout;          // the same of u^{k+1}; null: not wanted
};

template <int N>
struct MFCfg {
  static constexpr int NP = (N + 1) * (N + 2) / 2;
  static constexpr int Q = N + 1;
  static constexpr int R = 2 * NP;
  static constexpr int KS = (NP + 3) / 4;       // k steps over the modes
  static constexpr int MT = (NP + 7) / 8;       // row tiles of the modes
  static constexpr int RQ = 3 * Q;              // edge points of an element
  static constexpr int TT = (RQ + 7) / 8;       // row tiles of the edge points
  static constexpr int KL = (3 * RQ + 3) / 4;   // k steps of the lift: F, H_0, H_1 at the edge points
  // Tables in fragment order, one double per lane: volume [ab][MT][KS],
  // lift [MT][KL], traces [value, d/d0, d/d1][TT][KS].
  static constexpr int VOL = 4 * MT * KS * 32;
  static constexpr int LIFT = MT * KL * 32;
  static constexpr int TRC = 3 * TT * KS * 32;
  static constexpr int TABLES = VOL + LIFT + TRC;
  // Per warp: rows of eight elements (fluxes, then u^{k+1}), face records.
  static constexpr int ROWS = 4 * KL > 8 * MT ? 4 * KL : 8 * MT;
  static constexpr int FP = 38;                 // pitch of an element's face records; its inverse mass at 36
  static constexpr int warps(int fb) {
    const int n = (227 * 1024 / 8 - TABLES) / (2 * ROWS * 8 + fb * 8 * FP + 1);
    return N <= 4 ? 8 : n > 12 ? 12 : n;
  }
  // The next tile's records are requested a tile ahead where a second buffer
  // costs no warp.
  static constexpr int FB = warps(2) == warps(1) ? 2 : 1;
  static constexpr int WS = 2 * ROWS * 8 + FB * 8 * FP;
  static constexpr int WARPS = warps(FB);
  static constexpr size_t smem_bytes() { return size_t(TABLES + WARPS * WS + WARPS) * sizeof(double); }
  static constexpr int fit() {
    int n = int(228 * 1024 / (smem_bytes() + 1024));
    while (n * WARPS > 16 && n > 1) --n;
    return n < 1 ? 1 : n;
  }
  static constexpr int CTAS = fit();  // per SM
};

// Position of element e in row k of a shared-memory B operand.
__device__ __forceinline__ int mf_at(int k, int e) { return k * 8 + (e ^ ((k & 2) << 1)); }

// Per-element constants of the step from geometry and materials (once per handle).
__global__ void k_matfree_geometry(int ne, const double* __restrict__ invJ, const double* __restrict__ detJ,
                                   const double* __restrict__ lam_, const double* __restrict__ mu_,
                                   const double* __restrict__ elen, const double* __restrict__ enrm,
                                   const int* __restrict__ neigh, const int* __restrict__ nedge, double pen_n2,
                                   double* __restrict__ alpha, double* __restrict__ face) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += gridDim.x * blockDim.x) {
    const double lam = lam_[e], mu = mu_[e], adet = fabs(detJ[e]);
    const double* iJ = invJ + 4 * size_t(e);  // iJ[a + 2 k] = invJ(a, k)
    const double C[4][4] = {{lam + 2 * mu, 0, 0, mu}, {0, lam, mu, 0}, {0, mu, lam, 0}, {mu, 0, 0, lam + 2 * mu}};
    auto al = [&](int mn, int a, int b) {
      double s = 0.0;
      for (int k = 0; k < 2; ++k)
        for (int l = 0; l < 2; ++l) s += C[mn][k * 2 + l] * iJ[a + 2 * k] * iJ[b + 2 * l];
      return adet * s;
    };
    double* o = alpha + 10 * size_t(e);
    o[0] = al(0, 0, 0), o[1] = al(0, 0, 1), o[2] = al(0, 1, 1);
    o[3] = al(3, 0, 0), o[4] = al(3, 0, 1), o[5] = al(3, 1, 1);
    o[6] = al(1, 0, 0), o[7] = al(1, 0, 1), o[8] = al(1, 1, 0), o[9] = al(1, 1, 1);
    for (int l = 0; l < 3; ++l) {
      double* f = face + 36 * size_t(e) + 12 * l;
      const int nb = neigh[3 * size_t(e) + l];
      const double n0 = enrm[6 * size_t(e) + 2 * l], n1 = enrm[6 * size_t(e) + 2 * l + 1];
      const double hL = 0.5 * elen[3 * size_t(e) + l];
      double h_l = 0.0, h_m = 0.0;
      if (nb >= 0) {
        h_l = harm(lam, lam_[nb]);
        h_m = harm(mu, mu_[nb]);
      }
      f[0] = pen_n2 * ((h_l + 2 * h_m) * n0 * n0 + 2 * h_m * n1 * n1);
      f[1] = pen_n2 * (h_l * n0 * n1);
      f[2] = pen_n2 * ((h_l + 2 * h_m) * n1 * n1 + 2 * h_m * n0 * n0);
      f[3] = __longlong_as_double(nb < 0 ? -1 : 4 * nb + nedge[3 * size_t(e) + l]);
      const double tau[4][2] = {{(lam + 2 * mu) * n0, mu * n1}, {lam * n1, mu * n0}, {mu * n1, lam * n0},
                                {mu * n0, (lam + 2 * mu) * n1}};
      for (int mn = 0; mn < 4; ++mn)
        for (int a = 0; a < 2; ++a) f[4 + mn * 2 + a] = hL * (tau[mn][0] * iJ[a] + tau[mn][1] * iJ[a + 2]);
    }
  }
}

// Face records and inverse masses of the tile's elements into the warp's
// shared memory, in flight until mf_faces_landed.
template <int N>
__device__ __forceinline__ void mf_load_faces(const MatFreeParams& q, const double* minv, int e8, int ne, int lane,
                                              double* fc) {
  const int n2 = min(8, ne - e8) * 18;
  const double* src = q.face + 36 * size_t(e8);
#pragma unroll
  for (int i = lane; i < 8 * 18; i += 32) {
    const int el = i / 18;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     smem_u32(fc + el * MFCfg<N>::FP + 2 * (i - el * 18))),
                 "l"(i < n2 ? src + 2 * i : q.face), "r"(i < n2 ? 16 : 0)
                 : "memory");
  }
  if (minv != nullptr && lane < 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(fc + lane * MFCfg<N>::FP + 36)),
                 "l"(minv + min(e8 + lane, ne - 1))
                 : "memory");
}
__device__ __forceinline__ void mf_faces_landed() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// Values and tractions at the edge points of the tile's elements from the
// coefficients in un ([2][ROWS][8]), written to d.
template <int N>
__device__ __forceinline__ void mf_traces(const double* trc, const double* un, const double* fc, int e8, int ne,
                                          int lane, double* d) {
  typedef MFCfg<N> CF;
  constexpr int KS = CF::KS, TT = CF::TT, RQ = CF::RQ, Q = CF::Q;
  const int g = lane >> 2, tg = lane & 3;
  double b0[KS], b1[KS];
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    b0[ks] = un[mf_at(4 * ks + tg, g)];
    b1[ks] = un[CF::ROWS * 8 + mf_at(4 * ks + tg, g)];
  }
#pragma unroll 1
  for (int t = 0; t < TT; ++t) {
    double c[3][2][2];  // value and two derivatives, component, element
#pragma unroll
    for (int w = 0; w < 3; ++w) c[w][0][0] = c[w][0][1] = c[w][1][0] = c[w][1][1] = 0.0;
    const double* tt = trc + t * KS * 32 + lane;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const double a = tt[(w * TT * KS + ks) * 32];
        dmma_m8n8k4(c[w][0][0], c[w][0][1], a, b0[ks]);
        dmma_m8n8k4(c[w][1][0], c[w][1][1], a, b1[ks]);
      }
    const int r = 8 * t + g;
    if (r < RQ) {
      const int l = r / Q;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int el = 2 * tg + h;
        if (e8 + el < ne) {
          const double* be = fc + el * CF::FP + 12 * l + 4;
          // T^m = sum_na beta^{nm}_a g^n_a
          const double2 b00 = *reinterpret_cast<const double2*>(be), b01 = *reinterpret_cast<const double2*>(be + 2);
          const double2 b10 = *reinterpret_cast<const double2*>(be + 4), b11 = *reinterpret_cast<const double2*>(be + 6);
          double* o = d + (size_t(e8 + el) * RQ + r) * 4;
          *reinterpret_cast<double2*>(o) = make_double2(c[0][0][h], c[0][1][h]);
          *reinterpret_cast<double2*>(o + 2) =
              make_double2(b00.x * c[1][0][h] + b00.y * c[2][0][h] + b10.x * c[1][1][h] + b10.y * c[2][1][h],
                           b01.x * c[1][0][h] + b01.y * c[2][0][h] + b11.x * c[1][1][h] + b11.y * c[2][1][h]);
        }
      }
    }
  }
}

// Edge values (dout) of a state given by its coefficients.
template <int N>
__global__ void __launch_bounds__(MFCfg<N>::WARPS * 32, MFCfg<N>::CTAS)
    k_matfree_traces(const double* __restrict__ x, int ne, const MatFreeParams q) {
  typedef MFCfg<N> CF;
  constexpr int NP = CF::NP, R = CF::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* tab = reinterpret_cast<double*>(smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* un = tab + CF::TRC + warp * CF::WS;
  double* fc = un + 2 * CF::ROWS * 8;
  const double2* src = reinterpret_cast<const double2*>(q.tables + CF::VOL + CF::LIFT);
  for (int i = threadIdx.x; i < CF::TRC / 2; i += CF::WARPS * 32) reinterpret_cast<double2*>(tab)[i] = __ldg(src + i);
  __syncthreads();
  const int tiles = (ne + 7) / 8;
  for (int tile = blockIdx.x + gridDim.x * warp; tile < tiles; tile += gridDim.x * CF::WARPS) {
    const int e8 = tile * 8;
    mf_load_faces<N>(q, nullptr, e8, ne, lane, fc);
    for (int i = lane; i < 2 * 4 * CF::KS * 8; i += 32) {
      const int el = i & 7, k = (i >> 3) % (4 * CF::KS), m = (i >> 3) / (4 * CF::KS);
      const int e = min(e8 + el, ne - 1);
      un[m * CF::ROWS * 8 + mf_at(k, el)] = k < NP ? x[size_t(e) * R + m * NP + k] : 0.0;
    }
    mf_faces_landed();
    mf_traces<N>(tab, un, fc, e8, ne, lane, q.dout);
    __syncwarp();
  }
}

template <int N>
__global__ void __launch_bounds__(MFCfg<N>::WARPS * 32, MFCfg<N>::CTAS)
    k_step_matfree(const StepParams p, const MatFreeParams q) {
  typedef MFCfg<N> CF;
  constexpr int NP = CF::NP, Q = CF::Q, R = CF::R, KS = CF::KS, MT = CF::MT, RQ = CF::RQ, KL = CF::KL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* tab = reinterpret_cast<double*>(smem_raw);
  const double* vol = tab;
  const double* lift = vol + CF::VOL;
  const double* trc = lift + CF::LIFT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, tg = lane & 3;
  double* rows = tab + CF::TABLES + warp * CF::WS;  // [2][ROWS][8]
  double* fc = rows + 2 * CF::ROWS * 8;             // [FB][8][FP]
  double* red = tab + CF::TABLES + CF::WARPS * CF::WS;

  {
    const double2* src = reinterpret_cast<const double2*>(q.tables);
    for (int i = threadIdx.x; i < CF::TABLES / 2; i += CF::WARPS * 32)
      reinterpret_cast<double2*>(tab)[i] = __ldg(src + i);
  }
  const int ne = p.ne, tiles = (ne + 7) / 8, first = blockIdx.x + gridDim.x * warp;
  if (first < tiles) mf_load_faces<N>(q, p.minv, first * 8, ne, lane, fc);
  __syncthreads();
  // Tables and geometry are constant: they are in place before the previous step ends.
  // The state and the edge values change under this grid until the wait, so
  // they are read by ordinary loads, not through the read-only path.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  const long long k = (p.step_base ? *p.step_base : 0) + p.rel;
  const bool stepping = p.mode == kModeStep || p.mode == kModeFirst;
  double en = 0.0, pw1 = 0.0, pw2 = 0.0;  // energy / power-iteration partials
  double chk = 0.0;  // NaN once a non-finite u^{k+1} was written (inf * 0 and NaN * 0 are NaN)
  const int src_e = stepping && p.src_of == nullptr && p.src_elem != nullptr ? src_elem_at(p, 0) : -1;
  for (int tile = first; tile < tiles; tile += gridDim.x * CF::WARPS) {
    const int e8 = tile * 8, e8n = (tile + gridDim.x * CF::WARPS) * 8;
    mf_faces_landed();
    // ---- B fragments of u^k and the element's elastic factors ----
    const int eg = min(e8 + g, ne - 1);
    double xb[KS][2], al[10];
    {
      const double* xg = p.x + size_t(eg) * R;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        const int kk = 4 * ks + tg;
        const bool in = NP % 4 == 0 || kk < NP;
        xb[ks][0] = in ? xg[kk] : 0.0;
        xb[ks][1] = in ? xg[NP + kk] : 0.0;
      }
      const double2* ag = reinterpret_cast<const double2*>(q.alpha + 10 * size_t(eg));
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const double2 v = __ldg(ag + i);
        al[2 * i] = v.x;
        al[2 * i + 1] = v.y;
      }
      if (p.mode == kModePower) {
        const double xsc = power_scale(p, eg);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          xb[ks][0] *= xsc;
          xb[ks][1] *= xsc;
        }
      }
    }
    // ---- numerical fluxes at the edge points: lane = (element, every fourth point) ----
    {
      const int el = lane & 7, e = min(e8 + el, ne - 1);
      int nb[3];
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        nb[l] = int(__double_as_longlong(fc[el * CF::FP + 12 * l + 3]));
        if (nb[l] >= 0) nb[l] = (TSP_INDEX(nb[l] >> 2, 0, ne, kSiteNeigh) << 2) | (nb[l] & 3);
      }
      double xsc = 1.0;
      if (p.mode == kModePower) xsc = power_scale(p, e);
#pragma unroll
      for (int r = lane >> 3; r < RQ; r += 4) {
        const int l = r >= 2 * Q ? 2 : r >= Q ? 1 : 0, kq = r - l * Q;
        const int code = l == 0 ? nb[0] : l == 1 ? nb[1] : nb[2];
        double F0 = 0.0, F1 = 0.0, H00 = 0.0, H01 = 0.0, H10 = 0.0, H11 = 0.0;
        if (code >= 0) {
          const double2* de = reinterpret_cast<const double2*>(q.din + (size_t(e) * RQ + r) * 4);
          const double2* dn =
              reinterpret_cast<const double2*>(q.din + (size_t(code >> 2) * RQ + (code & 3) * Q + Q - 1 - kq) * 4);
          const double2 ue = de[0], te = de[1], un = dn[0], tn = dn[1];
          const double* f = fc + el * CF::FP + 12 * l;
          double J0 = ue.x - un.x, J1 = ue.y - un.y, D0 = te.x - tn.x, D1 = te.y - tn.y;
          if (p.mode == kModePower) {
            J0 *= xsc;
            J1 *= xsc;
            D0 *= xsc;
            D1 *= xsc;
          }
          const double2 c0 = *reinterpret_cast<const double2*>(f);
          const double c11 = f[2];
          F0 = c0.x * J0 + c0.y * J1 - D0;
          F1 = c0.y * J0 + c11 * J1 - D1;
          const double2 b00 = *reinterpret_cast<const double2*>(f + 4), b01 = *reinterpret_cast<const double2*>(f + 6);
          const double2 b10 = *reinterpret_cast<const double2*>(f + 8), b11 = *reinterpret_cast<const double2*>(f + 10);
          H00 = -(b00.x * J0 + b01.x * J1);  // H^m_a, m = 0: a = 0, 1
          H01 = -(b00.y * J0 + b01.y * J1);
          H10 = -(b10.x * J0 + b11.x * J1);
          H11 = -(b10.y * J0 + b11.y * J1);
        }
        rows[mf_at(r, el)] = F0;
        rows[mf_at(RQ + r, el)] = H00;
        rows[mf_at(2 * RQ + r, el)] = H01;
        rows[CF::ROWS * 8 + mf_at(r, el)] = F1;
        rows[CF::ROWS * 8 + mf_at(RQ + r, el)] = H10;
        rows[CF::ROWS * 8 + mf_at(2 * RQ + r, el)] = H11;
      }
      if constexpr (4 * KL > 3 * RQ) {  // k padding of the lift
        const int r = 3 * RQ + (lane >> 3);
        if (r < 4 * KL) rows[mf_at(r, el)] = rows[CF::ROWS * 8 + mf_at(r, el)] = 0.0;
      }
    }
    // ---- volume ----
    double acc[MT][2][2];
#pragma unroll
    for (int t = 0; t < MT; ++t) acc[t][0][0] = acc[t][0][1] = acc[t][1][0] = acc[t][1][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const double x0 = xb[ks][0], x1 = xb[ks][1];
      const double z0[4] = {al[0] * x0 + al[6] * x1, al[1] * x0 + al[7] * x1, al[1] * x0 + al[8] * x1,
                            al[2] * x0 + al[9] * x1};
      const double z1[4] = {al[6] * x0 + al[3] * x1, al[8] * x0 + al[4] * x1, al[7] * x0 + al[4] * x1,
                            al[9] * x0 + al[5] * x1};
#pragma unroll
      for (int ab = 0; ab < 4; ++ab)
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const double a = vol[((ab * MT + t) * KS + ks) * 32 + lane];
          dmma_m8n8k4(acc[t][0][0], acc[t][0][1], a, z0[ab]);
          dmma_m8n8k4(acc[t][1][0], acc[t][1][1], a, z1[ab]);
        }
    }
    __syncwarp();
    // Both levels of this lane's outputs (rows 8 t + g of elements 2 tg,
    // 2 tg + 1), in flight during the lift; also `out` may be `uprev`, so a
    // store would hold back every load after it.
    double uk[MT][2][2], upv[MT][2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const size_t at = size_t(min(e8 + 2 * tg + h, ne - 1)) * R;
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int i = 8 * t + g, r = m * NP + i;
          const bool row = NP % 8 == 0 || i < NP;
          uk[t][m][h] = row ? p.x[at + r] : 0.0;
          upv[t][m][h] = row && stepping && p.uprev != nullptr ? p.uprev[at + r] : 0.0;
        }
    }
    int t0 = 0, t1 = 0;
    if (stepping && p.rcv_ptr != nullptr) {
      t0 = rcv_ptr_at(p, e8);
      t1 = rcv_ptr_at(p, min(e8 + 8, ne));
    }
    double* fnext = fc;
    if constexpr (CF::FB == 2) {
      fnext = (fc - rows) > 2 * CF::ROWS * 8 ? fc - 8 * CF::FP : fc + 8 * CF::FP;
      if (e8n < ne) mf_load_faces<N>(q, p.minv, e8n, ne, lane, fnext);
    }
    // ---- lift of the fluxes (w_k is in the table) ----
#pragma unroll 2
    for (int ks = 0; ks < KL; ++ks) {
      const double f0 = rows[mf_at(4 * ks + tg, g)], f1 = rows[CF::ROWS * 8 + mf_at(4 * ks + tg, g)];
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        const double a = lift[(t * KL + ks) * 32 + lane];
        dmma_m8n8k4(acc[t][0][0], acc[t][0][1], a, f0);
        dmma_m8n8k4(acc[t][1][0], acc[t][1][1], a, f1);
      }
    }
    __syncwarp();
    // ---- update: this lane holds rows 8 t + g of elements 2 tg, 2 tg + 1 ----
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int el = 2 * tg + h, e = e8 + el;
      const bool in = e < ne;
      const int ec = in ? e : ne - 1;
      const double mi = fc[el * CF::FP + 36];
      const double dt = p.dt_elem ? p.dt_elem[ec] : p.dt;
      const int srow = !stepping ? -1 : p.src_of ? p.src_of[ec]
                                      : src_e == ec ? 0 : -1;
      const bool is_src = srow >= 0 && k < p.nF;
      const double xsc = p.mode != kModePower ? 1.0 : power_scale(p, ec);
      double* og = p.out + size_t(ec) * R;
      double pe0 = 0.0, pe1 = 0.0, pe2 = 0.0;
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        const int i = 8 * t + g;
        const bool row = NP % 8 == 0 || i < NP;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          double un = 0.0;
          if (row) {
            const int r = m * NP + i;
            const double y = acc[t][m][h];
            double u = uk[t][m][h];
            if (stepping) {
              const double f =
                  is_src ? p.F[(size_t(srow) * p.nF + k) * 2 + m] * p.src_phi[size_t(srow) * NP + i] : 0.0;
              const double up = upv[t][m][h];
              if (p.mode == kModeStep) un = (2 * u - up) + mi * ((-dt * dt) * (y - f));
              else un = (u + dt * up) - mi * (dt * dt / 2 * (y - f));
              if (in) {
                chk = __fma_rn(un, 0.0, chk);
                if (p.energy != nullptr) {
                  const double d = un - u;
                  en += 0.5 * (d * d) / (mi * dt * dt) + 0.5 * un * y;
                }
              }
            } else if (p.mode == kModeApply) {
              un = y;
            } else {  // kModePower
              u *= xsc;
              un = mi * y;
              if (in) {
                pe0 += u * y;
                pe1 += u * u / mi;
                pe2 += un * un;
              }
            }
            if (in) og[r] = un;
          }
          if (i < CF::ROWS) rows[m * CF::ROWS * 8 + mf_at(i, el)] = un;  // rows past NP: zero
        }
      }
      if (p.mode == kModePower) {
        if (p.mesh_of != nullptr) {
          // The eight lanes of this element (lane bits 2..4) sum, then one adds.
#pragma unroll
          for (int o = 4; o < 32; o <<= 1) {
            pe0 += __shfl_xor_sync(0xffffffffu, pe0, o);
            pe1 += __shfl_xor_sync(0xffffffffu, pe1, o);
            pe2 += __shfl_xor_sync(0xffffffffu, pe2, o);
          }
          if (g == 0 && in) {
            double* acc3 = p.acc + 3 * size_t(p.mesh_of[ec]);
            atomicAdd(acc3 + 0, pe0);
            atomicAdd(acc3 + 1, pe1);
            atomicAdd(acc3 + 2, pe2);
          }
        } else {
          en += pe0;
          pw1 += pe1;
          pw2 += pe2;
        }
      }
    }
    __syncwarp();
    // ---- receivers of the tile's elements: sample u^{k+1} ----
    if (t1 > t0) {
      const int mine = rcv_ptr_at(p, min(e8 + 1 + (lane & 7), ne));
      int end[7];  // first receiver position behind each element of the tile
#pragma unroll
      for (int j = 0; j < 7; ++j) end[j] = __shfl_sync(0xffffffffu, mine, j);
      sample_receivers<NP, NP>(p, t0, t1, k, 0, lane,
                           [&](int r) {
                             int el = 0;
#pragma unroll
                             for (int j = 0; j < 7; ++j) el += r >= end[j];
                             return el;
                           },
                           [&](int el, int c, int i) { return rows[c * CF::ROWS * 8 + mf_at(i, el)]; });
    }
    // ---- edge values of u^{k+1} for the next step ----
    if (q.dout != nullptr) mf_traces<N>(trc, rows, fc, e8, ne, lane, q.dout);
    __syncwarp();
    if (CF::FB == 1 && e8n < ne) mf_load_faces<N>(q, p.minv, e8n, ne, lane, fc);
    fc = fnext;
  }
  if (chk != chk && p.nonfinite != nullptr) *p.nonfinite = 1;
  const bool power = p.mode == kModePower && p.mesh_of == nullptr;
  if (power) {
    const double v0 = warp_sum(en), v1 = warp_sum(pw1), v2 = warp_sum(pw2);
    if (lane == 0) {
      atomicAdd(p.acc + 0, v0);
      atomicAdd(p.acc + 1, v1);
      atomicAdd(p.acc + 2, v2);
    }
  } else if (p.energy != nullptr && stepping) {
    const double v = warp_sum(en);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0.0;
      for (int w = 0; w < CF::WARPS; ++w) sum += red[w];
      atomicAdd(p.energy + (k % p.energy_cap), sum);
    }
  }
}

}  // namespace tsp
