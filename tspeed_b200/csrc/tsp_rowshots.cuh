// Step of a few shots over a symmetric block operator (FP64 or FP32 blocks),
// on the FP64 tensor cores (internal header of tspeed_b200).
//
// With few shots the step is bound by the bytes of the operator, not by its
// products, so it uses the storage of the single-shot ring kernel
// (tsp_rowring.cuh): one block per face, used transposed by the higher row,
// whose copy comes from L2. Per row Y[shot][r] = sum_b sum_k X_b[shot][k]
// B_b[r][k] runs on mma.sync m8n8k4.f64 (exact FP64 products, FP64
// accumulation) with tiles of 8, 16, 24 or 32 shots: the 32- and 64-shot tiles
// of the batched kernels would multiply mostly padding. FP32 blocks are
// widened as they leave the stage and multiply the FP64 state: half the bytes
// of FP64 blocks, and only the operator is rounded to FP32 (no FP32 shadow of
// the state, no FP32 sums).
//
// Roles: NG groups of WN consumer warps, each warp NTW tiles of 8 operator
// rows x all shots; group g owns every NG-th row of the CTA and a ring of its
// own, filled by lane g of the producer warp with two bulk copies per block
// (the stored block, pitch 2Np, and the neighbour's state tile; completion on
// mbarriers, no multicast). Operand fragments come straight from the stage:
// B[k][n] at column k, row n of the block, or transposed at column n, row k.
// Where 2Np is not a multiple of 4 the last k step's padding is masked in both
// operands; rows past 2Np only reach outputs that are dropped. The epilogue's
// u^{k-1} and the next row's references are requested before the products; its
// u^k likewise, or it is read from the state tile of the diagonal block
// (STAGED): L2 to shared memory carries 37 KB per row of 24 shots at 2Np = 30
// with FP32 blocks, u^k from memory 5.8 KB more, and 14,520 triangles take
// 132.0 us per step instead of 144.6.
//
// Every ring belongs to one group, in that group's row order, so use j / NSG
// of a stage is unambiguous for both sides. Every wait is bounded (about a
// second); on a timeout the CTA raises an abort flag, every role stops
// waiting, the producer waits (bounded) for its copies in flight, and
// err_flag tells the host that the results are void. Blocks and references
// are constant, the state is read after griddepcontrol.wait (programmatic
// dependent launch).
#pragma once

#include <stdint.h>

#include "tsp_rowring.cuh"

namespace tsp {

// Row tiles per warp and groups of a CTA. Measured on 4,900 triangles, us per
// step (tiles, groups): FP64 2Np = 20, 8 shots (1, 6) 17.0, (3, 12) 14.1; 42,
// 24 shots (1, 3) 95, (2, 4) 86; 72, 8 shots (1, 2) 108, (3, 2) 96; 90, 24
// shots (2, 1) 369, (1, 1) 288. FP32 2Np = 30, 8 shots (1, 4) 21.3, (4, 12)
// 18.8; 42, 24 shots (1, 3) 99, (2, 5) 91; 72, 8 shots (1, 2) 75.5, (3, 4)
// 71.8; 90, 24 shots (1, 1) 292, (2, 2) 285. More row tiles per warp read the
// state's fragments fewer times and leave more warps to other rows, until
// the accumulators and the requested state levels spill.
constexpr int rowshots_tiles(int R, int ST, bool fp64) {
  switch (R) {
    case 20: return ST == 8 ? 3 : 1;
    case 30: return ST == 8 && !fp64 ? 4 : ST <= 24 && fp64 ? 2 : 1;
    case 42: return 2;
    case 72: return ST == 8 ? 3 : 1;
    case 90: return fp64 ? 1 : 2;
    default: return 1;
  }
}
constexpr int rowshots_groups(int R, int ST, bool fp64) {
  switch (R) {
    case 20: return ST == 8 ? 12 : 6;
    case 30: return ST == 8 && !fp64 ? 12 : ST <= 24 && fp64 ? 6 : 4;
    case 42: return fp64 || ST == 32 ? 4 : 5;
    case 72: return ST == 8 && !fp64 ? 4 : 2;
    default: return 2;
  }
}

template <int R, int ST, typename BT>
struct RowShotsCfg {
  static constexpr int KS = (R + 3) / 4;
  static constexpr int NTL = (R + 7) / 8;
  static constexpr int MT = ST / 8;
  static constexpr int NTW = rowshots_tiles(R, ST, sizeof(BT) == 8);
  static constexpr int WN = (NTL + NTW - 1) / NTW;
  // u^k of the epilogue from the diagonal block's state tile instead of from
  // memory: less traffic, but read between the wait for the stage and the
  // products. It pays for the large tiles beside FP32 blocks; 4,900 triangles,
  // us per step, memory / stage: FP32 24 shots 2Np = 30 51.9 / 47.4, 42 91.4 /
  // 85.2, 56 126 / 130, 72 202 / 196; 32 shots 56 174 / 169, 72 248 / 251, 90 417 / 397; 16
  // shots 42 54.7 / 57.7, 56 89 / 95; FP64 24 shots 30 48.7 / 49.0, 90 305 /
  // 316; 8 shots 72 103 / 107.
  static constexpr bool STAGED = sizeof(BT) == 4 && ((ST == 32 && R != 72) || (ST == 24 && R != 56));
  static constexpr int BB = R * R * int(sizeof(BT));  // bytes: the block
  static constexpr int XB = ST * R * 8;               // the state tile
  static constexpr int STAGE = BB + XB;
  static_assert(BB % 16 == 0 && XB % 16 == 0, "16-byte aligned stages");
  static_assert(8 * NTL - R <= ST, "fragment rows past the block stay inside the stage");
  static_assert((8 * NTL - R) * R * int(sizeof(BT)) <= XB, "fragment rows past the block stay inside the stage");
  static constexpr int total() { return int((226 * 1024) / (STAGE + 16)); }
  // One group where two rings of two stages do not fit.
  static constexpr int NG0 = rowshots_groups(R, ST, sizeof(BT) == 8);
  static constexpr int NG = total() / NG0 >= 2 ? NG0 : 1;
  static constexpr int NSG = total() / NG > 6 ? 6 : total() / NG;
  static_assert(NSG >= 2, "two stages per group must fit");
  static constexpr int NST = NG * NSG;
  static constexpr int NT = (NG * WN + 1) * 32;
  static constexpr size_t smem_bytes() { return size_t(NST) * STAGE + size_t(2 * NST) * 8 + 16; }
};

template <int R, int ST, typename BT>
__global__ void __launch_bounds__(RowShotsCfg<R, ST, BT>::NT, 1) k_step_rowshots(const StepParams p, int* err_flag) {
  typedef RowShotsCfg<R, ST, BT> CF;
  constexpr int NP = R / 2, KS = CF::KS, NTL = CF::NTL, MT = CF::MT, NTW = CF::NTW, WN = CF::WN, NSG = CF::NSG;
  constexpr int NG = CF::NG, NST = CF::NST;
  constexpr bool MASK = R % 4 != 0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* stages = smem_raw;
  uint64_t* bfull = reinterpret_cast<uint64_t*>(stages + size_t(NST) * CF::STAGE);
  uint64_t* bempty = bfull + NST;
  volatile int* abort_s = reinterpret_cast<volatile int*>(bempty + NST);
  const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
  if (t == 0) {
    *abort_s = 0;
    for (int i = 0; i < NST; ++i) {
      fx_mbar_init(smem_u32(&bfull[i]), 1);
      fx_mbar_init(smem_u32(&bempty[i]), WN);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // State tiles of fewer than ST shots leave their last rows unwritten.
  for (int i = t; i < NST * CF::STAGE / 16; i += CF::NT) reinterpret_cast<int4*>(stages)[i] = make_int4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();

  const int S = p.S, ne = p.ne, G = int(gridDim.x);
  const int ntile = (S + ST - 1) / ST;
  // Items (row, tile) fit 32 bits: each holds at least 2Np doubles of state.
  const int nitems = ne * ntile, stride = NG * G;
  auto row_of = [&](int item) { return ntile == 1 ? item : item / ntile; };
  auto tile_of = [&](int item) { return ntile == 1 ? 0 : item % ntile; };
  const RowRefs* rows = reinterpret_cast<const RowRefs*>(p.rows);
  struct Refs {
    int4 a, b;  // (col, ref) of blocks 0, 1 and 2, 3
  };
  auto refs_of = [&](int item) {
    Refs r;
    r.a = r.b = make_int4(-1, 0, -1, 0);
    if (item < nitems) {
      const int e = row_of(item);
      r.a = __ldg(reinterpret_cast<const int4*>(rows + e));
      r.b = __ldg(reinterpret_cast<const int4*>(rows + e) + 1);
    }
    return r;
  };
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == NG * WN) {
    // ---------------- producers: lane g fills ring g ----------------
    if (lane < NG) {
      const int g = lane;
      uint64_t* gfull = bfull + g * NSG;
      uint64_t* gempty = bempty + g * NSG;
      const uint32_t gst = smem_u32(stages + size_t(g) * NSG * CF::STAGE);
      constexpr uint32_t bbytes = CF::BB;
      auto block_of = [&](const Refs& rr, int b) {
        return b == 0 ? make_int2(rr.a.x, rr.a.y) : b == 1 ? make_int2(rr.a.z, rr.a.w)
               : b == 2 ? make_int2(rr.b.x, rr.b.y) : make_int2(rr.b.z, rr.b.w);
      };
      auto tile_bytes = [&](int item) { return uint32_t(min(ST, S - tile_of(item) * ST)) * R * 8; };
      auto copy_block = [&](int2 cr, int s, uint32_t xbytes) {
        const int phys = TSP_INDEX(cr.y >> 1, 0, p.nphys, kSiteRow);
        fx_mbar_arrive_tx(smem_u32(&gfull[s]), bbytes + xbytes);
        fx_bulk_g2s(gst + uint32_t(s) * CF::STAGE,
                    reinterpret_cast<const unsigned char*>(p.blocks) + size_t(phys) * CF::BB, bbytes,
                    smem_u32(&gfull[s]));
      };
      auto copy_state = [&](int2 cr, int s, uint32_t xbytes, int tile) {
        const int c = TSP_INDEX(cr.x, 0, ne, kSiteCol);
        fx_bulk_g2s(gst + uint32_t(s) * CF::STAGE + CF::BB, p.x + (size_t(c) * S + size_t(tile) * ST) * R, xbytes,
                    smem_u32(&gfull[s]));
      };
      uint32_t j = 0;
      bool ok = true;
      int item = blockIdx.x + g * G;
      Refs nx = refs_of(item);
      // The first blocks before the previous step ends, their state tiles after.
      constexpr int AHEAD = NSG < 4 ? NSG : 4;
      int ahead = 0;
#pragma unroll
      for (int b = 0; b < AHEAD; ++b)
        if (block_of(nx, b).x >= 0) copy_block(block_of(nx, b), ahead++, tile_bytes(item));
      asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
      for (int b = 0; b < AHEAD; ++b)
        if (b < ahead) copy_state(block_of(nx, b), b, tile_bytes(item), tile_of(item));
      for (; item < nitems && ok; item += stride) {
        const Refs rr = nx;
        nx = refs_of(item + stride);
        const uint32_t xbytes = tile_bytes(item);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int2 cr = block_of(rr, b);
          if (cr.x < 0 || !ok) continue;
          if (int(j) < ahead) {  // under way (the first row's blocks are its leading ones)
            ++j;
            continue;
          }
          const int s = int(j % NSG);
          const uint32_t n = j / NSG;
          if (n > 0 && !fx_wait(smem_u32(&gempty[s]), (n - 1) & 1, abort_s)) {
            ok = false;
            continue;
          }
          copy_block(cr, s, xbytes);
          copy_state(cr, s, xbytes, tile_of(item));
          ++j;
        }
      }
      // Every issued copy lands before the CTA ends (bounded; copies complete).
      const long long t0 = clock64();
      for (int s = 0; s < NSG; ++s) {
        if (j <= uint32_t(s)) continue;
        const uint32_t uses = (j - 1 - s) / NSG + 1;
        while (!mbar_try(smem_u32(&gfull[s]), (uses - 1) & 1) && clock64() - t0 < (1ll << 31)) {
        }
      }
      if (clock64() - t0 >= (1ll << 31)) *abort_s = 1;
    } else {
      asm volatile("griddepcontrol.wait;" ::: "memory");
    }
  } else {
    // ---------------- consumers ----------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool off = *reinterpret_cast<volatile int*>(err_flag) != 0;  // an earlier launch of the run timed out
    const int grp = warp / WN, wn = warp % WN, tl = t - grp * WN * 32;
    const int g = lane >> 2, tg = lane & 3;
    // Fragment row g holds shot gs: with 2Np odd in pairs, even shots first
    // puts a half-warp's rows in distinct banks.
    const int gs = (R / 2) % 2 ? (((g & 3) << 1) | (g >> 2)) : g;
    const int nt0 = wn * NTW;
    const long long k = (p.step_base ? *p.step_base : 0) + p.rel;
    const double dt = p.dt;
    uint64_t* gfull = bfull + grp * NSG;
    uint64_t* gempty = bempty + grp * NSG;
    const unsigned char* gst = stages + size_t(grp) * NSG * CF::STAGE;
    double en = 0.0, chk = 0.0;  // chk: NaN once a non-finite u^{k+1} was written
    uint32_t j = 0;
    bool dead = off;
    int item = blockIdx.x + grp * G;
    Refs nx = refs_of(item);
    for (; item < nitems; item += stride) {
      const Refs rr = nx;
      nx = refs_of(item + stride);
      const int e = row_of(item), s0 = tile_of(item) * ST, nsv = min(ST, S - s0);
      const double mi = p.minv[e];
      int src_e[MT];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) src_e[mt] = 8 * mt + gs < nsv && k < p.nF ? src_elem_at(p, s0 + 8 * mt + gs) : -1;
      int q0 = 0, q1 = 0;
      if (p.rcv_ptr != nullptr) {
        q0 = rcv_ptr_at(p, e);
        q1 = rcv_ptr_at(p, e + 1);
      }
      // u^k and u^{k-1} of this lane's outputs, in flight during the products.
      // STAGED: u^k from memory only where the row has no diagonal block.
      const bool diag = CF::STAGED && (rr.a.x == e || rr.a.z == e || rr.b.x == e || rr.b.z == e);
      double2 uk[MT][NTW], up[MT][NTW];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int sh = 8 * mt + gs;
        const size_t me = (size_t(e) * S + s0 + (sh < nsv ? sh : 0)) * R;
#pragma unroll
        for (int q = 0; q < NTW; ++q) {
          const int r0 = (nt0 + q) * 8 + 2 * tg;
          const bool in = sh < nsv && nt0 + q < NTL && r0 < R;
          if (!diag) uk[mt][q] = in ? *reinterpret_cast<const double2*>(p.x + me + r0) : make_double2(0.0, 0.0);
          up[mt][q] = in && p.uprev ? *reinterpret_cast<const double2*>(p.uprev + me + r0) : make_double2(0.0, 0.0);
        }
      }
      double acc[MT][NTW][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int q = 0; q < NTW; ++q) acc[mt][q][0] = acc[mt][q][1] = 0.0;
#pragma unroll 1
      for (int b = 0; b < 4; ++b) {
        const int2 cr = b == 0 ? make_int2(rr.a.x, rr.a.y) : b == 1 ? make_int2(rr.a.z, rr.a.w)
                        : b == 2 ? make_int2(rr.b.x, rr.b.y) : make_int2(rr.b.z, rr.b.w);
        if (cr.x < 0 || dead) continue;
        const int s = int(j % NSG);
        const uint32_t n = j / NSG;
        ++j;
        const bool okw = fx_wait(smem_u32(&gfull[s]), n & 1, abort_s);
        if (__any_sync(0xffffffffu, !okw)) {
          dead = true;
          continue;
        }
        const BT* B = reinterpret_cast<const BT*>(gst + size_t(s) * CF::STAGE);
        const double* X = reinterpret_cast<const double*>(gst + size_t(s) * CF::STAGE + CF::BB) + gs * R + tg;
        if (CF::STAGED && cr.x == e) {
          const double* U = reinterpret_cast<const double*>(gst + size_t(s) * CF::STAGE + CF::BB) + gs * R + 2 * tg;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int q = 0; q < NTW; ++q)
              if ((nt0 + q) * 8 + 2 * tg < R)
                uk[mt][q] = *reinterpret_cast<const double2*>(U + mt * 8 * R + (nt0 + q) * 8);
        }
        // B[k][n]: column k, row n of the block; transposed: column n, row k.
        const bool tr = cr.y & 1;
        const BT* Bt = B + (tr ? (nt0 * 8 + g) * R + tg : tg * R + nt0 * 8 + g);
        const int bk = tr ? 4 : 4 * R, bq = tr ? 8 * R : 8;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          const bool in = !MASK || ks + 1 < KS || 4 * ks + tg < R;
          double a[MT], bb[NTW];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) a[mt] = in ? X[mt * 8 * R + 4 * ks] : 0.0;
#pragma unroll
          for (int q = 0; q < NTW; ++q) bb[q] = in && (NTL % NTW == 0 || nt0 + q < NTL) ? double(Bt[ks * bk + q * bq]) : 0.0;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int q = 0; q < NTW; ++q) dmma_m8n8k4(acc[mt][q][0], acc[mt][q][1], a[mt], bb[q]);
        }
        fx_reads_done();
        __syncwarp();
        if (lane == 0) fx_mbar_arrive(smem_u32(&gempty[s]));
      }
      // ---- epilogue (leap-frog, source, energy terms) ----
      if (!dead) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int sh = s0 + 8 * mt + gs;
          if (8 * mt + gs >= nsv) continue;
          const size_t me = (size_t(e) * S + sh) * R;
          const bool is_src = src_e[mt] == e;
          double F0 = 0.0, F1 = 0.0;
          if (is_src) {
            F0 = p.F[(size_t(sh) * p.nF + k) * 2];
            F1 = p.F[(size_t(sh) * p.nF + k) * 2 + 1];
          }
#pragma unroll
          for (int q = 0; q < NTW; ++q) {
            const int r0 = (nt0 + q) * 8 + 2 * tg;
            if (nt0 + q >= NTL || r0 >= R) continue;  // rows come in pairs (R is even)
            const double u[2] = {uk[mt][q].x, uk[mt][q].y}, upr[2] = {up[mt][q].x, up[mt][q].y};
            double un[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = r0 + h;
              const int cmp = r / NP, ii = r - cmp * NP;
              const double f = is_src ? (cmp ? F1 : F0) * p.src_phi[size_t(sh) * NP + ii] : 0.0;
              const double y = acc[mt][q][h];
              if (p.mode == kModeStep) un[h] = (2 * u[h] - upr[h]) + mi * ((-dt * dt) * (y - f));
              else un[h] = (u[h] + dt * upr[h]) - mi * (dt * dt / 2 * (y - f));  // kModeFirst, uprev = v0
              if (p.energy != nullptr) {
                const double d = un[h] - u[h];
                en += 0.5 * (d * d) / (mi * dt * dt) + 0.5 * un[h] * y;
              }
            }
            *reinterpret_cast<double2*>(p.out + me + r0) = make_double2(un[0], un[1]);
            chk = __fma_rn(un[0], 0.0, __fma_rn(un[1], 0.0, chk));
          }
        }
      }
      // ---- receivers (the condition is the same for every warp of the group) ----
      if (q1 > q0) {
        // u^{k+1} of this row is visible to the whole group.
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(WN * 32) : "memory");
        if (!dead) {
          const long long slot = k % p.seis_cap;
          for (int wk = tl; wk < (q1 - q0) * nsv * 2; wk += WN * 32) {
            const int cmp = wk & 1, sh = s0 + (wk >> 1) % nsv, q = q0 + (wk >> 1) / nsv;
            const int rid = rcv_id_at(p, q);
            const double* ph = p.rcv_phi + size_t(rid) * NP;
            const double* un = p.out + (size_t(e) * S + sh) * R + cmp * NP;
            double v = 0.0;
#pragma unroll(NP <= 21 ? NP : 9)
            for (int ii = 0; ii < NP; ++ii) v += ph[ii] * un[ii];
            p.seis[((size_t(sh) * p.seis_cap + slot) * p.nrcv + rid) * 2 + cmp] = v;
          }
        }
      }
    }
    if (chk != chk && p.nonfinite != nullptr) *p.nonfinite = 1;
    if (p.energy != nullptr) {
      const double v = warp_sum(en);
      if (lane == 0 && v != 0.0) atomicAdd(p.energy + (k % p.energy_cap), v);
    }
    // A launch that is off consumes nothing: its producers stop at their rings' end.
    if (off && lane == 0) *abort_s = 1;
  }
  __syncthreads();
  if (t == 0 && *abort_s) atomicExch(err_flag, 1);
}

}  // namespace tsp
