// Single-shot fused leap-frog step over a symmetric block operator, streamed
// through shared-memory rings (internal header of tspeed_b200).
//
// B is symmetric, so of the two blocks of a face only the one above the
// diagonal is stored; the row below uses it transposed. A block row then is
// a list of (physical block, transposed) references. The rows of the mesh
// advance in index order over the whole chip, so the second use of a block
// comes soon after the first and is served by L2: HBM carries
// ne + (nnzb - ne)/2 blocks per step instead of nnzb (62.5 % in the interior
// of a mesh). An operator that is not symmetric (handles built from foreign
// blocks) is stored in full and its references are never transposed.
//
// What bounds it: the bytes of the blocks, from HBM or from L2, and for small
// meshes the latency of one row. A team of four warps (one CTA) owns a row at
// a time, warp w its block w: the products of a row run side by side, few rows
// are open at once (so that the second use of a block finds it in L2), and a
// mesh of a thousand rows still fills the chip. Each warp streams its blocks
// through a ring of its own: column chunks of one bulk copy each
// (cp.async.bulk, completion on an mbarrier, no multicast), requested by its
// lane 0 as soon as the warp has consumed the slot. The warp waits only on
// copies it requested itself, in the order it requested them, so a slot's
// phase always names the chunk. The next row's state is requested into
// registers while the current row multiplies. The warps take turns with the
// epilogue: three arrive at the row's barrier and go on, the fourth waits for
// them there.
//
// Programmatic dependent launch: the blocks and row references never change,
// so a step's warps fill their rings before they wait for the previous step
// (griddepcontrol.wait); everything that a step writes or reads of the state
// comes after that wait, by ordinary loads: the read-only path does not hold
// for data that changes while the grid waits.
//
// Products: a chunk holds NC columns of the stored block (column-major, pitch
// 2Np). Untransposed, lanes own row pairs (G groups of lanes share the columns
// when 2Np <= 32) and keep their sums in registers over the block.
// Transposed, lanes own columns (PT lanes per column split the rows) and a
// column's dot product is complete within its chunk; columns start at
// staggered row pairs where the pitch would put them in the same banks.
#pragma once

#include <stdint.h>

#include <type_traits>

#include "tsp_kernels.cuh"
#include "tsp_tcfx.cuh"
#include "tsp_tcgen05.cuh"

namespace tsp {

// Row e of the operator: columns (-1: no block) and block references
// (physical block << 1 | transposed) of its blocks, diagonal first.
struct alignas(32) RowRefs {
  struct alignas(8) {
    int col, ref;
  } q[4];
};

// Bytes of stored blocks from which the rows are claimed instead of shared
// out: five times L2. us per step at 12,000 triangles, shared out / claimed:
// FP64 2Np = 56 (0.75 GB) 114.4 / 113.7, FP32 90 (0.97 GB) 182 / 166.
constexpr size_t row_queue_bytes = size_t(640) << 20;

template <int R, typename BT>
struct RowRingCfg {
  static constexpr int SZ = int(sizeof(BT));
  static constexpr int NPAIR = R / 2;
  static constexpr int W = 4;  // warps of a team: blocks of a row
  // Columns per chunk (whole columns, multiples of 16 bytes), slots per warp
  // (whole blocks of DEPTH rows ahead, or a part of a block) and teams per SM.
  // Large chunks cost fewer waits and requests per row; small ones, or a
  // single slot, leave room for more teams. Measured on 40,000 triangles, us
  // per step (columns, slots, teams): FP64 2Np = 30 (15, 2, 5) 119, (30, 1, 6)
  // 116; 42 (14, 3, 3) 208, (6, 7, 3) 291; 56 (14, 2, 3) 437, (28, 2, 2) 420;
  // 72 (12, 2, 3) 747, (24, 3, 1) 855; 90 (10, 3, 2) 1162, (6, 3, 3) 1313.
  // FP32 (columns, slots) 42 (42, 2) 125, (14, 3) 132, (42, 1) 120; 56 (14, 4)
  // 292, (28, 2) 228; 72 (12, 3) 404, (36, 2) 433 (12,000 triangles 141, 137;
  // 120,000 1274, 1289); 90 (18, 5) 929, (10, 3) 560.
  static constexpr bool F64 = SZ == 8;
  static constexpr int NC = F64 ? (R == 42 ? 14 : R == 56 ? 28 : R == 72 ? 12 : R == 90 ? 10 : R)
                                : (R == 56 ? 28 : R == 72 ? 36 : R == 90 ? 10 : R);
  static constexpr int NCH = R / NC;    // chunks per block
  static constexpr int CB = NC * R * SZ;
  static_assert(R % NC == 0 && CB % 16 == 0, "whole chunks, multiples of 16 bytes");
  static constexpr int NS = R <= 20 ? 2 : F64 ? (R == 42 ? 3 : R == 56 ? 2 : R == 72 ? 2 : R == 90 ? 3 : 1)
                                          : (R == 56 ? 2 : R == 72 ? 2 : R == 90 ? 3 : 1);
  static constexpr int DEPTH = NS >= NCH ? NS / NCH : 1;
  static constexpr int LAP = NS >= NCH ? 1 : NCH / NS;  // uses of a slot per block
  static_assert(NS >= NCH ? NS % NCH == 0 : NCH % NS == 0, "a chunk's slot is known at compile time");
  // FP32: sums in column order (see ORD in the kernel): no lane groups over the
  // columns, no parts of a column, no staggering.
  static constexpr bool ORD = !F64;
  static constexpr int PPL = (NPAIR + 31) / 32;              // row pairs per lane
  static constexpr int G = !ORD && NPAIR <= 16 ? 32 / NPAIR : 1;  // lane groups over columns
  static constexpr int CPL = (NC + 31) / 32;                 // transposed: columns per lane
  static_assert(NC % CPL == 0, "columns split evenly over the lanes");
  static constexpr int LC = NC / CPL;                        // transposed: lanes per row part
  static constexpr int PT = ORD ? 1 : 32 / LC < 3 ? 32 / LC : (NPAIR % 3 == 0 ? 3 : 2);  // transposed: lanes per column
  static constexpr int JN = (NPAIR + PT - 1) / PT;           // row pairs per lane, transposed
  static constexpr bool ROT = !ORD && NPAIR % 2 == 0;        // stagger columns over the banks
  static_assert(!ROT || NPAIR % PT == 0, "staggered parts are even");
  static constexpr int XB = ((R * int(sizeof(typename AccOf<BT>::type)) + 15) / 16) * 16;
  static constexpr int PER = NS * CB + XB;                   // one warp: ring and x of its block
  static constexpr int YB = 4 * W * R * 8;                   // row sums of four rows
  // Rows claimed as teams come free (see the row queue in the kernel), where
  // the blocks are of several times the size of L2 (row_queue_bytes). us per
  // step with a fixed share of rows / claimed, 40,000 triangles: FP64 2Np = 56
  // 414 / 362, 72 773 / 634; FP32 56 245 / 228, 72 451 / 433, 90 721 / 560;
  // 120,000 triangles: FP64 56 1495 / 1164, 72 2632 / 2084, FP32 56 800 / 687,
  // 72 1396 / 1289. Smaller rows lose: FP64 30 115 / 157, 42 211 / 221, FP32
  // 42 118 / 118 (before FP32 sums went in column order).
  static constexpr bool QUEUE = R >= 56;
  static constexpr int LOOK = DEPTH + 2;
  static constexpr int CLAIM = LOOK + 4;
  static_assert(!QUEUE || CLAIM <= 8, "queue of 16 rows");
  static constexpr size_t smem_bytes() { return size_t(W) * (PER + NS * 8) + YB + W * 3 * 8 + 16 + (QUEUE ? 16 * 4 : 0); }
  static constexpr int fit() {
    const int n = int((228 * 1024) / (smem_bytes() + 1024));
    const int most = R <= 20 ? 7 : R == 30 ? 6 : R == 42 && !F64 ? 5 : 4;
    return n > most ? most : n;
  }
  static constexpr int CTAS = fit();  // per SM
};

__device__ __forceinline__ void lds_pair(const double* p, double& a, double& b) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  a = v.x;
  b = v.y;
}
__device__ __forceinline__ void lds_pair(const float* p, float& a, float& b) {
  const float2 v = *reinterpret_cast<const float2*>(p);
  a = v.x;
  b = v.y;
}

// Barrier 1 + id of the team (128 threads): wait there, or arrive and go on.
// Immediate identifiers: a barrier named by a register reserves all sixteen of
// the CTA, which halved the CTAs per SM.
template <int ID>
__device__ __forceinline__ void row_barrier_id(bool wait) {
  if (wait) asm volatile("bar.sync %0, 128;" ::"n"(1 + ID) : "memory");
  else asm volatile("bar.arrive %0, 128;" ::"n"(1 + ID) : "memory");
}
__device__ __forceinline__ void row_barrier(int id, bool wait) {
  if (id == 0) row_barrier_id<0>(wait);
  else if (id == 1) row_barrier_id<1>(wait);
  else if (id == 2) row_barrier_id<2>(wait);
  else row_barrier_id<3>(wait);
}

// ORD (FP32 operators): every row's FP32 products are summed in column order,
// block by block, as k_step_rows does: the results are the same to the bit
// whichever storage the handle has. The freer order of the FP64 operators
// (lane groups over columns, columns started at staggered row pairs) is up to
// 15 % faster with FP32 blocks too (160,000 triangles N = 6 924 us per step
// against 997), but its rounding errors are other ones, and seismograms came
// out up to twice as far from 64-bit products.
template <int R, typename BT>
__global__ void __launch_bounds__(128, RowRingCfg<R, BT>::CTAS) k_step_rowring(const StepParams p, int* err_flag) {
  typedef RowRingCfg<R, BT> CF;
  typedef typename AccOf<BT>::type AT;
  constexpr bool ORD = CF::ORD, ROT = CF::ROT;
  constexpr int G = CF::G, PT = CF::PT, JN = CF::JN;
  constexpr int NP = R / 2, NPAIR = CF::NPAIR, NC = CF::NC, NCH = CF::NCH, NS = CF::NS, PPL = CF::PPL, W = CF::W;
  constexpr int DEPTH = CF::DEPTH, LAP = CF::LAP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0);
  unsigned char* mine = smem_raw + warp * CF::PER;
  AT* xs = reinterpret_cast<AT*>(mine + NS * CF::CB);                           // [R] x of the warp's block
  double* ysum = reinterpret_cast<double*>(smem_raw + W * CF::PER);             // [4][W][R]
  double* red = ysum + 4 * W * R;                                               // [W][3]
  uint64_t* bars = reinterpret_cast<uint64_t*>(red + W * 3) + warp * NS;
  volatile int* abort_s = reinterpret_cast<volatile int*>(reinterpret_cast<uint64_t*>(red + W * 3) + W * NS);
  volatile int* rowq = abort_s + 4;  // [16]
  const uint32_t ring_a = smem_u32(mine), bar_a = smem_u32(bars);

  const int ne = p.ne, grid = int(gridDim.x);
  const RowRefs* rows = reinterpret_cast<const RowRefs*>(p.rows);

  // Row queue: the team's first CLAIM rows are blockIdx + k grid, the later
  // ones are claimed from a counter by the warp whose turn it is, CLAIM rows
  // ahead. The rows in work then stay close together over the whole chip; with
  // a fixed share the teams drift apart and the second use of a block misses
  // L2. Entry n is written by turn n - CLAIM and read from row n - LOOK = n -
  // CLAIM + 4 on, before which every warp has met that turn (its own turn lies
  // in between). It is written again at turn n + 16 - CLAIM, when all warps
  // have come past row n. Claims are made in turn, so once one of them is
  // behind the last row, all later ones are.
  if (CF::QUEUE && threadIdx.x < 16) {
    const long long r = (long long)blockIdx.x + (long long)threadIdx.x * grid;
    rowq[threadIdx.x] = int(threadIdx.x) < CF::CLAIM && r < ne ? int(r) : ne;
  }
  const bool claiming = CF::QUEUE && p.row_counter != nullptr && (long long)CF::CLAIM * grid < ne;
  // Row number n of the team, ne behind its last.
  auto row_at = [&](int n) {
    if constexpr (CF::QUEUE) return int(rowq[n & 15]);
    const long long r = (long long)blockIdx.x + (long long)n * grid;
    return r < ne ? int(r) : ne;
  };
  if (threadIdx.x == 0) *abort_s = 0;
  if (lane == 0) {
    for (int i = 0; i < NS; ++i) fx_mbar_init(bar_a + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The warp's block of row e: column and reference, -1 where there is none.
  auto entry = [&](int e, int& col, int& ref) {
    col = ref = -1;
    if (e < ne) {
      const int2 v = __ldg(reinterpret_cast<const int2*>(&rows[e].q[warp]));
      col = v.x;
      ref = v.y;
#ifdef TSP_CHECKED
      if (col >= 0) {
        col = TSP_INDEX(col, 0, ne, kSiteCol);
        ref = (TSP_INDEX(ref >> 1, 0, p.nphys, kSiteRow) << 1) | (ref & 1);
      }
#endif
    }
  };
  if constexpr (CF::QUEUE) __syncthreads();
  int col[DEPTH + 2], ref[DEPTH + 2];  // rows i .. i + DEPTH + 1 of this team
#pragma unroll
  for (int d = 0; d < DEPTH + 2; ++d) entry(row_at(d), col[d], ref[d]);
  if constexpr (!CF::QUEUE) __syncthreads();

  auto block_at = [&](int rf) {
    return reinterpret_cast<const unsigned char*>(p.blocks) + size_t(unsigned(rf) >> 1) * size_t(R * R * CF::SZ);
  };
  auto request = [&](const unsigned char* src, int slot) {  // lane 0
    fx_mbar_arrive_tx(bar_a + 8 * slot, CF::CB);
    fx_bulk_g2s(ring_a + slot * CF::CB, src, CF::CB, bar_a + 8 * slot);
  };
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
#pragma unroll
      for (int ch = 0; ch < (NCH < NS ? NCH : NS); ++ch)
        if (col[d] >= 0) request(block_at(ref[d]) + ch * CF::CB, d * NCH + ch);
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool off = *reinterpret_cast<volatile int*>(err_flag) != 0;  // an earlier launch of the run timed out

  const long long k = (p.step_base ? *p.step_base : 0) + p.rel;
  const bool stepping = p.mode == kModeStep || p.mode == kModeFirst;

  double2 xv[PPL];  // x of the next row's block, in flight while this row multiplies
  auto fetch_x = [&](int c) {
    const double2* src = reinterpret_cast<const double2*>(p.x + size_t(unsigned(c < 0 ? 0 : c)) * R) + lane;
#pragma unroll
    for (int s = 0; s < PPL; ++s)
      if (lane + 32 * s < NPAIR) xv[s] = src[32 * s];
  };
  // What the epilogue of a row needs, requested a row ahead by the warp whose turn it is.
  double2 uk[PPL], up[PPL];
  double mi = 1.0, dt = p.dt;
  int srow = -1, r0 = 0, r1 = 0, nb_e = 0;
  auto fetch_row = [&](int e) {
    const double2* src = reinterpret_cast<const double2*>(p.x + size_t(e) * R) + lane;
    const double2* prv = reinterpret_cast<const double2*>(p.uprev + size_t(e) * R) + lane;
#pragma unroll
    for (int s = 0; s < PPL; ++s) {
      uk[s] = up[s] = make_double2(0.0, 0.0);
      if (lane + 32 * s < NPAIR) {
        uk[s] = src[32 * s];
        if (stepping && p.uprev != nullptr) up[s] = prv[32 * s];
      }
    }
    nb_e = TSP_INDEX(p.row_ptr[e + 1] - p.row_ptr[e], 1, 5, kSiteRow);
    mi = p.minv[e];
    if (p.dt_elem) dt = p.dt_elem[e];
    if (stepping) {
      srow = p.src_of ? p.src_of[e] : ((p.src_elem != nullptr && src_elem_at(p, 0) == e) ? 0 : -1);
      if (p.rcv_ptr != nullptr) {
        r0 = rcv_ptr_at(p, e);
        r1 = rcv_ptr_at(p, e + 1);
      }
    }
  };
  const double xsc_all = p.mode == kModePower && p.mesh_of == nullptr ? power_scale(p, 0) : 1.0;
  int e = row_at(0);
#pragma unroll
  for (int s = 0; s < PPL; ++s) xv[s] = make_double2(0.0, 0.0);
  if (e < ne && !off) {
    fetch_x(col[0]);
    if (warp == 0) fetch_row(e);
  }

  double en = 0.0, en2 = 0.0, en3 = 0.0;
  double chk = 0.0;  // NaN once a non-finite u^{k+1} was written (inf * 0 and NaN * 0 are NaN)
  uint32_t phase = 0;  // bit d: phase of the slots that rows i = d (mod DEPTH) use
  bool dead = off;
  int i = 0;
  for (; e < ne && !off; e = row_at(++i)) {
    const int d = DEPTH > 1 ? i % DEPTH : 0;
    double xsc = 1.0;
    if (p.mode == kModePower) {
      xsc = p.mesh_of != nullptr ? power_scale(p, e) : xsc_all;
#pragma unroll
      for (int s = 0; s < PPL; ++s) {
        xv[s].x *= xsc;
        xv[s].y *= xsc;
      }
    }
#pragma unroll
    for (int s = 0; s < PPL; ++s) {
      const int q = lane + 32 * s;
      if (q < NPAIR) {
        xs[2 * q] = AT(xv[s].x);
        xs[2 * q + 1] = AT(xv[s].y);
      }
    }
    __syncwarp();
    fetch_x(col[1]);
    int col_l, ref_l;
    entry(row_at(i + CF::LOOK), col_l, ref_l);

    double* y = ysum + ((i & 3) * W + warp) * R;
    const int cur = col[0], cref = ref[0];
    // Chunk ch is consumed: its slot takes the chunk NS further on (none if
    // that row has no such block).
    const unsigned char* here = block_at(cref);
    const unsigned char* next = block_at(ref[DEPTH]);
    const bool more = col[DEPTH] >= 0;
    auto refill = [&](int ch) {
      fx_reads_done();
      __syncwarp();
      if (lane == 0 && !dead) {
        if constexpr (NS < NCH) {
          if (ch + NS < NCH) request(here + (ch + NS) * CF::CB, ch % NS);
          else if (more) request(next + (ch + NS - NCH) * CF::CB, ch % NS);
        } else {
          if (more) request(next + ch * CF::CB, d * NCH + ch);
        }
      }
    };
    // Waits for chunk ch. After a wait gave up nothing is waited for or
    // requested any more and the products run on what the ring holds: the
    // results are void, the loops and barriers stay balanced.
    auto land = [&](int ch) {
      const int slot = NS < NCH ? ch % NS : d * NCH + ch;
      const uint32_t ph = ((phase >> d) + uint32_t(NS < NCH ? ch / NS : 0)) & 1;
      if (!__all_sync(0xffffffffu, mbar_try(bar_a + 8 * slot, ph)) && !dead)
        dead = !__all_sync(0xffffffffu, fx_wait(bar_a + 8 * slot, ph, abort_s));
      return reinterpret_cast<const BT*>(mine + slot * CF::CB);
    };
    if (cur < 0) {
      for (int ch = NS < NCH ? NCH - NS : 0; ch < NCH; ++ch) refill(ch);
    } else if (!(cref & 1)) {
      AT acc[PPL][2];
#pragma unroll
      for (int q = 0; q < PPL; ++q) acc[q][0] = acc[q][1] = AT(0);
      const int g = G > 1 ? lane / NPAIR : 0;
      const int pl = G > 1 ? lane - g * NPAIR : lane;
#pragma unroll 1
      for (int ch = 0; ch < NCH; ++ch) {
        const BT* st = land(ch) + 2 * pl;
        const AT* xc = xs + ch * NC;
        if constexpr (G > 1) {
          constexpr int CI = (NC + G - 1) / G;  // columns per group
          constexpr int UN = CI % 7 == 0 ? 7 : CI % 5 == 0 ? 5 : 6;
          if (g < G) {
#pragma unroll UN
            for (int ci = 0; ci < CI; ++ci) {
              const int cc = g + ci * G;
              if (NC % G == 0 || cc < NC) {
                AT w0, w1;
                lds_pair(st + cc * R, w0, w1);
                acc[0][0] = fma(w0, xc[cc], acc[0][0]);
                acc[0][1] = fma(w1, xc[cc], acc[0][1]);
              }
            }
          }
        } else {
          // Two columns per step: one load brings both x.
          static_assert(G > 1 || NC % 2 == 0, "column pairs");
          constexpr int UN = NC % 14 == 0 ? 7 : NC % 10 == 0 ? 5 : NC % 8 == 0 ? 4 : 3;
#pragma unroll UN
          for (int cc = 0; cc < NC; cc += 2) {
            AT x0, x1;
            lds_pair(xc + cc, x0, x1);
#pragma unroll
            for (int q = 0; q < PPL; ++q) {
              if (32 * (q + 1) <= NPAIR || lane + 32 * q < NPAIR) {
                AT w0, w1, z0, z1;
                lds_pair(st + cc * R + 64 * q, w0, w1);
                lds_pair(st + cc * R + R + 64 * q, z0, z1);
                acc[q][0] = fma(w0, x0, acc[q][0]);
                acc[q][1] = fma(w1, x0, acc[q][1]);
                acc[q][0] = fma(z0, x1, acc[q][0]);
                acc[q][1] = fma(z1, x1, acc[q][1]);
              }
            }
          }
        }
        refill(ch);
      }
#pragma unroll
      for (int q = 0; q < PPL; ++q) {
        double v0 = double(acc[q][0]), v1 = double(acc[q][1]);
        if constexpr (G > 1) {
          double t0 = v0, t1 = v1;
#pragma unroll
          for (int gg = 1; gg < G; ++gg) {
            t0 += __shfl_sync(0xffffffffu, v0, (pl + gg * NPAIR) & 31);
            t1 += __shfl_sync(0xffffffffu, v1, (pl + gg * NPAIR) & 31);
          }
          v0 = t0;
          v1 = t1;
        }
        const int pr = pl + 32 * q;
        if (g == 0 && pr < NPAIR) *reinterpret_cast<double2*>(y + 2 * pr) = make_double2(v0, v1);
      }
    } else {
      const int pt = lane / CF::LC, lc = lane - pt * CF::LC;
      const bool work = pt < PT;
      const int jb = work ? pt * JN : 0;
      const int len = NPAIR % PT == 0 ? JN : (NPAIR - jb < JN ? NPAIR - jb : JN);
#pragma unroll 1
      for (int ch = 0; ch < NCH; ++ch) {
        const BT* st = land(ch) + (work ? lc : 0) * R + 2 * jb;
        const AT* xc = xs + 2 * jb;
        AT s0[CF::CPL], s1[CF::CPL];
#pragma unroll
        for (int c = 0; c < CF::CPL; ++c) s0[c] = s1[c] = AT(0);
        int jj = ROT ? lc % JN : 0;
#pragma unroll 7
        for (int t = 0; t < JN; ++t) {
          const int o = ROT ? 2 * jj : 2 * t;
          if (NPAIR % PT == 0 || t < len) {
            AT x0, x1;
            lds_pair(xc + o, x0, x1);
#pragma unroll
            for (int c = 0; c < CF::CPL; ++c) {
              AT w0, w1;
              lds_pair(st + c * CF::LC * R + o, w0, w1);
              s0[c] = fma(w0, x0, s0[c]);
              if constexpr (ORD) s0[c] = fma(w1, x1, s0[c]);
              else s1[c] = fma(w1, x1, s1[c]);
            }
          }
          if (ROT) jj = jj + 1 == JN ? 0 : jj + 1;
        }
#pragma unroll
        for (int c = 0; c < CF::CPL; ++c) {
          const double v = double(s0[c]) + double(s1[c]);
          double tot = v;
#pragma unroll
          for (int q = 1; q < PT; ++q) tot += __shfl_sync(0xffffffffu, v, (lc + q * CF::LC) & 31);
          if (pt == 0) y[ch * NC + lc + c * CF::LC] = tot;
        }
        refill(ch);
      }
    }
    if (cur >= 0) phase ^= uint32_t(LAP & 1) << d;

    // Barrier 1 + i mod 4: the warp whose turn the epilogue is waits for the
    // other three, which go on. A warp writes a buffer (and arrives at a
    // barrier) again four rows later, after a turn of its own in between, at
    // which the buffer's reader had come past that epilogue.
    const bool turn = warp == (i & (W - 1));
    row_barrier(i & 3, turn);
    if (turn) {
      int claimed = ne;
      if (claiming && lane == 0) claimed = atomicAdd(p.row_counter, 1);
      // ---- epilogue: inverse mass, leap-frog, source ----
      double* yr = ysum + (i & 3) * W * R;
      const bool is_src = srow >= 0 && k < p.nF;
      double F0 = 0.0, F1 = 0.0;
      if (is_src) {
        F0 = p.F[(size_t(srow) * p.nF + k) * 2];
        F1 = p.F[(size_t(srow) * p.nF + k) * 2 + 1];
      }
      const bool listen = r1 > r0;
      double2 un2[PPL];
#pragma unroll
      for (int s = 0; s < PPL; ++s) {
        const int q = lane + 32 * s;
        un2[s] = make_double2(0.0, 0.0);
        if (q >= NPAIR) continue;
        typename std::conditional<ORD, AT, double>::type ya = 0, yb = 0;
        for (int b = 0; b < nb_e; ++b) {
          const double2 v = *reinterpret_cast<const double2*>(yr + b * R + 2 * q);
          ya += decltype(ya)(v.x);
          yb += decltype(yb)(v.y);
        }
        const double yy[2] = {double(ya), double(yb)};
        double u[2] = {uk[s].x, uk[s].y};
        if (p.mode == kModePower) {
          u[0] *= xsc;
          u[1] *= xsc;
        }
        const double upr[2] = {up[s].x, up[s].y};
        double un[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = 2 * q + h;
          const int cmp = r / NP, ii = r - cmp * NP;
          const double f = is_src ? (cmp ? F1 : F0) * p.src_phi[size_t(srow) * NP + ii] : 0.0;
          if (p.mode == kModeStep) un[h] = (2 * u[h] - upr[h]) + mi * ((-dt * dt) * (yy[h] - f));
          else if (p.mode == kModeFirst) un[h] = (u[h] + dt * upr[h]) - mi * (dt * dt / 2 * (yy[h] - f));
          else if (p.mode == kModeApply) un[h] = yy[h];
          else {  // kModePower
            un[h] = mi * yy[h];
            en += u[h] * yy[h];
            en2 += u[h] * u[h] / mi;
            en3 += un[h] * un[h];
          }
          if (stepping) chk = __fma_rn(un[h], 0.0, chk);
          if (p.energy != nullptr) {
            const double dd = un[h] - u[h];
            en += 0.5 * (dd * dd) / (mi * dt * dt) + 0.5 * un[h] * yy[h];
          }
        }
        un2[s] = make_double2(un[0], un[1]);
        *(reinterpret_cast<double2*>(p.out + size_t(e) * R) + q) = un2[s];
      }
      // ---- receivers: sample the new level of this element ----
      if (listen) {
        double* yw = yr;  // this row's sums are read: the buffer takes u^{k+1}
        __syncwarp();
#pragma unroll
        for (int s = 0; s < PPL; ++s) {
          const int q = lane + 32 * s;
          if (q < NPAIR) *reinterpret_cast<double2*>(yw + 2 * q) = un2[s];
        }
        __syncwarp();
        // Rounds that leave the registers of the products alone (2Np = 20 with
        // rounds of 5: 40,000 triangles 78.5 us per step instead of 76.7).
        constexpr int UN = NP == 45 ? 15 : NP == 36 ? 12 : NP % 7 == 0 ? 7 : NP == 10 ? 2 : 5;
        sample_receivers<NP, UN>(p, r0, r1, k, 0, lane, [](int) { return 0; },
                             [&](int, int c, int i) { return yw[c * NP + i]; });
      }
      // ---- per-mesh power-iteration sums (multi-mesh groups) ----
      if (p.mode == kModePower && p.mesh_of != nullptr) {
        const double a0 = warp_sum(en), a1 = warp_sum(en2), a2 = warp_sum(en3);
        en = en2 = en3 = 0.0;
        if (lane == 0) {
          double* acc3 = p.acc + 3 * size_t(p.mesh_of[e]);
          atomicAdd(acc3 + 0, a0);
          atomicAdd(acc3 + 1, a1);
          atomicAdd(acc3 + 2, a2);
        }
      }
      if (CF::QUEUE && lane == 0) {
        long long r = (long long)CF::CLAIM * grid + claimed;
        if (!claiming) r = (long long)blockIdx.x + (long long)(i + CF::CLAIM) * grid;
        rowq[(i + CF::CLAIM) & 15] = r < ne ? int(r) : ne;
      }
    }
    if (warp == ((i + 1) & (W - 1))) {
      const int en = row_at(i + 1);
      if (en < ne) fetch_row(en);
    }
#pragma unroll
    for (int t = 0; t < DEPTH + 1; ++t) {
      col[t] = col[t + 1];
      ref[t] = ref[t + 1];
    }
    col[DEPTH + 1] = col_l;
    ref[DEPTH + 1] = ref_l;
  }
  if (chk != chk && p.nonfinite != nullptr) *p.nonfinite = 1;
  // Every chunk that was requested has been consumed, unless this launch was
  // off or a wait gave up: then the copies in flight land first (bounded).
  if (dead && lane == 0) {
    const long long t0 = clock64();
    if (off) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d)
        for (int ch = 0; ch < (NCH < NS ? NCH : NS); ++ch)
          while (col[d] >= 0 && !mbar_try(bar_a + 8 * (d * NCH + ch), 0) && clock64() - t0 < (1ll << 31)) {
          }
    } else {
      while (clock64() - t0 < (1ll << 24)) {
      }
    }
  }
  const bool summing = (p.mode == kModePower && p.mesh_of == nullptr) || p.energy != nullptr;
  if (summing) {
    const double a0 = warp_sum(en), a1 = warp_sum(en2), a2 = warp_sum(en3);
    if (lane == 0) {
      red[warp * 3] = a0;
      red[warp * 3 + 1] = a1;
      red[warp * 3 + 2] = a2;
    }
  }
  __syncthreads();
  const int nred = p.mode == kModePower ? 3 : 1;
  if (summing && int(threadIdx.x) < nred) {
    double t = 0.0;
    for (int w = 0; w < W; ++w) t += red[w * 3 + threadIdx.x];
    if (p.mode == kModePower) atomicAdd(p.acc + threadIdx.x, t);
    else atomicAdd(p.energy + (k % p.energy_cap), t);
  }
  if (threadIdx.x == 0) {
    if (*abort_s) atomicExch(err_flag, 1);
    // The last team to end clears the counters for the next launch.
    if (claiming && atomicAdd(p.row_counter + 1, 1) == grid - 1) {
      p.row_counter[0] = 0;
      p.row_counter[1] = 0;
    }
  }
}

}  // namespace tsp
