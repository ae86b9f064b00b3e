// FP64 block-sparse contraction in one launch: gather, GEMM, scatter.
//
// C[out block] = sum over the matching (A block, B block) pairs, every output
// block cut into BM x BN tiles.  A CTA gathers its operand tiles straight from
// the operands' blocks (8-byte cp.async through per-block row and K axes: an
// affine stride or an offset table, so any leg order and extent is read in
// place) into a 4-stage shared-memory ring, multiplies on the FP64 tensor
// cores (mma.sync m8n8k4) and stores straight into the output block.
//
// What bounds it: the FP64 tensor pipe, 36.5 TFLOP/s measured (64 FMA per
// clock and SM).  A 64 x 64 x 16 step takes 1024 clocks of it and loads 16 KB,
// which an SM fetches in about 256 clocks, so gathering element by element
// costs less than a packed copy of each operand and of the result would: the
// packed path moved every operand three times (clear, write, read) and the
// result four times.  DMMAs are issued for valid 8-row and 8-column fragments
// and 4-deep K steps only; fragments are dealt to the warps cyclically so that
// a ragged tile keeps all four tensor pipes busy.
//
// Shapes with few output tiles and a long K (CTM projections: 80 x 80 x 1280)
// split K over the CTAs of one cluster, which add their partial tiles through
// distributed shared memory in rank order: no workspace, no atomics, and the
// same bits on every run.  A K too long for eight CTAs (the last product of a
// two-site density matrix: 4 x 4 x 102400, 1200 us with a cluster alone, 33 us)
// takes several clusters a tile, whose parts a second launch adds in order.
//
// Measured, CUDA events: 80 x 80 x 1280 76 us unsplit, 10.5 us; 1280 x 1280 x
// 80 18.8 us (14 TFLOP/s); 6400 x 1024 x 256 131 us (26 TFLOP/s); 4096^3 4.35
// ms (31.6 TFLOP/s; the packed path's GEMM alone 4.15 ms).  Below about a
// thousand tiles the last wave and one or two CTAs an SM are what is lost.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "contract_f64.hpp"
#include "kernels.cuh"

namespace tnx {

namespace {
constexpr int BK = 16;
constexpr int STAGES = 4;
constexpr int kSmemSpans = 32;  // span records kept in shared memory; the rest are read from global

__device__ __forceinline__ int64_t axis_off(const int32_t* __restrict__ tab, int32_t t, int32_t str, int i) {
  return t < 0 ? static_cast<int64_t>(i) * str : __ldg(tab + t + i);
}

// Asynchronous copies of 8 or 16 bytes, of which the first `bytes` are read and
// the rest is zero.  No memory clobber: they fill a stage that no fragment load
// touches before the next barrier, so the two may be interleaved.
__device__ __forceinline__ void cp8(uint32_t dst, const double* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp16(uint32_t dst, const double* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ double ld_peer(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

// One operand's tile of R rows x 16 K.  KF: K is the operand's fast axis; the
// tile is stored row-major with the XOR swizzle that spreads the fragment
// loads over all banks, and 16 lanes fetch one row's 16 consecutive K.
// Otherwise rows are the fast axis: the tile is stored K-major with a row
// pitch of R + 4 (bank-free fragment loads), consecutive lanes fetch
// consecutive rows.  VEC: elements 2i and 2i + 1 of the fast axis are adjacent
// and every pair starts on 16 bytes, so a lane fetches a pair: the copies' issue
// is what holds the tensor pipe below its rate.
template <int R, bool KF, bool VEC, int THREADS>
struct Operand {
  static constexpr int W = VEC ? 2 : 1;                         // elements a copy
  static constexpr int kPer = R * BK / W / THREADS;             // copies per thread and K tile
  static constexpr int kLanes = (KF ? BK : R) / W;              // lanes along the fast axis
  static constexpr int kRows = KF ? kPer : 1;                   // distinct rows per thread
  static constexpr int kTile = KF ? R * BK : BK * (R + 4);      // doubles per stage
  static_assert(kPer >= 1 && THREADS % kLanes == 0, "whole copies");
  const double* base;  // affine axes: the tile's own origin, so that 32-bit offsets span one tile
  int32_t kt, ks;
  int32_t rbytes;      // rows fast: bytes of this lane's copy that lie inside the block
  int32_t off[kRows];

  __device__ __forceinline__ void set_span(const double* p, const int32_t* tab, int32_t rt, int32_t rs, int32_t kt_,
                                           int32_t ks_, int row0, int rows) {
    base = rt < 0 ? p + static_cast<int64_t>(row0) * rs : p;
    kt = kt_;
    ks = ks_;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int r = KF ? static_cast<int>(threadIdx.x) / kLanes + THREADS / kLanes * i
                       : static_cast<int>(threadIdx.x) % kLanes * W;
      off[i] = r < rows ? (rt < 0 ? r * rs : __ldg(tab + rt + row0 + r)) : -1;  // -1: past the block, not loaded
      if (!KF) rbytes = 8 * min(W, rows - r);
    }
  }
  // TAB: the K axis is a table (several legs that do not merge), else a stride
  template <bool TAB>
  __device__ __forceinline__ void load_as(double* s, const int32_t* tab, int k0, int K) const {
    const double* b0 = TAB ? base : base + static_cast<int64_t>(k0) * ks;
    if constexpr (KF) {
      const int kk = static_cast<int>(threadIdx.x) % kLanes * W, r0 = static_cast<int>(threadIdx.x) / kLanes;
      const int bytes = 8 * max(0, min(W, K - k0 - kk));
      const double* p = b0 + (bytes ? (TAB ? __ldg(tab + kt + k0 + kk) : kk * ks) : 0);
      const uint32_t d = smem_u32(s) + 8 * (r0 * BK + (kk ^ ((r0 & 3) << 2)));
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        // rows r0 + i * THREADS / kLanes: a multiple of 4 apart, so one swizzle
        static_assert(THREADS / kLanes % 4 == 0, "rows of a thread share their swizzle");
        if (off[i] < 0) continue;
        if constexpr (VEC)
          cp16(d + 8 * i * (THREADS / kLanes) * BK, p + off[i], bytes);
        else
          cp8(d + 8 * i * (THREADS / kLanes) * BK, p + off[i], bytes);
      }
    } else {
      const int r = static_cast<int>(threadIdx.x) % kLanes * W, q = static_cast<int>(threadIdx.x) / kLanes;
      if (off[0] < 0) return;
      const double* p = b0 + off[0];
      const uint32_t d = smem_u32(s) + 8 * (q * (R + 4) + r);
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int kk = q + i * (THREADS / kLanes);
        const bool ok = k0 + kk < K;
        const int ko = ok ? (TAB ? __ldg(tab + kt + k0 + kk) : kk * ks) : 0;
        if constexpr (VEC)
          cp16(d + 8 * i * (THREADS / kLanes) * (R + 4), p + ko, ok ? rbytes : 0);
        else
          cp8(d + 8 * i * (THREADS / kLanes) * (R + 4), p + ko, ok ? 8 : 0);
      }
    }
  }
  __device__ __forceinline__ void load(double* s, const int32_t* tab, int k0, int K) const {
    if (kt < 0)
      load_as<false>(s, tab, k0, K);
    else
      load_as<true>(s, tab, k0, K);
  }
  static __device__ __forceinline__ double frag(const double* s, int r, int kk) {
    return KF ? s[r * BK + (kk ^ ((r & 3) << 2))] : s[kk * (R + 4) + r];
  }
};

// One 4-deep K step of a warp with MV x NV valid fragments.  The counts are
// compile-time: guarding each DMMA at run time cost 10 issued instructions per
// DMMA against 4 and held the 6400 x 256 x 1024 product at 53 % of the pipe.
template <int MV, int NV, int WM, int WN, class OpA, class OpB, int MI, int NI>
__device__ __forceinline__ void products(double (&acc)[MI][NI][2], const double* as, const double* bs, int wm, int wn,
                                         int lane, int k4) {
  {
    const int kk = k4 * 4 + (lane & 3);
    double af[MV], bf[NV];
#pragma unroll
    for (int i = 0; i < MV; ++i) af[i] = OpA::frag(as, (i * WM + wm) * 8 + (lane >> 2), kk);
#pragma unroll
    for (int j = 0; j < NV; ++j) bf[j] = OpB::frag(bs, (j * WN + wn) * 8 + (lane >> 2), kk);
#pragma unroll
    for (int i = 0; i < MV; ++i)
#pragma unroll
      for (int j = 0; j < NV; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
  }
}
template <int MV, int WM, int WN, class OpA, class OpB, int MI, int NI>
__device__ __forceinline__ void products_n(double (&acc)[MI][NI][2], const double* as, const double* bs, int wm,
                                           int wn, int lane, int nv, int n4) {
  if constexpr (MV <= MI) {
    for (int k4 = 0; k4 < n4; ++k4) {
      if (nv == 1) products<MV, 1, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, k4);
      if constexpr (NI >= 2)
        if (nv == 2) products<MV, 2, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, k4);
      if constexpr (NI >= 4) {
        if (nv == 3) products<MV, 3, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, k4);
        if (nv == 4) products<MV, 4, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, k4);
      }
    }
  }
}

template <int BM, int BN, bool AK, bool BKF>
constexpr int smem_doubles() {
  constexpr int ring = STAGES * (Operand<BM, AK, false, 128>::kTile + Operand<BN, BKF, false, 128>::kTile);
  constexpr int part = BM * (BN + 1);  // a split's partial tile reuses the ring
  return ring > part ? ring : part;
}

template <int BM, int BN, int WM, int WN, bool AK, bool BKF, bool AV, bool BV>
__global__ void __launch_bounds__(32 * WM * WN, (BM * BN >= 4096) ? 3 : 4)
    contract_f64_kernel(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C,
                        const ContractTile* __restrict__ tiles, const ContractSpan* __restrict__ spans,
                        const int32_t* __restrict__ tab, int split, int parts, double* __restrict__ ws,
                        const uint64_t* __restrict__ a_ptrs, const uint64_t* __restrict__ b_ptrs,
                        const uint64_t* __restrict__ c_ptrs, const int32_t* __restrict__ skip_flag) {
  constexpr int THREADS = 32 * WM * WN;
  pdl_trigger();
  constexpr int MI = BM / 8 / WM, NI = BN / 8 / WN;
  using OpA = Operand<BM, AK, AV, THREADS>;
  using OpB = Operand<BN, BKF, BV, THREADS>;
  extern __shared__ __align__(16) double ring[];
  __shared__ ContractSpan sspan[kSmemSpans];
  double* As = ring;
  double* Bs = ring + STAGES * OpA::kTile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp / WN, wn = warp % WN;
  const int rank = static_cast<int>(blockIdx.x) % split, part = static_cast<int>(blockIdx.x) / split % parts;
  const ContractTile t = tiles[blockIdx.x / (split * parts)];
  for (int i = tid; i < t.nspan * 4 && i < kSmemSpans * 4; i += THREADS)
    reinterpret_cast<int4*>(sspan)[i] = __ldg(reinterpret_cast<const int4*>(spans + t.span0) + i);
  pdl_wait();  // the tables are the plan's; operands, pointers and the skip flag are not
  if (skip_flag && *skip_flag) return;  // the whole cluster
  __syncthreads();
  const int rows = min(BM, t.M - t.m0), cols = min(BN, t.N - t.n0);
  // this CTA's K tiles: an even share of the output tile's
  const int share = part * split + rank, shares = split * parts;
  const int kt0 = static_cast<int>(static_cast<int64_t>(t.ktiles) * share / shares);
  const int nkt = static_cast<int>(static_cast<int64_t>(t.ktiles) * (share + 1) / shares) - kt0;
  // valid fragments of this warp, dealt cyclically
  const int mv = ((rows + 7) / 8 - wm + WM - 1) / WM, nv = ((cols + 7) / 8 - wn + WN - 1) / WN;

  double acc[MI][NI][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  OpA oa;
  OpB ob;
  int sp = 0, k0 = 0, K = 0;
  bool fresh = true;
  if (nkt > 0) {
    int skip = kt0;
    for (;; ++sp) {
      const int n = ((sp < kSmemSpans ? sspan[sp].K : spans[t.span0 + sp].K) + BK - 1) / BK;
      if (skip < n) break;
      skip -= n;
    }
    k0 = skip * BK;
  }
  uint32_t steps = 0;  // 4-deep K steps of each stage, one byte a stage
  // the next K tile's span, before its loads; then past it, after them
  auto begin = [&](int s) {
    if (fresh) {
      const ContractSpan g = sp < kSmemSpans ? sspan[sp] : spans[t.span0 + sp];
      K = g.K;
      const double* pa = a_ptrs ? reinterpret_cast<const double*>(a_ptrs[g.a_slot]) : A;
      const double* pb = b_ptrs ? reinterpret_cast<const double*>(b_ptrs[g.b_slot]) : B;
      oa.set_span(pa + g.a_off, tab, g.ar_tab, g.ar_str, g.ak_tab, g.ak_str, t.m0, rows);
      ob.set_span(pb + g.b_off, tab, g.br_tab, g.br_str, g.bk_tab, g.bk_str, t.n0, cols);
      fresh = false;
    }
    const uint32_t n4 = static_cast<uint32_t>((min(BK, K - k0) + 3) / 4);
    steps = (steps & ~(0xffu << (8 * s))) | (n4 << (8 * s));
  };
  auto finish = [&]() {
    k0 += BK;
    if (k0 >= K) {
      k0 = 0;
      ++sp;
      fresh = true;
    }
  };
  auto issue = [&](int s) {
    begin(s);
    oa.load(As + s * OpA::kTile, tab, k0, K);
    ob.load(Bs + s * OpB::kTile, tab, k0, K);
    finish();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nkt) issue(s);
    cp_commit();
  }
  for (int kt = 0; kt < nkt; ++kt) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int s = kt % STAGES, sn = (kt + STAGES - 1) % STAGES;
    const int n4 = static_cast<int>((steps >> (8 * s)) & 0xffu);
    const bool more = kt + STAGES - 1 < nkt;
    const double* as = As + s * OpA::kTile;
    const double* bs = Bs + s * OpB::kTile;
    if (more) issue(sn);
    cp_commit();
    if (mv == MI && nv == NI && n4 == BK / 4) {
#pragma unroll
      for (int k4 = 0; k4 < BK / 4; ++k4) products<MI, NI, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, k4);
    } else {
      switch (mv) {
        case 1: products_n<1, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, nv, n4); break;
        case 2: products_n<2, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, nv, n4); break;
        case 3: products_n<3, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, nv, n4); break;
        case 4: products_n<4, WM, WN, OpA, OpB>(acc, as, bs, wm, wn, lane, nv, n4); break;
        default: break;  // no valid row fragment
      }
    }
  }
  cp_wait<0>();
  double* out = (c_ptrs ? reinterpret_cast<double*>(c_ptrs[t.out_slot]) : C) + t.out_off;
  if (split == 1) {
    int64_t co[NI][2];
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        co[j][h] = axis_off(tab, t.c_tab, t.c_str, t.n0 + min(cols - 1, (j * WN + wn) * 8 + (lane & 3) * 2 + h));
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int r = (i * WM + wm) * 8 + (lane >> 2);
      if (r >= rows) continue;
      double* row = out + axis_off(tab, t.r_tab, t.r_str, t.m0 + r);
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const int c = (j * WN + wn) * 8 + (lane & 3) * 2;
        if (c < cols) row[co[j][0]] = acc[i][j][0] * t.scale;
        if (c + 1 < cols) row[co[j][1]] = acc[i][j][1] * t.scale;
      }
    }
    return;
  }
  // split K: partial tiles through distributed shared memory, added in rank
  // order; each CTA finishes every split-th row
  __syncthreads();
  constexpr int P = BN + 1;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = (i * WM + wm) * 8 + (lane >> 2);
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int c = (j * WN + wn) * 8 + (lane & 3) * 2;
      ring[r * P + c] = acc[i][j][0];
      ring[r * P + c + 1] = acc[i][j][1];
    }
  }
  cluster_sync();
  const int mine = (rows - rank + split - 1) / split;  // rows rank, rank + split, ...
  const bool rfast = t.c_str != 1 && t.r_str == 1;     // lanes along whichever axis the output has contiguous
  double* wpart = parts > 1 ? ws + static_cast<int64_t>(blockIdx.x / split) * (BM * BN) : nullptr;
  for (int e = tid; e < mine * cols; e += THREADS) {
    const int q = rfast ? e % mine : e / cols;
    const int c = rfast ? e / mine : e - q * cols;
    const int r = rank + q * split;
    const uint32_t sa = smem_u32(ring + r * P + c);
    double v = ld_peer(sa, 0);
    for (int p = 1; p < split; ++p) v += ld_peer(sa, p);
    if (parts > 1)
      wpart[r * BN + c] = v;
    else
      out[axis_off(tab, t.r_tab, t.r_str, t.m0 + r) + axis_off(tab, t.c_tab, t.c_str, t.n0 + c)] = v * t.scale;
  }
  cluster_sync();  // no CTA leaves while a peer reads its shared memory
}

// The parts of every output tile added in order (a K too long for one cluster).
__global__ void __launch_bounds__(256)
    contract_parts_kernel(const double* __restrict__ ws, double* __restrict__ C, const ContractTile* __restrict__ tiles,
                          const int32_t* __restrict__ tab, int parts, int bm, int bn) {
  const ContractTile t = tiles[blockIdx.x];
  const int rows = min(bm, t.M - t.m0), cols = min(bn, t.N - t.n0);
  const double* w = ws + static_cast<int64_t>(blockIdx.x) * parts * bm * bn;
  for (int e = blockIdx.y * 256 + threadIdx.x; e < rows * cols; e += gridDim.y * 256) {
    const int r = e / cols, c = e - r * cols;
    double v = 0.0;
    for (int p = 0; p < parts; ++p) v += w[static_cast<int64_t>(p) * bm * bn + r * bn + c];
    C[t.out_off + axis_off(tab, t.r_tab, t.r_str, t.m0 + r) + axis_off(tab, t.c_tab, t.c_str, t.n0 + c)] = v * t.scale;
  }
}

template <int BM, int BN, int WM, int WN, bool AK, bool BKF, bool AV, bool BV>
cudaError_t go(const ContractLaunch& L, cudaStream_t st) {
  constexpr int smem = smem_doubles<BM, BN, AK, BKF>() * static_cast<int>(sizeof(double));
  auto kernel = contract_f64_kernel<BM, BN, WM, WN, AK, BKF, AV, BV>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  double* ws = nullptr;
  if (L.parts > 1) {
    // partial tiles of this call, from the stream-ordered pool: safe with any
    // number of streams and threads, returned as soon as the sum is queued
    e = cudaMallocAsync(&ws, sizeof(double) * BM * BN * static_cast<size_t>(L.n_tiles) * L.parts, st);
    if (e != cudaSuccess) return e;
  }
  // a tile is a few us: the launch overlap still shows at 10^4 tiles (an
  // environment update's three steps, chi = 512: 93 us without it, 85 with)
  e = launch_pdl(kernel, static_cast<unsigned>(L.n_tiles) * L.split * L.parts, 32 * WM * WN, smem, st, L.split,
                 L.n_tiles / 16, L.a, L.b, L.c, L.tiles, L.spans, L.tab, L.split, L.parts, ws, L.a_ptrs, L.b_ptrs, L.c_ptrs, L.skip);
  if (L.parts > 1) {
    if (e == cudaSuccess) {
      contract_parts_kernel<<<dim3(L.n_tiles, (BM * BN + 255) / 256), 256, 0, st>>>(ws, L.c, L.tiles, L.tab, L.parts,
                                                                                  BM, BN);
      e = cudaGetLastError();
    }
    const cudaError_t f = cudaFreeAsync(ws, st);
    if (e == cudaSuccess) e = f;
  }
  return e;
}

// 16-byte copies of A alone or of both operands (a step where only B could
// have them reads both by 8 bytes)
template <int BM, int BN, int WM, int WN, bool AK, bool BKF>
cudaError_t go_vec(const ContractLaunch& L, cudaStream_t st) {
  const bool av = L.a_vec && reinterpret_cast<uintptr_t>(L.a) % 16 == 0;
  const bool bv = L.b_vec && reinterpret_cast<uintptr_t>(L.b) % 16 == 0;
  if (av && bv) return go<BM, BN, WM, WN, AK, BKF, true, true>(L, st);
  if (av) return go<BM, BN, WM, WN, AK, BKF, true, false>(L, st);
  return go<BM, BN, WM, WN, AK, BKF, false, false>(L, st);
}
template <int BM, int BN, int WM, int WN>
cudaError_t go_layout(const ContractLaunch& L, cudaStream_t st) {
  if (L.a_kfast)
    return L.b_kfast ? go_vec<BM, BN, WM, WN, true, true>(L, st) : go_vec<BM, BN, WM, WN, true, false>(L, st);
  return L.b_kfast ? go_vec<BM, BN, WM, WN, false, true>(L, st) : go_vec<BM, BN, WM, WN, false, false>(L, st);
}

struct Shape {
  int bm, bn, wm, wn, resident;
  double eff;  // tensor-pipe rate against 64 x 64 tiles (2000^3: 29.1, 25.4, 21.8, 26.7 TFLOP/s)
};
// 64 x 64: the DMMA-bound shape; 64 x 32 and 32 x 32: few tiles or small
// blocks; 128 x 16: narrow column blocks (an MPO leg), whose rows are many
constexpr Shape kShapes[kContractShapes] = {
    {64, 64, 2, 2, 3, 1.0}, {32, 32, 2, 2, 4, 0.87}, {128, 16, 4, 1, 3, 0.75}, {64, 32, 2, 2, 4, 0.95}};
static_assert(BK == kTileK && kShapes[2].bm == kTileRows, "the 32-bit offsets of a tile");

// What a step's blocks come to in one tile shape: clocks of all CTAs and of the
// longest, output elements, CTAs, K tiles of the longest.  A template, because
// a division by a tile extent is then a shift: it runs for every block of every
// new operator.
struct ShapeWork {
  double sum = 0.0, work_max = 0.0, cells = 0.0;
  int64_t n = 0, kmax = 0;
};
template <int S>
ShapeWork shape_work(const std::vector<ContractBlk>& blks) {
  constexpr uint32_t bm = kShapes[S].bm, bn = kShapes[S].bn, wm = kShapes[S].wm, wn = kShapes[S].wn;
  ShapeWork w;
  for (const ContractBlk& b : blks) {
    w.kmax = std::max(w.kmax, b.ktiles);
    const uint32_t M = static_cast<uint32_t>(b.M), N = static_cast<uint32_t>(b.N);
    const int64_t fm = M / bm, fn = N / bn;  // full tiles, then the ragged edges
    const uint32_t em = M % bm, en = N % bn;
    auto add = [&](int64_t count, uint32_t r, uint32_t c) {
      if (count <= 0 || r == 0 || c == 0) return;
      const uint32_t fr = ((r + 7) / 8 + wm - 1) / wm, fc = ((c + 7) / 8 + wn - 1) / wn;
      const double mma = 16.0 * static_cast<double>(fr * fc) * static_cast<double>(b.k4);
      const double mem = static_cast<double>((r + c) * b.ktiles) * 16.0 * 8.0 / 48.0;
      const double x = std::max(mma, mem);
      w.sum += static_cast<double>(count) * x;
      w.work_max = std::max(w.work_max, x);
      w.cells += static_cast<double>(count * r * c);
      w.n += count;
    };
    add(fm * fn, bm, bn);
    add(fn, em, bn);
    add(fm, bm, en);
    add(em > 0 && en > 0 ? 1 : 0, em, en);
  }
  return w;
}

}  // namespace

// Estimated clocks of a step for every tile shape and number of K shares (up
// to 8 in one cluster, beyond that parts of 8 summed by a second launch); the
// smallest wins.  A CTA's work is its longest warp's DMMA chain (16 clocks
// each) or its operand loads (about 48 bytes a clock and SM).  The step takes
// an even spread of that over the SMs, whose pipes are 0.6 busy with one CTA
// and 0.9 with three, plus what the longest share overhangs it by; at least the
// longest share alone (700 to 1000 clocks a K tile of latency and issue); and the
// prologues and epilogues, where a split writes and reads back every partial.
// Against both sides measured on 20 dense products of 0.02 to 16 GFLOP (every
// shape, 1 to 16 shares) the choice is within 12 % of the best.
void contract_choose(const std::vector<ContractBlk>& blks, int n_sm, int min_split, int max_split, int* shape,
                     int* split, int* parts) {
  double best = -1.0;
  *shape = 0;
  *split = std::min(min_split, 8);
  *parts = min_split / *split;
  for (int s : {1, 3, 2, 0}) {  // the smallest tile of equal estimates
    const Shape& h = kShapes[s];
    const ShapeWork w = s == 0 ? shape_work<0>(blks) : s == 1 ? shape_work<1>(blks) : s == 2 ? shape_work<2>(blks) : shape_work<3>(blks);
    const double sum = w.sum, work_max = w.work_max, cells = w.cells;
    const int64_t n = w.n, kmax = w.kmax;
    if (n == 0) continue;
    const double cell = cells / static_cast<double>(n);
    for (int sp = min_split; sp <= max_split; sp *= 2) {
      if (sp > min_split && kmax < 2 * sp) break;
      const double ctas = static_cast<double>(n) * sp;
      const double per_sm = std::min(static_cast<double>(h.resident), std::max(1.0, ctas / n_sm));
      const double eff = std::min(0.9, 0.45 + 0.15 * per_sm) * h.eff;
      const double over = sp == 1 ? 2500.0 + 0.8 * cell : 4500.0 + (0.8 / sp + 1.5) * cell;
      const double waves = std::max(1.0, ctas / (static_cast<double>(n_sm) * h.resident));
      const double alone = std::max(work_max / (0.6 * h.eff), (400.0 + 4.6 * (h.bm + h.bn)) * static_cast<double>(kmax)) / sp;
      const double est = std::max(sum / n_sm / eff + 0.6 * work_max / sp, alone) + over * waves +
                         (sp > 8 ? 6000.0 : 0.0);
      if (best < 0.0 || est < best) {
        best = est;
        *shape = s;
        *split = std::min(sp, 8);
        *parts = sp / *split;
      }
    }
  }
}

int64_t contract_tiles(const std::vector<ContractTile>& proto, const std::vector<ContractBlk>& blks, int shape,
                       std::vector<uint8_t>& dst) {
  const int bm = kShapes[shape].bm, bn = kShapes[shape].bn;
  // a block's tiles fall into four rectangles of one cost each (interior, last
  // column, last row, corner): these are sorted, not the tiles, into classes of
  // costs within 1/32 of each other (binary exponent and five bits), longest
  // first, in the blocks' order inside a class
  struct Rect {
    int32_t blk, m0, m1, n0, n1, cls;
  };
  constexpr int kClasses = 64 * 32;
  std::vector<Rect> rects;
  rects.reserve(4 * proto.size());
  std::vector<int32_t> first(kClasses + 1, 0);
  int64_t n = 0;
  for (size_t i = 0; i < proto.size(); ++i) {
    const int32_t M = proto[i].M, N = proto[i].N, mf = M & ~(bm - 1), nf = N & ~(bn - 1);
    auto add = [&](int32_t m0, int32_t m1, int32_t n0, int32_t n1) {
      if (m0 >= m1 || n0 >= n1) return;
      const uint64_t fm = (std::min(bm, m1 - m0) + 7) / 8, fn = (std::min(bn, n1 - n0) + 7) / 8;
      const uint64_t cost = static_cast<uint64_t>(blks[i].k4) * fm * fn;
      const int e = cost ? 63 - __builtin_clzll(cost) : 0;
      const int fine = static_cast<int>((e >= 5 ? cost >> (e - 5) : cost << (5 - e)) & 31);
      rects.push_back({static_cast<int32_t>(i), m0, m1, n0, n1, kClasses - 1 - (e * 32 + fine)});
      ++first[rects.back().cls + 1];
      // M and N are below 2^31, so m1 - m0 + bm - 1 is not
      n += ((static_cast<int64_t>(m1) - m0 + bm - 1) / bm) * ((static_cast<int64_t>(n1) - n0 + bn - 1) / bn);
    };
    add(0, mf, 0, nf);
    add(0, mf, nf, N);
    add(mf, M, 0, nf);
    add(mf, M, nf, N);
  }
  for (int c = 0; c < kClasses; ++c) first[c + 1] += first[c];
  std::vector<int32_t> order(rects.size());
  for (size_t r = 0; r < rects.size(); ++r) order[first[rects[r].cls]++] = static_cast<int32_t>(r);
  size_t at = dst.size();
  dst.resize(at + static_cast<size_t>(n) * sizeof(ContractTile));
  for (int32_t o : order) {
    const Rect& r = rects[o];
    ContractTile t = proto[r.blk];
    for (int64_t m0 = r.m0; m0 < r.m1; m0 += bm)
      for (int64_t n0 = r.n0; n0 < r.n1; n0 += bn) {
        t.m0 = static_cast<int32_t>(m0);
        t.n0 = static_cast<int32_t>(n0);
        std::memcpy(dst.data() + at, &t, sizeof(t));
        at += sizeof(t);
      }
  }
  return n;
}

cudaError_t launch_contract_f64(const ContractLaunch& L, cudaStream_t st) {
  if (L.n_tiles <= 0) return cudaSuccess;
  switch (L.shape) {
    case 0: return go_layout<64, 64, 2, 2>(L, st);
    case 1: return go_layout<32, 32, 2, 2>(L, st);
    case 2: return go_layout<128, 16, 4, 1>(L, st);
    default: return go_layout<64, 32, 2, 2>(L, st);
  }
}

}  // namespace tnx
