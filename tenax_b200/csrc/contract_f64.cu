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
// same bits on every run.  contract_choose() picks tile and split from a cost
// model of the step's tiles.
#include <algorithm>

#include "common.cuh"
#include "contract_f64.hpp"
#include "kernels.cuh"

namespace tnx {

namespace {
constexpr int BK = 16;
constexpr int STAGES = 4;
constexpr int THREADS = 128;
constexpr int kSmemSpans = 16;  // span records kept in shared memory; the rest are read from global

__device__ __forceinline__ int axis_off(const int32_t* __restrict__ tab, int32_t t, int32_t str, int i) {
  return t < 0 ? i * str : __ldg(tab + t + i);
}

// 8-byte asynchronous copy; ok = false writes a zero without reading
__device__ __forceinline__ void cp8(double* dst, const double* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 8 : 0)
               : "memory");
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
// consecutive rows.
template <int R, bool KF>
struct Operand {
  static constexpr int kPer = R * BK / THREADS;                 // elements per thread and K tile
  static constexpr int kRows = KF ? kPer : 1;                   // distinct rows per thread
  static constexpr int kTile = KF ? R * BK : BK * (R + 4);      // doubles per stage
  const double* base;
  int32_t kt, ks;
  int32_t off[kRows];

  __device__ __forceinline__ void set_span(const double* p, const int32_t* tab, int32_t rt, int32_t rs, int32_t kt_,
                                           int32_t ks_, int row0, int rows) {
    base = p;
    kt = kt_;
    ks = ks_;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int r = KF ? (static_cast<int>(threadIdx.x) >> 4) + 8 * i : static_cast<int>(threadIdx.x) % R;
      off[i] = r < rows ? axis_off(tab, rt, rs, row0 + r) : -1;  // -1: past the block, not loaded
    }
  }
  __device__ __forceinline__ void load(double* s, const int32_t* tab, int k0, int K) const {
    if constexpr (KF) {
      const int kk = threadIdx.x & 15;
      const bool ok = k0 + kk < K;
      const int ko = ok ? axis_off(tab, kt, ks, k0 + kk) : 0;
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int r = (static_cast<int>(threadIdx.x) >> 4) + 8 * i;
        if (off[i] >= 0) cp8(s + r * BK + (kk ^ ((r & 3) << 2)), base + (off[i] + ko), ok);
      }
    } else {
      const int r = static_cast<int>(threadIdx.x) % R;
      if (off[0] < 0) return;
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int kk = static_cast<int>(threadIdx.x) / R + i * (THREADS / R);
        const bool ok = k0 + kk < K;
        const int ko = ok ? axis_off(tab, kt, ks, k0 + kk) : 0;
        cp8(s + kk * (R + 4) + r, base + (off[0] + ko), ok);
      }
    }
  }
  static __device__ __forceinline__ double frag(const double* s, int r, int kk) {
    return KF ? s[r * BK + (kk ^ ((r & 3) << 2))] : s[kk * (R + 4) + r];
  }
};

template <int BM, int BN, bool AK, bool BKF>
constexpr int smem_doubles() {
  constexpr int ring = STAGES * (Operand<BM, AK>::kTile + Operand<BN, BKF>::kTile);
  constexpr int part = BM * (BN + 1);  // a split's partial tile reuses the ring
  return ring > part ? ring : part;
}

template <int BM, int BN, int WM, int WN, bool AK, bool BKF>
__global__ void __launch_bounds__(THREADS, (BM * BN >= 4096) ? 3 : 4)
    contract_f64_kernel(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C,
                        const ContractTile* __restrict__ tiles, const ContractSpan* __restrict__ spans,
                        const int32_t* __restrict__ tab, int split) {
  static_assert(WM * WN == 4, "four warps");
  constexpr int MI = BM / 8 / WM, NI = BN / 8 / WN;
  using OpA = Operand<BM, AK>;
  using OpB = Operand<BN, BKF>;
  extern __shared__ __align__(16) double ring[];
  __shared__ ContractSpan sspan[kSmemSpans];
  double* As = ring;
  double* Bs = ring + STAGES * OpA::kTile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp / WN, wn = warp % WN;
  const int rank = static_cast<int>(blockIdx.x) % split;
  const ContractTile t = tiles[blockIdx.x / split];
  for (int i = tid; i < t.nspan * 4 && i < kSmemSpans * 4; i += THREADS)
    reinterpret_cast<int4*>(sspan)[i] = __ldg(reinterpret_cast<const int4*>(spans + t.span0) + i);
  __syncthreads();
  const int rows = min(BM, t.M - t.m0), cols = min(BN, t.N - t.n0);
  // this CTA's K tiles: an even share of the cluster's
  const int kt0 = static_cast<int>(static_cast<int64_t>(t.ktiles) * rank / split);
  const int nkt = static_cast<int>(static_cast<int64_t>(t.ktiles) * (rank + 1) / split) - kt0;
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
  auto issue = [&](int s) {
    if (fresh) {
      const ContractSpan g = sp < kSmemSpans ? sspan[sp] : spans[t.span0 + sp];
      K = g.K;
      oa.set_span(A + g.a_off, tab, g.ar_tab, g.ar_str, g.ak_tab, g.ak_str, t.m0, rows);
      ob.set_span(B + g.b_off, tab, g.br_tab, g.br_str, g.bk_tab, g.bk_str, t.n0, cols);
      fresh = false;
    }
    oa.load(As + s * OpA::kTile, tab, k0, K);
    ob.load(Bs + s * OpB::kTile, tab, k0, K);
    const uint32_t n4 = static_cast<uint32_t>((min(BK, K - k0) + 3) / 4);
    steps = (steps & ~(0xffu << (8 * s))) | (n4 << (8 * s));
    k0 += BK;
    if (k0 >= K) {
      k0 = 0;
      ++sp;
      fresh = true;
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nkt) issue(s);
    cp_commit();
  }
  for (int kt = 0; kt < nkt; ++kt) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int s = kt % STAGES;
    const int n4 = static_cast<int>((steps >> (8 * s)) & 0xffu);
    if (kt + STAGES - 1 < nkt) issue((kt + STAGES - 1) % STAGES);
    cp_commit();
    const double* as = As + s * OpA::kTile;
    const double* bs = Bs + s * OpB::kTile;
#pragma unroll
    for (int k4 = 0; k4 < BK / 4; ++k4) {
      if (k4 >= n4) break;
      const int kk = k4 * 4 + (lane & 3);
      double af[MI], bf[NI];
#pragma unroll
      for (int i = 0; i < MI; ++i) af[i] = OpA::frag(as, (i * WM + wm) * 8 + (lane >> 2), kk);
#pragma unroll
      for (int j = 0; j < NI; ++j) bf[j] = OpB::frag(bs, (j * WN + wn) * 8 + (lane >> 2), kk);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        if (i >= mv) break;
#pragma unroll
        for (int j = 0; j < NI; ++j) {
          if (j >= nv) break;
          dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
      }
    }
  }
  cp_wait<0>();
  double* out = C + t.out_off;
  if (split == 1) {
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int r = (i * WM + wm) * 8 + (lane >> 2);
      if (r >= rows) continue;
      const int ro = axis_off(tab, t.r_tab, t.r_str, t.m0 + r);
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const int c = (j * WN + wn) * 8 + (lane & 3) * 2;
        if (c < cols) out[ro + axis_off(tab, t.c_tab, t.c_str, t.n0 + c)] = acc[i][j][0];
        if (c + 1 < cols) out[ro + axis_off(tab, t.c_tab, t.c_str, t.n0 + c + 1)] = acc[i][j][1];
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
  for (int e = tid; e < mine * cols; e += THREADS) {
    const int q = rfast ? e % mine : e / cols;
    const int c = rfast ? e / mine : e - q * cols;
    const int r = rank + q * split;
    const uint32_t sa = smem_u32(ring + r * P + c);
    double v = ld_peer(sa, 0);
    for (int p = 1; p < split; ++p) v += ld_peer(sa, p);
    out[axis_off(tab, t.r_tab, t.r_str, t.m0 + r) + axis_off(tab, t.c_tab, t.c_str, t.n0 + c)] = v;
  }
  cluster_sync();  // no CTA leaves while a peer reads its shared memory
}

template <int BM, int BN, int WM, int WN, bool AK, bool BKF>
cudaError_t go(const ContractLaunch& L, cudaStream_t st) {
  constexpr int smem = smem_doubles<BM, BN, AK, BKF>() * static_cast<int>(sizeof(double));
  auto kernel = contract_f64_kernel<BM, BN, WM, WN, AK, BKF>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(L.n_tiles) * L.split);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  if (L.split > 1) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = L.split;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, L.a, L.b, L.c, L.tiles, L.spans, L.tab, L.split);
}

template <int BM, int BN, int WM, int WN>
cudaError_t go_layout(const ContractLaunch& L, cudaStream_t st) {
  if (L.a_kfast) return L.b_kfast ? go<BM, BN, WM, WN, true, true>(L, st) : go<BM, BN, WM, WN, true, false>(L, st);
  return L.b_kfast ? go<BM, BN, WM, WN, false, true>(L, st) : go<BM, BN, WM, WN, false, false>(L, st);
}

struct Shape {
  int bm, bn, wm, wn, resident;
};
// 64 x 64: the DMMA-bound shape; 32 x 32: few tiles or small blocks; 128 x 16:
// narrow column blocks (an MPO leg), whose rows are many
constexpr Shape kShapes[kContractShapes] = {{64, 64, 2, 2, 3}, {32, 32, 2, 2, 4}, {128, 16, 4, 1, 3}};
}  // namespace

void contract_tile_shape(int shape, int* bm, int* bn) {
  *bm = kShapes[shape].bm;
  *bn = kShapes[shape].bn;
}

// Estimated clocks of a step for every (tile shape, K split); the smallest
// wins.  Per CTA: the longest warp's DMMA chain (16 clocks each) or its
// operand loads (about 48 bytes a clock and SM), and a fixed 2500 clocks of
// table reads, ring fill and stores, overlapped over the resident CTAs; a
// split adds 2000 clocks for its exchange.  Fitted to: 80 x 80 x 1280 in
// 64 x 64 tiles without a split 48 us, and the 6400 x 256 x 256 product 30 us.
void contract_choose(const std::vector<ContractBlk>& blks, int n_sm, int* shape, int* split) {
  double best = -1.0;
  *shape = 0;
  *split = 1;
  for (int s = 0; s < kContractShapes; ++s) {
    const Shape& h = kShapes[s];
    double sum = 0.0, longest = 0.0;
    int64_t n = 0, kmax = 0;
    for (const ContractBlk& b : blks) {
      kmax = std::max(kmax, b.ktiles);
      const int64_t fm = b.M / h.bm, fn = b.N / h.bn;  // full tiles, then the ragged edges
      const int64_t em = b.M % h.bm, en = b.N % h.bn;
      auto add = [&](int64_t count, int64_t r, int64_t c) {
        if (count <= 0 || r <= 0 || c <= 0) return;
        const int64_t fr = ((r + 7) / 8 + h.wm - 1) / h.wm, fc = ((c + 7) / 8 + h.wn - 1) / h.wn;
        const double mma = 16.0 * static_cast<double>(fr * fc) * static_cast<double>(b.k4);
        const double mem = static_cast<double>((r + c) * b.ktiles) * 16.0 * 8.0 / 48.0;
        const double x = std::max(mma, mem);
        sum += static_cast<double>(count) * x;
        longest = std::max(longest, x);
        n += count;
      };
      add(fm * fn, h.bm, h.bn);
      add(fn, em, h.bn);
      add(fm, h.bm, en);
      add(em > 0 && en > 0 ? 1 : 0, em, en);
    }
    for (int sp = 1; sp <= 8; sp *= 2) {
      if (sp > 1 && kmax < 2 * sp) break;
      const double over = 2500.0 + (sp > 1 ? 2000.0 : 0.0);
      const double waves = std::max(1.0, static_cast<double>(n * sp) / (static_cast<double>(n_sm) * h.resident));
      const double est = std::max(sum / n_sm, longest / sp) + over * waves;
      if (best < 0.0 || est < best) {
        best = est;
        *shape = s;
        *split = sp;
      }
    }
  }
}

cudaError_t launch_contract_f64(const ContractLaunch& L, cudaStream_t st) {
  if (L.n_tiles <= 0) return cudaSuccess;
  switch (L.shape) {
    case 0: return go_layout<64, 64, 2, 2>(L, st);
    case 1: return go_layout<32, 32, 2, 2>(L, st);
    default: return go_layout<128, 16, 4, 1>(L, st);
  }
}

}  // namespace tnx
