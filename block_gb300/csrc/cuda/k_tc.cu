// tcgen05 building blocks: a single-tile GEMM used to check the operand
// layout, descriptors and TMEM read-back against a host product.
#include <algorithm>
#include <type_traits>

#include "k_tc.cuh"
#include "tc.cuh"

namespace bgpu {
namespace dev {

using namespace tc;

// D (128 x N, row-major f32) = A (128 x K, row-major bf16) * B (N x K, row-major bf16)^T
__global__ void __launch_bounds__(128) tc_tile_kernel(const __nv_bfloat16* __restrict__ A,
                                                       const __nv_bfloat16* __restrict__ B, float* __restrict__ D,
                                                       int N, int K, int* status) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5;
  uint8_t* sA = smem;
  uint8_t* sB = smem + 128 * K * 2;
  if (warp == 0) {
    tmem_alloc(&tbase, 256);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  for (int idx = tid; idx < 128 * K; idx += 128)
    *(__nv_bfloat16*)(sA + kmajor_off(idx / K, idx % K, 128)) = A[idx];
  for (int idx = tid; idx < N * K; idx += 128) *(__nv_bfloat16*)(sB + kmajor_off(idx / K, idx % K, N)) = B[idx];
  fence_async_smem();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t d = tbase;
  if (tid == 0) {
    const uint32_t idesc = idesc_bf16(128, N);
    for (int j = 0; j < K / 16; ++j) {
      const uint64_t ad = smem_desc(smem_u32(sA) + j * 2 * 128 * 16, 128 * 16, 128);
      const uint64_t bd = smem_desc(smem_u32(sB) + j * 2 * N * 16, N * 16, 128);
      mma_bf16(d, ad, bd, idesc, j > 0 ? 1u : 0u);
    }
    mma_commit(&bar);
  }
  __syncwarp();
  bool ok = mbar_wait_bounded(&bar, 0, 1000000000ull);
  ok = __syncthreads_and(ok) != 0;
  fence_after_sync();
  if (ok) {
    const int row = warp * 32 + (tid & 31);
    for (int c = 0; c < N; c += 16) {
      float v[16];
      tmem_ld16(d + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) D[(int64_t)row * N + c + i] = v[i];
    }
  } else {
    if (tid == 0) atomicExch(status, 1);
    mbar_wait_bounded(&bar, 0, 1000000000ull);  // let the MMAs drain before freeing TMEM
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, 256);
}

// Same product with both operands pre-packed in global memory as K-chunks of
// 64 columns in the K-major core-matrix order (chunk c of a R-row operand at
// element R * 64 * c), each chunk moved to shared memory by one bulk copy.
__global__ void __launch_bounds__(128) tc_tile_bulk_kernel(const __nv_bfloat16* __restrict__ Ap,
                                                            const __nv_bfloat16* __restrict__ Bp,
                                                            float* __restrict__ D, int N, int K, int* status) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full, done;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5;
  uint8_t* sA = smem;              // 128 x 64
  uint8_t* sB = smem + 128 * 128;  // N x 64
  if (warp == 0) {
    tmem_alloc(&tbase, 256);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(&full, 1);
    mbar_init(&done, 1);
    mbar_fence_init();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t d = tbase;
  bool ok = true;
  if (tid == 0) {
    const uint32_t idesc = idesc_bf16(128, N);
    const int nck = (K + 63) / 64;
    for (int c = 0; c < nck && ok; ++c) {
      const int w = min(64, K - 64 * c);
      mbar_expect_tx(&full, (uint32_t)(128 + N) * w * 2);
      bulk_g2s(sA, Ap + (int64_t)128 * 64 * c, 128 * w * 2, &full);
      bulk_g2s(sB, Bp + (int64_t)N * 64 * c, N * w * 2, &full);
      ok = mbar_wait_bounded(&full, c & 1, 1000000000ull);
      if (!ok) break;
      fence_after_sync();
      for (int j = 0; j < w / 16; ++j) {
        const uint64_t ad = smem_desc(smem_u32(sA) + j * 2 * 128 * 16, 128 * 16, 128);
        const uint64_t bd = smem_desc(smem_u32(sB) + j * 2 * N * 16, N * 16, 128);
        mma_bf16(d, ad, bd, idesc, (c > 0 || j > 0) ? 1u : 0u);
      }
      mma_commit(&done);
      ok = mbar_wait_bounded(&done, c & 1, 1000000000ull);  // stage reused by the next chunk
    }
    if (!ok) atomicExch(status, 1);
  }
  ok = __syncthreads_and(ok) != 0;
  fence_after_sync();
  if (ok) {
    const int row = warp * 32 + (tid & 31);
    for (int c = 0; c < N; c += 16) {
      float v[16];
      tmem_ld16(d + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) D[(int64_t)row * N + c + i] = v[i];
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, 256);
}

cudaError_t launch_tc_tile_bulk(const __nv_bfloat16* Ap, const __nv_bfloat16* Bp, float* D, int N, int K,
                                int* status, cudaStream_t s) {
  if (N < 16 || N > 256 || N % 16 || K < 16 || K > 256 || K % 16) return cudaErrorInvalidValue;
  const size_t smem = 200 * 1024;  // operands use (128 + N) * 128 bytes
  cudaError_t e = cudaFuncSetAttribute(tc_tile_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  tc_tile_bulk_kernel<<<1, 128, smem, s>>>(Ap, Bp, D, N, K, status);
  return cudaGetLastError();
}

cudaError_t launch_tc_tile(const __nv_bfloat16* A, const __nv_bfloat16* B, float* D, int N, int K, int* status,
                           cudaStream_t s) {
  if (N < 16 || N > 256 || N % 16 || K < 16 || K > 64 || K % 16) return cudaErrorInvalidValue;
  // the operands need (128 + N) * K * 2 bytes; the allocation is larger so
  // that every address the descriptors can form stays inside it
  const size_t smem = 200 * 1024;
  cudaError_t e = cudaFuncSetAttribute(tc_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  tc_tile_kernel<<<1, 128, smem, s>>>(A, B, D, N, K, status);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- sigma

// p[i] for a small kernel-parameter array, by selects (dynamic indexing
// would copy the parameter block to local memory)
template <class T, int N>
__device__ __forceinline__ T pick(const T (&p)[N], int i) {
  T r = p[0];
#pragma unroll
  for (int k = 1; k < N; ++k)
    if (i == k) r = p[k];
  return r;
}

// Packs FP64 blocks into split bf16 operands.  Each thread writes one
// 16-byte core-matrix row (8 consecutive K values of one operand row) of the
// hi and of the lo slice; for transposed views consecutive threads take
// consecutive rows so that the FP64 reads stay coalesced.
__global__ void __launch_bounds__(256) tc_pack_kernel(TcBufs b, const TcPack* __restrict__ units) {
  const TcPack u = units[blockIdx.x];
  const double* src = pick(b.src, u.src) + u.src_off;
  __nv_bfloat16* dst = pick(b.pool, u.pool) + u.dst_off;
  const int kg = u.kp >> 3;
  const int64_t total = (int64_t)u.rows_p * kg;
  for (int64_t g = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.y * blockDim.x) {
    int r, k0;
    if (u.trans) {
      r = (int)(g % u.rows_p);
      k0 = (int)(g / u.rows_p) * 8;
    } else {
      r = (int)(g / kg);
      k0 = (int)(g % kg) * 8;
    }
    uint32_t hw[4], lw[4];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int k = k0 + e;
      double x = 0.0;
      if (r < u.rows_v && k < u.cols_v) x = u.trans ? src[(int64_t)k * u.ld + r] : src[(int64_t)r * u.ld + k];
      uint32_t bh, bl;
      split16(x, b.fp16 != 0, bh, bl);
      if (e & 1) {
        hw[e >> 1] |= bh << 16;
        lw[e >> 1] |= bl << 16;
      } else {
        hw[e >> 1] = bh;
        lw[e >> 1] = bl;
      }
    }
    // row R of the destination operand (of H rows; a stack member starts at row0)
    const int H = u.dst_rows > 0 ? u.dst_rows : u.rows_p, R = u.row0 + r;
    const int t = R / u.rt, c = k0 / kTcKC;
    const int rest = H - u.rt * t;
    const int h = rest < u.rt ? rest : u.rt;
    const int w = min(kTcKC, u.kp - kTcKC * c);
    const int64_t off = 2 * tc_block_off(H, u.kp, t, c, u.rt) + (kmajor_off(R - u.rt * t, k0 % kTcKC, h) >> 1);
    *(uint4*)(dst + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    *(uint4*)(dst + off + (int64_t)h * w) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
  }
}

cudaError_t launch_tc_pack(const TcBufs& b, const TcPack* units, int nunits, cudaStream_t s, int split) {
  if (nunits > 0) tc_pack_kernel<<<dim3(nunits, split), 256, 0, s>>>(b, units);
  return cudaGetLastError();
}

namespace {

// Pipeline shape by output-tile width NB (the B operands' row tile): with
// NB = 64 two independent blocks share an SM (256 TMEM columns and half the
// shared memory each); with NB = 128 one block owns the SM.  The ring holds as
// many stages as fit for the plan's largest piece (tc_ring).
// Epilogue: one warp per 32 rows and 64 columns.
template <int NB>
struct TcCfg {
  static constexpr int kRing = (NB == 64 ? 4 : 6) * 2 * (kTcRowsA + NB) * kTcKC * 2;
  // an MMA reads 128 rows of A and a multiple of 16 of B, also of a shorter piece
  static constexpr int kSmem = kRing + 128 * 16 + 16 * 16;
  static constexpr int kEpiWarps = NB / 16;
  static constexpr int kThreads = 32 * (kEpiWarps + 2);
  static constexpr int kProducer = kEpiWarps, kIssuer = kEpiWarps + 1;
  static constexpr int kAcc = 4;                     // accumulators of NB TMEM columns
  static constexpr uint32_t kTmemCols = kAcc * NB;
  static constexpr int kBlocksPerSm = NB == 64 ? 2 : 1;
};
constexpr int kTcSlots = 16;  // stages at most
constexpr int kTcMaxAcc = 4;

struct TcShared {
  uint64_t full[kTcSlots], empty[kTcSlots], acc_full[kTcMaxAcc], acc_empty[kTcMaxAcc], drain;
  uint32_t tbase;
  int abort_flag;
};

// bounded wait that also gives up when another role gave up
__device__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, uint64_t limit_ns) {
  // polled without the clock first: a read of the global timer takes about a
  // microsecond, longer than most waits
  for (int i = 0; i < kSpinPolls; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (globaltimer_ns() - t0 > limit_ns) {
      *abort_flag = 1;
      atomicExch(status, 1);
      return false;
    }
  }
  return true;
}

// hi + lo += x, with the rounding error of the sum kept in lo (TwoSum), two
// values at a time
__device__ __forceinline__ void two_sum_acc(uint64_t& hi, uint64_t& lo, uint64_t x) {
  const uint64_t s = add2(hi, x);
  const uint64_t bp = sub2(s, hi);
  const uint64_t err = add2(sub2(hi, sub2(s, bp)), sub2(x, bp));
  hi = s;
  lo = add2(lo, err);
}

}  // namespace

// Work records are read straight into registers, the next ones while the
// present one is processed, and prefetched into L1 ahead of that.  (Records
// held one per lane and handed out by shuffles cost 130 to 290 clocks a
// shuffle in the one-thread roles' divergent code: 1000 to 2000 clocks an
// item, more than its copies and MMAs.)
constexpr int kWorkAhead = 6;  // records prefetched into L1
__device__ __forceinline__ void prefetch_work(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ int64_t join64(int lo, int hi) {
  return (int64_t)(((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo);
}
// what the producer needs of record i (zeros from end on)
struct CopyRec {
  int4 base;  // a_base, b_base
  int kp, hw, pf;
};
__device__ __forceinline__ CopyRec load_copy(const TcWork* __restrict__ w, int i, int end) {
  CopyRec r{};
  if (i < end) {
    const int4* p = reinterpret_cast<const int4*>(w + i);
    r.base = __ldg(p);
    r.kp = __ldg(&w[i].kp);
    r.hw = __ldg(reinterpret_cast<const int*>(p + 2));
    r.pf = __ldg(reinterpret_cast<const int*>(p + 3));
    if (i + kWorkAhead < end) prefetch_work(w + i + kWorkAhead);
  }
  return r;
}
// the MMA issuer
struct MmaRec {
  int kp, hw, pf;
};
__device__ __forceinline__ MmaRec load_mma(const TcWork* __restrict__ w, int i, int end) {
  MmaRec r{};
  if (i < end) {
    const int4* p = reinterpret_cast<const int4*>(w + i);
    r.kp = __ldg(&w[i].kp);
    r.hw = __ldg(reinterpret_cast<const int*>(p + 2));
    r.pf = __ldg(reinterpret_cast<const int*>(p + 3));
    if (i + kWorkAhead < end) prefetch_work(w + i + kWorkAhead);
  }
  return r;
}
// the epilogue (every lane reads the same record)
struct EpiRec {
  int4 q1, q2;  // out_base, kp, alpha; h_a | h_b << 16, valid rows | columns << 16, out_ld, col0
  int pf;
};
__device__ __forceinline__ EpiRec load_epi(const TcWork* __restrict__ w, int i, int end) {
  EpiRec r{};
  if (i < end) {
    const int4* p = reinterpret_cast<const int4*>(w + i);
    r.q1 = __ldg(p + 1);
    r.q2 = __ldg(p + 2);
    r.pf = __ldg(reinterpret_cast<const int*>(p + 3));
    if (i + kWorkAhead < end) prefetch_work(w + i + kWorkAhead);
  }
  return r;
}

// Grouped split-precision GEMM over packed operands on tcgen05: per K=16
// step three MMAs (hi*hi + hi*lo + lo*hi) into an f32 TMEM accumulator of
// 128 x NB; the items of an accumulation group share the accumulator, four
// accumulators rotate between groups.  Operand pieces are streamed by bulk
// copies through the shared-memory ring.  Persistent: block j walks the work
// records [ranges[j].x, ranges[j].y), and the pipeline runs across task
// boundaries; one lane produces, one warp issues the MMAs.
// The epilogue folds each group sum into a compensated (hi, lo) f32 pair per
// element, 64 columns a thread, two values an instruction (168 registers a
// thread, 68 bytes of them spilled).  With the pairs in TMEM and four warps
// phase 2 took 680 us at 24 orbitals, M=500; 441 now.
// Bound, of the issuer's clocks in phase 2: 24 orbitals M=500 (spin 0: all
// factors are 1, nine items a group) MMAs 48 %, waits for operand pieces 36 %,
// for an accumulator 11 %; 18 orbitals M=1000 65, 28 and 9 %.  Targets with
// spin: a stage-1 product read by several couplings keeps its factor and is a
// group by itself (triplet M=101: waits for an accumulator, that is the folds,
// 48 %, MMAs 15 %).
template <int PHASE, int NB>
__global__ void __launch_bounds__(TcCfg<NB>::kThreads, TcCfg<NB>::kBlocksPerSm)
    tc_sigma_kernel(TcBufs b, const TcWork* __restrict__ work, const int2* __restrict__ ranges,
                    double* __restrict__ sigma, uint64_t limit_ns, int slots, uint32_t stage_bytes, int piece_k) {
  using Cfg = TcCfg<NB>;
  constexpr int kTcProducer = Cfg::kProducer, kTcIssuer = Cfg::kIssuer, kTcAcc = Cfg::kAcc;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ TcShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int2 rg = ranges[blockIdx.x];
  if (warp == kTcIssuer) {
    tmem_alloc(&sh.tbase, Cfg::kTmemCols);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < slots; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 1);
    }
    for (int i = 0; i < kTcAcc; ++i) {
      mbar_init(&sh.acc_full[i], 1);
      mbar_init(&sh.acc_empty[i], Cfg::kEpiWarps);
    }
    mbar_init(&sh.drain, 1);
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sh.tbase;
  volatile int* abort_flag = &sh.abort_flag;

  if (warp == kTcProducer) {
    // ---- producer (lane 0): streams the operand pieces (up to piece_k columns
    // of one item, per K-chunk A hi, A lo, then B hi, B lo) through the stages
    if (lane == 0) {
      uint32_t k = 0;  // pieces issued
      int slot = 0;
      uint32_t ph = 0;
      bool ok = true;
      CopyRec n0 = load_copy(work, rg.x, rg.y), n1 = load_copy(work, rg.x + 1, rg.y);
      for (int i = rg.x; i < rg.y && ok; ++i) {
        const CopyRec r = n0;
        n0 = n1;
        n1 = load_copy(work, i + 2, rg.y);
        if ((r.pf >> 16) & kTcEmpty) continue;
        const uint32_t a4 = 4u * (r.hw & 0xffff), b4 = 4u * ((r.hw >> 16) & 0xffff);  // bytes per column
        const uint8_t* pa = reinterpret_cast<const uint8_t*>(join64(r.base.x, r.base.y));
        const uint8_t* pb = reinterpret_cast<const uint8_t*>(join64(r.base.z, r.base.w));
        for (int left = r.kp; left > 0; left -= piece_k, ++k) {
          const uint32_t w = (uint32_t)min(piece_k, left);  // its K-chunks lie one after another
          const uint32_t abytes = a4 * w, bbytes = b4 * w;
          if (!tc_wait(&sh.empty[slot], ph ^ 1u, abort_flag, b.status, limit_ns)) {
            ok = false;
            break;
          }
          uint8_t* dst = smem + (uint32_t)slot * stage_bytes;
          mbar_expect_tx(&sh.full[slot], abytes + bbytes);
          bulk_g2s(dst, pa, abytes, &sh.full[slot]);
          bulk_g2s(dst + abytes, pb, bbytes, &sh.full[slot]);
          pa += abytes;
          pb += bbytes;
          if (++slot == slots) {
            slot = 0;
            ph ^= 1u;
          }
        }
      }
      const uint32_t ns = (uint32_t)slots;
      if (!ok) {
        // copies already issued still land in shared memory: wait for them
        for (uint32_t i = (k > ns ? k - ns : 0); i < k; ++i)
          mbar_wait_bounded(&sh.full[i % ns], (i / ns) & 1u, limit_ns);
      }
    }
  } else if (warp == kTcIssuer) {
    // ---- MMA issuer: the whole warp walks the records and one lane issues
    // (mma_bf16_if).  The issue of an MMA blocks while the one before it runs
    // (64 clocks at 128 x 128, 48 at 128 x 64), so that every clock spent
    // between two pieces is lost to the tensor core: the next piece's record,
    // place and descriptors are worked out between the MMAs of this one.
    const bool on = elect_one();
    int slot = 0;
    uint32_t ph = 0;
    int ab = 0;
    uint32_t aph = 0;
    const uint32_t sm0 = smem_u32(smem) >> 4, stage16 = stage_bytes >> 4;
    const uint32_t idesc0 = b.fp16 ? idesc_f16(128, 0) : idesc_bf16(128, 0);
    // low words of the operands' descriptors: address / 16 and rows (the
    // leading byte offset / 16); the high word is the same for all
    constexpr uint64_t kDescHi = smem_desc_hi();
    // records i (uniform in u_*), i + 1 (n0) and i + 2 (n1) are on their way
    MmaRec n0 = load_mma(work, rg.x, rg.y), n1 = load_mma(work, rg.x + 1, rg.y);
    int u_kp = uniform(n0.kp), u_hw = uniform(n0.hw), u_pf = uniform(n0.pf);
    n0 = n1;
    n1 = load_mma(work, rg.x + 2, rg.y);
    int i = rg.x, kp = 0, k0 = 0, flags = 0, w = 0;
    uint32_t ha = 0, hb = 0, idesc = 0, la = 0, lb = 0;
    auto next_item = [&]() {  // false at the end of the records
      do {
        if (i >= rg.y) return false;
        kp = u_kp;
        ha = (uint32_t)u_hw & 0xffffu;
        hb = (uint32_t)u_hw >> 16;
        flags = (u_pf >> 16) & 0xff;
        ++i;
        u_kp = uniform(n0.kp);
        u_hw = uniform(n0.hw);
        u_pf = uniform(n0.pf);
        n0 = n1;
        n1 = load_mma(work, i + 2, rg.y);
      } while (flags & kTcEmpty);
      idesc = idesc0 | ((((hb + 15u) & ~15u) >> 3) << 17);
      k0 = 0;
      return true;
    };
    auto place = [&]() {  // the piece at k0, in stage `slot`
      w = min(piece_k, kp - k0);
      const uint32_t a0 = sm0 + (uint32_t)slot * stage16;
      la = a0 | (ha << 16);
      lb = (a0 + (ha * (uint32_t)w >> 2)) | (hb << 16);
    };
    bool more = next_item(), ready = false;
    if (more) place();
    while (more) {
      const bool gstart = k0 == 0 && (flags & kTcGStart);
      if (gstart && !__all_sync(0xffffffffu, tc_wait(&sh.acc_empty[ab], aph ^ 1u, abort_flag, b.status, limit_ns)))
        break;
      if (!ready && !__all_sync(0xffffffffu, tc_wait(&sh.full[slot], ph, abort_flag, b.status, limit_ns))) break;
      fence_after_sync();
      const uint32_t d = tmem + (uint32_t)ab * (uint32_t)NB, id = idesc;
      const int w0 = min(kTcKC, w), w1 = w - w0;
      // a slice of h rows x w0 columns is h w0 / 8 units; one K=16 step 2 h
      const uint64_t dah = kDescHi | la, dal = dah + (ha * (uint32_t)w0 >> 3);
      const uint64_t dbh = kDescHi | lb, dbl = dbh + (hb * (uint32_t)w0 >> 3);
      const uint64_t sa = 2 * ha, sb = 2 * hb;
      const uint64_t ea = dah + 4 * sa, eb = dbh + 4 * sb;  // second chunk
      const uint64_t eal = ea + (ha * (uint32_t)w1 >> 3), ebl = eb + (hb * (uint32_t)w1 >> 3);
      const bool gend = (flags & kTcGEnd) && k0 + w >= kp;
      const int slot_c = slot, ab_c = ab;
      mma_bf16_if(on, d, dah, dbh, id, gstart ? 0u : 1u);
      k0 += w;
      if (gend && ++ab == kTcAcc) {
        ab = 0;
        aph ^= 1u;
      }
      if (++slot == slots) {
        slot = 0;
        ph ^= 1u;
      }
      mma_bf16_if(on, d, dah, dbl, id, 1u);
      if (k0 >= kp) more = next_item();
      mma_bf16_if(on, d, dal, dbh, id, 1u);
      if (more) place();
      if (w0 == kTcKC) {
        mma_bf16_if(on, d, dah + sa, dbh + sb, id, 1u);
        mma_bf16_if(on, d, dah + sa, dbl + sb, id, 1u);
        mma_bf16_if(on, d, dal + sa, dbh + sb, id, 1u);
      }
      if (w1 > 0) {
        mma_bf16_if(on, d, ea, eb, id, 1u);
        mma_bf16_if(on, d, ea, ebl, id, 1u);
        mma_bf16_if(on, d, eal, eb, id, 1u);
        if (w1 == kTcKC) {
          mma_bf16_if(on, d, ea + sa, eb + sb, id, 1u);
          mma_bf16_if(on, d, ea + sa, ebl + sb, id, 1u);
          mma_bf16_if(on, d, eal + sa, eb + sb, id, 1u);
        }
      }
      const bool probe = mbar_test(&sh.full[slot], ph);
      mma_commit_if(on, &sh.empty[slot_c]);
      if (gend) mma_commit_if(on, &sh.acc_full[ab_c]);
      ready = __all_sync(0xffffffffu, probe);
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4).., columns
    // 64 (w / 4)..; thread `row` holds the sums of its row's 64 columns, two
    // to a register pair
    const int row = 32 * (warp & 3) + lane;
    const int cw = 64 * (warp >> 2);  // first column of this warp
    const uint32_t lane_base = ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)cw;
    int ab = 0;
    uint32_t aph = 0;
    bool ok = true, first = true;
    uint64_t vh[PHASE == 2 ? 32 : 1], vl[PHASE == 2 ? 32 : 1];
    // the row map of a stacked phase-1 tile is read one record ahead as well
    auto load_row = [&](const EpiRec& x) {
      const bool st = PHASE == 1 && ((x.pf >> 16) & kTcStacked) && row < (x.q2.x & 0xffff);
      return st ? __ldg(reinterpret_cast<const int4*>(b.rows + join64(x.q1.x, x.q1.y) + row)) : make_int4(0, 0, 0, 0);
    };
    EpiRec n0 = load_epi(work, rg.x, rg.y), n1{};
    int4 row_next = load_row(n0);
    if (PHASE == 1) n1 = load_epi(work, rg.x + 1, rg.y);
    for (int i = rg.x; i < rg.y && ok; ++i) {
      const EpiRec r = n0;
      const int4 row_map = row_next;
      if (PHASE == 1) {
        n0 = n1;
        n1 = load_epi(work, i + 2, rg.y);
        row_next = load_row(n0);
      } else {
        n0 = load_epi(work, i + 1, rg.y);
      }
      const int flags = (r.pf >> 16) & 0xff;
      if (!(flags & (kTcFirst | kTcLast | kTcGEnd))) continue;
      const float alpha = __int_as_float(r.q1.w);
      const int hw = r.q2.x;
      const int h_a = hw & 0xffff, h_b = (hw >> 16) & 0xffff;
      // 16-column groups of the accumulator in this warp's columns
      const int ng = min(max((((h_b + 15) & ~15) - cw) >> 4, 0), 4);
      if (flags & kTcFirst) first = true;
      const bool have = (flags & kTcGEnd) && !(flags & kTcEmpty);
      const bool last = (flags & kTcLast) != 0;
      const uint32_t d = tmem + (uint32_t)ab * (uint32_t)NB + lane_base;
      if (have) {
        ok = __all_sync(0xffffffffu, tc_wait(&sh.acc_full[ab], aph, abort_flag, b.status, limit_ns));
        if (!ok) break;  // TMEM loads below need the whole warp
        fence_after_sync();
      }
      if constexpr (PHASE == 2) {
        if (have) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (g < ng) {
              float v[16];
              tmem_ld16(d + 16u * (uint32_t)g, v);
              if (g == ng - 1) {
                // accumulator read: the MMA issuer may reuse it
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.acc_empty[ab]);
              }
              if (first) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  vh[8 * g + e] = scale2(alpha, v[2 * e], v[2 * e + 1]);
                  vl[8 * g + e] = 0ull;
                }
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  two_sum_acc(vh[8 * g + e], vl[8 * g + e], scale2(alpha, v[2 * e], v[2 * e + 1]));
              }
            }
          }
          if (ng == 0 && lane == 0) mbar_arrive(&sh.acc_empty[ab]);
        } else if (first) {  // a task without items writes zeros
#pragma unroll
          for (int e = 0; e < 32; ++e) vh[e] = vl[e] = 0ull;
        }
        if (last) {
          const int64_t out_base = join64(r.q1.x, r.q1.y);
          const int vrc = r.q2.y, out_ld = r.q2.z;
          const bool direct = (flags & kTcDirect) != 0;
          const int rows = direct ? vrc & 0xffff : h_a;
          const int cols = (direct ? (vrc >> 16) & 0xffff : h_b) - cw;
          if (row < rows) {
            double* out = sigma + out_base + (int64_t)row * out_ld + cw;
            float2* outp = b.partials + out_base + (int64_t)row * h_b + cw;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (2 * e < cols) {
                float h0, h1, l0, l1;
                unpack2(vh[e], h0, h1);
                unpack2(vl[e], l0, l1);
                if (direct) {
                  out[2 * e] = f32_to_f64(h0) + f32_to_f64(l0);
                  if (2 * e + 1 < cols) out[2 * e + 1] = f32_to_f64(h1) + f32_to_f64(l1);
                } else {  // h_b is even
                  outp[2 * e] = make_float2(h0, l0);
                  outp[2 * e + 1] = make_float2(h1, l1);
                }
              }
            }
          }
        }
        if (have || last) first = false;
      } else if (have) {
        // phase 1: S tile written as a packed operand (rows of this tile,
        // K columns col0.. of S; row s_row of an s_h-row operand); a
        // stacked tile's rows go to their members' operands and scales
        const int64_t out_base = join64(r.q1.x, r.q1.y);
        const int out_ld = r.q2.z, col0 = r.q2.w;
        int64_t s_base = out_base;
        int s_h = h_a, s_row = row;
        float s_alpha = alpha;
        if ((flags & kTcStacked) && row < h_a) {
          s_base = join64(row_map.x, row_map.y);
          s_h = row_map.z & 0xffff;
          s_row = (row_map.z >> 16) & 0xffff;
          s_alpha = __int_as_float(row_map.w);
        }
        const bool mine = row < h_a && s_h > 0;
        const int c_s = col0 + cw;                      // S column of this warp's first
        const int ncols = min(NB, out_ld - col0) - cw;  // its S columns (a multiple of 8)
        // element of the row in the first 8-column group of its K-chunk; the
        // next group is 8 s_h on, the lo slice s_h wc, the next chunk 64 s_h
        __nv_bfloat16* sp = b.pool[kTcPoolS] + s_base + 2 * (int64_t)s_h * c_s + (s_row >> 3) * 64 + (s_row & 7) * 8;
        auto store = [&](auto fp16) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float v[16];
            if (g < ng) {
              tmem_ld16(d + 16u * (uint32_t)g, v);
              if (g == ng - 1) {
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.acc_empty[ab]);
              }
            }
            const int cc = 32 * (g / 2);
            const int wc = min(kTcKC, out_ld - c_s - cc);
#pragma unroll
            for (int g8 = 0; g8 < 2; ++g8) {
              const int c0 = 16 * g + 8 * g8;  // column in this warp's 64
              if (mine && c0 < ncols) {
                // columns of the accumulator beyond h_b (a multiple of 8) are
                // another operand's: zeros
                const bool zero = cw + c0 >= h_b;
                uint32_t hw4[4], lw4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const uint64_t x = zero ? 0ull : scale2(s_alpha, v[8 * g8 + 2 * e], v[8 * g8 + 2 * e + 1]);
                  split16x2(x, decltype(fp16)::value, hw4[e], lw4[e]);
                }
                __nv_bfloat16* q = sp + 2 * cc * s_h + (c0 - cc) * s_h;
                *(uint4*)q = make_uint4(hw4[0], hw4[1], hw4[2], hw4[3]);
                *(uint4*)(q + wc * s_h) = make_uint4(lw4[0], lw4[1], lw4[2], lw4[3]);
              }
            }
          }
        };
        if (b.fp16) store(std::true_type{});
        else store(std::false_type{});
        if (ng == 0 && lane == 0) mbar_arrive(&sh.acc_empty[ab]);
      }
      if (have && ++ab == kTcAcc) {
        ab = 0;
        aph ^= 1u;
      }
    }
  }
  __syncthreads();
  if (warp == kTcIssuer) {
    // every MMA of this block has completed before TMEM is released
    __syncwarp();
    if (elect_one()) {  // the lane that issued them
      mma_commit(&sh.drain);
      mbar_wait_bounded(&sh.drain, 0, limit_ns);
    }
    __syncwarp();
    fence_after_sync();
    tmem_dealloc(tmem, TcCfg<NB>::kTmemCols);
  }
}

// Columns per piece and stages of the ring for pieces of at most rows rows (A
// and B together) and kp columns: two K-chunks a piece, which halves the
// barrier round trips, where three stages of them fit, else one.
struct TcRing {
  int piece_k, stage, slots;
};
template <int NB>
static TcRing tc_ring(int rows, int kp) {
  TcRing r;
  for (r.piece_k = 2 * kTcKC;; r.piece_k = kTcKC) {
    r.stage = (4 * rows * std::min(r.piece_k, kp) + 127) / 128 * 128;
    r.slots = std::min(kTcSlots, TcCfg<NB>::kRing / r.stage);
    if (r.slots >= 3 || r.piece_k == kTcKC) return r;
  }
}

template <int PHASE, int NB>
static cudaError_t launch_tc_sigma_nb(const TcBufs& b, const TcWork* work, const int2* ranges, int nblocks,
                                      double* sigma, uint64_t limit_ns, cudaStream_t s, int2 most) {
  constexpr int smem = TcCfg<NB>::kSmem;
  if (most.x <= 0 || most.x > kTcRowsA + NB || most.y <= 0) return cudaErrorInvalidValue;
  const TcRing r = tc_ring<NB>(most.x, most.y);
  cudaError_t e = cudaFuncSetAttribute(tc_sigma_kernel<PHASE, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  tc_sigma_kernel<PHASE, NB>
      <<<nblocks, TcCfg<NB>::kThreads, smem, s>>>(b, work, ranges, sigma, limit_ns, r.slots, (uint32_t)r.stage, r.piece_k);
  return cudaGetLastError();
}

cudaError_t launch_tc_sigma(int phase, int nb, const TcBufs& b, const TcWork* work, const int2* ranges, int nblocks,
                            double* sigma, uint64_t limit_ns, cudaStream_t s, int2 most) {
  if (nblocks <= 0) return cudaGetLastError();
  if (phase == 1 && nb == 64) return launch_tc_sigma_nb<1, 64>(b, work, ranges, nblocks, sigma, limit_ns, s, most);
  if (phase == 2 && nb == 64) return launch_tc_sigma_nb<2, 64>(b, work, ranges, nblocks, sigma, limit_ns, s, most);
  if (phase == 1 && nb == 128) return launch_tc_sigma_nb<1, 128>(b, work, ranges, nblocks, sigma, limit_ns, s, most);
  if (phase == 2 && nb == 128) return launch_tc_sigma_nb<2, 128>(b, work, ranges, nblocks, sigma, limit_ns, s, most);
  return cudaErrorInvalidValue;
}

int tc_blocks_per_sm(int nb) { return nb == 64 ? TcCfg<64>::kBlocksPerSm : TcCfg<128>::kBlocksPerSm; }

// Bound by the latency of the slot reads: few tiles (56 at 24 orbitals,
// M=500) with tens of partials each, so every thread keeps eight reads in
// flight and a 128 x 128 tile is spread over 32 blocks.
__global__ void __launch_bounds__(256) tc_reduce_kernel(const float2* __restrict__ partials,
                                                         const TcTile* __restrict__ tiles,
                                                         const int64_t* __restrict__ slots, double* __restrict__ sigma) {
  const TcTile t = tiles[blockIdx.x];
  const int n = t.h * t.w;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < n; e += gridDim.y * blockDim.x) {
    double acc = 0.0;
    const int r = e / t.w, c = e % t.w;
    const float2* src = partials + (int64_t)r * t.pad + c;  // slots are h_a x h_b, row stride pad
    int p = t.pbeg;
    // eight partials in flight per thread, summed in slot order
    for (; p + 8 <= t.pend; p += 8) {
      float2 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = src[slots[p + i]];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc += f32_to_f64(v[i].x) + f32_to_f64(v[i].y);
    }
    for (; p < t.pend; ++p) {
      const float2 v = src[slots[p]];
      acc += f32_to_f64(v.x) + f32_to_f64(v.y);
    }
    sigma[t.s_off + (int64_t)(t.r0 + r) * t.lds + t.c0 + c] = acc;
  }
}

cudaError_t launch_tc_reduce(const TcBufs& b, const TcTile* tiles, const int64_t* slots, int ntiles, double* sigma,
                             cudaStream_t s, int split) {
  if (ntiles > 0) tc_reduce_kernel<<<dim3(ntiles, split), 256, 0, s>>>(b.partials, tiles, slots, sigma);
  return cudaGetLastError();
}

// Waits on an mbarrier that nothing arrives at, through the same bounded
// wait the sigma kernels use; the wait must give up after limit_ns and set
// *status.  out[0] = 1 if the wait reported failure, out[1] = elapsed ns.
__global__ void tc_wait_selftest_kernel(int* status, unsigned long long* out, uint64_t limit_ns) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    abort_flag = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint64_t t0 = globaltimer_ns();
    const bool ok = tc_wait(&bar, 0, &abort_flag, status, limit_ns);
    out[0] = ok ? 0ull : 1ull;
    out[1] = globaltimer_ns() - t0;
  }
}

cudaError_t launch_tc_wait_selftest(int* status, unsigned long long* out, uint64_t limit_ns, cudaStream_t s) {
  tc_wait_selftest_kernel<<<1, 32, 0, s>>>(status, out, limit_ns);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace bgpu
