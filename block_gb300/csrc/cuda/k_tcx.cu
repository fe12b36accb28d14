// Exact-slice products on tcgen05 (see k_tc.cuh, "exact"): row exponents,
// six-digit packing, the two sigma phases and the FP64 reduction of split
// tiles.
#include "k_tc.cuh"
#include "tc.cuh"

namespace bgpu {
namespace dev {

using namespace tc;

namespace {

template <class T, int N>
__device__ __forceinline__ T pick_x(const T (&p)[N], int i) {
  T r = p[0];
#pragma unroll
  for (int k = 1; k < N; ++k)
    if (i == k) r = p[k];
  return r;
}

// unbiased binary exponent of a normal FP64 number (kTcxNoExp for zero and
// subnormal values, which the digits treat as zero)
__device__ __forceinline__ int exp_of(double x) {
  const int e = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  return e == 0 ? kTcxNoExp : e - 1023;
}

// the six balanced base-128 digits of x / 2^e (e > exponent of x), most
// significant first: x = 2^e sum_s d[s] 2^-7(s+1) up to 2^(e-43)
__device__ __forceinline__ void digits6(double x, int e, int (&d)[kTcxSlices]) {
  const uint64_t bits = (uint64_t)__double_as_longlong(x);
  const int be = (int)((bits >> 52) & 0x7ff);
  uint64_t M = 0;
  if (be != 0) {
    const uint64_t mant = (bits & ((1ull << 52) - 1)) | (1ull << 52);
    // |x| = mant 2^(be-1023-52);  M = round(|x| 2^(42-e)) = mant >> sh
    const int sh = e - (be - 1023) + 10;  // >= 11
    if (sh < 64) M = (mant + (1ull << (sh - 1))) >> sh;
  }
  // offset 64 in each of the five lower digits makes them balanced
  constexpr uint64_t C = 64ull * (1ull + (1ull << 7) + (1ull << 14) + (1ull << 21) + (1ull << 28));
  const uint64_t Mp = M + C;
  const int sg = (bits >> 63) ? -1 : 1;
  d[0] = sg * (int)(Mp >> 35);
#pragma unroll
  for (int s = 1; s < kTcxSlices; ++s) d[s] = sg * ((int)((Mp >> (7 * (5 - s))) & 127) - 64);
}

// the bf16 bits of two integers below 2^8: x in the low half (the addition of
// 1.5 2^23 puts an integer in the low bits of a float; the conversion unit
// takes an eighth of the adders' rate)
__device__ __forceinline__ uint32_t bf16x2_of(int x, int y) {
  const float fx = __int_as_float(0x4B400000 + x) - 12582912.f, fy = __int_as_float(0x4B400000 + y) - 12582912.f;
  return __byte_perm(__float_as_uint(fx), __float_as_uint(fy), 0x7632);
}

// Row exponents of one packed operand per block: rows of a row-major view
// one warp each (lanes along K), rows of a transposed view one thread each
// (threads along the source's contiguous rows).
__global__ void __launch_bounds__(256) tcx_rowexp_kernel(TcxBufs b, const TcPack* __restrict__ units) {
  const TcPack u = units[blockIdx.x];
  const double* src = pick_x(b.src, u.src) + u.src_off;
  int* ex = pick_x(b.ex, u.pool) + u.ex_off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!u.trans) {
    for (int r = warp + 8 * blockIdx.y; r < u.rows_p; r += 8 * gridDim.y) {
      int m = kTcxNoExp;
      if (r < u.rows_v)
        for (int k = lane; k < u.cols_v; k += 32) m = max(m, exp_of(src[(int64_t)r * u.ld + k]));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) ex[r] = m;
    }
  } else {
    for (int r = tid + 256 * blockIdx.y; r < u.rows_p; r += 256 * gridDim.y) {
      int m = kTcxNoExp;
      if (r < u.rows_v)
        for (int k = 0; k < u.cols_v; ++k) m = max(m, exp_of(src[(int64_t)k * u.ld + r]));
      ex[r] = m;
    }
  }
}

// Six digit slices per element; each thread writes one 16-byte core-matrix
// row (8 consecutive K of one row) of every slice.  Within the block of a
// K-chunk (h rows x w columns, six slices), each 16-column half is one K-major
// core-matrix operand of 6 h rows, slice s in rows s h.. : one bulk copy moves
// the operand piece of one K=16 step, and an MMA takes any run of slices of B
// as its columns.
// Bound by memory (8 bytes read and 12 written an element).  Consecutive
// threads take consecutive rows, so that a slice's rows are written 512 bytes
// at a time; a row-major source is then read 64 bytes a thread, which needs
// 32-byte reads: other row-major sources are taken along K (T of 20 orbitals
// M=300, 42 M elements: 180 us; 327 along K).
__global__ void __launch_bounds__(256) tcx_pack_kernel(TcxBufs b, const TcPack* __restrict__ units) {
  const TcPack u = units[blockIdx.x];
  const double* src = pick_x(b.src, u.src) + u.src_off;
  __nv_bfloat16* dst = pick_x(b.pool, u.pool) + u.dst_off;
  const int* ex = pick_x(b.ex, u.pool) + u.ex_off;
  const int kg = u.kp >> 3;
  const bool wide = !u.trans && (u.ld & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 31) == 0;
  const bool by_row = u.trans || wide;
  const int64_t total = (int64_t)u.rows_p * kg;
  for (int64_t g = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.y * blockDim.x) {
    const int d = by_row ? u.rows_p : kg;
    int q, m;  // g / d, g % d
    if (total <= UINT32_MAX) {
      q = (int)((uint32_t)g / (uint32_t)d);
      m = (int)((uint32_t)g - (uint32_t)q * (uint32_t)d);
    } else {
      q = (int)(g / d);
      m = (int)(g % d);
    }
    const int r = by_row ? m : q, k0 = 8 * (by_row ? q : m);
    const int em = ex[r];
    const bool live = em > kTcxNoExp / 2 && r < u.rows_v;
    double x[8];
    if (live && wide && k0 + 8 <= u.cols_v) {
      const double* p = src + (int64_t)r * u.ld + k0;
#pragma unroll
      for (int e = 0; e < 8; e += 4)
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[e]), "=d"(x[e + 1]), "=d"(x[e + 2]), "=d"(x[e + 3]) : "l"(p + e));
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int k = k0 + e;
        x[e] = live && k < u.cols_v ? (u.trans ? src[(int64_t)k * u.ld + r] : src[(int64_t)r * u.ld + k]) : 0.0;
      }
    }
    uint32_t w[kTcxSlices][4];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      int d0[kTcxSlices], d1[kTcxSlices];
      digits6(x[e], live ? em + 1 : 0, d0);
      digits6(x[e + 1], live ? em + 1 : 0, d1);
#pragma unroll
      for (int s = 0; s < kTcxSlices; ++s) w[s][e >> 1] = bf16x2_of(d0[s], d1[s]);
    }
    const int t = r / u.rt, c = k0 / kTcKC, kk = k0 % kTcKC;
    const int rest = u.rows_p - u.rt * t;
    const int h = rest < u.rt ? rest : u.rt;
    const int64_t off = (int64_t)kTcxSlices * (tc_block_off(u.rows_p, u.kp, t, c, u.rt) + (int64_t)(kk >> 3) * h * 8) +
                        (int64_t)(r - u.rt * t) * 8;
#pragma unroll
    for (int s = 0; s < kTcxSlices; ++s)
      *(uint4*)(dst + off + (int64_t)s * h * 8) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
  }
}

constexpr int kTcxSlots = 5;  // stages of one K=16 step
constexpr uint32_t kTcxStageBytes = (uint32_t)kTcxSlices * (kTcRowsA + kTcxNB) * kTcxKS * 2;
// TMEM: two halves of 256 columns, each for the six accumulators of a block of
// MMAs, in turn
constexpr uint32_t kTcxTmemCols = 512, kTcxTmemHalf = 256;
static_assert(kTcxSlices * kTcxNB <= (int)kTcxTmemHalf && kTcxNB % 16 == 0, "six accumulators in half of TMEM");
// warps 0-15 epilogue (warp w: TMEM lanes 32 (w % 4).., quarter w / 4 of the
// tile columns), 16 producer, 17 MMA issuer
constexpr int kTcxEpiWarps = 16;
constexpr int kTcxThreads = 32 * (kTcxEpiWarps + 2);
constexpr int kTcxProducer = kTcxEpiWarps, kTcxIssuer = kTcxEpiWarps + 1;
constexpr int kTcxCols = kTcxNB / 4;  // tile columns per epilogue thread, at most
constexpr int kTcxStepsPerBlock = kTcxKBlock / kTcxKS;

// the epilogue's part of an item: its record and the exponents of the tile's
// rows and columns
struct __align__(16) TcxItem {
  TcxWork w;
  int ea[kTcRowsA], eb[kTcxNB];
};
constexpr int kTcxItems = 8;  // in flight
// joined accumulators of an item, by thread: in registers they and the sums did
// not fit (1348 us in place of 1324 at 20 orbitals M=300)
constexpr int kTcxJoin = kTcxCols * 32 * kTcxEpiWarps * 8;
// shared memory: joined accumulators, items, stages.  An MMA reads 128 rows of A, also of a shorter
// tile and of one that goes to the lanes from row0 on: up to 1.5 KB before its
// stage and, of a tile of few rows, 2 KB behind it, inside the stage.
constexpr int kTcxRing = kTcxJoin + kTcxItems * (int)sizeof(TcxItem);
static_assert(kTcxRing >= 96 * 16 && kTcxRing % 16 == 0, "rows read before the first stage");
constexpr int kTcxSmem = kTcxRing + kTcxSlots * (int)kTcxStageBytes;

struct TcxShared {
  uint64_t full[kTcxSlots], empty[kTcxSlots];
  uint64_t acc_full[2][4], acc_empty[2][4];  // by TMEM half and lane quarter
  uint64_t item_full[kTcxItems], item_empty[kTcxItems], drain;
  uint32_t tbase;
  int abort_flag;
};

__device__ bool tcx_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, uint64_t limit_ns) {
  for (int i = 0; i < kSpinPolls; ++i)  // without the clock first (tc_wait)
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

// Each role reads what it needs of a record straight into registers, the next
// ones ahead (handing out records held one per lane by shuffles takes longer
// than the copies of a small item).
constexpr int kTcxAhead = 4;  // records prefetched into L1
// the producer and the MMA issuer: operand places (the producer's), K, tile
// heights h_a | h_b << 16, pools and flags
struct XCopy {
  int4 base;
  int kp, a_ex, b_ex, hw, pf;
};
__device__ __forceinline__ XCopy load_xcopy(const TcxWork* __restrict__ w, int i, int end, bool places) {
  XCopy r{};
  if (i < end) {
    const int4* p = reinterpret_cast<const int4*>(w + i);
    if (places) {
      r.base = __ldg(p);
      r.a_ex = __ldg(&w[i].a_ex);
      r.b_ex = __ldg(&w[i].b_ex);
    }
    r.kp = __ldg(&w[i].kp);
    r.hw = __ldg(reinterpret_cast<const int*>(p + 3) + 2);
    r.pf = __ldg(reinterpret_cast<const int*>(p + 4));
    if (i + kTcxAhead < end) asm volatile("prefetch.global.L1 [%0];" ::"l"(w + i + kTcxAhead));
  }
  return r;
}

// reads of an item, kept in their place between its wait and item_read
__device__ __forceinline__ int4 lds_v4(const void* p) {
  int4 r;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(smem_u32(p)) : "memory");
  return r;
}
__device__ __forceinline__ int lds(const void* p) {
  int r;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(r) : "r"(smem_u32(p)) : "memory");
  return r;
}

// The place of an item whose fields this warp has read goes back to the producer,
// whose bulk copies fill it again.  Those writes belong to the async proxy: the
// proxy fence puts a lane's reads before them, __syncwarp the other lanes' fences
// before lane 0's arrival, and the arrival comes before the producer's wait and its
// copies.  (20 orbitals M=300: 1181 us a product; with the exponents read into
// registers and the place given back before the sums 1272.)
__device__ __forceinline__ void item_read(uint64_t* bar, int lane) {
  fence_async_smem();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// 32 lanes x 4 columns of six accumulators hb columns apart, one wait (which
// names the values, so that nothing made of them can come before it)
__device__ __forceinline__ void tmem_ld4x6(uint32_t t, uint32_t hb, uint32_t (&r)[kTcxSlices][4]) {
#pragma unroll
  for (int q = 0; q < kTcxSlices; ++q) {
    const uint32_t a = t + (uint32_t)q * hb;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[q][0]), "=r"(r[q][1]), "=r"(r[q][2]), "=r"(r[q][3])
                 : "r"(a));
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0][0]), "+r"(r[0][1]), "+r"(r[0][2]), "+r"(r[0][3]),
                 "+r"(r[1][0]), "+r"(r[1][1]), "+r"(r[1][2]), "+r"(r[1][3]),
                 "+r"(r[2][0]), "+r"(r[2][1]), "+r"(r[2][2]), "+r"(r[2][3]),
                 "+r"(r[3][0]), "+r"(r[3][1]), "+r"(r[3][2]), "+r"(r[3][3]),
                 "+r"(r[4][0]), "+r"(r[4][1]), "+r"(r[4][2]), "+r"(r[4][3]),
                 "+r"(r[5][0]), "+r"(r[5][1]), "+r"(r[5][2]), "+r"(r[5][3])
               :
               : "memory");
}

// 32 bytes of FP64 values (32-byte aligned)
__device__ __forceinline__ void st_global_v4(double* p, double x, double y, double z, double w) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(w) : "memory");
}

// the six accumulators of an element (integers: J_0 below 2^23, J_4 128 + J_5
// below 2^31) as one: sum_q J_q 128^(5-q), below 2^59.  The conversion unit
// takes an eighth of the rate of the adders, so that accumulators below 2^22
// (SMALL: at most 2^15 per K, so 128 K) become integers by the addition of
// 1.5 2^23, which leaves them in the low bits of the sum.
template <bool SMALL>
__device__ __forceinline__ int as_int(uint32_t f) {
  if (SMALL) return __float_as_int(__uint_as_float(f) + 12582912.f) - 0x4B400000;
  return __float2int_rn(__uint_as_float(f));
}
template <bool SMALL>
__device__ __forceinline__ long long join6(const uint32_t (&r)[kTcxSlices][4], int e) {
  const int p0 = as_int<SMALL>(r[0][e]) * 128 + as_int<SMALL>(r[1][e]);
  const int p1 = as_int<SMALL>(r[2][e]) * 128 + as_int<SMALL>(r[3][e]);
  const int p2 = as_int<SMALL>(r[4][e]) * 128 + as_int<SMALL>(r[5][e]);
  return (long long)p0 * (1ll << 28) + ((long long)p1 * (1ll << 14) + p2);
}

// a 2^k (|a| < 2^62, |k| <= 960), rounded as (double)a is, by integer
// operations: the conversion would take a slot of the FP64 pipe, which the sums
// need
__device__ __forceinline__ double scaled(long long a, int k) {
  const long long s = a >> 63;
  const unsigned long long m = (unsigned long long)((a ^ s) - s);
  const int lz = __clzll((long long)m);
  unsigned long long t = m << (lz - 1 < 0 ? 0 : lz - 1);  // leading bit 62
  t += 0x1ff + ((t >> 10) & 1);                           // to 53 bits, to nearest, ties to even
  const long long bits = (long long)(t >> 10) + ((long long)(1085 - lz + k) << 52);
  return __longlong_as_double(a == 0 ? 0ll : bits | (s & (1ll << 63)));
}

}  // namespace

// Persistent grouped exact-slice GEMM: per K=16 step the 21 digit products
// (s, u), s + u <= 5, into accumulator s + u; accumulators are read out after
// every kTcxKBlock K of an item and at its end.  Phase 1 writes the T tiles
// (FP64) and reduces their row exponents; phase 2 sums the items of a task in
// FP64 registers and writes sigma or a partial tile.
// Tiles are 128 x 32: the six accumulators fill half of TMEM, so that one item
// is read out while the next is multiplied (20 orbitals M=300, 1245 us a product
// in place of 1386 with tiles of 64 columns, which need all of TMEM).
template <int PHASE>
__global__ void __launch_bounds__(kTcxThreads, 1)
    tcx_sigma_kernel(TcxBufs b, const TcxWork* __restrict__ work, const int2* __restrict__ ranges,
                     double* __restrict__ sigma, uint64_t limit_ns) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ TcxShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int2 rg = ranges[blockIdx.x];
  if (warp == kTcxIssuer) {
    tmem_alloc(&sh.tbase, kTcxTmemCols);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < kTcxSlots; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 1);
    }
    for (int i = 0; i < kTcxItems; ++i) {
      mbar_init(&sh.item_full[i], 1);
      mbar_init(&sh.item_empty[i], kTcxEpiWarps);
    }
    for (int i = 0; i < 8; ++i) {
      mbar_init(&sh.acc_full[i >> 2][i & 3], 1);
      mbar_init(&sh.acc_empty[i >> 2][i & 3], kTcxEpiWarps / 4);
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
  TcxItem* itm = reinterpret_cast<TcxItem*>(smem + kTcxJoin);
  uint8_t* ring = smem + kTcxRing;

  if (warp == kTcxProducer) {
    // ---- producer (lane 0): the epilogue's part of every item, and one stage
    // per K=16 step, A then B
    if (lane == 0) {
      uint32_t k = 0, items = 0;  // stages and items filled
      int slot = 0;
      uint32_t ph = 0;
      bool ok = true;
      XCopy n0 = load_xcopy(work, rg.x, rg.y, true), n1 = load_xcopy(work, rg.x + 1, rg.y, true);
      for (int i = rg.x; i < rg.y && ok; ++i) {
        const XCopy r = n0;
        n0 = n1;
        n1 = load_xcopy(work, i + 2, rg.y, true);
        const bool empty = ((r.pf >> 16) & kTcEmpty) != 0;
        const int ni = i - rg.x, it = ni % kTcxItems;
        if (!tcx_wait(&sh.item_empty[it], ((ni / kTcxItems) & 1u) ^ 1u, abort_flag, b.status, limit_ns)) {
          ok = false;
          break;
        }
        // (rows and columns come in multiples of 8: 32 bytes of exponents)
        const uint32_t ra = empty ? 0u : 4u * (r.hw & 0xffff), rb = empty ? 0u : 4u * ((r.hw >> 16) & 0xffff);
        mbar_expect_tx(&sh.item_full[it], (uint32_t)sizeof(TcxWork) + ra + rb);
        bulk_g2s(&itm[it].w, work + i, (uint32_t)sizeof(TcxWork), &sh.item_full[it]);
        ++items;
        if (empty) continue;
        bulk_g2s(itm[it].ea, pick_x(b.ex, r.pf & 0xff) + r.a_ex, ra, &sh.item_full[it]);
        bulk_g2s(itm[it].eb, pick_x(b.ex, (r.pf >> 8) & 0xff) + r.b_ex, rb, &sh.item_full[it]);
        const uint32_t abytes = (uint32_t)kTcxSlices * (r.hw & 0xffff) * kTcxKS * 2;
        const uint32_t bbytes = (uint32_t)kTcxSlices * ((r.hw >> 16) & 0xffff) * kTcxKS * 2;
        const int64_t oa = (int64_t)(((uint64_t)(uint32_t)r.base.y << 32) | (uint32_t)r.base.x);
        const int64_t ob = (int64_t)(((uint64_t)(uint32_t)r.base.w << 32) | (uint32_t)r.base.z);
        const uint8_t* pa = reinterpret_cast<const uint8_t*>(pick_x(b.pool, r.pf & 0xff) + oa);
        const uint8_t* pb = reinterpret_cast<const uint8_t*>(pick_x(b.pool, (r.pf >> 8) & 0xff) + ob);
        for (int left = r.kp; left > 0; left -= kTcxKS, ++k) {
          if (!tcx_wait(&sh.empty[slot], ph ^ 1u, abort_flag, b.status, limit_ns)) {
            ok = false;
            break;
          }
          uint8_t* dst = ring + (uint32_t)slot * kTcxStageBytes;
          mbar_expect_tx(&sh.full[slot], abytes + bbytes);
          bulk_g2s(dst, pa, abytes, &sh.full[slot]);
          bulk_g2s(dst + abytes, pb, bbytes, &sh.full[slot]);
          pa += abytes;
          pb += bbytes;
          if (++slot == kTcxSlots) {
            slot = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok) {  // no copy in flight when the block ends
        for (uint32_t i = (k > kTcxSlots ? k - kTcxSlots : 0); i < k; ++i)
          mbar_wait_bounded(&sh.full[i % kTcxSlots], (i / kTcxSlots) & 1u, limit_ns);
        for (uint32_t i = (items > kTcxItems ? items - kTcxItems : 0); i < items; ++i)
          mbar_wait_bounded(&sh.item_full[i % kTcxItems], (i / kTcxItems) & 1u, limit_ns);
      }
    }
  } else if (warp == kTcxIssuer) {
    // ---- MMA issuer: the whole warp walks the records, one lane issues
    // (mma_bf16_if).  Slice s of A meets slices 0 .. 5 - s of B, which lie row
    // after row, in one MMA of 6 - s times the tile's columns; product (s, u)
    // lands in the columns of accumulator s + u by itself.  Six MMAs a K=16 step
    // take 384 clocks at 128 x 32 (an MMA for each of the 21 products, issued by
    // one lane: 1700 at 128 x 64).
    const bool on = elect_one();
    const uint32_t sm0 = smem_u32(ring) >> 4;
    constexpr uint64_t kDescHi = smem_desc_hi();
    constexpr uint32_t kIdesc0 = idesc_bf16(128, 0);
    int slot = 0;
    uint32_t ph = 0, aph = 0, sel = 0, tm = tmem;
    uint32_t busy[2] = {0, 0};  // lane quarters that have yet to read a half's last block
    bool ok = true, ready = false;
    XCopy n0 = load_xcopy(work, rg.x, rg.y, false), n1 = load_xcopy(work, rg.x + 1, rg.y, false);
    for (int i = rg.x; i < rg.y && ok; ++i) {
      const int kp = uniform(n0.kp), hw = uniform(n0.hw), pf = uniform(n0.pf);
      n0 = n1;
      n1 = load_xcopy(work, i + 2, rg.y, false);
      if ((pf >> 16) & kTcEmpty) continue;
      const uint32_t ha = (uint32_t)hw & 0xffffu, hb = (uint32_t)hw >> 16, row0 = (uint32_t)pf >> 24;
      const uint32_t quarters = ((1u << (ha + 31) / 32) - 1) << row0 / 32;  // lane quarters of the tile's rows
      const uint32_t id = (hb >> 3) << 17;  // instruction descriptor of hb columns, less the rest
      const int nst = kp / kTcxKS;
      for (int st = 0; st < nst; ++st) {
        const int at = st % kTcxStepsPerBlock;
        const bool last = at == kTcxStepsPerBlock - 1 || st == nst - 1;
        if (at == 0) {  // the other half of TMEM
          tm = tmem + sel * kTcxTmemHalf;
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h)
            if (sel == h) {
#pragma unroll
              for (uint32_t q = 0; q < 4; ++q)
                if (busy[h] >> q & 1) {
                  ok = ok && __all_sync(0xffffffffu, tcx_wait(&sh.acc_empty[h][q], aph >> (4 * h + q) & 1, abort_flag, b.status, limit_ns));
                  aph ^= 1u << (4 * h + q);
                }
              busy[h] = quarters;
            }
          if (!ok) break;
        }
        if (!ready && !__all_sync(0xffffffffu, tcx_wait(&sh.full[slot], ph, abort_flag, b.status, limit_ns))) {
          ok = false;
          break;
        }
        fence_after_sync();
        // rows of a half, six slices: the leading byte offset is 6 h 16 bytes;
        // A read from row0 rows before the tile: its rows land in TMEM lanes row0..
        const uint32_t a0 = sm0 + (uint32_t)slot * (kTcxStageBytes >> 4);
        const uint64_t da = kDescHi | (a0 - row0) | (6 * ha << 16);
        const uint64_t db = kDescHi | (a0 + 12 * ha) | (6 * hb << 16);
        const int slot_c = slot;
        const uint32_t acc = at == 0 ? 0u : 1u;
        mma_bf16_if(on, tm, da, db, kIdesc0 | 6 * id, acc);               // s = 0
        mma_bf16_if(on, tm + 5 * hb, da + 5 * ha, db, kIdesc0 | id, 1u);  // s = 5
        if (++slot == kTcxSlots) {
          slot = 0;
          ph ^= 1u;
        }
#pragma unroll
        for (uint32_t s = 4; s > 0; --s) mma_bf16_if(on, tm + s * hb, da + s * ha, db, kIdesc0 | (6 - s) * id, 1u);
        const bool probe = mbar_test(&sh.full[slot], ph);
        mma_commit_if(on, &sh.empty[slot_c]);
        if (last) {
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q)
            if (quarters >> q & 1) mma_commit_if(on, &sh.acc_full[sel][q]);
          sel ^= 1u;
        }
        ready = __all_sync(0xffffffffu, probe);
      }
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4).. and quarter w / 4 of
    // the tile's columns; a thread keeps the FP64 sums of its row and columns in
    // registers.  The MMAs wait for the read-out only, which joins the six
    // accumulators of an element into one integer; rounding to FP64 and the sums
    // run beside the MMAs of the items that follow.  A tile of few rows takes the
    // TMEM lanes, and the warps that read them, from row0 on: tasks side by side
    // in the records take different ones.  This work bounds the kernel where K
    // is short (20 orbitals M=300, tiles of 34 rows, 24 columns and K = 60 on
    // average: 3300 clocks an item, 1300 of them MMAs).  With 8 warps, of twice
    // the columns, it took 1.15 times as long; code that spilled registers
    // up to twice, since little L1 is left beside the stages.
    // FP64 operations take 63 clocks a warp, and shared-memory reads queue behind
    // them, so that an item's record is read before its sums.
    const int lane_row = 32 * (warp & 3) + lane;
    long long* joined = reinterpret_cast<long long*>(smem) + tid;  // column c at 32 kTcxEpiWarps c
    const uint32_t lane_base = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    uint32_t aph = 0, sel = 0;
    bool ok = true;
    double acc[kTcxCols];
#pragma unroll
    for (int c = 0; c < kTcxCols; ++c) acc[c] = 0.0;
    for (int i = rg.x; i < rg.y && ok; ++i) {
      const int ni = i - rg.x, it = ni % kTcxItems;
      ok = __all_sync(0xffffffffu, tcx_wait(&sh.item_full[it], (ni / kTcxItems) & 1u, abort_flag, b.status, limit_ns));
      if (!ok) break;
      const TcxItem& x = itm[it];
      const int pf = lds(&x.w.a_pool), hw = lds(&x.w.h_a), kp = lds(&x.w.kp);
      const int flags = (pf >> 16) & 0xff, ha = hw & 0xffff, hb = hw >> 16;
      const int own = hb >> 2, cb = (warp >> 2) * own;  // this warp's columns
      const int row = lane_row - (int)((uint32_t)pf >> 24);
      const bool mine = row >= 0 && row < ha;
      if (!__any_sync(0xffffffffu, mine)) {  // another quarter's item
        if (!(flags & kTcEmpty)) sel ^= ((uint32_t)(kp + kTcxKBlock - 1) / kTcxKBlock) & 1u;
        item_read(&sh.item_empty[it], lane);
        continue;
      }
      const int4 q1 = lds_v4(&x.w.out_base), q2 = lds_v4(&x.w.kp), q3 = lds_v4(&x.w.b_ex);
      const double alpha = __hiloint2double(q1.w, q1.z);
      // the thread's row and first column in T, sigma or the partial tile; the
      // place of the row's exponent, or the valid rows and columns
      const int64_t at = (int64_t)(((uint64_t)(uint32_t)q1.y << 32) | (uint32_t)q1.x) + (int64_t)row * q2.y + cb + (PHASE == 1 ? q2.z : 0);
      const int aux = PHASE == 1 ? q3.y : q3.w;
      if (flags & kTcFirst) {
#pragma unroll
        for (int c = 0; c < kTcxCols; ++c) acc[c] = 0.0;
      }
      if (!(flags & kTcEmpty)) {
        // zero rows and columns have zero digits, whatever their exponent
        const int ea = mine ? lds(x.ea + row) : kTcxNoExp, ec = lane < own ? lds(x.eb + cb + lane) : kTcxNoExp;
        const int ka = (ea > kTcxNoExp / 2 ? ea : 0) + 2 - 7 * (kTcxSlices + 1);
        const bool far = __any_sync(0xffffffffu, (ea > kTcxNoExp / 2 && abs(ea) > 440) || (ec > kTcxNoExp / 2 && abs(ec) > 440));
        for (int left = kp; left > 0; left -= kTcxKBlock) {
          ok = __all_sync(0xffffffffu, tcx_wait(&sh.acc_full[sel][warp & 3], aph >> sel & 1u, abort_flag, b.status, limit_ns));
          if (!ok) break;
          aph ^= 1u << sel;
          fence_after_sync();
#pragma unroll 1
          for (int g = 0; g < own; g += 4) {
            uint32_t v[kTcxSlices][4];
            tmem_ld4x6(lane_base + sel * kTcxTmemHalf + (uint32_t)(cb + g), (uint32_t)hb, v);
            long long* j = joined + g * (32 * kTcxEpiWarps);
            if (left <= 128) {
#pragma unroll
              for (int e = 0; e < 4; ++e) j[e * (32 * kTcxEpiWarps)] = join6<true>(v, e);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) j[e * (32 * kTcxEpiWarps)] = join6<false>(v, e);
            }
          }
          // accumulators read: the MMA issuer may use their half again
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.acc_empty[sel][warp & 3]);
          __syncwarp();
          sel ^= 1u;
#pragma unroll
          for (int g = 0; g < kTcxCols; g += 4) {
            if (g >= own) break;
            const int4 e4 = lds_v4(x.eb + cb + g);
            const int eb[4] = {e4.x, e4.y, e4.z, e4.w};
            double y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int k = ka + (eb[e] > kTcxNoExp / 2 ? eb[e] : 0);
              y[e] = scaled(joined[(g + e) * (32 * kTcxEpiWarps)], max(-960, min(960, k)));
            }
            if (far) {  // the rest of a scale out of the range of one factor
              asm volatile("");  // (else all products are formed in any case, and dropped)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int k = ka + (eb[e] > kTcxNoExp / 2 ? eb[e] : 0), k2 = k - max(-960, min(960, k));
                y[e] *= __longlong_as_double((long long)(1023 + max(-1022, min(1023, k2))) << 52);
              }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[g + e] = fma(y[e], alpha, acc[g + e]);
          }
        }
        if (!ok) break;
      }
      item_read(&sh.item_empty[it], lane);
      if (!(flags & kTcLast)) continue;
      // the task's tile is complete in this thread's row and columns
      if (PHASE == 1) {
        if (mine) {  // 32-byte aligned: rows and tiles of T are multiples of 16 columns
          double* out = b.t + at;
          int m = kTcxNoExp;
#pragma unroll
          for (int c = 0; c < kTcxCols; c += 4)
            if (c < own) {
              st_global_v4(out + c, acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
#pragma unroll
              for (int e = 0; e < 4; ++e) m = max(m, exp_of(acc[c + e]));
            }
          if (m > kTcxNoExp / 2) atomicMax(b.ex[kTcPoolS] + aux + row, m);
        }
      } else if (flags & kTcDirect) {
        if (row >= 0 && row < (aux & 0xffff)) {
          const int nc = min((aux >> 16) - cb, own);
          double* out = sigma + at;
#pragma unroll
          for (int c = 0; c < kTcxCols; ++c)
            if (c < nc) out[c] = acc[c];
        }
      } else if (mine) {
        double* out = b.partials + at;
#pragma unroll
        for (int c = 0; c < kTcxCols; c += 4)
          if (c < own) st_global_v4(out + c, acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      }
    }
  }
  __syncthreads();
  if (warp == kTcxIssuer) {
    // every MMA of this block has completed before TMEM is released
    if (elect_one()) {  // the lane that issued them
      mma_commit(&sh.drain);
      mbar_wait_bounded(&sh.drain, 0, limit_ns);
    }
    __syncwarp();
    fence_after_sync();
    tmem_dealloc(tmem, kTcxTmemCols);
  }
}

__global__ void __launch_bounds__(256) tcx_reduce_kernel(const double* __restrict__ partials,
                                                          const TcTile* __restrict__ tiles,
                                                          const int64_t* __restrict__ slots, double* __restrict__ sigma) {
  const TcTile t = tiles[blockIdx.x];
  const int n = t.h * t.w;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < n; e += gridDim.y * blockDim.x) {
    double acc = 0.0;
    const int r = e / t.w, c = e % t.w;
    const double* src = partials + (int64_t)r * t.pad + c;
    int p = t.pbeg;
    for (; p + 8 <= t.pend; p += 8) {  // eight partials in flight, summed in slot order
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = src[slots[p + i]];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc += v[i];
    }
    for (; p < t.pend; ++p) acc += src[slots[p]];
    sigma[t.s_off + (int64_t)(t.r0 + r) * t.lds + t.c0 + c] = acc;
  }
}

__global__ void fill_int_kernel(int* x, int64_t n, int v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] = v;
}

cudaError_t launch_tcx_rowexp(const TcxBufs& b, const TcPack* units, int nunits, cudaStream_t s, int split) {
  if (nunits > 0) tcx_rowexp_kernel<<<dim3(nunits, split), 256, 0, s>>>(b, units);
  return cudaGetLastError();
}

cudaError_t launch_tcx_pack(const TcxBufs& b, const TcPack* units, int nunits, cudaStream_t s, int split) {
  if (nunits > 0) tcx_pack_kernel<<<dim3(nunits, split), 256, 0, s>>>(b, units);
  return cudaGetLastError();
}

template <int PHASE>
static cudaError_t launch_tcx_phase(const TcxBufs& b, const TcxWork* work, const int2* ranges, int nblocks,
                                    double* sigma, uint64_t limit_ns, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(tcx_sigma_kernel<PHASE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcxSmem);
  if (e != cudaSuccess) return e;
  tcx_sigma_kernel<PHASE><<<nblocks, kTcxThreads, kTcxSmem, s>>>(b, work, ranges, sigma, limit_ns);
  return cudaGetLastError();
}

cudaError_t launch_tcx_sigma(int phase, const TcxBufs& b, const TcxWork* work, const int2* ranges, int nblocks,
                             double* sigma, uint64_t limit_ns, cudaStream_t s) {
  if (nblocks <= 0) return cudaGetLastError();
  if (phase == 1) return launch_tcx_phase<1>(b, work, ranges, nblocks, sigma, limit_ns, s);
  if (phase == 2) return launch_tcx_phase<2>(b, work, ranges, nblocks, sigma, limit_ns, s);
  return cudaErrorInvalidValue;
}

int tcx_blocks_per_sm() { return 1; }

cudaError_t launch_tcx_reduce(const TcxBufs& b, const TcTile* tiles, const int64_t* slots, int ntiles, double* sigma,
                              cudaStream_t s, int split) {
  if (ntiles > 0) tcx_reduce_kernel<<<dim3(ntiles, split), 256, 0, s>>>(b.partials, tiles, slots, sigma);
  return cudaGetLastError();
}

cudaError_t launch_fill_int(int* x, int64_t n, int v, cudaStream_t s) {
  if (n > 0) fill_int_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, s>>>(x, n, v);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace bgpu
