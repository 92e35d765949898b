// FP32 block matmul on the tensor cores.
//
// An f32 value is the exact sum of three bf16 values (8 significant bits each):
//     a = a0 + 2^-8 a1 + 2^-16 a2,   a0 = bf16(a), a1 = bf16((a - a0) 2^8), ...
// The planes are scaled so that each has a0's exponent range: no plane
// underflows before a itself does. A product a b is then
//     a0 b0 + 2^-8 (a0 b1 + a1 b0) + 2^-16 (a0 b2 + a1 b1 + a2 b0) + O(2^-26 |a b|),
// six bf16 products that tcgen05.mma forms exactly and accumulates in f32. The
// three dropped products are below a quarter of an ulp of a b.
//
// Accumulation. The tensor core truncates when it accumulates, so a long K loop
// in one accumulator loses about K * 2^-26 (relative, measured: 1.0e-6 at K = 1024, 4.0e-6
// at K = 4096, where the FMA chain of k_gemm_f32 loses 5.7e-7 and 1.2e-6). Here
// the MMA accumulates only kF3BK = 64 steps of K: the 2^-16 products first, then the
// accumulator is scaled by 2^-8 in the MMA itself (scale-input-d) and takes the
// 2^-8 products, then once more and the leading product, so only the last four
// MMAs truncate at the size of the result. The epilogue warps add each chunk to
// FP32 registers with round-to-nearest while the next chunk runs in the other
// TMEM buffer.
//
// Operands are read from their split planes (k_f32_split): TMA tiles of one
// plane through a 3-D map (columns, rows, plane * batch + b), in whichever
// major-ness the block has. A stage holds the six plane tiles of a chunk (128
// rows x 64 of K, 16 KiB each), two stages fill the shared memory, and each tile is
// handed back on its own as soon as the last product that reads it retires.
//
// Shapes: PAIR, a 256 x 256 tile on two SMs (cta_group::2: each SM loads 128
// rows of A and of B), and a 128 x 128 tile on one SM for groups with too few tiles to
// fill the chip with pairs. Both compute each output by the same chain of
// operations, so the shape changes no bit of the result. Shared memory sets the pace of
// the smaller: per chunk of K its MMAs read 24 x 8 KiB and the TMA writes 96 KiB at
// 128 bytes a cycle, 2300 cycles where the tensor pipe needs 1536 (measured 2190); the pair
// spreads the same traffic over the 3072 cycles of a tile twice as wide (measured 3600;
// a 256 x 128 pair measured 2950, more per output than either).
//
// The producer and MMA warps run converged, with one elected lane issuing, so that
// the TMA and MMA operands are uniform; a problem's fields are read once per tile
// into registers, from the kernel parameters when there is a single problem.
//
// A problem whose operands could leave the range of the scheme (non-finite, or
// large enough that a partial sum could overflow where an FP32 FMA chain does
// not; see f3_in_range) is skipped by every warp's main loop and computed after
// it by the epilogue warps, with FP32 FMAs in K order and k_gemm_f32_v's tiling
// (f3_plain_tiles). No bounded wait spans that: the tensor-core part is over.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include "gemm_f32.cuh"
#include "ptx.cuh"
#include "tile_order.h"

namespace bbx {

constexpr int kF3BK = 64;
constexpr int kF3Tile = 128 * kF3BK * 2;      // one plane tile of 128 rows, 16 KiB
constexpr int kF3Stage = 6 * kF3Tile;         // A0 A1 A2 B0 B1 B2
constexpr int kF3MaxProblems = 256;           // per launch
constexpr int kF3EpiPitch = 20;               // floats; 80-byte rows keep 16-byte accesses conflict-free
constexpr int kF3EpiSlot = 32 * kF3EpiPitch * 4;
constexpr int kF3EpiWarps = 8;
constexpr int kF3Threads = 64 + 32 * kF3EpiWarps;
constexpr int kF3Smem =
    2 * kF3Stage + 1024 /* align slack */ + kF3EpiWarps * kF3EpiSlot + 256 /* barriers */ + kF3MaxProblems * 16;
static_assert(kF3Smem <= 232448, "dynamic shared memory per CTA");

// One (batched) product. 64-byte alignment is required by the tensor maps.
struct F3Fields {
  const __nv_bfloat16* a;      // plane 0 of the operands, for problems out of range
  const __nv_bfloat16* b;
  float* c;
  const float* bias;
  const uint32_t* amax_a;      // na / nb partial maxima of |a| and |b| (float bits), written by the split
  const uint32_t* amax_b;
  // element (row, k) of A's plane p: a + p * a_plane + batch * a_batch + row * a_row + k * a_k, and so on
  long long a_plane, a_row, a_k, a_batch, b_plane, b_col, b_k, b_batch, ldc, c_batch;
  int m, n, k, batch;
  int na, nb;
  int tile_start, tiles_m, tiles_n;
  int a_mn, b_mn;              // operand tiles are MN-major
  int c_col;                   // element (i, j) of C at c[i + j * ldc], else c[i * ldc + j]
  float alpha, beta;
};
struct alignas(64) F3Problem {
  CUtensorMap tmap_a, tmap_b;  // split planes, box 64 columns x 128 rows (K-major) or 64 x 64 (MN-major)
  F3Fields f;
};

struct F3Args {
  const F3Problem* table;  // device table, or nullptr: `one`
  int num_problems;
  int total_tiles;
  uint32_t* status;
  F3Problem one;
};

// |a| < 2^ea, |b| < 2^eb for the maxima's exponents. The largest partial sum of
// the scheme is below 3 K 2^(ea + eb) < 2^(ea + eb + lk + 2): kept below 2^127, so nothing
// overflows that an FMA chain would not. The upper limit on each operand keeps
// bf16(a) finite. Products that are all below 2^-80 are left to the FMA chain,
// which rounds them to f32 subnormals as the reference does.
__host__ __device__ __forceinline__ bool f3_in_range(uint32_t amax, uint32_t bmax, int k) {
  if (amax >= 0x7F7F8000u || bmax >= 0x7F7F8000u) return false;  // also inf and NaN
  if (amax == 0 || bmax == 0) return true;
  const int ea = (int)(amax >> 23) - 126, eb = (int)(bmax >> 23) - 126;
#ifdef __CUDA_ARCH__
  const int lk = 32 - __clz(k - 1);  // 2^lk >= k
#else
  int lk = 0;
  while ((1ll << lk) < k) ++lk;
#endif
  return ea + eb + lk + 2 <= 127 && ea + eb >= -80;
}

// ------------------------------------------------------------------ split into planes
// One matrix (or gathered tensor) to split: rows indexed by up to three outer
// dimensions, `len` elements along a row.
struct F3Split {
  const float* src;
  __nv_bfloat16* dst;          // plane p at dst + p * plane
  long long plane;             // elements
  long long odims[3], istride[3], ostride[3];  // outer dims, outermost first; unused ones have extent 1
  long long len, inner, oinner;  // elements of a row, their source and destination strides
  long long items;             // rows * ceil(len / 8)
  long long items_per_chunk;
  uint32_t* amax;              // one word per chunk
  int chunk_start;             // first chunk of this record in the launch
  int rank_s;                  // modes summed at each element (0: none)
  long long sdims[4], sstride[4];
};

struct F3SplitArgs {
  const F3Split* table;        // device table, or nullptr: `inl`
  int count;
  F3Split inl[2];
};

// bf16 of a finite value, rounded to nearest, but never to infinity.
__device__ __forceinline__ __nv_bfloat16 f3_bf16_finite(float x) {
  const __nv_bfloat16 p = __float2bfloat16_rn(x);
  return fabsf(__bfloat162float(p)) <= 3.3895314e38f ? p : __ushort_as_bfloat16((unsigned short)(__float_as_uint(x) >> 16));
}

// The planes of any f32 value: f3_join2 gives the value back exactly (a NaN as a NaN).
__device__ __forceinline__ void f3_split1(float x, __nv_bfloat16& p0, __nv_bfloat16& p1, __nv_bfloat16& p2) {
  const uint32_t mag = __float_as_uint(x) & 0x7FFFFFFFu;
  if (mag >= 0x7F800000u) {
    p0 = __float2bfloat16_rn(x);
    p1 = p2 = __ushort_as_bfloat16(0);
    return;
  }
  p0 = mag < 0x7F000000u ? __float2bfloat16_rn(x) : f3_bf16_finite(x);
  const float r1 = __fmul_rn(__fsub_rn(x, __bfloat162float(p0)), 256.f);  // exact
  p1 = mag < 0x7F000000u ? __float2bfloat16_rn(r1) : f3_bf16_finite(r1);
  p2 = __float2bfloat16_rn(__fmul_rn(__fsub_rn(r1, __bfloat162float(p1)), 256.f));
}

// Two neighbouring elements from the words that hold their planes.
__device__ __forceinline__ float2 f3_join2(uint32_t p0, uint32_t p1, uint32_t p2) {
  auto join = [](uint32_t a, uint32_t b, uint32_t c) {  // bf16 values in the upper halves
    const float lo = __fadd_rn(__fmul_rn(__uint_as_float(b), 1.f / 256.f), __fmul_rn(__uint_as_float(c), 1.f / 65536.f));
    return __fadd_rn(__uint_as_float(a), lo);
  };
  return make_float2(join(p0 << 16, p1 << 16, p2 << 16), join(p0 & 0xFFFF0000u, p1 & 0xFFFF0000u, p2 & 0xFFFF0000u));
}

// The planes of eight elements as 16-byte pieces, and the maximum of their magnitudes.
__device__ __forceinline__ void f3_split8(const float (&v)[8], uint4 (&p)[3], uint32_t& mx) {
  uint32_t w[3][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    __nv_bfloat16 x[3], y[3];
    mx = max(mx, max(__float_as_uint(v[2 * u]) & 0x7FFFFFFFu, __float_as_uint(v[2 * u + 1]) & 0x7FFFFFFFu));
    f3_split1(v[2 * u], x[0], x[1], x[2]);
    f3_split1(v[2 * u + 1], y[0], y[1], y[2]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
      w[q][u] = (uint32_t)__bfloat16_as_ushort(x[q]) | ((uint32_t)__bfloat16_as_ushort(y[q]) << 16);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) p[q] = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
}

// Each CTA writes the maximum of |x| over its chunk as one word, so no counter
// has to be cleared before the launch. All 256 threads.
__device__ __forceinline__ void f3_chunk_max(uint32_t mx, uint32_t* out) {
  mx = __reduce_max_sync(0xffffffffu, mx);
  __shared__ uint32_t wm[8];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) mx = max(mx, wm[w]);
    *out = mx;
  }
}

__device__ __forceinline__ const F3Split& f3_split_record(const F3SplitArgs& args, int chunk) {
  const F3Split* const recs = args.table ? args.table : args.inl;
  int lo = 0, hi = args.count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (recs[mid].chunk_start <= chunk) lo = mid; else hi = mid - 1;
  }
  return recs[lo];
}

// Chunk blockIdx.x of the launch: its record's items [i0, i1), eight elements
// each. 4 bytes read and 6 written per element: HBM-bound.
// Flat records (a whole number of items, contiguous and 16-byte aligned on both
// sides: every block whose row length is a multiple of 8): two items a thread
// in flight, 16-byte accesses, few registers so that 48 warps fit an SM. The general form
// below moved the same records at 2.5 TB/s (64-bit index arithmetic, 80 registers).
__global__ void __launch_bounds__(256, 6) k_f32_split_flat(const __grid_constant__ F3SplitArgs args) {
  griddep_launch();
  const F3Split& r = f3_split_record(args, blockIdx.x);
  const float* __restrict__ src = r.src;
  __nv_bfloat16* const dst = r.dst;
  const long long plane = r.plane, per = r.items_per_chunk;
  uint32_t* const out = r.amax + (blockIdx.x - r.chunk_start);
  const long long i0 = (blockIdx.x - r.chunk_start) * per;
  const int n = (int)min(per, r.items - i0);
  const float4* const sp = (const float4*)src + 2 * i0;
  uint4* const dp = (uint4*)dst + i0;
  const long long pw = plane / 8;
  uint32_t mx = 0;
  griddep_wait();
  for (int it = threadIdx.x; it < n; it += 512) {
    const bool two = it + 256 < n;
    const float4 a = __ldg(sp + 2 * it), b = __ldg(sp + 2 * it + 1);
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f), d = c;
    if (two) {
      c = __ldg(sp + 2 * it + 512);
      d = __ldg(sp + 2 * it + 513);
    }
    uint4 p[3];
    f3_split8({a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}, p, mx);
#pragma unroll
    for (int w = 0; w < 3; ++w) dp[it + w * pw] = p[w];
    if (two) {
      f3_split8({c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w}, p, mx);
#pragma unroll
      for (int w = 0; w < 3; ++w) dp[it + 256 + w * pw] = p[w];
    }
  }
  f3_chunk_max(mx, out);
}

// Row records: rows of consecutive elements on both sides, one row stride each,
// 16-byte aligned rows in the planes (pitches are multiples of 8), any alignment in the source.
// An item's eight elements come from the two or three aligned 16-byte pieces that
// hold them (a lane's eight element loads touched each sector eight times: rows of a
// contraction's operands moved at 1.7 TB/s), except at the ends of the tensor,
// where a piece could reach outside it.
__global__ void __launch_bounds__(256, 5) k_f32_split_rows(const __grid_constant__ F3SplitArgs args) {
  griddep_launch();
  const F3Split& r = f3_split_record(args, blockIdx.x);
  const float* __restrict__ src = r.src;
  __nv_bfloat16* const dst = r.dst;
  const long long plane = r.plane, istr = r.istride[2], ostr = r.ostride[2];
  uint32_t* const out = r.amax + (blockIdx.x - r.chunk_start);
  const uint32_t len = (uint32_t)r.len, per_row = (len + 7) / 8;
  const uint32_t i0 = (uint32_t)((blockIdx.x - r.chunk_start) * r.items_per_chunk);
  const uint32_t i1 = (uint32_t)min((long long)i0 + r.items_per_chunk, r.items);
  const float* const last = src + (r.odims[2] - 1) * istr + len;  // one past the tensor
  uint32_t mx = 0;
  griddep_wait();
  for (uint32_t it = i0 + threadIdx.x; it < i1; it += 256) {
    const uint32_t row = it / per_row, e = (it - row * per_row) * 8;
    const int cnt = (int)min(8u, len - e);
    const float* const sp = src + row * istr + e;
    const int mis = (int)(((uintptr_t)sp >> 2) & 3);
    float v[8];
    if (sp - mis >= src && sp - mis + 12 <= last) {
      const float4* const w = (const float4*)(sp - mis);
      const float4 a = __ldg(w), b = __ldg(w + 1), c = mis ? __ldg(w + 2) : make_float4(0.f, 0.f, 0.f, 0.f);
      float x[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
#pragma unroll
      for (int u = 0; u < 11; ++u) x[u] = (mis & 1) ? x[u + 1] : x[u];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = (mis & 2) ? x[u + 2] : x[u];
#pragma unroll
      for (int u = 1; u < 8; ++u) v[u] = u < cnt ? v[u] : 0.f;
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = u < cnt ? __ldg(sp + u) : 0.f;
    }
    uint4 p[3];
    f3_split8(v, p, mx);
    __nv_bfloat16* const dp = dst + row * ostr + e;
    // a row's last piece ends in its padding (pitch >= len rounded up to 8): zeros there
#pragma unroll
    for (int w = 0; w < 3; ++w) *(uint4*)(dp + w * plane) = p[w];
  }
  f3_chunk_max(mx, out);
}

// Any record: strided rows, gathers, summed modes, unaligned rows.
__global__ void __launch_bounds__(256) k_f32_split(const __grid_constant__ F3SplitArgs args) {
  griddep_launch();
  const int chunk = blockIdx.x;
  const F3Split& r = f3_split_record(args, chunk);
  const float* __restrict__ src = r.src;
  __nv_bfloat16* const dst = r.dst;
  const long long plane = r.plane, len = r.len, inner = r.inner;
  const long long per_row = (len + 7) >> 3;
  const long long i0 = (chunk - r.chunk_start) * r.items_per_chunk;
  const long long i1 = min(i0 + r.items_per_chunk, r.items);
  const long long od1 = r.odims[1], od2 = r.odims[2];
  const long long is0 = r.istride[0], is1 = r.istride[1], is2 = r.istride[2];
  const long long os0 = r.ostride[0], os1 = r.ostride[1], os2 = r.ostride[2];
  const bool small = r.items < (1ll << 31) && od1 * od2 < (1ll << 31);
  uint32_t mx = 0;
  griddep_wait();
  for (long long it = i0 + threadIdx.x; it < i1; it += blockDim.x) {
    long long row, c8;
    if (small) {  // 32-bit division
      row = (uint32_t)it / (uint32_t)per_row;
      c8 = it - row * per_row;
    } else {
      row = it / per_row;
      c8 = it - row * per_row;
    }
    long long q, d2, d1;
    if (small) {
      q = (uint32_t)row / (uint32_t)od2;
      d2 = row - q * od2;
      const long long q1 = (uint32_t)q / (uint32_t)od1;
      d1 = q - q1 * od1;
      q = q1;
    } else {
      q = row / od2;
      d2 = row - q * od2;
      const long long q1 = q / od1;
      d1 = q - q1 * od1;
      q = q1;
    }
    const long long e = c8 * 8;
    const int cnt = (int)min(8ll, len - e);
    const float* sp = src + q * is0 + d1 * is1 + d2 * is2 + e * inner;
    float v[8];
    if (r.rank_s > 0) {
      long long ns = 1;
      for (int d = 0; d < r.rank_s; ++d) ns *= r.sdims[d];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        v[u] = 0.f;
        if (u < cnt)
          for (long long s = 0; s < ns; ++s) {
            long long rem = s, off = 0;
            for (int d = 0; d < r.rank_s; ++d) {
              off += (rem % r.sdims[d]) * r.sstride[d];
              rem /= r.sdims[d];
            }
            v[u] += sp[u * inner + off];
          }
      }
    } else if (cnt == 8 && inner == 1 && (((uintptr_t)sp) & 15) == 0) {
      const float4 a = __ldg((const float4*)sp), b = __ldg((const float4*)sp + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = u < cnt ? __ldg(sp + u * inner) : 0.f;
    }
    uint4 p[3];
    f3_split8(v, p, mx);
    const long long oi = r.oinner;
    __nv_bfloat16* dp = dst + q * os0 + d1 * os1 + d2 * os2 + e * oi;
    if (cnt == 8 && oi == 1 && (((uintptr_t)dp) & 15) == 0) {  // plane strides are multiples of 8 elements
#pragma unroll
      for (int w = 0; w < 3; ++w) *(uint4*)(dp + w * plane) = p[w];
    } else {
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const uint32_t x[4] = {p[w].x, p[w].y, p[w].z, p[w].w};
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (u < cnt) dp[w * plane + u * oi] = __ushort_as_bfloat16((unsigned short)(x[u >> 1] >> (16 * (u & 1))));
      }
    }
  }
  f3_chunk_max(mx, r.amax + (chunk - r.chunk_start));
}

// ------------------------------------------------------------------ product
// The fields of problem p; a single problem's come from the kernel parameters.
__device__ __forceinline__ F3Fields f3_fields(const F3Args& args, int p) {
  if (!args.table) return args.one.f;
  return args.table[p].f;
}

struct F3Where { int p, b, tm, tn, k; };  // k < 0: out of range, -k is the extent

// meta[p] = (tile_start, tiles_m, tiles_n, k or -k)
__device__ __forceinline__ F3Where f3_locate(const int4* meta, int num, int t) {
  int lo = 0, hi = num - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (meta[mid].x <= t) lo = mid; else hi = mid - 1;
  }
  const int4 e = meta[lo];
  F3Where w;
  w.p = lo;
  w.k = e.w;
  const int per = e.y * e.z, lt = t - e.x;
  w.b = lt / per;
  band_tile(lt - w.b * per, e.y, e.z, w.tm, w.tn);
  return w;
}

// What the epilogue needs of a problem.
struct F3Out {
  float* c;          // of the tile's batch
  const float* bias;
  long long ldc;
  int m, n;
  float alpha, beta;
  bool plain, c_col;
};

__device__ __forceinline__ F3Out f3_out(const F3Args& args, int p, int batch) {
  const F3Fields f = f3_fields(args, p);
  F3Out o;
  o.c = f.c + batch * f.c_batch;
  o.bias = f.bias;
  o.ldc = f.ldc;
  o.m = f.m;
  o.n = f.n;
  o.alpha = f.alpha;
  o.beta = f.beta;
  o.plain = f.beta == 0.f && !f.bias;
  o.c_col = f.c_col != 0;
  return o;
}

__device__ __forceinline__ float f3_finish(const F3Out& o, float acc, const float* cp, int col) {
  float v = o.alpha * acc;
  if (o.plain) return v;
  if (o.beta != 0.f) v += o.beta * *cp;
  if (o.bias) v += o.bias[col];
  return v;
}

// The out-of-range problems' tiles of this CTA, by the 256 epilogue threads: 128 x 128
// outputs at a time, 8 x 8 a thread in packed pairs, one FMA chain over k per output (the SIMT
// kernels' order and bits). Operands come from the split planes, which join to the f32 values exactly and
// have one layout for dense blocks and gathered tensors: a thread loads one aligned piece of eight
// elements (three 16-byte loads) of A or B per eight steps of K, a step before it joins them into the
// free one of two shared-memory buffers (the epilogue's, which no TMA writes).
// Issue and barriers bound it, two warps a scheduler: 1024^3 with one infinity 162 us, 4096^3 4.3 ms;
// k_gemm_f32_v, which reads f32, takes 105 us and 2.7 ms; one thread a row straight from the
// planes took 7.7 ms for 1024^3. 16 steps a barrier (in the stages' memory): 4.4 ms. Joining at the
// end of a step: 4.7.
// Elements past the end of a row are masked: a row's padding in the planes may be unwritten.
constexpr int kF3PlainBK = 8;
constexpr int kF3PlainLd = 132;
static_assert(2 * 2 * kF3PlainBK * kF3PlainLd * 4 <= kF3EpiWarps * kF3EpiSlot, "plain tiles' shared memory");
static_assert(kF3EpiWarps == 8, "plain tiles take 256 threads");

template <bool PAIR>
__device__ __noinline__ void f3_plain_tiles(const F3Args& args, uint32_t stage_at, uint32_t meta_at, int unit, int units,
                                            int rank) {
  constexpr int BM = PAIR ? 256 : 128, BN = BM, BUF = kF3PlainBK * kF3PlainLd;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  float* const As = (float*)(smem_raw + stage_at);  // [2][BK][Ld]
  float* const Bs = As + 2 * BUF;
  const int4* const meta = (const int4*)(smem_raw + meta_at);
  const int tid = threadIdx.x - 64, tx = tid & 15, ty = tid >> 4;
  const bool of_b = tid >= 128;  // the operand that this thread loads
  const int lt = tid & 127;
  float* const put = of_b ? Bs : As;
  auto sync = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
  sync();  // every warp is done with its part of that memory
  for (int t0 = unit, rr = 0; t0 < args.total_tiles; t0 += units, ++rr) {
    const F3Where w = f3_locate(meta, args.num_problems, snake_tile_of(t0, rr, args.total_tiles, unit, units));
    if (w.k >= 0) continue;
    const int k = -w.k;
    const F3Fields f = f3_fields(args, w.p);
    const F3Out o = f3_out(args, w.p, w.b);
    const __nv_bfloat16* const src = of_b ? f.b + w.b * f.b_batch : f.a + w.b * f.a_batch;
    const long long plane = of_b ? f.b_plane : f.a_plane;
    const bool mn = (of_b ? f.b_mn : f.a_mn) != 0;
    const long long pitch = of_b ? (mn ? f.b_k : f.b_col) : (mn ? f.a_k : f.a_row);
    const int extent = of_b ? o.n : o.m;
    const int m0 = w.tm * BM + rank * 128;
    if (m0 >= o.m) continue;
    for (int n0 = w.tn * BN; n0 < min(w.tn * BN + BN, o.n); n0 += 128) {
      const int e0 = of_b ? n0 : m0;
      // K-major: steps k0 .. k0 + 7 of row e0 + lt; MN-major: step k0 + lt / 16 of elements e0 + 8 (lt % 16) .. + 7
      const int row0 = mn ? lt >> 4 : e0 + lt, col0 = mn ? e0 + 8 * (lt & 15) : 0;
      // a piece has min(8, left) elements; left counts down along K where the steps do
      const __nv_bfloat16* p = src + row0 * pitch + col0;
      const long long step = mn ? kF3PlainBK * pitch : kF3PlainBK;
      int left = mn ? extent - col0 : e0 + lt < extent ? k : 0;
      int rows = mn ? k - row0 : 1;  // MN-major: steps left
      uint4 q[3];
      int have;
      auto load = [&]() {
        have = rows > 0 ? left : 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) q[i] = have > 0 ? __ldg((const uint4*)(p + i * plane)) : make_uint4(0u, 0u, 0u, 0u);
        p += step;
        if (mn) rows -= kF3PlainBK; else left -= kF3PlainBK;
      };
      auto store = [&](int buf) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t *x = &q[0].x, *y = &q[1].x, *z = &q[2].x;
          const float2 g = f3_join2(x[i], y[i], z[i]);
          v[2 * i] = g.x;
          v[2 * i + 1] = g.y;
        }
        if (have < 8) {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = i < have ? v[i] : 0.f;
        }
        float* const b = put + buf * BUF;
        if (mn) {
          float* const r = b + (lt >> 4) * kF3PlainLd + 8 * (lt & 15);
          *(float4*)r = make_float4(v[0], v[1], v[2], v[3]);
          *(float4*)(r + 4) = make_float4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) b[i * kF3PlainLd + lt] = v[i];
        }
      };
      f32pair acc[8][4];  // columns 2 j and 2 j + 1
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
      load();
      store(0);
      load();  // past the end: zeros
      sync();
      for (int k0 = 0, buf = 0; k0 < k; k0 += kF3PlainBK, buf ^= 1) {
        store(buf ^ 1);  // read last before the barrier that ended the step before
        load();
        const float *a = As + buf * BUF + 4 * ty, *b = Bs + buf * BUF + 4 * tx;
#pragma unroll
        for (int kk = 0; kk < kF3PlainBK; ++kk) {
          const float4 a0 = *(const float4*)(a + kk * kF3PlainLd), a1 = *(const float4*)(a + kk * kF3PlainLd + 64);
          const ulonglong2 b0 = *(const ulonglong2*)(b + kk * kF3PlainLd), b1 = *(const ulonglong2*)(b + kk * kF3PlainLd + 64);
          const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          const f32pair bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const f32pair ai = pair_of(av[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) fma_pair(acc[i][j], ai, bv[j]);
          }
        }
        sync();
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = m0 + 4 * ty + (i & 3) + 64 * (i >> 2);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = n0 + 4 * tx + (j & 3) + 64 * (j >> 2);
          if (row >= o.m || col >= o.n) continue;
          float* const cp = o.c + (o.c_col ? row + col * o.ldc : row * o.ldc + col);
          const float2 v = unpack_pair(acc[i][j >> 1]);
          *cp = f3_finish(o, j & 1 ? v.y : v.x, cp, col);
        }
      }
    }
  }
}

// One warp's 32 rows x NC columns of C from its accumulators (lane l holds row
// row0 + l). Row-major C goes through the warp's 32 x 16 buffer, so that each
// store writes whole 64-byte row segments: 4 lanes x 16 bytes of 8 rows, or, where
// C's rows are not 16-byte aligned (or there is a beta or a bias), 16 lanes of
// 2 rows (4-byte stores of 8 rows each, every lane its own 16 bytes, made a lone
// 501^3 product 27.6 us, now 25.0). Columns of a column-major C are already 32
// consecutive elements across the lanes.
template <int NC>
__device__ __forceinline__ void f3_store(const F3Out& o, int row0, int col0, int lane, float* stage, const float (&acc)[NC]) {
  if (row0 >= o.m) return;
  if (o.c_col) {
    if (row0 + lane >= o.m) return;
    float* cp = o.c + row0 + lane + (long long)col0 * o.ldc;
#pragma unroll
    for (int j0 = 0; j0 < NC; j0 += 32) {
      const int left = o.n - col0 - j0;
      if (left >= 32 && o.plain) {  // no test per column
#pragma unroll
        for (int j = 0; j < 32; ++j, cp += o.ldc) *cp = o.alpha * acc[j0 + j];
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j, cp += o.ldc)
          if (j < left) *cp = f3_finish(o, acc[j0 + j], cp, col0 + j0 + j);
      }
    }
    return;
  }
  const bool vec = ((((uintptr_t)o.c) & 15) == 0) && (o.ldc & 3) == 0 && (o.n & 3) == 0;
  const int rr = lane >> 2, cc = (lane & 3) * 4;
  float* const crow = o.c + (long long)(row0 + rr) * o.ldc + col0 + cc;
#pragma unroll
  for (int j = 0; j < NC / 16; ++j) {
    if (col0 + 16 * j >= o.n) break;  // warp-uniform
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *(float4*)(stage + lane * kF3EpiPitch + 4 * q) =
          make_float4(acc[16 * j + 4 * q], acc[16 * j + 4 * q + 1], acc[16 * j + 4 * q + 2], acc[16 * j + 4 * q + 3]);
    __syncwarp();
    if (vec && o.plain) {
      const int col = col0 + 16 * j + cc;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const float4 x = *(const float4*)(stage + (8 * s + rr) * kF3EpiPitch + cc);
        if (row0 + 8 * s + rr < o.m && col < o.n)
          *(float4*)(crow + 8 * s * o.ldc + 16 * j) = make_float4(o.alpha * x.x, o.alpha * x.y, o.alpha * x.z, o.alpha * x.w);
      }
    } else {
      const int r0 = lane >> 4, c1 = lane & 15, col = col0 + 16 * j + c1;
      float* cp = o.c + (long long)(row0 + r0) * o.ldc + col;
      const int rows = col < o.n ? o.m - row0 - r0 : 0;
#pragma unroll 8
      for (int e = 0; e < 32; e += 2, cp += 2 * o.ldc)
        if (e < rows) *cp = f3_finish(o, stage[(e + r0) * kF3EpiPitch + c1], cp, col);
    }
    __syncwarp();
  }
}

template <bool PAIR>
__device__ __forceinline__ void f3_tma(uint8_t* dst, const void* tmap, uint64_t* full, uint32_t full_pair, int x, int y, int z) {
  if constexpr (PAIR) tma_load_3d_2sm(dst, tmap, full_pair, x, y, z);
  else tma_load_3d(dst, tmap, full, x, y, z);
}

template <bool PAIR>
__device__ __forceinline__ void f3_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
  if constexpr (PAIR) umma_f16_2sm(d, da, db, idesc, accum);
  else umma_f16(d, da, db, idesc, accum);
}

template <bool PAIR>
__device__ __forceinline__ void f3_commit(uint64_t* bar) {
  if constexpr (PAIR) umma_commit_2sm(bar, 0x3);
  else umma_commit(bar);
}

// Four MMAs (K = 16 each) of one pair of plane tiles; ka, kb: a K step of the
// descriptors. FIRST: how the first one treats the accumulator: 0 adds to it, 1
// starts it, 2 scales it by 2^-8.
template <bool PAIR, int FIRST>
__device__ __forceinline__ void f3_product(uint32_t d, uint64_t da, uint64_t db, uint32_t ka, uint32_t kb, uint32_t idesc) {
  if constexpr (FIRST == 2) {
    if constexpr (PAIR) umma_f16_2sm_shift_d<8>(d, da, db, idesc);
    else umma_f16_shift_d<8>(d, da, db, idesc);
  } else {
    f3_mma<PAIR>(d, da, db, idesc, FIRST == 1 ? 0u : 1u);
  }
#pragma unroll
  for (int kk = 1; kk < 4; ++kk) f3_mma<PAIR>(d, da + kk * ka, db + kk * kb, idesc, 1u);
}

template <bool PAIR>
__device__ __forceinline__ void f3_gemm_body(const F3Args& args) {
  constexpr int BM = PAIR ? 256 : 128, BN = BM;
  constexpr int NC = BN / 2;  // columns per epilogue warp
  constexpr int TMEM_COLS = 2 * BN;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* epi = (float*)(smem + 2 * kF3Stage);
  uint64_t* bars = (uint64_t*)(smem + 2 * kF3Stage + kF3EpiWarps * kF3EpiSlot);
  uint64_t* full = bars;              // [2]
  uint64_t* empty = bars + 2;         // [2][5]
  uint64_t* tfull = bars + 12;        // [2]
  uint64_t* tempty = bars + 14;       // [2]
  uint32_t* tmem_slot = (uint32_t*)(bars + 16);
  int4* meta = (int4*)((uint8_t*)bars + 256);
  volatile uint32_t* status = args.status;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const bool leader = rank == 0;
  const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int units = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;

  if (warp == 0) {
    if (lane == 0) {
      for (int s = 0; s < 2; ++s) {
        mbar_init(&full[s], 1);
        for (int e = 0; e < 5; ++e) mbar_init(&empty[5 * s + e], 1);
        mbar_init(&tfull[s], 1);
        mbar_init(&tempty[s], (PAIR ? 2 : 1) * kF3EpiWarps);
      }
      fence_mbar_init();
      if (!args.table) {
        prefetch_tensormap(&args.one.tmap_a);
        prefetch_tensormap(&args.one.tmap_b);
      }
    }
  } else if (warp == 1) {
    if constexpr (PAIR) tmem_alloc_2sm(tmem_slot, TMEM_COLS);
    else tmem_alloc(tmem_slot, TMEM_COLS);
  }
  griddep_launch();
  griddep_wait();  // the maxima below are the split's
  int plain = 0;   // a problem is out of range
  if (warp >= 2) {
    // one warp per problem: its tiles, and whether its operands are in range
    for (int p = warp - 2; p < args.num_problems; p += kF3EpiWarps) {
      const F3Fields f = f3_fields(args, p);
      const uint32_t *xa = f.amax_a, *xb = f.amax_b;
      const int na = f.na, nb = f.nb, k = f.k;
      uint32_t ma = 0, mb = 0;
      for (int i = lane; i < max(na, nb); i += 32) {
        if (i < na) ma = max(ma, xa[i]);
        if (i < nb) mb = max(mb, xb[i]);
      }
      ma = __reduce_max_sync(0xffffffffu, ma);
      mb = __reduce_max_sync(0xffffffffu, mb);
      const bool in_range = f3_in_range(ma, mb, k);
      plain |= !in_range;
      if (lane == 0) meta[p] = make_int4(f.tile_start, f.tiles_m, f.tiles_n, in_range ? k : -k);
    }
  }
  tc_fence_before();
  plain = __syncthreads_or(plain);
  if constexpr (PAIR) {
    __syncwarp();
    cluster_sync();
  }
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // tile of this unit in a round; the same in every lane
  auto locate = [&](int t0, int round) {
    F3Where w = f3_locate(meta, args.num_problems, snake_tile_of(t0, round, args.total_tiles, unit, units));
    w.p = warp_uniform(w.p);
    w.b = warp_uniform(w.b);
    w.tm = warp_uniform(w.tm);
    w.tn = warp_uniform(w.tn);
    w.k = warp_uniform(w.k);
    return w;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    uint32_t c = 0;  // chunks so far: stage c & 1
    bool ok = true;
    int last_p = -1;
    for (int t0 = unit, rr = 0; t0 < args.total_tiles && ok; t0 += units, ++rr) {
      const F3Where w = locate(t0, rr);
      if (w.k <= 0) continue;
      const F3Fields f = f3_fields(args, w.p);
      const CUtensorMap* const map_a = args.table ? &args.table[w.p].tmap_a : &args.one.tmap_a;
      const CUtensorMap* const map_b = args.table ? &args.table[w.p].tmap_b : &args.one.tmap_b;
      const bool a_mn = warp_uniform(f.a_mn) != 0, b_mn = warp_uniform(f.b_mn) != 0;
      const int nb = warp_uniform(f.batch);
      const int row_a = w.tm * BM + (int)rank * 128, row_b = w.tn * BN + (int)rank * 128;
      if (args.table && w.p != last_p) {
        if (elect_one()) {
          tensormap_acquire(map_a);
          tensormap_acquire(map_b);
        }
        last_p = w.p;
      }
      for (int k0 = 0; k0 < w.k && ok; k0 += kF3BK, ++c) {
        const uint32_t s = c & 1, ph = (c >> 1) & 1;
        uint8_t* const sa = smem + s * kF3Stage;
        uint8_t* const sb = sa + 3 * kF3Tile;
        uint64_t* const fb = &full[s];
        uint64_t* const eb = &empty[5 * s];
        const uint32_t fp = PAIR ? mapa_shared(smem_u32(fb), 0) : 0u;
        auto load_a = [&](int plane) {
          uint8_t* const dst = sa + plane * kF3Tile;
          if (a_mn) {
            f3_tma<PAIR>(dst, map_a, fb, fp, row_a, k0, plane * nb + w.b);
            f3_tma<PAIR>(dst + kF3BK * 128, map_a, fb, fp, row_a + 64, k0, plane * nb + w.b);
          } else {
            f3_tma<PAIR>(dst, map_a, fb, fp, k0, row_a, plane * nb + w.b);
          }
        };
        auto load_b = [&](int plane) {
          uint8_t* const dst = sb + plane * kF3Tile;
          if (b_mn) {
            f3_tma<PAIR>(dst, map_b, fb, fp, row_b, k0, plane * nb + w.b);
            f3_tma<PAIR>(dst + kF3BK * 128, map_b, fb, fp, row_b + 64, k0, plane * nb + w.b);
          } else {
            f3_tma<PAIR>(dst, map_b, fb, fp, k0, row_b, plane * nb + w.b);
          }
        };
        // in the order in which the products hand the tiles back
        if (!(ok = mbar_wait_warp(&eb[0], ph ^ 1, status, DEV_TIMEOUT_EMPTY))) break;
        if (elect_one()) {
          if (leader) mbar_arrive_expect_tx(fb, (PAIR ? 2 : 1) * kF3Stage);
          load_b(2);
        }
        if (!(ok = mbar_wait_warp(&eb[1], ph ^ 1, status, DEV_TIMEOUT_EMPTY))) break;
        if (elect_one()) load_a(2);
        if (!(ok = mbar_wait_warp(&eb[2], ph ^ 1, status, DEV_TIMEOUT_EMPTY))) break;
        if (elect_one()) load_b(1);
        if (!(ok = mbar_wait_warp(&eb[3], ph ^ 1, status, DEV_TIMEOUT_EMPTY))) break;
        if (elect_one()) load_a(1);
        if (!(ok = mbar_wait_warp(&eb[4], ph ^ 1, status, DEV_TIMEOUT_EMPTY))) break;
        if (elect_one()) {
          load_a(0);
          load_b(0);
        }
      }
    }
    // every issued load has landed and been read before the CTA may exit
    for (int i = 0; i < 2 && ok; ++i, ++c)
      for (int e = 0; e < 5 && ok; ++e) ok = mbar_wait_warp(&empty[5 * (c & 1) + e], ((c >> 1) & 1) ^ 1, status, DEV_TIMEOUT_EMPTY);
    if (lane == 0 && *status != DEV_OK) {
      const long long t0 = clock64();
      while (clock64() - t0 < 200000) {}
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the pair's leader)
    if (leader) {
      uint32_t c = 0;
      bool ok = true;
      for (int t0 = unit, rr = 0; t0 < args.total_tiles && ok; t0 += units, ++rr) {
        const F3Where w = locate(t0, rr);
        if (w.k <= 0) continue;
        const F3Fields f = f3_fields(args, w.p);
        const bool a_mn = warp_uniform(f.a_mn) != 0, b_mn = warp_uniform(f.b_mn) != 0;
        const uint32_t idesc = make_idesc(BM, BN, 1u, a_mn, b_mn);
        // descriptors of plane 0's first K step in stage 0; their low words count 16-byte units
        const uint32_t s0 = smem_u32(smem);
        const uint64_t da0 = smem_desc_sw128(s0, a_mn ? kF3BK * 128 : 16, 1024);
        const uint64_t db0 = smem_desc_sw128(s0 + 3 * kF3Tile, b_mn ? kF3BK * 128 : 16, 1024);
        const uint32_t ka = (a_mn ? 2048 : 32) >> 4, kb = (b_mn ? 2048 : 32) >> 4;
        constexpr uint32_t P = kF3Tile >> 4;  // to the next plane
        for (int k0 = 0; k0 < w.k; k0 += kF3BK, ++c) {
          const uint32_t s = c & 1, ph = (c >> 1) & 1;
          if (!(ok = mbar_wait_warp(&tempty[s], ph ^ 1, status, DEV_TIMEOUT_TMEM_EMPTY))) break;
          if (!(ok = mbar_wait_warp(&full[s], ph, status, DEV_TIMEOUT_FULL))) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t d = tmem_base + s * BN;
            const uint64_t da = da0 + s * (kF3Stage >> 4), db = db0 + s * (kF3Stage >> 4);
            uint64_t* const e = empty + 5 * s;
            f3_product<PAIR, 1>(d, da, db + 2 * P, ka, kb, idesc);       // a0 b2
            f3_commit<PAIR>(&e[0]);
            f3_product<PAIR, 0>(d, da + 2 * P, db, ka, kb, idesc);       // a2 b0
            f3_commit<PAIR>(&e[1]);
            f3_product<PAIR, 0>(d, da + P, db + P, ka, kb, idesc);      // a1 b1
            f3_product<PAIR, 2>(d, da, db + P, ka, kb, idesc);           // a0 b1
            f3_commit<PAIR>(&e[2]);
            f3_product<PAIR, 0>(d, da + P, db, ka, kb, idesc);           // a1 b0
            f3_commit<PAIR>(&e[3]);
            f3_product<PAIR, 2>(d, da, db, ka, kb, idesc);                // a0 b0
            f3_commit<PAIR>(&e[4]);
            f3_commit<PAIR>(&tfull[s]);
          }
          __syncwarp();
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float* stage = epi + (warp - 2) * (kF3EpiSlot / 4);
    const uint32_t te[2] = {PAIR ? mapa_shared(smem_u32(&tempty[0]), 0) : 0u, PAIR ? mapa_shared(smem_u32(&tempty[1]), 0) : 0u};
    uint32_t c = 0;
    bool ok = true;
    for (int t0 = unit, rr = 0; t0 < args.total_tiles && ok; t0 += units, ++rr) {
      const F3Where w = locate(t0, rr);
      if (w.k <= 0) continue;
      const int row0 = w.tm * BM + (int)rank * 128 + 32 * quarter, col0 = w.tn * BN + half * NC;
      const F3Out o = f3_out(args, w.p, w.b);
      float acc[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[j] = 0.f;
      for (int k0 = 0; k0 < w.k; k0 += kF3BK, ++c) {
        const uint32_t s = c & 1, ph = (c >> 1) & 1;
        const bool got = mbar_wait(&tfull[s], ph, status, DEV_TIMEOUT_TMEM_FULL);
        if (!(ok = __all_sync(0xffffffffu, got))) break;
        tc_fence_after();
        const uint32_t t_row = tmem_base + s * BN + half * NC + ((uint32_t)(32 * quarter) << 16);
#pragma unroll
        for (int j = 0; j < NC / 32; ++j) {
          uint32_t r0[16], r1[16];
          tmem_ld16_nowait(t_row + 32 * j, r0);
          tmem_ld16_nowait(t_row + 32 * j + 16, r1);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            acc[32 * j + q] = __fadd_rn(acc[32 * j + q], __uint_as_float(r0[q]));
            acc[32 * j + 16 + q] = __fadd_rn(acc[32 * j + 16 + q], __uint_as_float(r1[q]));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (PAIR) mbar_arrive_cluster(te[s]);
          else mbar_arrive(&tempty[s]);
        }
      }
      if (!ok) break;
      f3_store<NC>(o, row0, col0, lane, stage, acc);
    }
    // all eight warps, whatever their waits came to
    if (plain)
      f3_plain_tiles<PAIR>(args, (uint32_t)((uint8_t*)epi - smem_raw), (uint32_t)((uint8_t*)meta - smem_raw), unit, units, (int)rank);
  }

  // in a pair the leader's MMAs read the peer's shared memory: neither CTA may
  // release TMEM or exit before both are done
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {
    __syncwarp();
    cluster_sync();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_2sm(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kF3Threads, 1)
    f32_gemm_pair_kernel(const __grid_constant__ F3Args args) {
  f3_gemm_body<true>(args);
}

__global__ void __launch_bounds__(kF3Threads, 1) f32_gemm_kernel(const __grid_constant__ F3Args args) {
  f3_gemm_body<false>(args);
}

}  // namespace bbx
