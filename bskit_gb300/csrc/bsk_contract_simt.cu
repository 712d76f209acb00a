// SIMT triple-product contraction: the plain-FP32 path and the FP64 yardstick.
//
// The FP64 variants (FP32 or FP64 fields, FP64 products and sums):
// Work item = (sub-tile of 128 pair rows x 32 third-shell columns, K slice).
// Per 32-point chunk the block forms the 128 pair products P[r][x] =
// F1[i_r](x) * F2[j_r](x) and the 32 column values F3[l](x) in shared memory
// (double buffered, register prefetch of the next chunk), then a 4x4
// register-tiled outer-product loop accumulates C[r][c] += P[r][x] * F3[c][x].
// At the end of the slice the tile sums are added to the FP64 output with
// atomics (only entries that are triangle bins); warps whose 16 x 32 entries hold
// no bin skip the multiply-adds.  Items are ordered slice-major
// so that blocks running at the same time share field data in L2.
#include <algorithm>
#include <type_traits>

#include "bsk_internal.cuh"

namespace bsk {
namespace {

constexpr int KC = 32;     // points per chunk
constexpr int ROWS = 128;  // pair rows per sub-tile
constexpr int COLS = 32;   // columns per sub-tile
constexpr int APAD = 4;
constexpr int BPAD = 4;
constexpr int THREADS = 256;

template <typename Tin, typename Tacc>
__device__ __forceinline__ Tacc prod(Tin a, Tin b) {
  return (Tacc)a * (Tacc)b;
}

template <typename Tin, typename Tacc>
__global__ void __launch_bounds__(THREADS) contract_simt_kernel(
    const TileDesc* __restrict__ tiles, const int2* __restrict__ subs, int n_sub,
    const int16_t* __restrict__ row_i, const int16_t* __restrict__ row_j,
    const int32_t* __restrict__ map, const Tin* __restrict__ f1, const Tin* __restrict__ f2,
    const Tin* __restrict__ f3, int n_shells, int64_t K, int64_t k_begin, int64_t k_end,
    int64_t slice, int64_t n_slices, double* __restrict__ out, double scale) {
  extern __shared__ __align__(16) unsigned char simt_smem[];
  typedef Tacc ATile[KC][ROWS + APAD];
  typedef Tacc BTile[KC][COLS + BPAD];
  ATile* As = reinterpret_cast<ATile*>(simt_smem);
  BTile* Bs = reinterpret_cast<BTile*>(simt_smem + 2 * sizeof(ATile));
  const int tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;          // micro-tile rows ty*4.., cols tx*4..
  const int ar = tid & (ROWS - 1), ah = tid >> 7;  // A-gen: row ar, points ah*16 .. +16
  const int bc = tid >> 3, bp = (tid & 7) * 4;     // B-gen: column bc, points bp .. +4
  const int64_t n_items = (int64_t)n_sub * n_slices;

  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int64_t sl = item / n_sub;
    const int2 sub = subs[item % n_sub];
    const TileDesc td = tiles[sub.x];
    const int c0 = sub.y;
    const int ri = row_i[td.row_off + ar];
    const int rj = row_j[td.row_off + ar];
    const int lcol = td.l0 + c0 + bc;
    const bool bvalid = (c0 + bc < td.nc) && (lcol < n_shells);
    const Tin* pa = f1 + (int64_t)(ri >= 0 ? ri : 0) * K;
    const Tin* pb = f2 + (int64_t)(ri >= 0 ? rj : 0) * K;
    const Tin* pc = f3 + (int64_t)(bvalid ? lcol : 0) * K;
    const int64_t x_begin = k_begin + sl * slice;
    const int64_t x_end = min(k_end, x_begin + slice);

    Tacc acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = (Tacc)0;
    // A warp (16 rows x 32 columns) whose entries hold no triangle bin skips the
    // multiply-adds; it still loads its share of the tiles the whole block uses.
    bool mine = false;
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = c0 + tx * 4 + q;
        if (c < td.nc && map[td.map_off + c * ROWS + ty * 4 + p] >= 0) mine = true;
      }
    const bool warp_busy = __any_sync(0xffffffffu, mine);

    Tacc ra[16], rc[4];
    auto load = [&](int64_t x0) {
      const int64_t xa = x0 + ah * 16;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        int64_t x = xa + e;
        ra[e] = (ri >= 0 && x < x_end) ? prod<Tin, Tacc>(__ldg(pa + x), __ldg(pb + x)) : (Tacc)0;
      }
      const int64_t xc = x0 + bp;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int64_t x = xc + e;
        rc[e] = (bvalid && x < x_end) ? (Tacc)__ldg(pc + x) : (Tacc)0;
      }
    };
    auto store = [&](int buf) {
#pragma unroll
      for (int e = 0; e < 16; ++e) As[buf][ah * 16 + e][ar] = ra[e];
#pragma unroll
      for (int e = 0; e < 4; ++e) Bs[buf][bp + e][bc] = rc[e];
    };

    load(x_begin);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int64_t x0 = x_begin; x0 < x_end; x0 += KC) {
      const bool more = x0 + KC < x_end;
      if (more) load(x0 + KC);
#pragma unroll 8
      for (int k = 0; k < KC && warp_busy; ++k) {
        Tacc a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a[q] = As[buf][k][ty * 4 + q];
          b[q] = Bs[buf][k][tx * 4 + q];
        }
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[p][q] += a[p] * b[q];
      }
      if (more) store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }

#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int r = ty * 4 + p;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = c0 + tx * 4 + q;
        if (c < td.nc) {
          const int t = map[td.map_off + c * ROWS + r];
          if (t >= 0) atomicAdd(out + t, (double)acc[p][q] * scale);
        }
      }
    }
  }
}

// ---------------------------------------------------------------- plain FP32 path
// FP32 pair products P = F1_i F2_j, FP32 multiply-adds in point order over 8192-point slices,
// FP64 atomics across slices; one warp per (8 TR rows x 4 TC columns of a tile, slice).  No
// block barriers: a block is one warp.  Source and column rows of the next chunks are copied
// with cp.async (16 bytes; 4 where a shard's range starts off a 16-byte boundary) while the
// current chunk is formed and multiplied.
//
// Long grids (TR = 16: all 128 rows x up to 32 columns).  Operand loads bound the outer
// product: a float delivered to a warp costs a shared-memory wavefront whatever is broadcast,
// so a thread tile of R rows x C columns costs (R + C) / (R C) wavefronts a multiply-add: 0.19
// for 16 x 8, 0.375 for the 8 x 4 that four warps sharing the tile have.  Columns come in the
// tile's own width, multiply-adds packed by two rows (fma.rn.f32x2).  250 registers, eight
// warps an SM (168 or 200 of them spill: +60%).  256^3 (31 shells, 3 tiles): 4.15 ms, where a
// block of four warps a tile took 6.5.
//
// Short grids and sparse sets (TR = 4: 32 rows x up to 16 columns).  A slice is a chain of 8192
// dependent multiply-adds an entry, so with few items the chain's pace is the time (48^3, 14
// items: 144 cycles a point with four warps and three barriers a chunk, 623 us): more, smaller
// items, and copies three chunks ahead (250 us).  Forming the next chunk's products before the
// current chunk's multiply-adds, to save a barrier, was 7% slower.  The items are the parts of the
// tiles that hold bins, listed with the schedule (f32_parts), each with its own source shells, so
// that sparse sets do no work for the rest of their tiles: 60 equilateral bins on 192^3 take
// 1.6 ms, as whole tiles 4.4, and 3.4 where a block of four warps a tile skipped what held no
// bin.  (Skipping empty parts in this kernel saved nothing: a block met the full ones every round.)
namespace f32 {
constexpr int ROWS = 128, COLS = 32, SRC = 64;
constexpr int64_t SLICE = 8192;

template <int TR_, int KC_, int ST_, int COLS_, bool kTwoSrc_, bool kAligned_>
struct Cfg {
  static constexpr int TR = TR_, KC = KC_, ST = ST_;  // rows a thread, points a chunk, chunks held
  static constexpr int COLS = COLS_;                  // columns of an item at most
  static constexpr bool kTwoSrc = kTwoSrc_, kAligned = kAligned_;
  static constexpr int PITCH = KC + 4;                // 16-byte pieces of 8 rows on distinct banks
  static constexpr int APITCH = 8 * TR + 4;
  // A[KC][APITCH] pair products of the chunk, B[ST][COLS][PITCH] column rows, then S1 and S2
  // [ST][src][PITCH] source rows (src: the widest source range of the launch's tiles)
  static constexpr int A_FLOATS = KC * APITCH, B_FLOATS = ST * COLS * PITCH;
  static size_t smem(int src) {
    return (A_FLOATS + B_FLOATS + (kTwoSrc ? 2 : 1) * ST * src * PITCH) * sizeof(float);
  }
};
template <bool kTwoSrc, bool kAligned>
using Long = Cfg<16, 8, 2, 32, kTwoSrc, kAligned>;
template <bool kTwoSrc, bool kAligned>
using Short = Cfg<4, 16, 4, 16, kTwoSrc, kAligned>;

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src),
               "r"(ok ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ unsigned long long dup2(float x) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
  return d;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a,
                                     unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Columns c0 + 4 e + (lane & 3), e < TC; rows r0 + TR (lane >> 2) .. + TR - 1.
template <class C, int TC>
__device__ __forceinline__ void run_item(float* sm, int src, const TileDesc& td, int r0, int c0,
                                         const int16_t* row_i, const int16_t* row_j,
                                         const int32_t* map, const float* f1, const float* f2,
                                         const float* f3, int n_shells, int64_t K,
                                         int64_t x_begin, int64_t x_end, bool one_src,
                                         double* out, double scale) {
  constexpr int TR = C::TR, KC = C::KC, ST = C::ST, PITCH = C::PITCH, AP = C::APITCH;
  float* sA = sm;
  float* sB = sA + C::A_FLOATS;
  float* s1 = sB + C::B_FLOATS;
  float* s2 = C::kTwoSrc && !one_src ? s1 + ST * src * PITCH : s1;
  const int lane = threadIdx.x, cg = lane & 3, rg = lane >> 2;
  // pair products: rows r0 + lane + 32 g
  int p1[TR / 4], p2[TR / 4];
#pragma unroll
  for (int g = 0; g < TR / 4; ++g) {
    const int at = td.row_off + r0 + lane + 32 * g;
    const int ri = row_i[at], rj = row_j[at];
    p1[g] = ri >= 0 ? ri - td.i0 : 0;  // rows past the tile's pairs: any (their sums are not read)
    p2[g] = ri >= 0 ? rj - td.j0 : 0;
  }
  // copies of one chunk in 16-byte pieces, lanes on consecutive ones; points past the slice zero
  auto copy_rows = [&](float* dst, const float* f, int s0, int rows, int64_t x0) {
    constexpr int W = C::kAligned ? 4 : 1;  // points a copy
    for (int i = lane; i < KC / W * rows; i += 32) {
      const int row = i / (KC / W), k = i % (KC / W) * W, s = s0 + row;
      const int64_t left = s < n_shells ? (x_end - (x0 + k)) * 4 : 0;
      const int bytes = (int)min((int64_t)(4 * W), max((int64_t)0, left));
      const float* p = bytes ? f + (int64_t)s * K + x0 + k : f;
      if constexpr (C::kAligned) cp_async16(dst + row * PITCH + k, p, bytes);
      else cp_async4(dst + row * PITCH + k, p, bytes != 0);
    }
  };
  auto stage = [&](int buf, int64_t x0) {
    if (x0 < x_end) {
      copy_rows(s1 + buf * src * PITCH, f1, td.i0, td.ni, x0);
      if (C::kTwoSrc && !one_src) copy_rows(s2 + buf * src * PITCH, f2, td.j0, td.nj, x0);
      copy_rows(sB + buf * C::COLS * PITCH, f3, td.l0 + c0, 4 * TC, x0);
    }
    cp_async_commit();
  };
  unsigned long long acc[TR / 2][TC];  // rows 2 m, 2 m + 1
#pragma unroll
  for (int m = 0; m < TR / 2; ++m)
#pragma unroll
    for (int e = 0; e < TC; ++e) acc[m][e] = 0ull;
#pragma unroll
  for (int q = 0; q < ST - 1; ++q) stage(q, x_begin + q * KC);
  int buf = 0;
  for (int64_t x0 = x_begin; x0 < x_end; x0 += KC, buf = (buf + 1) % ST) {
    cp_async_wait<ST - 2>();
    __syncwarp();  // the chunk has landed; the previous one and its products have been used
    stage((buf + ST - 1) % ST, x0 + (ST - 1) * KC);
    const float* S1 = s1 + buf * src * PITCH;
    const float* S2 = s2 + buf * src * PITCH;
#pragma unroll
    for (int g = 0; g < TR / 4; ++g)
#pragma unroll
      for (int k = 0; k < KC; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(S1 + p1[g] * PITCH + k);
        const float4 b = *reinterpret_cast<const float4*>(S2 + p2[g] * PITCH + k);
        float* A = sA + k * AP + lane + 32 * g;
        A[0] = a.x * b.x;
        A[AP] = a.y * b.y;
        A[2 * AP] = a.z * b.z;
        A[3 * AP] = a.w * b.w;
      }
    __syncwarp();
    const float* A = sA + TR * rg;
    const float* B = sB + buf * C::COLS * PITCH + cg * PITCH;
#pragma unroll
    for (int k0 = 0; k0 < KC; k0 += 2) {
      float2 bv[TC];
#pragma unroll
      for (int e = 0; e < TC; ++e)
        bv[e] = *reinterpret_cast<const float2*>(B + 4 * e * PITCH + k0);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        ulonglong2 av[TR / 4];
#pragma unroll
        for (int m = 0; m < TR / 4; ++m)
          av[m] = *reinterpret_cast<const ulonglong2*>(A + (k0 + k) * AP + 4 * m);
#pragma unroll
        for (int e = 0; e < TC; ++e) {
          const unsigned long long b = dup2(k ? bv[e].y : bv[e].x);
#pragma unroll
          for (int m = 0; m < TR / 4; ++m) {
            fma2(acc[2 * m][e], av[m].x, b);
            fma2(acc[2 * m + 1][e], av[m].y, b);
          }
        }
      }
    }
  }
  cp_async_wait<0>();
  __syncwarp();  // the next item's copies overwrite the buffers
#pragma unroll
  for (int e = 0; e < TC; ++e)
#pragma unroll
    for (int r = 0; r < TR; ++r) {
      const int t = __ldg(map + td.map_off + (c0 + 4 * e + cg) * kTileRows + r0 + TR * rg + r);
      const uint32_t bits = (uint32_t)(acc[r / 2][e] >> (r & 1 ? 32 : 0));
      if (t >= 0) atomicAdd(out + t, (double)__uint_as_float(bits) * scale);
    }
}

// Long grids: item = (slice, sub-tile of 32 columns).
template <class C>
__global__ void __launch_bounds__(32)
    contract_f32_kernel(const TileDesc* __restrict__ tiles, const int2* __restrict__ subs,
                        int n_sub, const int16_t* __restrict__ row_i,
                        const int16_t* __restrict__ row_j, const int32_t* __restrict__ map,
                        const float* __restrict__ f1, const float* __restrict__ f2,
                        const float* __restrict__ f3, int n_shells, int64_t K, int64_t k_begin,
                        int64_t k_end, int64_t n_slices, int src, double* __restrict__ out,
                        double scale) {
  extern __shared__ __align__(16) float f32_smem[];
  float* sm = f32_smem;
  for (int64_t item = blockIdx.x; item < n_slices * n_sub; item += gridDim.x) {
    const int64_t sl = item / n_sub;
    const int2 sub = subs[(int)(item - sl * n_sub)];
    const TileDesc td = tiles[sub.x];
    // the tile's columns in as many equal runs, multiples of 8, as it has 32-column sub-tiles
    const int runs = (td.nc + COLS - 1) / COLS, width = ((td.nc + runs - 1) / runs + 7) / 8 * 8;
    const int c0 = sub.y / COLS * width, nc = min(width, td.nc - c0), r0 = 0;
    const bool one_src = !C::kTwoSrc || (f1 == f2 && td.i0 == td.j0);
    const int64_t x_begin = k_begin + sl * SLICE;
    const int64_t x_end = min(k_end, x_begin + SLICE);
    if (nc <= 8)
      run_item<C, 2>(sm, src, td, r0, c0, row_i, row_j, map, f1, f2, f3, n_shells, K, x_begin,
                     x_end, one_src, out, scale);
    else if (nc <= 16)
      run_item<C, 4>(sm, src, td, r0, c0, row_i, row_j, map, f1, f2, f3, n_shells, K, x_begin,
                     x_end, one_src, out, scale);
    else if (nc <= 24)
      run_item<C, 6>(sm, src, td, r0, c0, row_i, row_j, map, f1, f2, f3, n_shells, K, x_begin,
                     x_end, one_src, out, scale);
    else
      run_item<C, 8>(sm, src, td, r0, c0, row_i, row_j, map, f1, f2, f3, n_shells, K, x_begin,
                     x_end, one_src, out, scale);
  }
}

// Short grids and sparse sets: item = (slice, part).
template <class C>
__global__ void __launch_bounds__(32)
    contract_f32_parts_kernel(const TileDesc* __restrict__ tiles,
                              const F32Part* __restrict__ parts, int n_parts,
                              const int16_t* __restrict__ row_i,
                              const int16_t* __restrict__ row_j, const int32_t* __restrict__ map,
                              const float* __restrict__ f1, const float* __restrict__ f2,
                              const float* __restrict__ f3, int n_shells, int64_t K,
                              int64_t k_begin, int64_t k_end, int64_t n_slices, int src,
                              double* __restrict__ out, double scale) {
  extern __shared__ __align__(16) float f32_smem[];
  float* sm = f32_smem;
  for (int64_t item = blockIdx.x; item < n_slices * n_parts; item += gridDim.x) {
    const int64_t sl = item / n_parts;
    const F32Part p = parts[(int)(item - sl * n_parts)];
    TileDesc td = tiles[p.tile];
    td.i0 = p.i0;
    td.ni = p.ni;
    td.j0 = p.j0;
    td.nj = p.nj;
    const bool one_src = !C::kTwoSrc || (f1 == f2 && td.i0 == td.j0);
    const int64_t x_begin = k_begin + sl * SLICE;
    const int64_t x_end = min(k_end, x_begin + SLICE);
    if (p.nc <= 8)
      run_item<C, 2>(sm, src, td, p.r0, p.c0, row_i, row_j, map, f1, f2, f3, n_shells, K, x_begin,
                     x_end, one_src, out, scale);
    else
      run_item<C, 4>(sm, src, td, p.r0, p.c0, row_i, row_j, map, f1, f2, f3, n_shells, K, x_begin,
                     x_end, one_src, out, scale);
  }
}

// Parts of one column block as long as the SMs hold them all at once, twice the items with half
// the chain: then of two.  Both sides measured, us, pairs / single blocks, at that many single
// blocks an SM: one source range 2: 369 / 273, 7.1: 468 / 339, 10.1: 482 / 420, 13.2: 479 / 540 and
// 551 / 852; two ranges or arrays 7.1: 532 / 421, 8.1: 521 / 706, 11.0: 602 / 867.
template <class C>
constexpr int64_t kNarrowPerSm = C::kTwoSrc ? 8 : 11;

template <class Kern>
unsigned blocks(Kern kern, size_t smem, size_t most_smem, int64_t items, int num_sms) {
  BSK_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)most_smem));
  int per_sm = 0;
  BSK_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32, smem));
  return (unsigned)std::min<int64_t>((int64_t)num_sms * std::max(per_sm, 1), items);
}

template <class C>
void launch(const DeviceSchedule& s, const float* f1, const float* f2, const float* f3,
            int n_shells, int64_t K, int64_t k_begin, int64_t k_end, double* out, int num_sms,
            cudaStream_t st, double scale) {
  const int64_t n_slices = (k_end - k_begin + SLICE - 1) / SLICE;
  if constexpr (C::TR == 16) {
    int src = 8;
    for (const TileDesc& d : s.h_tiles) src = std::max(src, std::max(d.ni, d.nj));
    auto kern = contract_f32_kernel<C>;
    const size_t smem = C::smem(src);
    kern<<<blocks(kern, smem, C::smem(SRC), n_slices * s.n_sub, num_sms), 32, smem, st>>>(
        s.tiles, s.subs, s.n_sub, s.row_i, s.row_j, s.map, f1, f2, f3, n_shells, K, k_begin, k_end,
        n_slices, src, out, scale);
  } else {
    const int list = n_slices * s.n_parts[kNarrowParts] <= kNarrowPerSm<C> * num_sms ? kNarrowParts
                                                                                 : kWideParts;
    const F32Part* parts = s.parts + (list == kNarrowParts ? s.n_parts[kWideParts] : 0);
    auto kern = contract_f32_parts_kernel<C>;
    const size_t smem = C::smem(s.part_src);
    kern<<<blocks(kern, smem, C::smem(SRC), n_slices * s.n_parts[list], num_sms), 32, smem, st>>>(
        s.tiles, parts, s.n_parts[list], s.row_i, s.row_j, s.map, f1, f2, f3, n_shells, K, k_begin,
        k_end, n_slices, s.part_src, out, scale);
  }
  BSK_CHECK_CUDA(cudaGetLastError());
}
}  // namespace f32

template <typename Tin, typename Tacc>
void launch_simt(const DeviceSchedule& s, const Tin* f1, const Tin* f2, const Tin* f3,
                 int n_shells, int64_t K, int64_t k_begin, int64_t k_end, int64_t slice,
                 double* out, int num_sms, cudaStream_t st, double scale) {
  if (s.n_sub == 0 || k_end <= k_begin) return;
  const size_t smem = 2 * sizeof(Tacc) * KC * ((ROWS + APAD) + (COLS + BPAD));
  BSK_CHECK_CUDA(cudaFuncSetAttribute(contract_simt_kernel<Tin, Tacc>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  BSK_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &per_sm, contract_simt_kernel<Tin, Tacc>, THREADS, smem));
  if (per_sm < 1) per_sm = 1;
  const int64_t n_slices = (k_end - k_begin + slice - 1) / slice;
  const int64_t n_items = n_slices * s.n_sub;
  int64_t grid = (int64_t)num_sms * per_sm;
  if (grid > n_items) grid = n_items;
  contract_simt_kernel<Tin, Tacc><<<(unsigned)grid, THREADS, smem, st>>>(
      s.tiles, s.subs, s.n_sub, s.row_i, s.row_j, s.map, f1, f2, f3, n_shells, K, k_begin, k_end,
      slice, n_slices, out, scale);
  BSK_CHECK_CUDA(cudaGetLastError());
}

}  // namespace

// Whole-tile items from four an SM on (both sides measured, us, parts / whole tiles; one array,
// different arrays): 500 items 1122 / 1132, 1323 / 1334; 730 items 1714 / 1947, 2511 / 2013; 864
// items 1884 / 1682, 2096 / 1927; 2916 items 5794 / 3948, 7104 / 4739 ...
constexpr int64_t kLongItemsPerSm = 4;
// ... unless the parts have few columns between them: with 1.9 times the tiles' columns
// 110 400 / 103 500 (every seventh bin of 90 shells, 216^3), with 2.4 times 108 000 / 97 200 (all
// of them), but with no more than the tiles' (equilateral and squeezed sets: only the diagonal of
// a tile holds bins) 837 / 2002 (30 shells, 192^3), 1570 / 4382 (60), 5217 / 12 840 (60, 288^3).
constexpr double kLongDensity = 1.75;

// FP32 products and tile sums (8192-point slices), FP64 cross-slice sum.
void launch_contract_simt_f32(const DeviceSchedule& s, const float* f1, const float* f2,
                              const float* f3, int n_shells, int64_t K, int64_t k_begin,
                              int64_t k_end, double* out, int num_sms, cudaStream_t st,
                              double scale) {
  if (s.n_tiles == 0 || k_end <= k_begin) return;
  const int64_t n_slices = (k_end - k_begin + f32::SLICE - 1) / f32::SLICE;
  const bool is_long = n_slices * s.n_sub >= kLongItemsPerSm * num_sms &&
                       s.part_cols >= kLongDensity * s.sum_nc;
  bool two_src = f1 != f2 || (!is_long && s.part_two);
  if (is_long)
    for (const TileDesc& d : s.h_tiles) two_src = two_src || d.i0 != d.j0;
  const bool aligned = k_begin % 4 == 0 && K % 4 == 0 &&
                       ((uintptr_t)f1 | (uintptr_t)f2 | (uintptr_t)f3) % 16 == 0;
  const auto pick = [&](auto two, auto al) {
    constexpr bool kTwo = decltype(two)::value, kAl = decltype(al)::value;
    return is_long ? f32::launch<f32::Long<kTwo, kAl>> : f32::launch<f32::Short<kTwo, kAl>>;
  };
  const auto yes = std::true_type{};
  const auto no = std::false_type{};
  auto run = aligned ? (two_src ? pick(yes, yes) : pick(no, yes))
                     : (two_src ? pick(yes, no) : pick(no, no));
  run(s, f1, f2, f3, n_shells, K, k_begin, k_end, out, num_sms, st, scale);
}

// FP64 products and sums of FP32 fields (the yardstick of the precision study).
void launch_contract_simt_f64(const DeviceSchedule& s, const float* f1, const float* f2,
                              const float* f3, int n_shells, int64_t K, int64_t k_begin,
                              int64_t k_end, double* out, int num_sms, cudaStream_t st,
                              double scale) {
  launch_simt<float, double>(s, f1, f2, f3, n_shells, K, k_begin, k_end, 65536, out, num_sms, st,
                             scale);
}

// FP64 fields (grid information).
void launch_contract_simt_d64(const DeviceSchedule& s, const double* f1, const double* f2,
                              const double* f3, int n_shells, int64_t K, int64_t k_begin,
                              int64_t k_end, double* out, int num_sms, cudaStream_t st,
                              double scale) {
  launch_simt<double, double>(s, f1, f2, f3, n_shells, K, k_begin, k_end, 65536, out, num_sms, st,
                              scale);
}

}  // namespace bsk
