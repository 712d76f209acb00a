// Grid information (triangle counts and mean |k| per bin) from residues modulo small primes.
//
// The sums that bsk_gridinfo_enum.cu evaluates by enumeration,
//   N_tri(a, b, c) = #{q1 in a, q2 in b, q3 in c : q1 + q2 + q3 = 0}
//   S(a; b, c)     = sum over those triangles of w(q1),  w(q) = |q| 2^44 rounded to an integer,
// are cyclic convolutions at zero of integer arrays, and no triangle wraps around a grid of side
// N > 3 qmax.  So in any field that has an N-th root of unity omega
//   N^3 N_tri(a, b, c) = sum_x n_a(x) n_b(x) n_c(x),  n_s(x) = sum_{q in s} omega^(q . x),
// and likewise for S with k_s(x) = sum_{q in s} w(q) omega^(q . x).  In the integers modulo a
// prime p = 1 (mod N) everything is exact; a handful of primes below 1448 determines the
// values (the Chinese remainder theorem) because they are non-negative and bounded by the
// mode counts.  The whole evaluation is then three small dense transforms per shell and the
// triple-product contraction of the tensor-core kernel (launch_contract_mod), instead of a
// visit to every pair of modes: ~qmax^6 pairs against ~qmax^3 points times bins.  At 512^3 (63
// shells to |q| = 127) 1.81 s -> 90 ms (contraction 41, last axis 23, first two 17), at 256^3 (31
// shells to 63) 41 -> 5.3 ms, at |q| <= 40 (14 shells) 3.9 -> 1.8 ms; the enumeration's two
// launches are kept below that (kMinQ).
//
// Symmetry.  Membership and w do not change under sign flips of a component or the x <-> y swap
// (bsk_gridinfo_enum.cu), so n_s and k_s are even in every coordinate and symmetric in (x, y):
// they are evaluated at 0 <= y <= x, z <= N / 2 only (1/16 of the grid), a point's weight
// (1 or 2 per coordinate, 2 for x != y) multiplied into the column fields.  An even transform
// is E[x][q] = omega^(q x) + omega^(-q x) (1 for q = 0).
//
// Arithmetic.  Residues are kept as FP32 integers of magnitude at most (p - 1) / 2 <= 723; a
// product is below 2^19.1, so 32 of them add exactly in FP32 before a reduction.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "bsk_internal.cuh"

namespace bsk {
namespace gmod {

constexpr int kMaxPrimes = 16;
constexpr int kFrac = 44;       // fractional bits of w, as in the enumeration
constexpr int kMinQ = 40, kMaxQ = 159;  // kMaxQ: shared memory of the transforms
// Below kFewQ the enumeration is the faster one for plans of few modes too (us, enumeration /
// residues): one shell of 21 000 modes at 41 956 / 1094, of 31 000 at 50 1391 / 1522, but of
// 250 000 at 41 2511 / 1444 and of 41 000 at 57 1850 / 1747; two shells of 12 000 at 40 893 / 1077,
// of 20 000 1294 / 1096; six of 4600 1026 / 1072, of 15 000 1246 / 1089.
constexpr int kFewQ = 53;
inline int64_t few_modes(int n_shells) { return n_shells == 1 ? 80000 : 24000 / n_shells; }
constexpr int kRun = 32;        // products added between reductions

struct Prime {
  int p, N, h, hz;      // h = N / 2 + 1 points an axis, hz = h rounded up to even
  int np;               // (x, y) pairs, h (h + 1) / 2
  int64_t K;            // np hz rounded up to 128
  int inv_n3;           // N^-3 mod p
  void size() {
    h = N / 2 + 1;
    hz = (h + 1) & ~1;
    np = h * (h + 1) / 2;
    K = ((int64_t)np * hz + 127) / 128 * 128;
  }
};

struct Garner {         // inv[j][k] = p_j^-1 mod p_k (j < k)
  int n;
  int p[kMaxPrimes], inv_n3[kMaxPrimes];
  int inv[kMaxPrimes][kMaxPrimes];
};

int pow_mod(int64_t b, int64_t e, int p) {
  int64_t r = 1;
  for (b %= p; e; e >>= 1, b = b * b % p)
    if (e & 1) r = r * b % p;
  return (int)r;
}

bool is_prime(int n) {
  for (int d = 2; d * d <= n; ++d)
    if (n % d == 0) return false;
  return n > 1;
}

// Primes p = 1 (mod N) below kModMaxPrime with the smallest N > 3 qmax each has, cheapest first
// (points per bit), until their product exceeds 2^bits.
std::vector<Prime> choose_primes(int qmax, double bits) {
  std::vector<Prime> all;
  for (int p = 3; p < kModMaxPrime; p += 2) {
    if (!is_prime(p)) continue;
    for (int N = 3 * qmax + 1; N < p; ++N)
      if ((p - 1) % N == 0) {
        Prime q{};
        q.p = p;
        q.N = N;
        all.push_back(q);
        break;
      }
  }
  auto cost = [](const Prime& q) { return std::pow((double)q.N, 3) / std::log2((double)q.p); };
  std::sort(all.begin(), all.end(), [&](const Prime& a, const Prime& b) {
    const double ca = cost(a), cb = cost(b);
    return ca != cb ? ca < cb : a.p > b.p;
  });
  std::vector<Prime> out;
  double have = 0;
  for (Prime q : all) {
    if (have > bits) break;
    if ((int)out.size() == kMaxPrimes) return {};
    q.size();
    q.inv_n3 = pow_mod(pow_mod(q.N, 3, q.p), q.p - 2, q.p);
    have += std::log2((double)q.p);
    out.push_back(q);
  }
  if (have <= bits) return {};
  // without the smallest prime that the others do not need
  std::sort(out.begin(), out.end(), [](const Prime& a, const Prime& b) { return a.p > b.p; });
  while (!out.empty() && have - std::log2((double)out.back().p) > bits) {
    have -= std::log2((double)out.back().p);
    out.pop_back();
  }
  return out;
}

__device__ __forceinline__ float mod_red(float v, float p, float inv) {
  return fmaf(-rintf(v * inv), p, v);
}

__device__ __forceinline__ float centred(int v, int p) {  // 0 <= v < p
  return (float)(2 * v > p ? v - p : v);
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ unsigned long long mod_red2(unsigned long long v, float p, float inv) {
  const float2 f = unpack2(v);
  return pack2(mod_red(f.x, p, inv), mod_red(f.y, p, inv));
}

// E[q][x] (rows of ep, zero past h) and its prefix sums over q, thread = x; om: omega's powers.
__global__ void table_kernel(const int* __restrict__ om, int N, int h, int ep, int q1, int p,
                             float* __restrict__ E, float* __restrict__ prefix) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= ep) return;
  int sum = 0, r = 0;
  prefix[x] = 0.f;
  for (int a = 0; a < q1; ++a) {
    int v = 0;
    if (x < h) {
      v = a == 0 ? 1 : om[r] + om[r ? N - r : 0];
      if (v >= p) v -= p;
      sum += v;
      if (sum >= p) sum -= p;
      r += x;  // a x mod N
      if (r >= N) r -= N;
    }
    E[(int64_t)a * ep + x] = centred(v, p);
    prefix[(int64_t)(a + 1) * ep + x] = centred(sum, p);
  }
}

// w(q) mod p, centred, for 0 <= q_a, q_b, q_c <= qmax: the correctly rounded |q| 2^44.
__global__ void weight_kernel(int q1, int p, int16_t* __restrict__ w) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y, a = blockIdx.z;
  if (c >= q1) return;
  const double v = __dsqrt_rn((double)(a * a + b * b + c * c)) * 17592186044416.0;  // 2^44
  int r = (int)(llround(v) % p);
  if (2 * r > p) r -= p;
  w[((int64_t)a * q1 + b) * q1 + c] = (int16_t)r;
}

// First axis of the |k| fields: out[s][x][b][c] = sum over the shell's q_a of E[x][q_a] w(q_a, b,
// c), rows of cp; thread = column (b, c) of a shell, eight x at a time, so that a column's
// weights are read once for eight x (a block per x read them from L2 for each: 1.1 of 2.1 ms).
__global__ void __launch_bounds__(128)
    column_kernel(const uint32_t* __restrict__ range, const int16_t* __restrict__ w,
                  const float* __restrict__ E, int ep, int q1, int h, int cp,
                  const int* __restrict__ radius, float p, float inv, int16_t* __restrict__ out) {
  const int c = blockIdx.z * blockDim.x + threadIdx.x, b = blockIdx.x, s = blockIdx.y;
  if (b > radius[s] || c >= cp) return;
  const uint32_t r = c < q1 ? range[((int64_t)s * q1 + b) * q1 + c] : kEmptyRange;
  const int a0 = (int)(r & 0xFFFF), a1 = (int)(r >> 16);
  int16_t* o = out + ((int64_t)s * h * q1 + b) * cp + c;
  for (int x0 = 0; x0 < h; x0 += 8) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
    int run = 0;
    for (int a = a0; a <= a1; ++a) {
      const float wa = (float)w[((int64_t)a * q1 + b) * q1 + c];
      const float4 e0 = __ldg(reinterpret_cast<const float4*>(E + (int64_t)a * ep + x0));
      const float4 e1 = __ldg(reinterpret_cast<const float4*>(E + (int64_t)a * ep + x0 + 4));
      const float ev[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = fmaf(ev[e], wa, v[e]);
      if (++run == kRun - 1) {  // with the residue carried on, kRun terms at most
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = mod_red(v[e], p, inv);
        run = 0;
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (x0 + e < h) o[(int64_t)(x0 + e) * q1 * cp] = (int16_t)mod_red(v[e], p, inv);
  }
}

// First two axes: block = (x, shell).  The plane A[b][c] (first axis done) goes to shared memory:
// for the count fields sum_{q_a in s} E[x][q_a], a difference of E's prefix sums, for the |k|
// fields column_kernel's.  Then out[pair(x, y)][c] = sum_b E[y][b] A[b][c], y <= x: a warp takes
// 8 y, a lane 4 c, 16 packed multiply-adds (by two y) for one 16-byte shared-memory load and
// two broadcast loads of E.
constexpr int kXyThreads = 256;
template <bool kWeighted>
__global__ void __launch_bounds__(kXyThreads)
    xy_kernel(const uint32_t* __restrict__ range, const int16_t* __restrict__ plane,
              const float* __restrict__ E /*[q][ep]*/, const float* __restrict__ prefix, int ep,
              int q1, const int* __restrict__ radius, int np, int cp, float p, float inv,
              float* __restrict__ out) {
  extern __shared__ __align__(16) float sA[];  // [R + 1][cp]
  __shared__ float sE[kMaxQ + 2];
  const int h = (int)gridDim.x;
  const int x = h - 1 - (int)blockIdx.x;  // the longest blocks first
  const int s = blockIdx.y;
  const int R = radius[s], nb = R + 1;
  if (kWeighted) {
    const int16_t* src = plane + ((int64_t)s * h + x) * q1 * cp;
    for (int i = threadIdx.x * 4; i < nb * cp; i += kXyThreads * 4) {
      const short4 v = *reinterpret_cast<const short4*>(src + i);
      *reinterpret_cast<float4*>(sA + i) = make_float4(v.x, v.y, v.z, v.w);
    }
  } else {
    for (int a = threadIdx.x; a < q1 + 1; a += kXyThreads) sE[a] = prefix[(int64_t)a * ep + x];
    __syncthreads();
    const uint32_t* rg = range + (int64_t)s * q1 * q1;
    for (int b = threadIdx.x >> 5; b < nb; b += kXyThreads / 32)
      for (int c = threadIdx.x & 31; c < cp; c += 32) {
        const uint32_t r = c < nb ? rg[b * q1 + c] : kEmptyRange;
        sA[b * cp + c] = r == kEmptyRange
                             ? 0.f
                             : mod_red(sE[(int)(r >> 16) + 1] - sE[(int)(r & 0xFFFF)], p, inv);
      }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* o = out + ((int64_t)s * np + (int64_t)x * (x + 1) / 2) * cp;
  for (int y0 = warp * 8; y0 <= x; y0 += (kXyThreads / 32) * 8) {
    for (int c = lane * 4; c < cp; c += 128) {
      unsigned long long acc[4][4];  // y pair, c
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[y][e] = 0ull;
      for (int b0 = 0; b0 < nb; b0 += kRun - 1) {
        const int b1 = min(nb, b0 + kRun - 1);
#pragma unroll 4
        for (int b = b0; b < b1; ++b) {
          const float4 av = *reinterpret_cast<const float4*>(sA + b * cp + c);
          const ulonglong2 e0 = __ldg(reinterpret_cast<const ulonglong2*>(E + (int64_t)b * ep + y0));
          const ulonglong2 e1 =
              __ldg(reinterpret_cast<const ulonglong2*>(E + (int64_t)b * ep + y0 + 4));
          const unsigned long long ev[4] = {e0.x, e0.y, e1.x, e1.y};
          const unsigned long long ad[4] = {pack2(av.x, av.x), pack2(av.y, av.y),
                                            pack2(av.z, av.z), pack2(av.w, av.w)};
#pragma unroll
          for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[y][e] = fma2(ev[y], ad[e], acc[y][e]);
        }
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[y][e] = mod_red2(acc[y][e], p, inv);
      }
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const float2 v[4] = {unpack2(acc[y][0]), unpack2(acc[y][1]), unpack2(acc[y][2]),
                             unpack2(acc[y][3])};
        float* oy = o + (int64_t)(y0 + 2 * y) * cp + c;
        if (y0 + 2 * y <= x)
          *reinterpret_cast<float4*>(oy) = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
        if (y0 + 2 * y + 1 <= x)
          *reinterpret_cast<float4*>(oy + cp) = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
      }
    }
  }
}

// Last axis: out[pair][z] = sum_c H[pair][c] E[z][c] for kPairs pairs at a time, persistent blocks
// (E stays in shared memory).  A warp takes 32 pairs x 64 z, a thread 8 x 8, as 32 multiply-adds
// packed by two z: per c 8 values of H (broadcast in a quarter warp) and 4 x 8 bytes of E, 16
// shared-memory wavefronts.  Writes the FP32 field (pair factors) and / or the weighted
// field's split (columns).
template <int kPairs>
__global__ void __launch_bounds__(4 * kPairs, 1)
    z_kernel(const float* __restrict__ H, const float* __restrict__ E, int ep, int q1,
             const int* __restrict__ radius, int n_shells, Prime pr, int cp, float p, float inv,
             float* __restrict__ field, __nv_bfloat16* __restrict__ split) {
  extern __shared__ __align__(16) float smz[];
  constexpr int kThreads = 4 * kPairs, kWarpRows = kPairs / 32;
  const int zp = (pr.hz + 63) / 64 * 64;
  float* sE = smz;                    // [q1 + 1][zp], the last row zero (an odd count's second c)
  float* sH = sE + (size_t)(q1 + 1) * zp;   // [kPairs][cp + 4]
  const int hp = cp + 4;
  for (int i = threadIdx.x; i < (q1 + 1) * zp; i += kThreads) {
    const int c = i / zp, z = i - c * zp;
    sE[i] = z < pr.h && c < q1 ? E[(int64_t)c * ep + z] : 0.f;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pg = warp % kWarpRows * 32 + (lane >> 3) * 8;  // this thread's 8 pairs
  const int zl = (lane & 7) * 2;                     // its z: zl + {0, 1} + 16 j of each 64
  const int tiles = (pr.np + kPairs - 1) / kPairs;
  // the next tile's rows are copied while the current one is reduced and stored
  auto fetch = [&](int u) {
    if (u >= tiles * n_shells) return;
    const int s = u / tiles, t0 = (u - s * tiles) * kPairs;
    const int nc4 = (radius[s] + 4) & ~3;
    for (int r = threadIdx.x >> 2; r < kPairs; r += kThreads / 4) {
      const int pair = min(t0 + r, pr.np - 1);  // past the last pair: any (not stored)
      const float* src = H + ((int64_t)s * pr.np + pair) * cp;
      for (int c = (threadIdx.x & 3) * 4; c < nc4; c += 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(sH + r * hp + c)),
                     "l"(src + c)
                     : "memory");
    }
  };
  fetch(blockIdx.x);
  for (int u = blockIdx.x; u < tiles * n_shells; u += gridDim.x) {
    const int s = u / tiles, t0 = (u - s * tiles) * kPairs;
    const int nc = radius[s] + 1, nc2 = (nc + 1) & ~1;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the rows have landed (and E, the first time)
    const int z0 = warp / kWarpRows * 64;  // 4 x 64 points cover hz (at most 256)
    unsigned long long acc[8][4];  // pair, z pair
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[a][j] = 0ull;
    // 28 products and a residue between reductions
    for (int c0 = 0; c0 < nc && z0 < pr.hz; c0 += 28) {
      const int c1 = min(nc2, c0 + 28);
      for (int c = c0; c < c1; c += 2) {
        float2 hv[8];
#pragma unroll
        for (int a = 0; a < 8; ++a)
          hv[a] = *reinterpret_cast<const float2*>(sH + (pg + a) * hp + c);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          unsigned long long ev[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ev[j] = *reinterpret_cast<const unsigned long long*>(sE + (c + k) * zp + z0 + zl +
                                                                 16 * j);
#pragma unroll
          for (int a = 0; a < 8; ++a) {
            const float h = k == 0 ? hv[a].x : hv[a].y;
            const unsigned long long hd = pack2(h, h);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[a][j] = fma2(hd, ev[j], acc[a][j]);
          }
        }
      }
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[a][j] = mod_red2(acc[a][j], p, inv);
    }
    __syncthreads();  // every warp has read the rows
    fetch(u + gridDim.x);
    // (x, y) of the thread's first pair
    int x, y;
    {
      const int pair = min(t0 + pg, pr.np - 1);
      x = (int)((sqrtf(8.f * pair + 1.f) - 1.f) * 0.5f);
      while ((x + 1) * (x + 2) / 2 <= pair) ++x;
      while (x * (x + 1) / 2 > pair) --x;
      y = pair - x * (x + 1) / 2;
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int pair = t0 + pg + a;
      if (pair >= pr.np) break;
      const float wxy = (x == 0 || 2 * x == pr.N ? 1.f : 2.f) *
                        (y == 0 || 2 * y == pr.N ? 1.f : 2.f) * (x != y ? 2.f : 1.f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int z = z0 + zl + 16 * j;
        if (z >= pr.hz) continue;
        const float2 v = unpack2(acc[a][j]);
        const float v0 = v.x, v1 = v.y;
        const int64_t pt = (int64_t)pair * pr.hz + z;
        if (field)
          *reinterpret_cast<float2*>(field + (int64_t)s * pr.K + pt) = make_float2(v0, v1);
        if (split) {
          const float w0 = wxy * (z == 0 || 2 * z == pr.N ? 1.f : 2.f);
          const float w1 = wxy * (2 * (z + 1) == pr.N ? 1.f : 2.f);
          const float u0 = mod_red(v0 * w0, p, inv), u1 = mod_red(v1 * w1, p, inv);
          const float h0 = 8.f * rintf(u0 * 0.125f), h1 = 8.f * rintf(u1 * 0.125f);
          *reinterpret_cast<__nv_bfloat162*>(split + split_index(0, s, pt, n_shells)) =
              __floats2bfloat162_rn(h0, h1);
          *reinterpret_cast<__nv_bfloat162*>(split + split_index(1, s, pt, n_shells)) =
              __floats2bfloat162_rn(u0 - h0, u1 - h1);
        }
      }
      if (++y > x) {
        ++x;
        y = 0;
      }
    }
  }
}

// The non-negative integer below the product of the first n primes with the given residues.
__device__ unsigned __int128 crt(const Garner& g, int n, const int* r) {
  int d[kMaxPrimes];  // mixed-radix digits
  for (int k = 0; k < n; ++k) {
    int v = r[k];
    for (int j = 0; j < k; ++j) {
      v = (v - d[j]) % g.p[k];
      if (v < 0) v += g.p[k];
      v = (int)((int64_t)v * g.inv[j][k] % g.p[k]);
    }
    d[k] = v;
  }
  unsigned __int128 x = 0;
  for (int k = n - 1; k >= 0; --k) x = x * (unsigned)g.p[k] + (unsigned)d[k];
  return x;
}

// Per triangle: its count and three |k| sums from their residues (cnt [n_cnt][ne], sum
// [g.n][ns]: integers congruent to N^3 times them).
__global__ void modular_finish_kernel(int64_t T, const int4* __restrict__ idx, Garner g,
                                      int n_cnt, int ne, int ns,
                                      const long long* __restrict__ cnt,
                                      const long long* __restrict__ sum, double kf,
                                      double* __restrict__ ntri, double* __restrict__ kmean) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 4 * T) return;
  const int64_t t = i >> 2;
  const int role = (int)(i & 3);  // 0: the count, 1 .. 3: the |k| sums (lanes of one triangle)
  const int4 id = idx[t];
  int r[kMaxPrimes];
  const int n = role ? g.n : n_cnt;
  const int e = role == 0 ? id.x : role == 1 ? id.y : role == 2 ? id.z : id.w;
  for (int k = 0; k < n; ++k) {
    long long v = (role ? sum[(int64_t)k * ns + e] : cnt[(int64_t)k * ne + e]) % g.p[k];
    if (v < 0) v += g.p[k];
    r[k] = (int)(v * g.inv_n3[k] % g.p[k]);
  }
  const unsigned __int128 x = crt(g, n, r);
  const double value = (double)(unsigned long long)(x >> 64) * 18446744073709551616.0 +
                       (double)(unsigned long long)x;
  // 4 T is a multiple of 4, so a triangle's four lanes are all here
  const unsigned lanes = 0xFu << (threadIdx.x & 28);
  const double count = __shfl_sync(lanes, value, 0, 4);
  if (role == 0) {
    ntri[t] = value;
  } else {
    kmean[3 * t + role - 1] =
        count != 0.0 ? value * (1.0 / (double)(1ull << kFrac)) / count * kf : nan("");
  }
}

struct Upload {  // host arrays gathered into one device block
  std::vector<unsigned char> host;
  size_t add(const void* src, size_t bytes) {
    const size_t at = (host.size() + 255) / 256 * 256;
    host.resize(at + bytes);
    if (bytes) memcpy(host.data() + at, src, bytes);
    return at;
  }
};

struct UploadedSchedule {
  size_t tiles, ri, rj, map;
  HostSchedule h;
  void add(Upload& up) {
    tiles = up.add(h.tiles.data(), h.tiles.size() * sizeof(TileDesc));
    ri = up.add(h.ri.data(), h.ri.size() * sizeof(int16_t));
    rj = up.add(h.rj.data(), h.rj.size() * sizeof(int16_t));
    map = up.add(h.map.data(), h.map.size() * sizeof(int32_t));
  }
  void bind(unsigned char* base, DeviceSchedule& s) const {
    s.n_tiles = (int)h.tiles.size();
    s.tiles = (TileDesc*)(base + tiles);
    s.row_i = (int16_t*)(base + ri);
    s.row_j = (int16_t*)(base + rj);
    s.map = (int32_t*)(base + map);
    s.h_tiles = h.tiles;
  }
};

size_t z_smem(const Prime& q, int q1, int cp, int pairs) {
  return ((size_t)(q1 + 1) * ((q.hz + 63) / 64 * 64) + (size_t)pairs * (cp + 4)) * sizeof(float);
}
constexpr size_t kMaxSmem = 227 * 1024;

}  // namespace gmod

bool gridinfo_modular(bsk_plan* p, const std::vector<HostTriangle>& tri, double* ntri,
                      double* kmean, cudaStream_t st) {
  using namespace gmod;
  if (!gridinfo_enum_supported(p) || p->qmax < kMinQ || p->qmax > kMaxQ) return false;
  const int n = p->n, q1 = p->qmax + 1;
  const int64_t T = (int64_t)tri.size();
  if (T > (int64_t)1 << 28) return false;
  int64_t modes = 0;
  for (int64_t c : p->counts) modes += c;
  if (p->qmax < kFewQ && modes <= few_modes(n)) return false;
  const int cp = (q1 + 3) / 4 * 4;
  if (p->mem_budget) {  // the least that any primes need, before the 130 us of choosing them
    Prime q{};
    q.N = 3 * p->qmax + 1;
    q.size();
    const size_t least = (size_t)n * (q.np * (size_t)cp + q.K) * sizeof(float) +
                         split_elems(n, q.K) * sizeof(__nv_bfloat16);
    if (device_bytes(p) + (int64_t)least > (int64_t)p->mem_budget) return false;
  }

  // distinct counts (shells sorted) and distinct |k| sums (pair (y >= z), the weighted shell x)
  std::vector<HostTriangle> ec, es;
  std::vector<int> at_c((size_t)n * n * n, -1), at_s(at_c);
  std::vector<int4> idx(T);
  auto entry = [&](std::vector<int>& at, std::vector<HostTriangle>& list, int i, int j, int l) {
    int& e = at[((size_t)i * n + j) * n + l];
    if (e < 0) {
      e = (int)list.size();
      list.push_back(HostTriangle{i, j, l});
    }
    return e;
  };
  double bound = 1.0;  // on any count: the product of a bin's two smallest mode counts
  double kmax = 1.0;
  for (int64_t t = 0; t < T; ++t) {
    int a[3] = {tri[t].i, tri[t].j, tri[t].l};
    int id[3];
    for (int role = 0; role < 3; ++role) {
      const int y = a[(role + 1) % 3], z = a[(role + 2) % 3];
      id[role] = entry(at_s, es, std::max(y, z), std::min(y, z), a[role]);
    }
    std::sort(a, a + 3);
    const int c = entry(at_c, ec, a[2], a[1], a[0]);
    idx[t] = make_int4(c, id[0], id[1], id[2]);
    double m[3] = {(double)p->counts[a[0]], (double)p->counts[a[1]], (double)p->counts[a[2]]};
    std::sort(m, m + 3);
    bound = std::max(bound, m[0] * m[1]);
  }
  kmax = (p->qmax + 1) * std::ldexp(1.0, kFrac);
  const std::vector<Prime> primes = choose_primes(p->qmax, std::log2(bound * kmax) + 1.0);
  if (primes.empty()) return false;
  const int n_pr = (int)primes.size();
  int n_cnt = 0;
  double have = 0;
  while (n_cnt < n_pr && have <= std::log2(bound) + 1.0) have += std::log2((double)primes[n_cnt++].p);
  int64_t max_k = 0, max_np = 0;
  for (const Prime& q : primes) {
    if (q.hz > 256 || z_smem(q, q1, cp, 64) > kMaxSmem) return false;
    max_k = std::max(max_k, q.K);
    max_np = std::max<int64_t>(max_np, q.np);
  }

  // host tables: schedules, shell radii, triangle entries, powers of omega per prime
  Upload up;
  UploadedSchedule sc, ss;
  tile_schedule(ec, n, nullptr, sc.h);
  tile_schedule(es, n, nullptr, ss.h);
  sc.add(up);
  ss.add(up);
  const size_t o_idx = up.add(idx.data(), T * sizeof(int4));
  const size_t o_rad = up.add(p->shell_r.data(), n * sizeof(int));
  std::vector<size_t> o_om(n_pr);
  std::vector<int> ep(n_pr);
  Garner g{};
  g.n = n_pr;
  for (int k = 0; k < n_pr; ++k) {
    const Prime& q = primes[k];
    g.p[k] = q.p;
    g.inv_n3[k] = q.inv_n3;
    for (int j = 0; j < k; ++j) g.inv[j][k] = pow_mod(primes[j].p, q.p - 2, q.p);
    int gen = 2;  // a generator of the field: its (p - 1) / f powers differ from 1 for every prime f
    for (;; ++gen) {
      bool ok = true;
      for (int f = 2, m = q.p - 1; m > 1; ++f)
        if (m % f == 0) {
          while (m % f == 0) m /= f;
          ok = ok && pow_mod(gen, (q.p - 1) / f, q.p) != 1;
        }
      if (ok) break;
    }
    std::vector<int> om(q.N);  // powers of omega
    const int omega = pow_mod(gen, (q.p - 1) / q.N, q.p);
    om[0] = 1;
    for (int i = 1; i < q.N; ++i) om[i] = (int)((int64_t)om[i - 1] * omega % q.p);
    ep[k] = (q.h + 7) / 8 * 8;
    o_om[k] = up.add(om.data(), om.size() * sizeof(int));
  }

  // device scratch in one stream-ordered block
  const int ne = (int)ec.size(), ns = (int)es.size();
  size_t total = 0;
  auto take = [&](size_t bytes) {
    const size_t at = total;
    total += (bytes + 1023) / 1024 * 1024;
    return at;
  };
  const size_t a_up = take(up.host.size());
  const size_t a_range = take((size_t)n * q1 * q1 * sizeof(uint32_t));
  const size_t a_w = take((size_t)q1 * q1 * q1 * sizeof(int16_t));
  const size_t a_out = take(((size_t)n_cnt * ne + (size_t)n_pr * ns) * sizeof(long long) + 8);
  int max_ep = 0;
  for (int e : ep) max_ep = std::max(max_ep, e);
  const size_t a_e = take((size_t)(2 * q1 + 1) * max_ep * sizeof(float));
  const size_t a_h = take((size_t)n * max_np * cp * sizeof(float));
  const size_t a_f = take((size_t)n * max_k * sizeof(float));
  // column_kernel's planes lie where the split of the same prime's |k| field goes later
  size_t planes = 0;
  for (const Prime& q : primes) planes = std::max(planes, (size_t)n * q.h * q1 * cp);
  const size_t a_s = take(std::max(split_elems(n, max_k) * sizeof(__nv_bfloat16),
                                   planes * sizeof(int16_t)));
  if (p->mem_budget && device_bytes(p) + (int64_t)total > (int64_t)p->mem_budget) return false;
  unsigned char* base = nullptr;
  if (cudaMallocAsync((void**)&base, total, st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  struct Free {
    void* w;
    cudaStream_t s;
    ~Free() { cudaFreeAsync(w, s); }
  } free_base{base, st};
  BSK_CHECK_CUDA(cudaMemcpyAsync(base + a_up, up.host.data(), up.host.size(),
                                 cudaMemcpyHostToDevice, st));
  uint32_t* range = (uint32_t*)(base + a_range);
  int16_t* w = (int16_t*)(base + a_w);
  long long* cnt = (long long*)(base + a_out);
  long long* sum = cnt + (size_t)n_cnt * ne;
  int* flag = (int*)(sum + (size_t)n_pr * ns);
  float* H = (float*)(base + a_h);
  float* field = (float*)(base + a_f);
  __nv_bfloat16* split = (__nv_bfloat16*)(base + a_s);
  const int* radius = (const int*)(base + a_up + o_rad);
  BSK_CHECK_CUDA(cudaMemsetAsync(cnt, 0, (char*)(flag + 2) - (char*)cnt, st));
  launch_shell_range(p, range, flag, st);
  int hflag = 0, gave_up = 0;
  BSK_CHECK_CUDA(cudaMemcpyAsync(&hflag, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  tc_error_flag_async(&gave_up, st);
  BSK_CHECK_CUDA(cudaStreamSynchronize(st));
  BSK_REQUIRE(hflag == 0, BSK_ERR_STATE, "internal: a mode lies in more than two shells");
  if (gave_up) return false;  // set by an earlier launch: it cuts the waits of later ones short

  DeviceSchedule dc, ds;
  sc.bind(base + a_up, dc);
  ss.bind(base + a_up, ds);
  float* E = (float*)(base + a_e);
  float* pre = E + (size_t)q1 * max_ep;
  const size_t xy_smem = (size_t)q1 * cp * sizeof(float);
  BSK_CHECK_CUDA(cudaFuncSetAttribute(xy_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)xy_smem));
  BSK_CHECK_CUDA(cudaFuncSetAttribute(xy_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)xy_smem));
  for (auto z : {z_kernel<64>, z_kernel<128>})
    BSK_CHECK_CUDA(cudaFuncSetAttribute(z, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kMaxSmem));
  for (int k = 0; k < n_pr; ++k) {
    const Prime& q = primes[k];
    table_kernel<<<(ep[k] + 31) / 32, 32, 0, st>>>((const int*)(base + a_up + o_om[k]), q.N, q.h,
                                                   ep[k], q1, q.p, E, pre);
    BSK_CHECK_CUDA(cudaGetLastError());
    const float pf = (float)q.p, inv = 1.f / pf;
    const int64_t points = (int64_t)q.np * q.hz;
    // the points past the last pair: zero in the fields, and so is the last chunk's split
    if (q.K > points)
      BSK_CHECK_CUDA(cudaMemset2DAsync(field + points, q.K * sizeof(float), 0,
                                       (q.K - points) * sizeof(float), n, st));
    const int pairs = z_smem(q, q1, cp, 128) <= kMaxSmem ? 128 : 64;
    const size_t zs = z_smem(q, q1, cp, pairs);
    const int z_grid = std::min(p->num_sms, (q.np + pairs - 1) / pairs * n);
    const auto last_axis = [&](float* f, __nv_bfloat16* planes_out) {
      if (planes_out)
        BSK_CHECK_CUDA(cudaMemsetAsync(split + split_elems(n, q.K - 128), 0,
                                       (split_elems(n, q.K) - split_elems(n, q.K - 128)) *
                                           sizeof(__nv_bfloat16), st));
      auto z = pairs == 128 ? z_kernel<128> : z_kernel<64>;
      z<<<z_grid, 4 * pairs, zs, st>>>(H, E, ep[k], q1, radius, n, q, cp, pf, inv, f, planes_out);
      BSK_CHECK_CUDA(cudaGetLastError());
    };
    xy_kernel<false><<<dim3(q.h, n), kXyThreads, xy_smem, st>>>(range, nullptr, E, pre, ep[k], q1,
                                                               radius, q.np, cp, pf, inv, H);
    BSK_CHECK_CUDA(cudaGetLastError());
    last_axis(field, k < n_cnt ? split : nullptr);
    if (k < n_cnt)
      launch_contract_mod(dc, field, split, n, q.K, q.p,
                          (unsigned long long*)cnt + (size_t)k * ne, p->num_sms, st);
    weight_kernel<<<dim3((q1 + 63) / 64, q1, q1), 64, 0, st>>>(q1, q.p, w);
    int16_t* plane = (int16_t*)split;
    column_kernel<<<dim3(q1, n, (cp + 127) / 128), 128, 0, st>>>(range, w, E, ep[k], q1, q.h, cp,
                                                                 radius, pf, inv, plane);
    xy_kernel<true><<<dim3(q.h, n), kXyThreads, xy_smem, st>>>(range, plane, E, pre, ep[k], q1,
                                                              radius, q.np, cp, pf, inv, H);
    BSK_CHECK_CUDA(cudaGetLastError());
    last_axis(nullptr, split);
    launch_contract_mod(ds, field, split, n, q.K, q.p,
                        (unsigned long long*)sum + (size_t)k * ns, p->num_sms, st);
  }
  const double kf = 2.0 * 3.14159265358979323846 / p->L;
  modular_finish_kernel<<<(unsigned)((4 * T + 127) / 128), 128, 0, st>>>(
      T, (const int4*)(base + a_up + o_idx), g, n_cnt, ne, ns, cnt, sum, kf, ntri, kmean);
  BSK_CHECK_CUDA(cudaGetLastError());
  dc.tiles = ds.tiles = nullptr;  // in the scratch block: nothing to release
  // a contraction that gave up has left sums out, and any residues make a count of some kind
  tc_error_flag_async(&gave_up, st);
  BSK_CHECK_CUDA(cudaStreamSynchronize(st));  // the host tables must outlive their copy
  return !gave_up;
}

}  // namespace bsk
