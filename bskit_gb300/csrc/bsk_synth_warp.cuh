// Field synthesis: FFT arithmetic and the warp-per-lines passes of compiled lengths.
//
// A compiled length N = RA RB is transformed in two register stages by one warp working on L
// lines of its own: stage A, RB butterflies of radix RA a line, whose inputs come straight from
// global memory, and stage B, RA groups of RB points (one radix, or two done one after the
// other in registers), whose outputs go straight to global memory.  One shared-memory exchange
// lies between them, and only warp barriers: a block's warps drift apart, so that one's loads,
// another's butterflies and a third's stores overlap.  (Blocks of 256 threads with a barrier
// around each pass kept the three apart: the Z pass of 384^3 ran at 0.69 of the HBM rate when
// writing fields and planes, and no faster, 0.79 ms a batch, when writing planes alone.)
// The exchange holds element (j, r) of stage A's butterfly j at j (RA + 1) + r: RA + 1 is
// odd, so the writes (consecutive j) and the reads (consecutive r) are free of bank conflicts.
//
// The butterflies, their order and their twiddles (a table computed in double precision) are
// those of the Stockham passes of run-time lengths (plan_radix), so a length gives the same bits
// on either path.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>

#include "bsk_internal.cuh"

namespace bsk {
namespace synth {

__device__ __forceinline__ int fft_freq(int a, int n) { return a < (n + 1) / 2 ? a : a - n; }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// multiply by +i
__device__ __forceinline__ float2 mul_i(float2 a) { return make_float2(-a.y, a.x); }

// Unnormalised R-point DFT with sign +1 in registers: v[q] <- sum_r v[r] e^{+2 pi i r q / R}.
// roots[R][k] = e^{+2 pi i k / R}.
__device__ __forceinline__ void dft2(float2* v) {
  const float2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}
__device__ __forceinline__ void dft4(float2* v) {
  const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
  const float2 s13 = cadd(v[1], v[3]), d13 = mul_i(csub(v[1], v[3]));
  v[0] = cadd(s02, s13);
  v[2] = csub(s02, s13);
  v[1] = cadd(d02, d13);
  v[3] = csub(d02, d13);
}
__device__ __forceinline__ void dft8(float2* v) {
  // two 4-point DFTs of the even and odd samples, combined with e^{+2 pi i k / 8}
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  dft4(e);
  dft4(o);
  const float h = 0.70710678118654752f;
  const float2 w1 = make_float2(h, h), w3 = make_float2(-h, h);
  const float2 t0 = o[0], t1 = cmul(o[1], w1), t2 = mul_i(o[2]), t3 = cmul(o[3], w3);
  v[0] = cadd(e[0], t0);
  v[4] = csub(e[0], t0);
  v[1] = cadd(e[1], t1);
  v[5] = csub(e[1], t1);
  v[2] = cadd(e[2], t2);
  v[6] = csub(e[2], t2);
  v[3] = cadd(e[3], t3);
  v[7] = csub(e[3], t3);
}
__device__ __forceinline__ void dft16(float2* v) {
  // 16 = 4 x 4: DFT4 over a of v[4a + b], twiddle e^{2 pi i b c / 16}, DFT4 over b
  float2 y[4][4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    float2 t[4] = {v[b], v[4 + b], v[8 + b], v[12 + b]};
    dft4(t);
#pragma unroll
    for (int c = 0; c < 4; ++c) y[b][c] = t[c];
  }
  const float c1 = 0.92387953251128676f, s1 = 0.38268343236508977f;  // cos, sin(pi/8)
  const float h = 0.70710678118654752f;
  // e^{2 pi i k / 16} for k = b c: k = 1, 2, 3, 4, 6, 9
  y[1][1] = cmul(y[1][1], make_float2(c1, s1));
  y[1][2] = cmul(y[1][2], make_float2(h, h));
  y[1][3] = cmul(y[1][3], make_float2(s1, c1));
  y[2][1] = cmul(y[2][1], make_float2(h, h));
  y[2][2] = mul_i(y[2][2]);
  y[2][3] = cmul(y[2][3], make_float2(-h, h));
  y[3][1] = cmul(y[3][1], make_float2(s1, c1));
  y[3][2] = cmul(y[3][2], make_float2(-h, h));
  y[3][3] = cmul(y[3][3], make_float2(-c1, -s1));
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float2 t[4] = {y[0][c], y[1][c], y[2][c], y[3][c]};
    dft4(t);
#pragma unroll
    for (int d = 0; d < 4; ++d) v[c + 4 * d] = t[d];
  }
}
template <int R>
__device__ __forceinline__ void dft_generic(float2* v, const float2* roots) {
  float2 out[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    float2 acc = v[0];
#pragma unroll
    for (int r = 1; r < R; ++r) acc = cadd(acc, cmul(v[r], roots[(r * q) % R]));
    out[q] = acc;
  }
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = out[q];
}

struct FftPlan {
  int n;
  int np;
  int radix[8];  // 16, 24, 12, 8, 6, 4, 2, 3 or 5
  float2 root3[3];
  float2 root5[5];
  float2 rootc[24];  // e^{+2 pi i k / Rc} of the plan's composite radix Rc (24, 12 or 6)
};

template <int R>
__device__ __forceinline__ void dft_small(float2* v, const FftPlan& pl) {
  if (R == 8) dft8(v);
  else if (R == 4) dft4(v);
  else if (R == 2) dft2(v);
  else if (R == 3) dft_generic<3>(v, pl.root3);
  else dft_generic<5>(v, pl.root5);
}

// R = R1 R2 point DFT: input r = R2 a + b, output q = c + R1 d:
// X[c + R1 d] = sum_b e^{2 pi i b d / R2} e^{2 pi i b c / R} sum_a v[R2 a + b] e^{2 pi i a c / R1}.
template <int R1, int R2>
__device__ __forceinline__ void dft_comp(float2* v, const FftPlan& pl) {
  float2 y[R2][R1];
#pragma unroll
  for (int b = 0; b < R2; ++b) {
    float2 t[R1];
#pragma unroll
    for (int a = 0; a < R1; ++a) t[a] = v[R2 * a + b];
    dft_small<R1>(t, pl);
#pragma unroll
    for (int c = 0; c < R1; ++c) y[b][c] = b && c ? cmul(t[c], pl.rootc[b * c]) : t[c];
  }
#pragma unroll
  for (int c = 0; c < R1; ++c) {
    float2 t[R2];
#pragma unroll
    for (int b = 0; b < R2; ++b) t[b] = y[b][c];
    dft_small<R2>(t, pl);
#pragma unroll
    for (int d = 0; d < R2; ++d) v[c + R1 * d] = t[d];
  }
}

// Radix plan of a length: 16s, then one of 24 / 12 / 8 / 6 / 4 / 2, then 3s and 5s (constexpr, so that a
// compile-time length gets a fully unrolled pass sequence).
// The p-th radix of a length's plan (0 past the end, -1 when the length does not factor).
__host__ __device__ constexpr int plan_radix(int n, int p) {
  int k = 0;
  while (n % 16 == 0) { n /= 16; if (k++ == p) return 16; }
  const int comp[6] = {24, 12, 8, 6, 4, 2};  // at most one of these, 2^a 3 first
  for (int c : comp)
    if (n % c == 0) { n /= c; if (k++ == p) return c; break; }
  while (n % 3 == 0) { n /= 3; if (k++ == p) return 3; }
  while (n % 5 == 0) { n /= 5; if (k++ == p) return 5; }
  return n == 1 ? 0 : -1;
}
__host__ __device__ constexpr int plan_np(int n) {
  int p = 0;
  while (plan_radix(n, p) > 0) ++p;
  return plan_radix(n, p) == 0 ? p : -1;
}

template <int R>
__device__ __forceinline__ void dft_radix(float2* v, const FftPlan& pl) {
  if (R == 16) dft16(v);
  else if (R == 24) dft_comp<8, 3>(v, pl);
  else if (R == 12) dft_comp<4, 3>(v, pl);
  else if (R == 6) dft_comp<2, 3>(v, pl);
  else dft_small<R>(v, pl);
}

// Index of the i-th kept frequency of an axis: the `nk` frequencies |q| <= R around 0
// (all n of them when 2R + 1 >= n).
__device__ __forceinline__ int kept_index(int i, int nk, int R, int n) {
  return nk == n ? i : (i - R + n) % n;
}

struct SynthArgs {
  int N, H, R, nk, Cp, s0, ns;
  int out0;                // shell written at fields[0] (and hi/lo[0])
  int fields_from;         // the FP32 field is written for shells s0 + s >= fields_from only
  const float2* spec;      // [a][b][c] slot spectrum
  const uint16_t* table;   // [a][b][c] shell codes (run-time lengths)
  const int* radius;       // [shell] largest |q_c| of each shell, at most R of the batch's
  const uint32_t* range;   // [shell][|b|][c] |q_a| interval (compiled lengths), q1 values an axis
  int q1;
  float2* G;               // [s][x][bk][c]   (c < Cp)
  float2* Hh;              // [s][x][y][c]
  float* fields;           // [shell][N^3], shell index s0 + s
  __nv_bfloat16* split;    // optional chunk-major hi / lo split of split_shells shells
  int split_shells;
  int split_to;            // the split is written for shells s0 + s < split_to only
  const float2* tw;        // [N] e^{+2 pi i k / N}
};

// The two stages of a compiled length.
template <int N>
struct Len {
  static constexpr int RA = plan_radix(N, 0), M = N / RA;  // M = RB: butterflies of stage A
  static constexpr int RB = M;
  static constexpr int R2 = plan_radix(N, 1), R3 = plan_radix(N, 2) ? plan_radix(N, 2) : 1;
  static_assert(plan_np(N) == 2 || plan_np(N) == 3, "two or three radices");
  static_assert(RA * R2 * R3 == N && R2 * R3 == RB, "the plan's radices");
  // stage B's twiddles: [(r - 1) RA + k] of R2, then [((r - 1) R2 + r2) RA + k] of R3
  static constexpr int TW2 = (R2 - 1) * RA, TW = TW2 + (R3 - 1) * R2 * RA;
};

// Exchange buffer of a line: RB x (RA + 1) values, the line pitch such that a half warp's
// lines fall on different banks (lines fastest: an odd multiple of 16 / L apart; else of 8).
template <int N, int L, bool kLineFast>
constexpr int line_pitch() {
  const int want = kLineFast ? 16 / L : 8;
  int p = Len<N>::RB * (Len<N>::RA + 1);
  while (p % (2 * want) != want) ++p;
  return p;
}

// Twiddle table of stage B, filled by the whole block.
template <int N>
__device__ __forceinline__ void fill_twiddles(float2* t, const float2* __restrict__ tw) {
  using P = Len<N>;
  for (int i = threadIdx.x; i < P::TW; i += blockDim.x) {
    int e;
    if (i < P::TW2) {
      e = (i / P::RA + 1) * (i % P::RA) * P::R3;
    } else {
      const int q = i - P::TW2, k = q % P::RA, r2 = q / P::RA % P::R2, r = q / (P::RA * P::R2) + 1;
      e = r * (k + P::RA * r2);
    }
    t[i] = tw[e];
  }
}

// L lines: load(line, j, v) -> v[r] = input j + RB r of the line for every r; store(on, line, k,
// v): outputs k + RA q in v[q], of no line unless `on`; mid() runs between the stages, when every
// input has been read.  Each lane's butterflies are numbered with the line fastest or slowest
// (the layout of the global arrays decides which coalesces).
template <int N, int L, bool kLineFast, class Load, class Mid, class Store>
__device__ __forceinline__ void warp_fft(float2* __restrict__ buf, const float2* __restrict__ tw,
                                         const FftPlan& pl, Load load, Mid mid, Store store) {
  using P = Len<N>;
  constexpr int LP = line_pitch<N, L, kLineFast>();
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int t = lane; t < L * P::M; t += 32) {
    const int line = kLineFast ? t % L : t / P::M, j = kLineFast ? t / L : t % P::M;
    float2 v[P::RA];
    load(line, j, v);
    dft_radix<P::RA>(v, pl);
    float2* o = buf + line * LP + j * (P::RA + 1);
#pragma unroll
    for (int r = 0; r < P::RA; ++r) o[r] = v[r];
  }
  __syncwarp();
  mid();
  constexpr int rounds = (L * P::RA + 31) / 32;
#pragma unroll 1
  for (int i = 0; i < rounds; ++i) {
    const int t = lane + 32 * i;
    const bool on = (L * P::RA) % 32 == 0 || t < L * P::RA;
    const int line = kLineFast ? t % L : t / P::RA, k = kLineFast ? t / L : t % P::RA;
    float2 v[P::RB];
    if (on) {
      const float2* in = buf + line * LP + k;
      if constexpr (P::R3 == 1) {
#pragma unroll
        for (int m = 0; m < P::RB; ++m) v[m] = in[m * (P::RA + 1)];
#pragma unroll
        for (int m = 1; m < P::RB; ++m) v[m] = cmul(v[m], tw[(m - 1) * P::RA + k]);
        dft_radix<P::RB>(v, pl);
      } else {
        float2 y[P::R3][P::R2];
#pragma unroll
        for (int c = 0; c < P::R3; ++c) {
          float2 u[P::R2];
#pragma unroll
          for (int r = 0; r < P::R2; ++r) u[r] = in[(c + P::R3 * r) * (P::RA + 1)];
#pragma unroll
          for (int r = 1; r < P::R2; ++r) u[r] = cmul(u[r], tw[(r - 1) * P::RA + k]);
          dft_radix<P::R2>(u, pl);
#pragma unroll
          for (int r = 0; r < P::R2; ++r) y[c][r] = u[r];
        }
#pragma unroll
        for (int r2 = 0; r2 < P::R2; ++r2) {
          float2 u[P::R3];
#pragma unroll
          for (int c = 0; c < P::R3; ++c)
            u[c] = c ? cmul(y[c][r2], tw[P::TW2 + ((c - 1) * P::R2 + r2) * P::RA + k]) : y[c][r2];
          dft_radix<P::R3>(u, pl);
#pragma unroll
          for (int q = 0; q < P::R3; ++q) v[r2 + P::R2 * q] = u[q];
        }
      }
    }
    store(on, line, k, v);
  }
  __syncwarp();  // the next unit's stage A rewrites the buffer
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

constexpr int kWarps = 4;                      // warps a block
constexpr int kStagePad = 8;                   // staged rows of the Z pass fall on both bank halves
template <int N>
constexpr int lines_xy() { return N <= 192 ? 8 : 4; }  // 64- or 32-byte runs of q_c
template <int N>
constexpr int lines_z() { return N <= 64 ? 8 : N > 400 ? 2 : 4; }
template <int N>
constexpr int min_blocks() { return Len<N>::RB > 25 ? 3 : 4; }  // 168 or 128 registers
template <int N, int L, bool kLineFast>
constexpr size_t pass_smem() {
  return ((size_t)kWarps * L * line_pitch<N, L, kLineFast>() + Len<N>::TW + 1) / 2 * 2 * sizeof(float2);
}

// X pass: unit = L columns q_c of (shell, q_b); the masked spectrum along q_a (the shell's modes
// on the column are the |q_a| in one interval) -> G[s][x][bk][c].
template <int N>
__global__ void __launch_bounds__(32 * kWarps, min_blocks<N>())
    x_kernel(SynthArgs A, FftPlan pl, int runs, int units) {
  extern __shared__ float2 sm[];
  constexpr int L = lines_xy<N>();
  constexpr int LP = line_pitch<N, L, true>();
  float2* tw = sm + kWarps * L * LP;
  pdl_trigger();
  fill_twiddles<N>(tw, A.tw);  // written with the workspace, long before
  __syncthreads();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* buf = sm + warp * L * LP;
  const int nk = A.nk;
  for (int u = blockIdx.x * kWarps + warp; u < units; u += gridDim.x * kWarps) {
    const int run = u % runs, v = u / runs, bk = v % nk, s = v / nk;
    const int b = kept_index(bk, nk, A.R, N);
    const int c = run * L + lane % L;  // this lane's column in both stages (32 is a multiple of L)
    const int ab = b <= N / 2 ? b : N - b, R = A.radius[A.s0 + s];
    if (ab > R || run * L > R) continue;  // the Y pass does not read it
    uint32_t rg = kEmptyRange;
    if (c <= R) rg = A.range[((int64_t)(A.s0 + s) * A.q1 + ab) * A.q1 + c];
    const int a0 = (int)(rg & 0xFFFF), a1 = (int)(rg >> 16);
    float2* g = A.G + (((int64_t)s * N) * nk + bk) * A.Cp + c;
    const int64_t xs = (int64_t)nk * A.Cp;
    if (!__any_sync(0xffffffffu, a0 <= a1)) {  // outside the shell's disc: zeros
      for (int x = lane / L; x < N; x += 32 / L) g[x * xs] = make_float2(0.f, 0.f);
      continue;
    }
    const float2* spec = A.spec + (int64_t)b * A.H + c;
    warp_fft<N, L, true>(
        buf, tw, pl,
        [&](int, int j, float2* in) {
#pragma unroll
          for (int r = 0; r < Len<N>::RA; ++r) {
            const int q = j + r * Len<N>::M, aq = 2 * r < Len<N>::RA ? q : N - q;  // |q_a|
            in[r] = aq >= a0 && aq <= a1 ? spec[(int64_t)q * (N * (N / 2 + 1))]
                                         : make_float2(0.f, 0.f);
          }
        },
        [] {},
        [&](bool on, int, int k, const float2* out) {
          if (!on) return;
#pragma unroll
          for (int q = 0; q < Len<N>::RB; ++q) g[(k + Len<N>::RA * q) * xs] = out[q];
        });
  }
}

// Y pass: unit = L columns q_c of (shell, x); G along q_b -> Hh[s][x][y][c].  The unit's kept
// rows (nk runs of 8 L bytes) are copied to shared memory during the previous unit's stage B.
template <int N>
__global__ void __launch_bounds__(32 * kWarps, min_blocks<N>())
    y_kernel(SynthArgs A, FftPlan pl, int runs, int units) {
  extern __shared__ float2 sm[];
  constexpr int L = lines_xy<N>();
  constexpr int LP = line_pitch<N, L, true>();
  float2* tw = sm + kWarps * L * LP;
  pdl_trigger();
  fill_twiddles<N>(tw, A.tw);  // written with the workspace, long before
  __syncthreads();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* buf = sm + warp * L * LP;
  const int nk = A.nk;
  float2* stage = sm + pass_smem<N, L, true>() / sizeof(float2) + warp * L * nk;
  auto fetch = [&](int u) {
    if (u < units) {
      const int run = u % runs, sx = u / runs, R = A.radius[A.s0 + sx / N];
      const float2* src = A.G + (int64_t)sx * nk * A.Cp + run * L;
      // rows |q_b| <= R of the shell (in an array of all N frequencies, q_b < 0 comes last)
      const int lo = nk == N ? 0 : A.R - R, n_rows = run * L > R ? 0 : min(2 * R + 1, nk);
      for (int i = lane; i < n_rows * (L / 2); i += 32) {
        int bk = lo + i / (L / 2);
        const int e = i % (L / 2) * 2;
        if (nk == N && bk > R) bk += N - n_rows;
        cp_async16(stage + bk * L + e, src + bk * A.Cp + e);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(blockIdx.x * kWarps + warp);
  for (int u = blockIdx.x * kWarps + warp; u < units; u += gridDim.x * kWarps) {
    const int run = u % runs, sx = u / runs;  // sx = s N + x
    const int c = run * L + lane % L, R = A.radius[A.s0 + sx / N], RB = A.R;
    if (run * L > R) {  // columns past the shell: the Z pass does not read them
      __syncwarp();
      fetch(u + gridDim.x * kWarps);
      continue;
    }
    float2* h = A.Hh + (int64_t)sx * N * A.Cp + c;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    warp_fft<N, L, true>(
        buf, tw, pl,
        [&](int, int j, float2* in) {
#pragma unroll
          for (int r = 0; r < Len<N>::RA; ++r) {
            // the first half of the inputs are q_b >= 0, the second q_b = q - N < 0
            const int q = j + r * Len<N>::M;
            const bool kept = 2 * r < Len<N>::RA ? q <= R : q >= N - R;
            const int bk = nk == N ? q : 2 * r < Len<N>::RA ? q + RB : q - N + RB;
            in[r] = kept ? stage[bk * L + lane % L] : make_float2(0.f, 0.f);
          }
        },
        [&] { fetch(u + gridDim.x * kWarps); },
        [&](bool on, int, int k, const float2* out) {
          if (!on) return;
#pragma unroll
          for (int q = 0; q < Len<N>::RB; ++q) h[(k + Len<N>::RA * q) * A.Cp] = out[q];
        });
  }
}

// Z pass: unit = L pairs of rows (x, y), (x, y + 1) of a shell, packed as Z1 + i Z2 (the
// Hermitian extension along q_c of each), so that one complex transform gives both real rows.
// Lanes k, k + 1 (even k) hold points z, z + 1 of a line and exchange one value: the even lane
// stores row y's pair, the odd lane row y + 1's: 8-byte field and 4-byte hi / lo stores.
// The unit's 2 L rows are one contiguous block of Hh: it is copied to shared memory with
// cp.async while the previous unit is in stage B, so that stage A, which reads each value twice
// (at q_c and at N - q_c), waits for no load.
template <int N>
__global__ void __launch_bounds__(32 * kWarps, min_blocks<N>())
    z_kernel(SynthArgs A, FftPlan pl, int runs, int units) {
  extern __shared__ float2 sm[];
  constexpr int L = lines_z<N>();
  constexpr int LP = line_pitch<N, L, false>();
  float2* tw = sm + kWarps * L * LP;
  pdl_trigger();
  fill_twiddles<N>(tw, A.tw);  // written with the workspace, long before
  __syncthreads();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* buf = sm + warp * L * LP;
  const int Cp = A.Cp, sp = Cp + kStagePad;
  float2* stage = sm + pass_smem<N, L, false>() / sizeof(float2) + warp * 2 * L * sp;
  auto fetch = [&](int u) {
    if (u < units) {
      // rows y0 .. y0 + 2 L - 1 of (shell, x); a ragged last unit has fewer
      const int run = u % runs, sx = u / runs;
      const int rows = min(2 * L, N - run * 2 * L);
      const float2* src = A.Hh + ((int64_t)sx * N + run * 2 * L) * Cp;
      constexpr int per_row = 32 / (2 * L);  // lanes a row, 16 bytes each
      const int r = lane / per_row, R = A.radius[A.s0 + sx / N];
      if (r < rows)
        for (int c = lane % per_row * 2; c <= R; c += 2 * per_row)
          cp_async16(stage + r * sp + c, src + r * Cp + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(blockIdx.x * kWarps + warp);
  constexpr int64_t K = (int64_t)N * N * N;
  for (int u = blockIdx.x * kWarps + warp; u < units; u += gridDim.x * kWarps) {
    const int run = u % runs, sx = u / runs;
    const int s = sx / N, x = sx - s * N;
    const int y0 = run * 2 * L;  // first of the unit's 2 L rows
    const int cn = min(A.radius[A.s0 + s], N / 2) + 1;  // q_c = 0 .. cn - 1 can be nonzero
    const int sh = A.s0 + s - A.out0;  // shell index in the output arrays
    const bool fp32 = A.s0 + s >= A.fields_from;
    const bool planes = A.split && A.s0 + s < A.split_to;
    float* field = A.fields + (int64_t)sh * K;
    const int64_t row0 = ((int64_t)x * N + y0) * N;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    warp_fft<N, L, false>(
        buf, tw, pl,
        [&](int line, int j, float2* in) {
          const float2* h1 = stage + 2 * line * sp;
          const bool row = (N / 2) % L == 0 || y0 + 2 * line < N;
          float2 z1[Len<N>::RA], z2[Len<N>::RA];
#pragma unroll
          for (int r = 0; r < Len<N>::RA; ++r) {
            // inputs q < N / 2, then N / 2 and the mirror images q_c = N - q
            const int q = j + r * Len<N>::M, c = 2 * r < Len<N>::RA ? q : N - q;
            const bool in_r = c < cn && row;
            z1[r] = in_r ? h1[c] : make_float2(0.f, 0.f);
            z2[r] = in_r ? h1[sp + c] : make_float2(0.f, 0.f);
          }
#pragma unroll
          for (int r = 0; r < Len<N>::RA; ++r) {
            if (2 * r < Len<N>::RA)
              in[r] = make_float2(z1[r].x - z2[r].y, z1[r].y + z2[r].x);   // Z1 + i Z2
            else
              in[r] = make_float2(z1[r].x + z2[r].y, -z1[r].y + z2[r].x);  // conj(Z1) + i conj(Z2)
            if ((r == 0 || 2 * r == Len<N>::RA) && j == 0)                 // q = 0 or N / 2: real
              in[r] = make_float2(z1[r].x, z2[r].x);
          }
        },
        [&] { fetch(u + gridDim.x * kWarps); },
        [&](bool on, int line, int k, const float2* v) {
          const bool odd = k & 1;
          const int y = 2 * line + (odd ? 1 : 0);
          on = on && ((N / 2) % L == 0 || y0 + y < N);
          // point o = z & ~1 of the row at chunk o >> 7; the row's later points are RA q further
          const int64_t o = row0 + (int64_t)y * N + (k & ~1);
          float* fp = field + o;
          const int o127 = (int)(o & 127), cs = 256 * A.split_shells, lo_plane = 128 * A.split_shells;
          __nv_bfloat16* hp = A.split + (o >> 7) * (int64_t)cs + sh * 128;
#pragma unroll
          for (int q = 0; q < Len<N>::RB; ++q) {
            const float got = __shfl_xor_sync(0xffffffffu, odd ? v[q].x : v[q].y, 1);
            const float2 f = odd ? make_float2(got, v[q].y) : make_float2(v[q].x, got);
            if (on && fp32) *reinterpret_cast<float2*>(fp + Len<N>::RA * q) = f;
            if (on && planes) {
              const __nv_bfloat162 hi = __floats2bfloat162_rn(f.x, f.y);
              const float2 fb = __bfloat1622float2(hi);
              const __nv_bfloat162 lo = __floats2bfloat162_rn(f.x - fb.x, f.y - fb.y);
              // rows of a multiple of 128 points start a chunk: which one z is in is a constant
              const int e = N % 128 == 0 && 128 % Len<N>::RA == 0
                                ? (Len<N>::RA * q >> 7) * cs + (Len<N>::RA * q & 127) + o127
                                : (o127 + Len<N>::RA * q >> 7) * cs + (o127 + Len<N>::RA * q & 127);
              *reinterpret_cast<__nv_bfloat162*>(hp + e) = hi;
              *reinterpret_cast<__nv_bfloat162*>(hp + e + lo_plane) = lo;
            }
          }
        });
  }
}

// The three passes of a batch of ns shells (A.ns).
template <int N>
void run_passes(const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  constexpr int LX = lines_xy<N>(), LZ = lines_z<N>();
  const size_t smem[3] = {
      pass_smem<N, LX, true>(),
      pass_smem<N, LX, true>() + (size_t)kWarps * LX * A.nk * sizeof(float2),
      pass_smem<N, LZ, false>() + (size_t)kWarps * 2 * LZ * (A.Cp + kStagePad) * sizeof(float2)};
  int dev = 0, nsm = 0, sm_bytes = 0, reserved = 0;
  BSK_CHECK_CUDA(cudaGetDevice(&dev));
  BSK_REQUIRE(dev < 64, BSK_ERR_UNSUPPORTED, "device ordinal above 63");
  BSK_CHECK_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  BSK_CHECK_CUDA(cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  BSK_CHECK_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
  const void* kern[3] = {(const void*)x_kernel<N>, (const void*)y_kernel<N>,
                         (const void*)z_kernel<N>};
  // blocks an SM holds by registers (0: not asked yet)
  static std::atomic<int> by_regs[64][3];
  if (!by_regs[dev][2])
    for (int k = 0; k < 3; ++k) {
      BSK_CHECK_CUDA(cudaFuncSetAttribute(kern[k], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          227 * 1024));
      int n = 0;
      BSK_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern[k], 32 * kWarps, 0));
      by_regs[dev][k] = n;
    }
  // persistent passes: as many blocks as are resident at once
  const auto grid = [&](int k, int units) {
    const int fit = std::min<int>(by_regs[dev][k], sm_bytes / (int)(smem[k] + reserved));
    BSK_REQUIRE(fit > 0, BSK_ERR_STATE, "internal: a synthesis pass does not fit an SM");
    return std::max(1, std::min((units + kWarps - 1) / kWarps, fit * nsm));
  };
  const int runs = (A.R + LX) / LX;  // q_c = 0 .. R
  const int xu = A.ns * A.nk * runs, yu = A.ns * N * runs;
  const int zruns = (N / 2 + LZ - 1) / LZ, zu = A.ns * N * zruns;
  launch_pdl(N <= kPdlSide, x_kernel<N>, grid(0, xu), 32 * kWarps, smem[0], st, A, pl, runs, xu);
  launch_pdl(N <= kPdlSide, y_kernel<N>, grid(1, yu), 32 * kWarps, smem[1], st, A, pl, runs, yu);
  launch_pdl(N <= kPdlSide, z_kernel<N>, grid(2, zu), 32 * kWarps, smem[2], st, A, pl, zruns, zu);
}

// Compiled lengths, spread over translation units; false when N is not one of a unit's.
bool run_compiled_a(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st);
bool run_compiled_b(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st);
bool run_compiled_c(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st);
bool run_compiled_d(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st);
bool run_compiled_e(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st);
bool run_compiled_f(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st);

template <int... Ns>
bool run_one_of(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  return ((N == Ns && (run_passes<Ns>(A, pl, st), true)) || ...);
}

}  // namespace synth
}  // namespace bsk
