// Shell-field synthesis: I_s(x) = c2r[ dhat_k 1{k in shell s} ] for a batch of shells,
// as three pruned passes of length-Ng inverse FFTs written for this problem.
//
// A shell of radius r occupies |q_a|, |q_b|, q_c <= r of the half spectrum, so:
//   X pass: for every column (q_b, q_c) with |q_b|, q_c <= r, the masked spectrum along
//           q_a (only |q_a| <= r nonzero) -> G[s][x][q_b][q_c]   (reads the slot spectrum
//           and the shell table once for all shells of the batch);
//   Y pass: for every (x, q_c <= r), G along q_b -> Hh[s][x][y][q_c];
//   Z pass: for every two rows (x, y), (x, y+1), the Hermitian-extended sequences along
//           q_c packed as Z1 + i Z2 -> one complex inverse FFT whose real and imaginary
//           parts are the two real output rows; the rows are written as FP32 fields and,
//           when asked, as the bf16 hi / lo planes of the tensor-core contraction.
// Every array keeps q_c fastest, so the passes read and write 8- or 16-wide (64- or 128-byte)
// runs of it.
// The FFTs are radix-16/24/12/8/6/4/2/3/5 Stockham passes in shared memory (twiddles from a
// table computed in double precision on the host); unnormalised, sign +1, as cuFFT's C2R.
// Lengths of two or three radices are compiled (bsk_synth_warp.cuh); this file has the same
// passes for the other lengths, with the radix plan at run time.
#include "bsk_synth_warp.cuh"

namespace bsk {
namespace synth {
namespace {

constexpr int kLines = 16;   // lines (one 16-wide q_c run) per block of the Y pass
constexpr int kXLines = 8;   // X pass: half a q_c run per block (its staged spectrum columns
                             // need shared memory too; 8 lines let three blocks share an SM)
constexpr int kZLines = 16;  // lines (two output rows each) per block of the Z pass
constexpr int kThreads = 256;

__device__ __forceinline__ bool in_shell(uint16_t code, int s) {
  const int first = code & 0xFF;
  const int cnt = (code >> 8) + 1;
  return first != 0xFF && s >= first && s < first + cnt;
}

// Lines are kept in shared memory with a stride of n + 1 complex values, and consecutive
// threads take the same butterfly of consecutive lines: both keep the Stockham reads and
// writes of a warp on distinct banks.
__host__ __device__ constexpr int line_stride(int n) { return n + 1; }

// One Stockham pass of radix R over `lines` sequences of length n (src -> dst).  Input
// positions zlo .. zhi are known to be zero: they are neither read nor need to be written
// (the first pass of a pruned transform, whose inputs outside the kept frequencies are zero).
template <int R>
__device__ __forceinline__ void fft_pass(const float2* __restrict__ src, float2* __restrict__ dst,
                                         int lines, int n, int Ns, const float2* __restrict__ tw,
                                         const FftPlan& pl, int zlo = 1 << 30, int zhi = -1) {
  const int m = n / R;
  const int step = n / (Ns * R);
  const int ls = line_stride(n);
  for (int t = threadIdx.x; t < lines * m; t += blockDim.x) {
    const int j = t / lines;
    const int line = t - j * lines;
    const int k = j % Ns;
    const float2* in = src + line * ls;
    float2* o = dst + line * ls;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = j + r * m;
      v[r] = (q >= zlo && q <= zhi) ? make_float2(0.f, 0.f) : in[q];
    }
    if (Ns > 1) {  // the first pass has k = 0: unit twiddles
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw[r * k * step]);
    }
    dft_radix<R>(v, pl);
    const int idx = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) o[idx + r * Ns] = v[r];
  }
}

// Inverse FFT (sign +1, unnormalised) of L sequences of length n stored with line
// stride n + 1 in `a`; `b` is scratch of the same size.  Returns the buffer holding the
// result.
template <int L>
__device__ float2* fft_lines(float2* a, float2* b, const FftPlan& pl,
                             const float2* __restrict__ tw, int zlo = 1 << 30, int zhi = -1) {
  float2* src = a;
  float2* dst = b;
  {
    const int n = pl.n;
    int Ns = 1;
    for (int p = 0; p < pl.np; ++p) {
      const int R = pl.radix[p];
      const int zl = p == 0 ? zlo : 1 << 30, zh = p == 0 ? zhi : -1;
      switch (R) {
        case 16: fft_pass<16>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 24: fft_pass<24>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 12: fft_pass<12>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 6: fft_pass<6>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 8: fft_pass<8>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 4: fft_pass<4>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 2: fft_pass<2>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        case 3: fft_pass<3>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
        default: fft_pass<5>(src, dst, L, n, Ns, tw, pl, zl, zh); break;
      }
      __syncthreads();
      float2* t2 = src;
      src = dst;
      dst = t2;
      Ns *= R;
    }
  }
  return src;
}

// X pass: block (bk, c-run).  Spectrum and table columns are read once for all shells.
__global__ void __launch_bounds__(kThreads) synth_x_kernel(SynthArgs A, FftPlan pl) {
  extern __shared__ float2 sm[];
  const int N = A.N, nk = A.nk;
  const int ls = line_stride(N);
  float2* buf0 = sm;                       // kXLines lines
  float2* buf1 = buf0 + kXLines * ls;       // kXLines lines
  float2* tw = buf1 + kXLines * ls;         // N
  float2* sS = tw + N;                     // nk * kXLines
  uint16_t* sT = reinterpret_cast<uint16_t*>(sS + nk * kXLines);  // nk * kXLines
  const int bk = blockIdx.x;
  const int c0 = blockIdx.y * kXLines;
  const int b = kept_index(bk, nk, A.R, N);
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = A.tw[i];
  for (int i = threadIdx.x; i < nk * kXLines; i += blockDim.x) {
    const int ak = i / kXLines, l = i - ak * kXLines;
    const int a = kept_index(ak, nk, A.R, N);
    const int c = c0 + l;
    float2 v = make_float2(0.f, 0.f);
    uint16_t code = 0xFF;
    if (c < A.H && c <= A.R) {
      const int64_t m = ((int64_t)a * N + b) * A.H + c;
      v = A.spec[m];
      code = A.table[m];
    }
    sS[i] = v;
    sT[i] = code;
  }
  __syncthreads();
  // positions R + 1 .. N - R - 1 of a line (|q_a| > R) are zero: not written, not read
  const int zlo = nk == N ? 1 << 30 : A.R + 1, zhi = nk == N ? -1 : N - A.R - 1;
  for (int s = 0; s < A.ns; ++s) {
    for (int i = threadIdx.x; i < kXLines * nk; i += blockDim.x) {
      const int ak = i / kXLines, l = i - ak * kXLines;
      // kept frequency ak sits at position a of line l (frequency index a)
      const int a = kept_index(ak, nk, A.R, N);
      const float2 v = in_shell(sT[ak * kXLines + l], A.s0 + s) ? sS[ak * kXLines + l]
                                                                 : make_float2(0.f, 0.f);
      buf0[l * ls + a] = v;
    }
    __syncthreads();
    const float2* res = fft_lines<kXLines>(buf0, buf1, pl, tw, zlo, zhi);
    // G[s][x][bk][c0 + l]
    float2* g = A.G + (((int64_t)s * N) * nk + bk) * A.Cp + c0;
    for (int i = threadIdx.x; i < kXLines * N; i += blockDim.x) {
      const int x = i / kXLines, l = i - x * kXLines;
      g[(int64_t)x * nk * A.Cp + l] = res[l * ls + x];
    }
    __syncthreads();
  }
}

// The Y and Z passes are persistent: a block walks units (u, u + gridDim.x, ...) and,
// while the FFT of one unit runs, the global loads of its share of the next unit's input
// are already in flight into registers (kYPf / kZPf values per thread; inputs beyond
// that, only possible for the largest shells, are read when the unit starts).
constexpr int kYPf = 16;  // Y pass: kYPf * kThreads / kLines kept q_b per line
constexpr int kZPf = 8;   // Z pass: kZPf * kThreads / kZLines nonzero q_c per line

// Y pass: unit (x, c-run, shell).
__global__ void __launch_bounds__(kThreads, 2) synth_y_kernel(SynthArgs A, FftPlan pl, int units) {
  extern __shared__ float2 sm[];
  const int N = A.N, nk = A.nk;
  const int ls = line_stride(N);
  float2* buf0 = sm;
  float2* buf1 = buf0 + kLines * ls;
  float2* tw = buf1 + kLines * ls;
  const int nrun = A.Cp / kLines;
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = A.tw[i];
  // thread's inputs: i = threadIdx.x + k kThreads -> (bk = i / kLines, l = i % kLines)
  float2 pre[kYPf];
  auto src = [&](int u) {
    const int s = u / (N * nrun), r = u - s * (N * nrun);
    const int x = r / nrun, c0 = (r - x * nrun) * kLines;
    return A.G + (((int64_t)s * N + x) * nk) * A.Cp + c0;
  };
  auto fetch = [&](int u) {
    const float2* g = src(u);
#pragma unroll
    for (int k = 0; k < kYPf; ++k) {
      const int i = threadIdx.x + k * kThreads;
      const int bk = i / kLines, l = i - bk * kLines;
      pre[k] = bk < nk ? g[(int64_t)bk * A.Cp + l] : make_float2(0.f, 0.f);
    }
  };
  int u = blockIdx.x;
  if (u < units) fetch(u);
  for (; u < units; u += gridDim.x) {
    const float2* g = src(u);
    // kept frequencies (|q_b| <= R, or all) from the prefetch, the rest of the line zero
#pragma unroll
    for (int k = 0; k < kYPf; ++k) {
      const int i = threadIdx.x + k * kThreads;
      const int bk = i / kLines, l = i - bk * kLines;
      if (bk < nk) buf0[l * ls + kept_index(bk, nk, A.R, N)] = pre[k];
    }
    for (int i = threadIdx.x + kYPf * kThreads; i < nk * kLines; i += kThreads) {
      const int bk = i / kLines, l = i - bk * kLines;
      buf0[l * ls + kept_index(bk, nk, A.R, N)] = g[(int64_t)bk * A.Cp + l];
    }
    // positions R + 1 .. N - R - 1 (|q_b| > R) are zero: not written, not read
    __syncthreads();
    if (u + (int)gridDim.x < units) fetch(u + gridDim.x);
    const float2* res = nk < N ? fft_lines<kLines>(buf0, buf1, pl, tw, A.R + 1, N - A.R - 1)
                               : fft_lines<kLines>(buf0, buf1, pl, tw);
    const int s = u / (N * nrun), r = u - s * (N * nrun);
    const int x = r / nrun, c0 = (r - x * nrun) * kLines;
    float2* h = A.Hh + (((int64_t)s * N + x) * N) * A.Cp + c0;
    for (int i = threadIdx.x; i < kLines * N; i += kThreads) {
      const int y = i / kLines, l = i - y * kLines;
      h[(int64_t)y * A.Cp + l] = res[l * ls + y];
    }
    __syncthreads();
  }
}

// Z pass: unit (x, run of 2 kZLines rows y, shell).  Line l packs rows y0 + 2l, y0 + 2l + 1.
__global__ void __launch_bounds__(kThreads, 2) synth_z_kernel(SynthArgs A, FftPlan pl, int units) {
  extern __shared__ float2 sm[];
  const int N = A.N;
  const int ls = line_stride(N);
  float2* buf0 = sm;
  float2* buf1 = buf0 + kZLines * ls;
  float2* tw = buf1 + kZLines * ls;
  const int ny = (N + 2 * kZLines - 1) / (2 * kZLines);
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = A.tw[i];
  const int cn = min(A.R, N / 2) + 1;  // q_c = 0 .. cn - 1 can be nonzero
  // kThreads / kZLines threads per line, q_c strided by that
  constexpr int tpl = kThreads / kZLines;
  const int l = threadIdx.x / tpl, cl = threadIdx.x % tpl;
  float2 p1[kZPf], p2[kZPf];
  auto fetch = [&](int u) {
    const int s = u / (N * ny), r = u - s * (N * ny);
    const int x = r / ny, y1 = (r - x * ny) * 2 * kZLines + 2 * l;
    const float2* h = A.Hh + (((int64_t)s * N + x) * N + y1) * A.Cp;
#pragma unroll
    for (int k = 0; k < kZPf; ++k) {
      const int c = cl + k * tpl;
      p1[k] = (y1 < N && c < cn) ? h[c] : make_float2(0.f, 0.f);
      p2[k] = (y1 + 1 < N && c < cn) ? h[A.Cp + c] : make_float2(0.f, 0.f);
    }
  };
  // line value at q_c = c and its Hermitian partner at N - c
  auto put = [&](float2* line, int c, float2 z1, float2 z2) {
    if (c == 0 || 2 * c == N) {
      line[c] = make_float2(z1.x, z2.x);
    } else {
      line[c] = make_float2(z1.x - z2.y, z1.y + z2.x);       // Z1 + i Z2
      line[N - c] = make_float2(z1.x + z2.y, -z1.y + z2.x);  // conj(Z1) + i conj(Z2)
    }
  };
  int u = blockIdx.x;
  if (u < units) fetch(u);
  for (; u < units; u += gridDim.x) {
    const int s = u / (N * ny), r = u - s * (N * ny);
    const int x = r / ny, y0 = (r - x * ny) * 2 * kZLines;
    const int y1 = y0 + 2 * l;
    float2* line = buf0 + l * ls;
#pragma unroll
    for (int k = 0; k < kZPf; ++k) {
      const int c = cl + k * tpl;
      if (c < cn) put(line, c, p1[k], p2[k]);
    }
    if (cn > kZPf * tpl) {
      const float2* h = A.Hh + (((int64_t)s * N + x) * N + y1) * A.Cp;
      for (int c = cl + kZPf * tpl; c < cn; c += tpl) {
        const float2 z1 = y1 < N ? h[c] : make_float2(0.f, 0.f);
        const float2 z2 = y1 + 1 < N ? h[A.Cp + c] : make_float2(0.f, 0.f);
        put(line, c, z1, z2);
      }
    }
    // positions cn .. N - cn (|q_c| >= cn) are zero: not written, not read
    __syncthreads();
    if (u + (int)gridDim.x < units) fetch(u + gridDim.x);
    const int64_t K = (int64_t)N * N * N;
    const int sh = A.s0 + s - A.out0;  // shell index in the output arrays
    const int64_t row0 = ((int64_t)x * N) * N;
    {
      const float2* res = fft_lines<kZLines>(buf0, buf1, pl, tw, cn, N - cn);
      // four consecutive z per thread: 16-byte field stores, 8-byte hi / lo stores (N % 4 == 0)
      const int nq = N / 4;
      for (int i = threadIdx.x; i < 2 * kZLines * nq; i += kThreads) {
        const int rr = i / nq, z = (i - rr * nq) * 4;  // output row y0 + rr
        const int y = y0 + rr;
        if (y >= N) continue;
        const float2* w = res + (rr >> 1) * ls + z;
        float4 v;
        if (rr & 1) v = make_float4(w[0].y, w[1].y, w[2].y, w[3].y);
        else v = make_float4(w[0].x, w[1].x, w[2].x, w[3].x);
        const int64_t pt = row0 + (int64_t)y * N + z;
        if (A.s0 + s >= A.fields_from)
          *reinterpret_cast<float4*>(A.fields + (int64_t)sh * K + pt) = v;
        if (A.split && A.s0 + s < A.split_to) {
          const __nv_bfloat162 h01 = __floats2bfloat162_rn(v.x, v.y);
          const __nv_bfloat162 h23 = __floats2bfloat162_rn(v.z, v.w);
          const float2 f01 = __bfloat1622float2(h01), f23 = __bfloat1622float2(h23);
          const __nv_bfloat162 l01 = __floats2bfloat162_rn(v.x - f01.x, v.y - f01.y);
          const __nv_bfloat162 l23 = __floats2bfloat162_rn(v.z - f23.x, v.w - f23.y);
          uint2 hv, lv;
          hv.x = *reinterpret_cast<const uint32_t*>(&h01);
          hv.y = *reinterpret_cast<const uint32_t*>(&h23);
          lv.x = *reinterpret_cast<const uint32_t*>(&l01);
          lv.y = *reinterpret_cast<const uint32_t*>(&l23);
          *reinterpret_cast<uint2*>(A.split + split_index(0, sh, pt, A.split_shells)) = hv;
          *reinterpret_cast<uint2*>(A.split + split_index(1, sh, pt, A.split_shells)) = lv;
        }
      }
    }
    __syncthreads();
  }
}

void run_synth(const SynthArgs& A, const FftPlan& pl, int nk, int Cp, int ns, cudaStream_t st) {
  const int N = A.N;
  const size_t fft_smem = (2 * (size_t)kLines * (N + 1) + N) * sizeof(float2);
  const size_t x_smem = (2 * (size_t)kXLines * (N + 1) + N) * sizeof(float2) +
                        (size_t)nk * kXLines * (sizeof(float2) + sizeof(uint16_t));
  BSK_REQUIRE(x_smem <= 227 * 1024, BSK_ERR_UNSUPPORTED, "grid too large for the field synthesis");
  static std::atomic<bool> attr_done[64];  // zero-initialised: false
  int dev = 0;
  BSK_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && !attr_done[dev]) {
    const int maxs = 227 * 1024;
    BSK_CHECK_CUDA(cudaFuncSetAttribute(synth_x_kernel,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, maxs));
    BSK_CHECK_CUDA(cudaFuncSetAttribute(synth_y_kernel,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, maxs));
    BSK_CHECK_CUDA(cudaFuncSetAttribute(synth_z_kernel,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, maxs));
    attr_done[dev] = true;
  }
  synth_x_kernel<<<dim3(nk, Cp / kXLines), kThreads, x_smem, st>>>(A, pl);
  BSK_CHECK_CUDA(cudaGetLastError());
  // persistent Y and Z passes: as many blocks as are resident at once
  int nsm = 0, by = 0, bz = 0;
  BSK_CHECK_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const size_t z_smem = (2 * (size_t)kZLines * (N + 1) + N) * sizeof(float2);
  BSK_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&by, synth_y_kernel, kThreads,
                                                               fft_smem));
  BSK_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bz, synth_z_kernel, kThreads,
                                                               z_smem));
  const int y_units = N * (Cp / kLines) * ns;
  const int z_units = N * ((N + 2 * kZLines - 1) / (2 * kZLines)) * ns;
  const int y_grid = std::max(1, std::min(y_units, std::max(by, 1) * nsm));
  const int z_grid = std::max(1, std::min(z_units, std::max(bz, 1) * nsm));
  synth_y_kernel<<<y_grid, kThreads, fft_smem, st>>>(A, pl, y_units);
  BSK_CHECK_CUDA(cudaGetLastError());
  synth_z_kernel<<<z_grid, kThreads, z_smem, st>>>(A, pl, z_units);
  BSK_CHECK_CUDA(cudaGetLastError());
}

bool make_plan(int n, FftPlan& pl) {
  pl.n = n;
  pl.np = plan_np(n);
  if (pl.np <= 0 || pl.np > 8) return false;
  int rc = 0;
  for (int p = 0; p < pl.np; ++p) {
    pl.radix[p] = plan_radix(n, p);
    if (pl.radix[p] == 24 || pl.radix[p] == 12 || pl.radix[p] == 6) rc = pl.radix[p];
  }
  for (int k = 0; k < 3; ++k)
    pl.root3[k] = make_float2((float)std::cos(2 * M_PI * k / 3), (float)std::sin(2 * M_PI * k / 3));
  for (int k = 0; k < 5; ++k)
    pl.root5[k] = make_float2((float)std::cos(2 * M_PI * k / 5), (float)std::sin(2 * M_PI * k / 5));
  for (int k = 0; k < 24; ++k)
    pl.rootc[k] = rc ? make_float2((float)std::cos(2 * M_PI * k / rc), (float)std::sin(2 * M_PI * k / rc))
                     : make_float2(1.f, 0.f);
  return true;
}

bool run_compiled(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  return run_compiled_a(N, A, pl, st) || run_compiled_b(N, A, pl, st) ||
         run_compiled_c(N, A, pl, st) || run_compiled_d(N, A, pl, st) ||
         run_compiled_e(N, A, pl, st) || run_compiled_f(N, A, pl, st);
}

}  // namespace
}  // namespace synth

using namespace synth;

// The sides a grid level may have.
bool synth_fast_size(int n) {
  switch (n) {
    case 48: case 96: case 128: case 160: case 192: case 240: case 256: case 288: case 320:
    case 384: case 480:
      return true;
    default:
      return false;
  }
}

bool synth_supported(int n) {
  FftPlan pl;
  return n >= 8 && n <= 512 && n % 4 == 0 && make_plan(n, pl);
}

size_t synth_workspace_bytes(int n, int max_r, int batch) {
  const int nk = std::min(2 * max_r + 1, n);
  const int Cp = (max_r + 1 + kLines - 1) / kLines * kLines;
  return ((size_t)batch * n * nk * Cp + (size_t)batch * n * n * Cp) * sizeof(float2) +
         (size_t)n * sizeof(float2);
}

void synth_init_workspace(int N, void* work) {
  std::vector<float2> htw(N);
  for (int k = 0; k < N; ++k)
    htw[k] = make_float2((float)std::cos(2 * M_PI * k / N), (float)std::sin(2 * M_PI * k / N));
  BSK_CHECK_CUDA(cudaMemcpy(work, htw.data(), N * sizeof(float2), cudaMemcpyHostToDevice));
}

void launch_synth(int N, const cufftComplex* spec, const uint16_t* table, const uint32_t* range,
                  const int* radius, int q1, int s0, int ns, int R, void* work, float* fields,
                  __nv_bfloat16* split, int split_shells, cudaStream_t st, int out_s0,
                  int fields_from, int split_to) {
  FftPlan pl;
  BSK_REQUIRE(make_plan(N, pl), BSK_ERR_UNSUPPORTED, "no FFT plan for this grid size");
  BSK_REQUIRE(fields || s0 + ns <= fields_from, BSK_ERR_STATE,
              "internal: no FP32 fields to write a shell to");
  R = std::min(R, N / 2);
  const int nk = std::min(2 * R + 1, N);
  const int Cp = (R + 1 + kLines - 1) / kLines * kLines;
  SynthArgs A;
  A.N = N;
  A.H = N / 2 + 1;
  A.R = R;
  A.nk = nk;
  A.Cp = Cp;
  A.s0 = s0;
  A.ns = ns;
  A.out0 = out_s0;
  A.fields_from = fields_from;
  A.split_to = split_to;
  A.spec = reinterpret_cast<const float2*>(spec);
  A.table = table;
  A.range = range;
  A.radius = radius;
  A.q1 = q1;
  float2* tw = reinterpret_cast<float2*>(work);
  A.G = tw + N;
  A.Hh = A.G + (size_t)ns * N * nk * Cp;
  A.fields = fields;
  A.split = split;
  A.split_shells = split_shells;
  A.tw = tw;
  if (!run_compiled(N, A, pl, st)) run_synth(A, pl, nk, Cp, ns, st);
}

}  // namespace bsk
