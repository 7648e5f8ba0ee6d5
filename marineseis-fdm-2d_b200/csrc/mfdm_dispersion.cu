// Phase-shift dispersion imaging of a receiver gather on the GPU (the
// reference's tools/test.py:50-98, `dispersion_imaging`).
//
// For a gather g[t][x] (nt samples of ntr traces at signed offsets x_r) with
// sampling rate fs:
//   S[k][r] = sum_t g[t][r] exp(-2 pi i k t / nt),   k = 0 .. nt/2   (rfft)
//   P[k][r] = conj(S[k][r]) / |S[k][r]|               (0 where |S| = 0)
//   A[k][j] = | sum_r P[k][r] exp(-i w_k x_r / c_j) | / ntr,
// w_k = 2 pi k fs / nt, c_j = c_min + j dc for c_j <= c_max + dc / 2.
// Both kernels accumulate in FP64 like the reference's numpy code and are bound by
// the FP64 pipe; the call around them by the copies of the gather and the image.
//   spectrum: a direct DFT. The samples t and nt - t share their cosine and sine,
//     so the sums run over their sums and differences, and with even nt the
//     frequencies k and nt/2 - k share their terms up to signs: a quarter of the
//     multiply-adds. A block takes 64 traces x 32 frequencies, a thread 4 x 4,
//     twiddles from a table of the nt roots of unity (index k t mod nt).
//   image: exp(-i w_k x_r / c_j) of 16 consecutive k by recurrence from one
//     sine/cosine pair at the first (two interleaved chains of 8 products, error
//     below 2e-15) instead of one pair per (k, r, j).
// nt 2000, 400 traces, 301 velocities: spectrum 241 us (987 us with a thread per
// trace and frequency and every term), image 197 us (428 us with a sincos per
// term), the call 3.8 -> 0.86 ms with the pool below.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/mfdm.h"
#include "mfdm_kernels.h"

namespace {

constexpr int kMaxTableSmem = 4096;  // roots of unity held in shared memory (64 KB of double2)
constexpr int kDR = 64, kDK = 32;    // traces x frequencies of a spectrum block
constexpr int kDT = 32;              // sample pairs staged at a time
constexpr int kDGroup = (kDR / 4) * (kDK / 4);
constexpr int kDThreads = 2 * kDGroup;  // one group takes the odd samples, one the even
constexpr size_t kDSumSmem = size_t(2) * kDT * kDR * sizeof(double);
static_assert(kDGroup == 128 && kDT % 2 == 0, "spectrum block");

// The nt roots exp(-2 pi i m / nt).
__global__ void roots_kernel(double2* roots, int nt) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= nt) return;
  double sn, cs;
  sincospi(2.0 * double(m) / double(nt), &sn, &cs);
  roots[m] = make_double2(cs, -sn);
}

// S and P. sum/dif[p][r]: g[t] +- g[nt - t] of the staged pairs t = t0 + p. The
// first group sums the odd t, the second the even; with even nt the frequency
// nt/2 - k has the same terms as k with the sign (-1)^t, so a block covers k =
// 0..nt/4 only and gets both from the two groups' sum and difference.
// SMEM: the roots fit shared memory.
template <bool SMEM>
__global__ void __launch_bounds__(kDThreads) spectrum_kernel(const float* __restrict__ g, int nt,
                                                             int ntr, int nk,
                                                             const double2* __restrict__ roots,
                                                             double2* __restrict__ P) {
  extern __shared__ __align__(16) double2 smem[];
  double* const sum = reinterpret_cast<double*>(smem);
  double* const dif = sum + kDT * kDR;
  double2* const tab = smem + kDT * kDR;
  if (SMEM)
    for (int m = threadIdx.x; m < nt; m += kDThreads) tab[m] = roots[m];
  // a warp covers 8 x 4 threads, so that its reads touch few addresses
  const int half = threadIdx.x / kDGroup, warp = threadIdx.x % kDGroup / 32, lane = threadIdx.x % 32;
  const int tr = (warp % 2) * 8 + lane % 8, tk = (warp / 2) * 4 + lane / 8;
  const int r0 = blockIdx.x * kDR, k0 = blockIdx.y * kDK + tk * 4;
  double re[4][4] = {}, im[4][4] = {};  // [k][r]
  int m[4], kq[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    // this group's pairs t = 1 + half, 3 + half, ...: k t mod nt advances by 2k
    const int k = min(k0 + a, nk - 1);
    m[a] = int((long long)k * (1 + half) % nt);
    kq[a] = int(2LL * k % nt);
  }
  const int h = (nt - 1) / 2;  // pairs t = 1..h
  for (int t0 = 1; t0 <= h; t0 += kDT) {
    const int np = min(kDT, h + 1 - t0);
    __syncthreads();
    for (int e = threadIdx.x; e < np * kDR; e += kDThreads) {
      const int p = e / kDR, r = e % kDR;
      double a = 0.0, b = 0.0;
      if (r0 + r < ntr) {
        a = double(__ldg(g + size_t(t0 + p) * ntr + r0 + r));
        b = double(__ldg(g + size_t(nt - t0 - p) * ntr + r0 + r));
      }
      sum[e] = a + b;
      dif[e] = a - b;
    }
    __syncthreads();
    for (int p = half; p < np; p += 2) {
      const double2* sp = reinterpret_cast<const double2*>(sum + p * kDR + tr * 4);
      const double2* dp = reinterpret_cast<const double2*>(dif + p * kDR + tr * 4);
      const double2 s0 = sp[0], s1 = sp[1], d0 = dp[0], d1 = dp[1];
      const double sv[4] = {s0.x, s0.y, s1.x, s1.y}, dv[4] = {d0.x, d0.y, d1.x, d1.y};
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const double2 e = SMEM ? tab[m[a]] : __ldg(roots + m[a]);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          re[a][b] = fma(sv[b], e.x, re[a][b]);
          im[a][b] = fma(dv[b], e.y, im[a][b]);
        }
        m[a] += kq[a];
        if (m[a] >= nt) m[a] -= nt;
      }
    }
  }
  // the two groups exchange their sums; the second goes on with nt/2 - k
  const bool fold = nt % 2 == 0;
  const int me = threadIdx.x % kDGroup;
  for (int q = 0; q < 2; ++q) {
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
        sum[(half * 16 + a * 4 + b) * kDGroup + me] = q ? im[a][b] : re[a][b];
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const double other = sum[((1 - half) * 16 + a * 4 + b) * kDGroup + me];
        double& own = q ? im[a][b] : re[a][b];
        own = half == 0 ? own + other : (q ? other - own : own - other);
      }
  }
  if (half == 1 && !fold) return;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int r = r0 + tr * 4 + b;
      if (k0 + a >= nk || r >= ntr) continue;
      const int k = half == 0 ? k0 + a : nt / 2 - (k0 + a);
      if (half == 1 && k == k0 + a) continue;  // k = nt/4 is its own partner
      // the unpaired samples: t = 0 and, with even nt, t = nt/2. The product with the
      // sine of the root 1 stays: infinite samples make it NaN, and the trace silent
      // at that frequency, as at every other t whose root is 1.
      const double v0 = double(__ldg(g + r));
      double x = re[a][b] + v0, y = fma(v0, -0.0, im[a][b]);
      if (fold) {
        const double v = double(__ldg(g + size_t(nt / 2) * ntr + r));
        x += k % 2 ? -v : v;
        if (k % 2 == 0) y = fma(v, -0.0, y);
      }
      const double mag = sqrt(x * x + y * y);
      P[size_t(k) * ntr + r] = mag > 0.0 ? make_double2(x / mag, -y / mag) : make_double2(0.0, 0.0);
    }
}

// Frequencies a spectrum launch runs over (see spectrum_kernel).
int spectrum_rows(int nt) { return nt % 2 == 0 ? nt / 4 + 1 : nt / 2 + 1; }

constexpr int kIK = 16;       // consecutive frequencies per thread
constexpr int kIJ = 64;       // velocities per block
constexpr int kIS = 4;        // threads that share a velocity's traces
constexpr int kIR = 32;       // traces staged at a time

// A: kIS threads per velocity j and kIK frequencies, each taking every kIS-th
// trace (one thread per velocity leaves an SM four warps, too few to hide the
// sine's and the recurrence's latency: 266 us). Measured at nf 1001, nc 301,
// 400 traces: 197 us, the FP64 pipe 56 % busy.
__global__ void __launch_bounds__(kIJ * kIS) image_kernel(const double2* __restrict__ P,
                                                    const double* __restrict__ x, int ntr, int nf,
                                                    int nc, double dw, double c_min, double dc,
                                                    float* __restrict__ A) {
  __shared__ double2 ps[kIR][kIK];
  __shared__ double2 part[kIK][kIJ];
  __shared__ double xs[kIR];
  const int t = threadIdx.x % kIJ, q4 = threadIdx.x / kIJ;
  const int j = blockIdx.x * kIJ + t, k0 = blockIdx.y * kIK;
  const double c = c_min + double(min(j, nc - 1)) * dc;
  const double s0 = (double(k0) * dw) / c, s1 = dw / c;  // w_k0 / c_j, (w_k+1 - w_k) / c_j
  double re[kIK] = {}, im[kIK] = {};
  for (int rt = 0; rt < ntr; rt += kIR) {
    const int nr = min(kIR, ntr - rt);
    __syncthreads();
    for (int e = threadIdx.x; e < kIR * kIK; e += kIJ * kIS) {
      const int k = e / kIR, r = e % kIR;
      ps[r][k] = r < nr && k0 + k < nf ? P[size_t(k0 + k) * ntr + rt + r] : make_double2(0.0, 0.0);
    }
    if (threadIdx.x < nr) xs[threadIdx.x] = x[rt + threadIdx.x];
    __syncthreads();
    for (int r = q4; r < nr; r += kIS) {
      double2 z0, z1, q, q2;  // exp(-i s x) at k0 and k0 + 1; the steps of one and of two k
      sincos(-s0 * xs[r], &z0.y, &z0.x);
      sincos(-s1 * xs[r], &q.y, &q.x);
      z1 = make_double2(z0.x * q.x - z0.y * q.y, z0.x * q.y + z0.y * q.x);
      q2 = make_double2(q.x * q.x - q.y * q.y, 2.0 * q.x * q.y);
#pragma unroll
      for (int k = 0; k < kIK; k += 2) {
        const double2 p0 = ps[r][k], p1 = ps[r][k + 1];
        re[k] = fma(p0.x, z0.x, fma(-p0.y, z0.y, re[k]));
        im[k] = fma(p0.x, z0.y, fma(p0.y, z0.x, im[k]));
        re[k + 1] = fma(p1.x, z1.x, fma(-p1.y, z1.y, re[k + 1]));
        im[k + 1] = fma(p1.x, z1.y, fma(p1.y, z1.x, im[k + 1]));
        z0 = make_double2(z0.x * q2.x - z0.y * q2.y, z0.x * q2.y + z0.y * q2.x);
        z1 = make_double2(z1.x * q2.x - z1.y * q2.y, z1.x * q2.y + z1.y * q2.x);
      }
    }
  }
  for (int s = 1; s < kIS; ++s) {
    if (q4 == s) {
#pragma unroll
      for (int k = 0; k < kIK; ++k) part[k][t] = make_double2(re[k], im[k]);
    }
    __syncthreads();
    if (q4 == 0) {
#pragma unroll
      for (int k = 0; k < kIK; ++k) {
        re[k] += part[k][t].x;
        im[k] += part[k][t].y;
      }
    }
    __syncthreads();
  }
  if (j >= nc || q4 != 0) return;
#pragma unroll
  for (int k = 0; k < kIK; ++k)
    if (k0 + k < nf)
      A[size_t(k0 + k) * nc + j] = float(sqrt(re[k] * re[k] + im[k] * im[k]) / double(ntr));
}

int err(int code, const char* msg) { return mfdm::set_error(code, msg); }

// Device buffers come from a pool of each device that keeps up to kPoolKeep bytes
// between calls: cudaMalloc and cudaFree of one call's 12 MB took 0.6 ms, on a busy
// host several, against 0.45 ms of kernels (the call 1.5 ms with them, 0.84 without).
// What is above that goes back before the call returns, and the rest when an
// allocation of this library would fail otherwise (device_malloc): the driver does
// not take a pool's idle memory for another allocation by itself. Pools are safe to
// use from several threads.
constexpr unsigned long long kPoolKeep = 64ull << 20;
constexpr int kMaxDevices = 64;
// A pool goes with its context: after cudaDeviceReset the device has another one, of
// another id, and gets another pool (the old handle is dead and not touched).
struct Pool {
  cudaMemPool_t pool = nullptr;
  unsigned long long context = 0;
};
std::mutex g_pool_mutex;
Pool g_pool[kMaxDevices];

// The id, never used twice in a process, of the context current to this thread.
// The driver's calls come through the runtime (no libcuda link), looked up once.
void* driver_call(const char* name) {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  return cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess ? p : nullptr;
}
cudaError_t context_id(unsigned long long* id) {
  typedef CUresult (*GetCurrent)(CUcontext*);
  typedef CUresult (*GetId)(CUcontext, unsigned long long*);
  static const GetCurrent get_current = reinterpret_cast<GetCurrent>(driver_call("cuCtxGetCurrent"));
  static const GetId get_id = reinterpret_cast<GetId>(driver_call("cuCtxGetId"));
  CUcontext c = nullptr;
  if (!get_current || !get_id || get_current(&c) != CUDA_SUCCESS || get_id(c, id) != CUDA_SUCCESS)
    return cudaErrorInitializationError;
  return cudaSuccess;
}

// The pool of `device`, which is current.
cudaError_t pool_of(int device, cudaMemPool_t* pool) {
  if (device >= kMaxDevices) return cudaErrorInvalidDevice;
  unsigned long long id = 0;
  const cudaError_t e0 = context_id(&id);
  if (e0 != cudaSuccess) return e0;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (!g_pool[device].pool || g_pool[device].context != id) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t p = nullptr;
    cudaError_t e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) return e;
    unsigned long long keep = kPoolKeep;
    if ((e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
      cudaMemPoolDestroy(p);
      return e;
    }
    g_pool[device] = {p, id};
  }
  *pool = g_pool[device].pool;
  return cudaSuccess;
}

// Gives the pool's idle memory back to the driver but for `keep` bytes, once the
// frees queued on the default stream have run.
void trim(cudaMemPool_t pool, unsigned long long keep) {
  unsigned long long reserved = 0;
  if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
      reserved > keep && cudaStreamSynchronize(nullptr) == cudaSuccess)
    cudaMemPoolTrimTo(pool, keep);
}

struct DevBuf {
  cudaMemPool_t pool = nullptr;
  void* p = nullptr;
  ~DevBuf() {
    if (!p) return;
    cudaFreeAsync(p, nullptr);
    trim(pool, kPoolKeep);  // every call, so that the last of several at once does
  }
};

}  // namespace

namespace mfdm {
cudaError_t device_malloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  int device = 0;
  unsigned long long id = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device >= kMaxDevices || context_id(&id) != cudaSuccess)
    return e;
  {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (!g_pool[device].pool || g_pool[device].context != id) return e;
    trim(g_pool[device].pool, 0);
  }
  (void)cudaGetLastError();
  return cudaMalloc(p, bytes);
}
}  // namespace mfdm

extern "C" int mfdm_dispersion_velocities(double c_min, double c_max, double dc) {
  if (!(c_min > 0.0) || !(c_max >= c_min) || !(dc > 0.0) || !std::isfinite(c_max)) return 0;
  // numpy.arange(c_min, c_max + dc / 2, dc): ceil((stop - start) / step) values
  return int(std::ceil((c_max + dc / 2.0 - c_min) / dc));
}

extern "C" int mfdm_dispersion_image(const float* gather, int nt, int ntr, const double* offsets,
                                     double fs, double c_min, double c_max, double dc,
                                     float* amplitude, int device) {
  if (!gather || !offsets || !amplitude) return err(MFDM_ERR_ARG, "null argument");
  if (nt < 2 || ntr < 1) return err(MFDM_ERR_ARG, "need at least two samples and one trace");
  if (!(fs > 0.0) || !std::isfinite(fs)) return err(MFDM_ERR_ARG, "fs must be a positive finite value");
  const int nc = mfdm_dispersion_velocities(c_min, c_max, dc);
  if (nc <= 0) return err(MFDM_ERR_ARG, "velocities must satisfy 0 < c_min <= c_max and dc > 0");
  for (int r = 0; r < ntr; ++r)
    if (!std::isfinite(offsets[r])) return err(MFDM_ERR_ARG, "all offsets must be finite");
  const int nf = nt / 2 + 1;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
    return err(MFDM_ERR_ARG, "no such CUDA device");
  int prev = 0;
  cudaGetDevice(&prev);
  struct Restore {
    int d;
    ~Restore() { cudaSetDevice(d); }
  } restore{prev};
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return err(MFDM_ERR_CUDA, cudaGetErrorString(e));
  const int nk = spectrum_rows(nt), ktiles = (nk + kDK - 1) / kDK, kblocks = (nf + kIK - 1) / kIK;
  if (ktiles > 65535 || kblocks > 65535) return err(MFDM_ERR_ARG, "too many samples");
  // one allocation: gather, offsets, roots, phase spectrum, image
  auto up = [](size_t n) { return (n + 255) / 256 * 256; };
  const size_t gb = size_t(nt) * ntr * sizeof(float), rb = size_t(nt) * sizeof(double2),
               xb = size_t(ntr) * sizeof(double), pb = size_t(nf) * ntr * sizeof(double2),
               ab = size_t(nf) * nc * sizeof(float);
  DevBuf d;
  if ((e = pool_of(device, &d.pool)) != cudaSuccess) return err(MFDM_ERR_CUDA, cudaGetErrorString(e));
  const size_t bytes = up(gb) + up(xb) + up(rb) + up(pb) + ab;
  e = cudaMallocFromPoolAsync(&d.p, bytes, d.pool, nullptr);
  if (e == cudaErrorMemoryAllocation) {  // not while idle blocks of other sizes stay reserved
    (void)cudaGetLastError();
    trim(d.pool, 0);
    e = cudaMallocFromPoolAsync(&d.p, bytes, d.pool, nullptr);
  }
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return err(MFDM_ERR_NOMEM, cudaGetErrorString(e));
  }
  char* p = static_cast<char*>(d.p);
  float* const dg = reinterpret_cast<float*>(p);
  double* const dx = reinterpret_cast<double*>(p += up(gb));
  double2* const dr = reinterpret_cast<double2*>(p += up(xb));
  double2* const dP = reinterpret_cast<double2*>(p += up(rb));
  float* const dA = reinterpret_cast<float*>(p += up(pb));
  roots_kernel<<<unsigned((nt + 255) / 256), 256>>>(dr, nt);
  if ((e = cudaMemcpy(dg, gather, gb, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(dx, offsets, xb, cudaMemcpyHostToDevice)) != cudaSuccess)
    return err(MFDM_ERR_CUDA, cudaGetErrorString(e));
  const bool in_smem = nt <= kMaxTableSmem;
  const size_t smem = (in_smem ? rb : 0) + kDSumSmem;
  const dim3 grid(unsigned((ntr + kDR - 1) / kDR), unsigned(ktiles));
  if (in_smem) {
    // the limit is the kernel's, not the call's: every call sets it to the most any
    // call needs, so that none lowers it between another thread's setting and launch
    if ((e = cudaFuncSetAttribute(spectrum_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(kMaxTableSmem * sizeof(double2) + kDSumSmem))) != cudaSuccess)
      return err(MFDM_ERR_CUDA, cudaGetErrorString(e));
    spectrum_kernel<true><<<grid, kDThreads, smem>>>(dg, nt, ntr, nk, dr, dP);
  } else {
    spectrum_kernel<false><<<grid, kDThreads, smem>>>(dg, nt, ntr, nk, dr, dP);
  }
  const double dw = 2.0 * M_PI * fs / double(nt);
  image_kernel<<<dim3(unsigned((nc + kIJ - 1) / kIJ), unsigned(kblocks)), kIJ * kIS>>>(dP, dx, ntr, nf, nc,
                                                                               dw, c_min, dc, dA);
  if ((e = cudaGetLastError()) != cudaSuccess) return err(MFDM_ERR_CUDA, cudaGetErrorString(e));
  if ((e = cudaMemcpy(amplitude, dA, ab, cudaMemcpyDeviceToHost)) != cudaSuccess)
    return err(MFDM_ERR_CUDA, cudaGetErrorString(e));
  return MFDM_OK;
}
