// vibe-model_gb300/csrc/ckern.cu
//
// GPU implementation of the reference's C11 hot-kernel ABI
// (include/vibe/common/c_kernels.h). The host-pointer entry points copy their
// arrays to the device, run the kernel on an internal stream and copy the
// result back; the *_dev entry points work on device pointers on the
// caller's stream. Reductions (CFL max-scan, Neumaier sum) are two-level:
// warp shuffles inside a block, one partial per block in device scratch, and
// a single-block pass that merges the partials in block order, so results are
// deterministic run to run.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

#include "cabi_host.cuh"
#include "vibe_c_kernels.h"
#include "vibe_internal.cuh"

namespace {

thread_local std::string g_cerr;

bool device_ok(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return true;
  g_cerr = std::string(what) + ": " + cudaGetErrorString(e);
  return false;
}

int cur_dev() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}

// ---- per-thread call contexts (cabi_host.cuh) ----------------------------
constexpr int kMaxDev = 64;
std::atomic<unsigned long long> g_allocs{0};

struct Ctx {
  cudaStream_t st = nullptr;
  cudaEvent_t last = nullptr;  // recorded after the last launch that used scr
  bool has_last = false;
  char* pin = nullptr;         // pinned host staging
  size_t pin_n = 0;
  char* dbuf = nullptr;        // device staging of host-pointer calls
  size_t dbuf_n = 0;
  char* scr = nullptr;         // scratch of _dev calls
  size_t scr_n = 0;
};

// One context per (host thread, device); freed when the thread exits (the
// main thread's at process exit, before the CUDA runtime's own teardown).
struct Holder {
  Ctx* c[kMaxDev] = {};
  ~Holder() {
    for (auto*& x : c) {
      if (!x) continue;
      if (x->st) cudaStreamSynchronize(x->st);
      if (x->has_last) cudaEventSynchronize(x->last);
      if (x->pin) cudaFreeHost(x->pin);
      if (x->dbuf) cudaFree(x->dbuf);
      if (x->scr) cudaFree(x->scr);
      if (x->last) cudaEventDestroy(x->last);
      if (x->st) cudaStreamDestroy(x->st);
      delete x;
      x = nullptr;
    }
  }
};
thread_local Holder t_hold;

Ctx* ctx() {
  int d = -1;
  if (!device_ok(cudaGetDevice(&d), "cudaGetDevice")) return nullptr;
  if (d < 0 || d >= kMaxDev) { g_cerr = "device ordinal out of range"; return nullptr; }
  Ctx*& c = t_hold.c[d];
  if (!c) {
    Ctx* n = new Ctx();
    if (!device_ok(cudaStreamCreateWithFlags(&n->st, cudaStreamNonBlocking), "cudaStreamCreate") ||
        !device_ok(cudaEventCreateWithFlags(&n->last, cudaEventDisableTiming), "cudaEventCreate")) {
      if (n->st) cudaStreamDestroy(n->st);
      delete n;
      return nullptr;
    }
    c = n;
  }
  return c;
}

size_t grown(size_t have, size_t need) {
  size_t n = have ? have : (size_t)4096;
  while (n < need) n *= 2;
  return n;
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// ---------------------------------------------------------------------------
// Thomas: one thread per system. Contract c_kernels.h:38-55 with the
// recurrence of thomas_solve (src/time/helmholtz.cpp:71-85); NULL a/c read
// as 0; exact-zero pivots give VIBE_C_ERR_SINGULAR as c_kernels.c:26,34,40.
// cp (the modified super-diagonal) lives in `work` (n per system).
template <typename T>
__device__ int thomas_seq(const T* __restrict__ as, const T* __restrict__ bs, const T* __restrict__ cs,
                          const T* __restrict__ ds, int n, T* __restrict__ xs, T* __restrict__ cp) {
  if (n == 1) {
    if (bs[0] == (T)0) return VIBE_C_ERR_SINGULAR;
    xs[0] = ds[0] / bs[0];
    return VIBE_C_OK;
  }
  T denom = bs[0];
  if (denom == (T)0) return VIBE_C_ERR_SINGULAR;
  cp[0] = (cs ? cs[0] : (T)0) / denom;
  xs[0] = ds[0] / denom;
  for (int k = 1; k < n; ++k) {
    const T am = as ? as[k - 1] : (T)0;
    denom = bs[k] - am * cp[k - 1];
    if (denom == (T)0) return VIBE_C_ERR_SINGULAR;
    xs[k] = (ds[k] - am * xs[k - 1]) / denom;
    if (k < n - 1) cp[k] = (cs ? cs[k] : (T)0) / denom;
  }
  for (int k = n - 1; k-- > 0;) xs[k] = xs[k] - cp[k] * xs[k + 1];
  return VIBE_C_OK;
}

template <typename T>
__global__ void k_thomas_batched(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ c,
                                 const T* __restrict__ d, int n, int n_sys, T* __restrict__ x, T* __restrict__ work,
                                 int* __restrict__ status) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_sys) return;
  const int rc = thomas_seq<T>(a ? a + (size_t)s * (n - 1) : nullptr, b + (size_t)s * n,
                               c ? c + (size_t)s * (n - 1) : nullptr, d + (size_t)s * n, n, x + (size_t)s * n,
                               work + (size_t)s * n);
  if (status) status[s] = rc;
}

// ---------------------------------------------------------------------------
// The sweep staged on chip: one warp takes 32 consecutive systems, one per
// lane, with the recurrence of thomas_seq. In every array the rows of those
// systems are one contiguous span; a chunk of kStage levels (a 32-byte sector a
// system) comes in by cp.async with four (FP32: eight) lanes on consecutive
// elements, so each fetched sector is used, and is transposed by the odd row
// stride of the staging buffer (no bank conflicts when lanes read their own
// rows). Two chunks are in flight; chunks of two sectors leave room for fewer
// warps an SM (1.04 ms against 0.87 at 262144 x 80, where one thread per system
// took 2.50 and read DRAM 13 times over; 1.95 against 0.99 at 65536 x 200, one warp
// per system 9.08). The modified super-diagonal and the eliminated right-hand
// side stay in shared memory, level-major, and the back substitution stores x
// through the same staging, so DRAM sees each element once and no workspace is
// needed. FP64 takes one reciprocal per row and corrects each product with it by
// its residual num - q den (Markstein's quotient), which rounds as a division
// does: about 17 FP64 operations a row, the bound there, where two divisions take
// 25 (products alone, 13 operations, are 1.35 times as far from 64-bit results).
// Pivots and quotients outside the range where that holds divide. FP32 divides
// twice.
// A system with a zero pivot leaves x as it was.
template <typename T>
struct Sweep {
  static constexpr int kStage = 32 / (int)sizeof(T), kRow = kStage + 1;
  static constexpr int kArr = 32 * kRow;  // one array's chunk
  static size_t smem(int n) { return ((size_t)64 * n + 8 * kArr) * sizeof(T); }
};
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* smem, const T* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gmem), "n"((int)sizeof(T)) : "memory");
}
// one row: x_k = (d - a x_{k-1}) / den, c'_k = c / den
__device__ __forceinline__ bool ordinary(double x, unsigned lo, unsigned hi) {  // |x| by its upper word
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - lo < hi - lo;
}
__device__ __forceinline__ double quotient(double num, double den, double r) {  // r = 1 / den
  const double q = num * r;
  return fma(fma(-q, den, num), r, q);
}
__device__ __forceinline__ void sweep_row(double den, double num, double c, double& x, double& cp) {
  const double r = 1.0 / den;
  x = quotient(num, den, r);
  cp = quotient(c, den, r);
  // (a quotient that is not finite, or of a pivot under 1e-290 or past 2^1021)
  if (!ordinary(den, 0x03d00000u, 0x7fc00000u) || !ordinary(x, 0u, 0x7ff00000u) || !ordinary(cp, 0u, 0x7ff00000u)) {
    x = num / den;
    cp = c / den;
  }
}
__device__ __forceinline__ void sweep_row(float den, float num, float c, float& x, float& cp) {
  x = num / den;
  cp = c / den;
}
template <typename T>
__global__ void __launch_bounds__(32) k_thomas_sweep(const T* __restrict__ a, const T* __restrict__ b,
                                                     const T* __restrict__ c, const T* __restrict__ d, int n, int n_sys,
                                                     T* __restrict__ x, int* __restrict__ status) {
  constexpr int K = Sweep<T>::kStage, R = Sweep<T>::kRow, A = Sweep<T>::kArr;
  extern __shared__ __align__(16) char s_sweep[];
  T* Y = reinterpret_cast<T*>(s_sweep);  // n x 32
  T* CP = Y + (size_t)32 * n;            // n x 32
  T* st = CP + (size_t)32 * n;           // 2 buffers x (a, b, c, d)
  const int lane = threadIdx.x;
  const int s0 = blockIdx.x * 32, ns = n_sys - s0 < 32 ? n_sys - s0 : 32;
  const T* bs = b + (size_t)s0 * n;
  const T* ds = d + (size_t)s0 * n;
  const T* as = a ? a + (size_t)s0 * (n - 1) : nullptr;
  const T* cs = c ? c + (size_t)s0 * (n - 1) : nullptr;
  // an absent a or c reads zeros; idle lanes read a = 0, b = c = d = 1, as a zero
  // pivot or numerator would take their warp through the slow path of the
  // division on every row (FP32, 33 systems of 128 rows: 48 us, with ones 29)
  if (!as || !cs)
    for (int e = lane; e < 8 * A; e += 32) st[e] = (T)0;
  __syncwarp();
  if (lane >= ns)
    for (int e = 0; e < 8 * K; ++e) st[e / K * A + lane * R + e % K] = e / K % 4 == 0 ? (T)0 : (T)1;
  __syncwarp();
  const int nch = (n + K - 1) / K;
  auto load = [&](int ch) {
    T* q = st + (ch & 1) * 4 * A;
#pragma unroll
    for (int m = 0; m < K; ++m) {
      const int e = m * 32 + lane, sys = e / K, kk = e % K, k = ch * K + kk;
      if (sys < ns && k < n) {
        const int o = sys * R + kk;
        const size_t g = (size_t)sys * n + k, h = g - sys;  // h: row k of the (n - 1)-long arrays
        cp_async_elem(q + A + o, bs + g);
        cp_async_elem(q + 3 * A + o, ds + g);
        if (as && k >= 1) cp_async_elem(q + o, as + h - 1);
        if (cs && k < n - 1) cp_async_elem(q + 2 * A + o, cs + h);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  load(0);
  T xp = (T)0, cp = (T)0;
  bool sing = false;
  for (int ch = 0; ch < nch; ++ch) {
    if (ch + 1 < nch) {
      load(ch + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncwarp();
    const T* q = st + (ch & 1) * 4 * A + lane * R;
#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
      const int k = ch * K + kk;
      if (k < n) {
        const T am = k > 0 ? q[kk] : (T)0;
        const T den = q[A + kk] - am * cp;
        sing |= den == (T)0;
        if (n == 1) xp = q[3 * A] / den;
        else sweep_row(den, q[3 * A + kk] - am * xp, k + 1 < n ? q[2 * A + kk] : (T)0, xp, cp);
        Y[k * 32 + lane] = xp;
        CP[k * 32 + lane] = cp;
      }
    }
    __syncwarp();  // the buffer is free for the chunk after next
  }
  if (lane >= ns) sing = true;
  const unsigned bad = __ballot_sync(0xffffffffu, sing);
  if (status && lane < ns) status[s0 + lane] = sing ? VIBE_C_ERR_SINGULAR : VIBE_C_OK;
  xp = (T)0;
  T* xs = x + (size_t)s0 * n;
  for (int ch = nch - 1; ch >= 0; --ch) {
    T* q = st + (ch & 1) * A;
#pragma unroll
    for (int kk = K - 1; kk >= 0; --kk) {
      const int k = ch * K + kk;
      if (k < n) {
        xp = (k + 1 < n) ? Y[k * 32 + lane] - CP[k * 32 + lane] * xp : Y[k * 32 + lane];
        q[lane * R + kk] = xp;
      }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < K; ++m) {
      const int e = m * 32 + lane, sys = e / K, kk = e % K, k = ch * K + kk;
      if (!((bad >> sys) & 1u) && k < n) xs[(size_t)sys * n + k] = q[sys * R + kk];
    }
  }
}

// ---------------------------------------------------------------------------
// Tall systems (n > kTallN) that are few, or too tall for the on-chip sweep:
// one warp per system. The n rows split into 32
// contiguous chunks, one per lane; each lane factors its chunk once (the
// recurrence above) and solves it for three right-hand sides: the chunk's d
// (y), its coupling to the unknown left of the chunk (v, from a at the first
// row) and to the unknown right of it (w, from c at the last row), so that
// x_i = y_i - v_i x_left - w_i x_right on the chunk. The chunks' first and
// last unknowns z_j = (F_j, E_j) then satisfy a 2x2 block-tridiagonal system,
// z_j + [vF; vE]_j E_{j-1} + [wF; wE]_j F_{j+1} = [yF; yE]_j, which lane 0
// solves by block elimination (32 blocks); every lane then reads its two
// neighbours' interface values from shared memory and finishes its chunk.
// The elimination order differs from one sequential sweep, so results agree
// with it to rounding. A chunk starts from its raw diagonal b[r0], so its
// pivots are not the sweep's: a nonsingular system can have a zero or a
// tiny chunk pivot (b[r0] = 0, non-dominant diagonals) or a near-singular
// 2x2 interface block. Whenever a chunk pivot is at most tall_rel (1e-8 in
// FP64, 1e-3 in FP32) of its row's |a| + |b| + |c|, or a block determinant at
// most tall_rel of its terms, lane 0 solves that system again with the single sequential sweep, whose
// contract is the reference's (c_kernels.c:26,34,40): VIBE_C_ERR_SINGULAR
// only on an exactly zero sweep pivot. Scratch: 3n per system (c', v, w).
constexpr int kTallN = 128;
constexpr int kTallWarps = 4;  // systems per block
template <typename T>
__device__ __forceinline__ T tall_rel();
template <>
__device__ __forceinline__ double tall_rel<double>() { return 1e-8; }
template <>
__device__ __forceinline__ float tall_rel<float>() { return 1e-3f; }

template <typename T>
__global__ void __launch_bounds__(32 * kTallWarps) k_thomas_tall(const T* __restrict__ a, const T* __restrict__ b,
                                                                 const T* __restrict__ c, const T* __restrict__ d,
                                                                 int n, int n_sys, T* __restrict__ x,
                                                                 T* __restrict__ work, int* __restrict__ status) {
  __shared__ T sh[kTallWarps][32][6];  // per lane: yF, yE, vF, vE, wF, wE
  __shared__ T zs[kTallWarps][32][2];  // interface solution F_j, E_j
  __shared__ int seq[kTallWarps];  // 1: this system falls back to the sequential sweep
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = blockIdx.x * kTallWarps + wid;
  const bool live = s < n_sys;
  const int m = (n + 31) / 32;                   // rows per chunk
  const int r0 = min(lane * m, n), r1 = min(r0 + m, n), L = r1 - r0;
  const int nch = (n + m - 1) / m;               // chunks with rows (lanes >= nch hold none)
  if (lane == 0) seq[wid] = 0;
  __syncwarp();
  const T rel = tall_rel<T>();
  const T* as = (live && a) ? a + (size_t)s * (n - 1) : nullptr;
  const T* bs = live ? b + (size_t)s * n : nullptr;
  const T* cs = (live && c) ? c + (size_t)s * (n - 1) : nullptr;
  const T* ds = live ? d + (size_t)s * n : nullptr;
  T* xs = live ? x + (size_t)s * n : nullptr;
  T* cp = live ? work + (size_t)s * 3 * n : nullptr;
  T* vv = cp ? cp + n : nullptr;
  T* ww = cp ? cp + 2 * n : nullptr;
  bool ok = true;
  if (live && L > 0) {
    // forward elimination of the chunk with the three right-hand sides
    T den = bs[r0];
    const T a0 = (r0 > 0 && as) ? as[r0 - 1] : (T)0;   // coupling to x_{r0-1}
    const T cl = (r1 < n && cs) ? cs[r1 - 1] : (T)0;   // coupling to x_{r1}
    const T c0 = (r0 + 1 < n && cs) ? cs[r0] : (T)0;
    if (!(fabs(den) > rel * (fabs(a0) + fabs(den) + fabs(c0)))) ok = false;
    if (ok) {
      cp[r0] = (r0 + 1 < r1) ? ((cs ? cs[r0] : (T)0) / den) : (T)0;
      xs[r0] = ds[r0] / den;
      vv[r0] = a0 / den;
      ww[r0] = (L == 1) ? cl / den : (T)0;
      for (int k = r0 + 1; k < r1 && ok; ++k) {
        const T am = as ? as[k - 1] : (T)0;
        const T ck = (k + 1 < n && cs) ? cs[k] : (T)0;
        den = bs[k] - am * cp[k - 1];
        if (!(fabs(den) > rel * (fabs(am) + fabs(bs[k]) + fabs(ck)))) { ok = false; break; }
        xs[k] = (ds[k] - am * xs[k - 1]) / den;
        vv[k] = (-am * vv[k - 1]) / den;
        ww[k] = ((k == r1 - 1 ? cl : (T)0) - am * ww[k - 1]) / den;
        if (k < r1 - 1) cp[k] = (cs ? cs[k] : (T)0) / den;
      }
      if (ok)
        for (int k = r1 - 1; k-- > r0;) {
          xs[k] -= cp[k] * xs[k + 1];
          vv[k] -= cp[k] * vv[k + 1];
          ww[k] -= cp[k] * ww[k + 1];
        }
    }
    if (ok) {
      sh[wid][lane][0] = xs[r0];
      sh[wid][lane][1] = xs[r1 - 1];
      sh[wid][lane][2] = vv[r0];
      sh[wid][lane][3] = vv[r1 - 1];
      sh[wid][lane][4] = ww[r0];
      sh[wid][lane][5] = ww[r1 - 1];
    }
  }
  if (!ok) seq[wid] = 1;
  __syncwarp();
  // the interface system, block elimination by lane 0: z_j + Lj z_{j-1} + Uj z_{j+1} = Yj,
  // Lj = [[0, vF], [0, vE]] and Uj = [[wF, 0], [wE, 0]]
  if (live && lane == 0 && !seq[wid]) {
    T C[32][2][2], Y[32][2];
    for (int j = 0; j < nch; ++j) {
      const T* q = sh[wid][j];
      T D00 = 1, D01 = 0, D10 = 0, D11 = 1, r0v = q[0], r1v = q[1];
      if (j > 0) {  // D = I - Lj C_{j-1}, rhs = Yj - Lj Y_{j-1}; Lj picks row 1 (E) of the previous block
        D00 -= q[2] * C[j - 1][1][0];
        D01 -= q[2] * C[j - 1][1][1];
        D10 -= q[3] * C[j - 1][1][0];
        D11 -= q[3] * C[j - 1][1][1];
        r0v -= q[2] * Y[j - 1][1];
        r1v -= q[3] * Y[j - 1][1];
      }
      const T det = D00 * D11 - D01 * D10;
      if (!(fabs(det) > rel * (fabs(D00 * D11) + fabs(D01 * D10)))) { seq[wid] = 1; break; }
      const T i00 = D11 / det, i01 = -D01 / det, i10 = -D10 / det, i11 = D00 / det;
      // C_j = D^-1 Uj (Uj acts on F_{j+1}: column 0), Y_j = D^-1 rhs
      const T u0 = (j + 1 < nch) ? q[4] : (T)0, u1 = (j + 1 < nch) ? q[5] : (T)0;
      C[j][0][0] = i00 * u0 + i01 * u1;
      C[j][1][0] = i10 * u0 + i11 * u1;
      C[j][0][1] = 0;
      C[j][1][1] = 0;
      Y[j][0] = i00 * r0v + i01 * r1v;
      Y[j][1] = i10 * r0v + i11 * r1v;
    }
    if (!seq[wid])
      for (int j = nch - 1; j >= 0; --j) {
        T f = Y[j][0], e = Y[j][1];
        if (j + 1 < nch) {  // z_j = Y_j - C_j z_{j+1}, C_j acting on F_{j+1}
          f -= C[j][0][0] * zs[wid][j + 1][0];
          e -= C[j][1][0] * zs[wid][j + 1][0];
        }
        zs[wid][j][0] = f;
        zs[wid][j][1] = e;
      }
  }
  __syncwarp();
  if (seq[wid]) {  // the sequential sweep over the whole system, on lane 0
    if (live && lane == 0) {
      const int rc = thomas_seq<T>(as, bs, cs, ds, n, xs, cp);
      if (status) status[s] = rc;
    }
    return;
  }
  if (live && L > 0) {
    const T xl = (lane > 0) ? zs[wid][lane - 1][1] : (T)0;        // E of the chunk to the left
    const T xr = (lane + 1 < nch) ? zs[wid][lane + 1][0] : (T)0;  // F of the chunk to the right
    for (int k = r0; k < r1; ++k) xs[k] = xs[k] - vv[k] * xl - ww[k] * xr;
  }
  if (live && lane == 0 && status) status[s] = VIBE_C_OK;
}

// WENO5 (c_kernels.c:64-104), one thread per stencil
template <typename T>
__device__ void weno5_d(T qm2, T qm1, T q0, T q1, T q2, T* ql, T* qr) {
  const T eps = (T)1e-6, d0 = (T)0.1, d1 = (T)0.6, d2 = (T)0.3;
  const T t12 = (T)13 / (T)12, q4 = (T)0.25;
  const T v0 = ((T)2.0 * qm2 - (T)7.0 * qm1 + (T)11.0 * q0) / (T)6;
  const T v1 = (-qm1 + (T)5.0 * q0 + (T)2.0 * q1) / (T)6;
  const T v2 = ((T)2.0 * q0 + (T)5.0 * q1 - q2) / (T)6;
  const T b0 = t12 * (qm2 - (T)2.0 * qm1 + q0) * (qm2 - (T)2.0 * qm1 + q0) +
                    q4 * (qm2 - (T)4.0 * qm1 + (T)3.0 * q0) * (qm2 - (T)4.0 * qm1 + (T)3.0 * q0);
  const T b1 = t12 * (qm1 - (T)2.0 * q0 + q1) * (qm1 - (T)2.0 * q0 + q1) + q4 * (qm1 - q1) * (qm1 - q1);
  const T b2 = t12 * (q0 - (T)2.0 * q1 + q2) * (q0 - (T)2.0 * q1 + q2) +
                    q4 * ((T)3.0 * q0 - (T)4.0 * q1 + q2) * ((T)3.0 * q0 - (T)4.0 * q1 + q2);
  const T a0 = d0 / ((eps + b0) * (eps + b0)), a1 = d1 / ((eps + b1) * (eps + b1)),
               a2 = d2 / ((eps + b2) * (eps + b2));
  *ql = (a0 * v0 + a1 * v1 + a2 * v2) / (a0 + a1 + a2);
  const T u0 = ((T)2.0 * q2 - (T)7.0 * q1 + (T)11.0 * q0) / (T)6;
  const T u1 = (-q1 + (T)5.0 * q0 + (T)2.0 * qm1) / (T)6;
  const T u2 = ((T)2.0 * q0 + (T)5.0 * qm1 - qm2) / (T)6;
  const T g0 = t12 * (q2 - (T)2.0 * q1 + q0) * (q2 - (T)2.0 * q1 + q0) +
                    q4 * (q2 - (T)4.0 * q1 + (T)3.0 * q0) * (q2 - (T)4.0 * q1 + (T)3.0 * q0);
  const T g1 = t12 * (q1 - (T)2.0 * q0 + qm1) * (q1 - (T)2.0 * q0 + qm1) + q4 * (q1 - qm1) * (q1 - qm1);
  const T g2 = t12 * (q0 - (T)2.0 * qm1 + qm2) * (q0 - (T)2.0 * qm1 + qm2) +
                    q4 * ((T)3.0 * q0 - (T)4.0 * qm1 + qm2) * ((T)3.0 * q0 - (T)4.0 * qm1 + qm2);
  const T c0 = d0 / ((eps + g0) * (eps + g0)), c1 = d1 / ((eps + g1) * (eps + g1)),
               c2 = d2 / ((eps + g2) * (eps + g2));
  *qr = (c0 * u0 + c1 * u1 + c2 * u2) / (c0 + c1 + c2);
}
template <typename T>
__global__ void k_weno_batched(const T* __restrict__ q, size_t n, T* __restrict__ ql, T* __restrict__ qr) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    weno5_d(q[5 * e], q[5 * e + 1], q[5 * e + 2], q[5 * e + 3], q[5 * e + 4], ql + e, qr + e);
}

// bilinear (c_kernels.c:108-144) on one level plane held in `plane`
template <typename T>
__global__ void k_bilinear(const T* __restrict__ plane, int halo, int nsx, int nsy, T xi, T yj, T* out) {
  const int nxi = nsx - 2 * halo, nyi = nsy - 2 * halo;
  const int i0 = (int)floor(xi), j0 = (int)floor(yj);
  const T wx = xi - (T)i0, wy = yj - (T)j0;
  // the reference's clamp order (c_kernels.c:128-135): up to 0 first, then
  // down to n-1, so a grid without interior points reads its last halo point
  auto clamp = [](int v, int n) { v = v < 0 ? 0 : v; return v > n - 1 ? n - 1 : v; };
  const int ia = clamp(i0, nxi), ib = clamp(i0 + 1, nxi);
  const int ja = clamp(j0, nyi), jb = clamp(j0 + 1, nyi);
  auto at = [&](int i, int j) { return plane[(size_t)(j + halo) * nsx + (size_t)(i + halo)]; };
  const T q00 = at(ia, ja), q10 = at(ib, ja), q01 = at(ia, jb), q11 = at(ib, jb);
  *out = (q00 + wx * (q10 - q00)) + wy * ((q01 + wx * (q11 - q01)) - (q00 + wx * (q10 - q00)));
}

// ---- reductions ----------------------------------------------------------
template <typename T>
struct Neu {
  T s, c;
};
// Neumaier add of one value (c_kernels.c:195-203)
template <typename T>
__device__ __forceinline__ void neu_add(Neu<T>& a, T x) {
  const T t = a.s + x;
  if (fabs(a.s) >= fabs(x)) a.c += (a.s - t) + x;
  else a.c += (x - t) + a.s;
  a.s = t;
}
// merge of two compensated partial sums: add b.s with compensation, then b.c
template <typename T>
__device__ __forceinline__ Neu<T> neu_merge(Neu<T> a, Neu<T> b) {
  neu_add(a, b.s);
  a.c += b.c;
  return a;
}
constexpr int kNeuThreads = 256;
// the block's sum, in thread 0. Pairs of all lanes are merged by halves down to one
// warp, which finishes by shuffles: 12 warps' merges of some ten FP64 operations
// where shuffles in every warp take 45.
template <typename T>
__device__ Neu<T> neu_block(Neu<T> v) {
  __shared__ T sh_s[kNeuThreads], sh_c[kNeuThreads];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // (lanes with empty pairs, as the integer sums leave them, need no merging)
  if (__syncthreads_or(lane != 0 && (v.s != (T)0 || v.c != (T)0))) {
    sh_s[tid] = v.s;
    sh_c[tid] = v.c;
    for (int h = kNeuThreads / 2; h >= 32; h >>= 1) {
      __syncthreads();
      if (tid < h) {
        v = neu_merge(v, Neu<T>{sh_s[tid + h], sh_c[tid + h]});
        sh_s[tid] = v.s;
        sh_c[tid] = v.c;
      }
    }
  } else {
    if (lane == 0) {
      sh_s[warp] = v.s;
      sh_c[warp] = v.c;
    }
    __syncthreads();
    if (warp == 0) v = lane < kNeuThreads / 32 ? Neu<T>{sh_s[lane], sh_c[lane]} : Neu<T>{(T)0, (T)0};
  }
  if (warp == 0)
    for (int off = 16; off > 0; off >>= 1) {
      Neu<T> o;
      o.s = __shfl_down_sync(0xffffffffu, v.s, off);
      o.c = __shfl_down_sync(0xffffffffu, v.c, off);
      v = neu_merge(v, o);
    }
  return v;
}
// Exact sum of doubles in integers: each lane's 128-bit fixed-point accumulator
// holds multiples of 2^(base - 1075) of elements whose exponent field lies in
// [base, base + 54]; an element is its 53-bit mantissa shifted by its exponent
// over the base, ~20 integer instructions where Neumaier's addition takes six
// on the FP64 pipe, which issues 1/32 of the integer rate here. The window is
// common to the warp, so the lanes' accumulators add up in integers too: the
// FP64 work is one conversion per warp. 107 bits leave 2^20 additions of
// headroom, 2^13 a lane and 2^5 for the lanes used. Elements above the window
// move it (the accumulators go to the lanes' compensated pairs first);
// elements below it, subnormals, infinities and NaN are added to the lane's
// pair as before. value() is exact to the two doubles of a pair.
struct ExactSum {
  static constexpr int kSpan = 54, kAbove = 8, kRounds = 1024;
  static constexpr int kTopBase = 0x7fe - kSpan;  // a window ends at the largest finite exponent field
  unsigned long long lo = 0;
  long long hi = 0;
  int base = 1 << 20;  // no window yet
  __device__ __forceinline__ void plus(unsigned long long l, long long h) {
    const unsigned long long t = lo + l;
    hi += h + (long long)(t < lo);
    lo = t;
  }
  __device__ __forceinline__ Neu<double> value() const {
    Neu<double> v{0.0, 0.0};
    if (lo == 0 && hi == 0) return v;
    const bool neg = hi < 0;
    unsigned long long l = lo, h = (unsigned long long)hi;
    if (neg) {
      l = ~l + 1;
      h = ~h + (l == 0);
    }
    // three parts of at most 43 bits, each an exact double
    const double p[3] = {(double)(l & 0x7ffffffffffull), (double)((l >> 43) | ((h & 0x3fffffull) << 21)),
                         (double)(h >> 22)};
    const int w[3] = {0, 43, 86};
    for (int q = 2; q >= 0; --q) {
      if (p[q] == 0.0) continue;
      const double x = ldexp(p[q], base - 1075 + w[q]);
      neu_add(v, neg ? -x : x);
    }
    return v;
  }
  __device__ __forceinline__ void flush(Neu<double>& pair) {
    pair = neu_merge(pair, value());
    lo = 0;
    hi = 0;
  }
  static __device__ __forceinline__ int exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
  // top: the warp's largest finite exponent field among the elements to come
  __device__ __forceinline__ void window(int top, Neu<double>& pair) {
    if (top == 0 || (unsigned)(top - base) <= (unsigned)kSpan || (top < base && base < 4096)) return;
    flush(pair);
    base = min(top + kAbove - kSpan, kTopBase);
  }
  __device__ __forceinline__ bool fits(double x) const {
    const int ef = exponent(x);
    return ((unsigned)(ef - base) <= (unsigned)kSpan && ef != 0) || ((unsigned long long)__double_as_longlong(x) << 1) == 0;
  }
  // false: added to the pair
  __device__ __forceinline__ bool add(double x, Neu<double>& pair) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    const int ef = exponent(x);
    const unsigned s = (unsigned)(ef - base);
    if (s > (unsigned)kSpan || ef == 0) {
      if ((bits << 1) == 0) return true;  // (a zero adds nothing)
      neu_add(pair, x);
      return false;
    }
    const unsigned long long m = (bits & 0xfffffffffffffull) | 0x10000000000000ull;
    const unsigned long long sg = (unsigned long long)((long long)bits >> 63);  // all ones for negative elements
    // two's complement: the inverted bits of a negative element, and one
    plus((m << s) ^ sg, (long long)(((m >> 1) >> (63 - s)) ^ sg));
    plus(sg & 1, 0);
    return true;
  }
};
// each block sums a contiguous chunk; partials[2*block] = (s, c)
template <typename T>
__global__ void __launch_bounds__(kNeuThreads) k_neu_partial(const T* __restrict__ x, size_t n, size_t chunk,
                                                             T* __restrict__ partials) {
  const size_t lo = (size_t)blockIdx.x * chunk, hi = lo + chunk < n ? lo + chunk : n;
  Neu<T> v{(T)0, (T)0};
  constexpr int kU = 8;  // loads in flight per thread
  if constexpr (sizeof(T) == 8) {
    ExactSum acc;
    int rounds = 0;
    size_t e0 = lo;
    bool all = true;
    for (; e0 < hi && all; e0 += kU * kNeuThreads) {  // the same trips for every lane
      T q[kU];
      int top = 0;
#pragma unroll
      for (int m = 0; m < kU; ++m) {
        const size_t e = e0 + m * kNeuThreads + threadIdx.x;
        q[m] = e < hi ? x[e] : (T)0;
      }
#pragma unroll
      for (int m = 0; m < kU; ++m) {
        const int ef = ExactSum::exponent(q[m]);
        top = max(top, ef == 0x7ff ? 0 : ef);
      }
      acc.window(__reduce_max_sync(0xffffffffu, top), v);
      if (e0 == lo) {  // (looked at beforehand in the first round: most data show at once which way they go)
#pragma unroll
        for (int m = 0; m < kU; ++m) all &= acc.fits(q[m]);
        all = __all_sync(0xffffffffu, all);
        if (!all) break;
      }
      if (++rounds == ExactSum::kRounds) {
        acc.flush(v);
        rounds = 0;
      }
#pragma unroll
      for (int m = 0; m < kU; ++m) all &= acc.add(q[m], v);
      // elements that do not fit would take the warp through both additions from
      // here on: it goes on with the pairs alone (8.8 M elements of magnitudes 1e-300 to
      // 1e300 180 us with both, 142 so, 138 with pairs from the start)
      all = __all_sync(0xffffffffu, all);
    }
    for (; e0 < hi; e0 += kU * kNeuThreads) {
      double q[kU];
#pragma unroll
      for (int m = 0; m < kU; ++m) {
        const size_t e = e0 + m * kNeuThreads + threadIdx.x;
        q[m] = e < hi ? x[e] : 0.0;
      }
#pragma unroll
      for (int m = 0; m < kU; ++m)
        if (e0 + m * kNeuThreads + threadIdx.x < hi) neu_add(v, q[m]);
    }
    for (int off = 16; off > 0; off >>= 1)  // lane 0 gets the warp's sum
      acc.plus(__shfl_down_sync(0xffffffffu, acc.lo, off), __shfl_down_sync(0xffffffffu, acc.hi, off));
    // the warps' sums, one per lane of the first warp: one conversion for all
    __shared__ ExactSum part[kNeuThreads / 32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < kNeuThreads / 32) part[threadIdx.x].flush(v);
  } else {
    for (size_t e0 = lo + threadIdx.x; e0 < hi; e0 += kU * kNeuThreads) {
      T q[kU];
#pragma unroll
      for (int m = 0; m < kU; ++m) q[m] = e0 + m * kNeuThreads < hi ? x[e0 + m * kNeuThreads] : (T)0;
#pragma unroll
      for (int m = 0; m < kU; ++m) neu_add(v, q[m]);
    }
  }
  v = neu_block(v);
  if (threadIdx.x == 0) { partials[2 * blockIdx.x] = v.s; partials[2 * blockIdx.x + 1] = v.c; }
}
template <typename T>
__global__ void k_neu_final(const T* __restrict__ partials, int nb, T* __restrict__ out) {
  Neu<T> v{(T)0, (T)0};
  for (int b = threadIdx.x; b < nb; b += blockDim.x) v = neu_merge(v, Neu<T>{partials[2 * b], partials[2 * b + 1]});
  v = neu_block(v);
  if (threadIdx.x == 0) *out = v.s + v.c;
}

constexpr int kCflThreads = 256;
// CFL scan (c_kernels.c:148-186): per cell dz = max(dzeta[k]*scale, 1),
// speed = sqrt(u^2+v^2+w^2), cfl = dt*(|u|/dx + |v|/dy + |w|/dz); block maxima
// of (cfl, speed) and min of dz, then one block merges.
// The three are never negative nor NaN, so they order as their bits: the merges
// are integer comparisons (FP64 ones would issue at the FP64 rate).
__device__ __forceinline__ long long order_bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ int order_bits(float x) { return __float_as_int(x); }
__device__ __forceinline__ double from_order(long long b) { return __longlong_as_double(b); }
__device__ __forceinline__ float from_order(int b) { return __int_as_float(b); }
template <typename T>
__device__ __forceinline__ void max3_block(T& ta, T& tb, T& tc) {  // max, max, min
  using I = decltype(order_bits(T()));
  __shared__ I s1[32], s2[32], s3[32];
  I a = order_bits(ta), b = order_bits(tb), c = order_bits(tc);
  auto merge = [&]() {
    for (int off = 16; off > 0; off >>= 1) {
      const I x = __shfl_down_sync(0xffffffffu, a, off), y = __shfl_down_sync(0xffffffffu, b, off),
              z = __shfl_down_sync(0xffffffffu, c, off);
      a = x > a ? x : a;
      b = y > b ? y : b;
      c = z < c ? z : c;
    }
  };
  merge();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) { s1[warp] = a; s2[warp] = b; s3[warp] = c; }
  __syncthreads();
  if (warp == 0) {
    a = lane < nw ? s1[lane] : 0;
    b = lane < nw ? s2[lane] : 0;
    c = lane < nw ? s3[lane] : order_bits((T)1e30);
    merge();
  }
  ta = from_order(a);
  tb = from_order(b);
  tc = from_order(c);
}
// Most cells cannot raise a maximum, and finding that out in FP64 costs three
// divisions a cell. So a cell's CFL number and squared speed are first bounded
// from above in FP32 (within 2.1e-5), from the doubles' upper bits (integer
// instructions; a conversion would issue at the FP64 rate). A cell is evaluated
// in FP64 only if its bound exceeds the block's best so far and is not so far
// under the largest bound of the block's tile that the cell holding that one
// must win: a handful of cells per block. The maxima are those of the FP64
// values, bit for bit. The bounds assume ordinary positive dt, dx, dy
// (`plain`); else, and where a bound is not finite, cells are evaluated.
// What FP32 cannot hold makes a bound larger than the cell by any factor, so a
// tile whose largest bound is no more than such floors (winds count from 2^-126
// up) sets no limit, and a cell whose dzeta or depth is past 1e30, beside which
// the other may have been cut to zero, has no bound.
// The minimum of dz over a column is dz at the smallest (or, where the column's
// depth is negative, the largest) dzeta: a product rounds monotonically.
__device__ __forceinline__ float trunc_abs(double x) {  // |x| rounded toward zero; tiny values up to 2^-126
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu, l = (unsigned)__double2loint(x);
  if (h >= 0x47f00000u) return __int_as_float(0x7f800000);
  if (h < 0x38100000u) return (h | l) ? 1.17549435e-38f : 0.f;
  return __uint_as_float(((h - 0x38000000u) << 3) | (l >> 29));
}
__device__ __forceinline__ float trunc_abs(float x) { return fabsf(x); }
__device__ __forceinline__ float trunc_signed(double x) {  // rounded toward zero; NaN and 2^128 up: NaN, infinity
  const int h = __double2hiint(x), m = h & 0x7fffffff;
  float f = m < 0x38100000 ? 0.f : trunc_abs(x);
  if (m > 0x7ff00000 || (m == 0x7ff00000 && __double2loint(x))) f = __int_as_float(0x7fc00000);
  return copysignf(f, __int_as_float(h));
}
__device__ __forceinline__ float trunc_signed(float x) { return x; }
template <typename T>
__device__ __forceinline__ float round_down(T x) {  // of x >= 0
  return fminf(trunc_signed(x), 3.402823466e38f);
}
// What is left of FP64: one subtraction a thread and tile, the column's smallest dz
// in the bottom tiles, the cells evaluated. 384 x 384 x 60 (floor 31 us): 66 us; the
// extent of dzeta, the merges and the roots in every warp took 28 more (FP64 pipe
// 76 % busy).
constexpr int kCflLevels = 4;  // levels of one tile, half of them where that leaves SMs without one
// A block's best CFL number and squared speed (as order bits), and the inputs of
// the last cell of each thread that had the best of its time. Both round
// monotonically in |u|, |v|, |w| (and the first falls with dz), so a cell with none larger
// cannot raise them: in fields with many equal cells, a uniform wind above all,
// every bound lies above the best. FP64 cells near the best, of which a nearly
// uniform wind has many, are compared by products with the reciprocals (5 FP64
// operations, where the three divisions take 31) before they are evaluated. Both
// scan kernels, 384 x 384 x 60: white noise 69 us, a uniform wind 163 and a nearly uniform one 319,
// where every cell evaluated took 997 and 620 (and 1066 and 679 with the bounds alone).
template <typename T>
struct CflBest {
  using I = decltype(order_bits(T()));
  static constexpr int kOf = sizeof(T) == 8 ? kCflThreads : 1;  // (FP32: not used)
  I best[2], top_c[4][kOf], top_s[3][kOf];
  T up_dt, inv_dx, inv_dy;
};
template <typename T, int kL>
__global__ void __launch_bounds__(kCflThreads, 4) k_cfl_partial(const T* __restrict__ u, const T* __restrict__ v,
                                                             const T* __restrict__ w, const T* __restrict__ dzeta,
                                                             const T* __restrict__ zs, int nx, int ny, int nz, T dx,
                                                             T dy, T z_top, T dt, size_t tiles,
                                                             T* __restrict__ partials) {
  const size_t nxy = (size_t)nx * ny;  // (no negative dimension reaches here)
  const size_t ctiles = (nxy + kCflThreads - 1) / kCflThreads;
  const bool plain = dt >= (T)1e-30 && dt <= (T)1e30 && dx >= (T)1e-30 && dx <= (T)1e30 && dy >= (T)1e-30 && dy <= (T)1e30;
  const float up = 1.00002f;  // above the rounding of the bounds (a few 1e-6)
  const float bdt = (float)dt * up, bdx = 1.f / (float)dx, bdy = 1.f / (float)dy;
  const float cfloor = fmaxf(bdt * (bdx + bdy + 1.f) * 1e-30f, 1e-30f);
  // the largest squared speed, one square root at the end: a correctly
  // rounded square root is monotone, so the maximum of the roots is the root
  // of the maximum, bit for bit
  T mdz = (T)1e30;
  __shared__ CflBest<T> sh;
  __shared__ unsigned seen[2][2];  // a tile's largest bounds, as float bits (non-negative floats order as their bits)
  const int tid = threadIdx.x;
  if constexpr (sizeof(T) == 8) {
    for (int q = 0; q < 3; ++q) sh.top_c[q][tid] = sh.top_s[q][tid] = 0;
    sh.top_c[3][tid] = 0;
  }
  if (tid < 2) sh.best[tid] = 0, seen[0][tid] = 0u;
  if (tid == 0) sh.up_dt = dt * (T)(1.0 + 0x1p-48), sh.inv_dx = (T)1 / dx, sh.inv_dy = (T)1 / dy;
  int par = 0;
  __shared__ T dext[2];  // the smallest and the largest dzeta, for the blocks that have bottom tiles
  if (blockIdx.x < ctiles && threadIdx.x < 32) {
    T dlo = (T)NAN, dhi = (T)NAN;
    for (int k = threadIdx.x; k < nz; k += 32) {
      dlo = fmin(dlo, dzeta[k]);
      dhi = fmax(dhi, dzeta[k]);
    }
    for (int off = 16; off > 0; off >>= 1) {
      dlo = fmin(dlo, __shfl_xor_sync(0xffffffffu, dlo, off));
      dhi = fmax(dhi, __shfl_xor_sync(0xffffffffu, dhi, off));
    }
    if (threadIdx.x == 0) {
      dext[0] = dlo;
      dext[1] = dhi;
    }
  }
  __syncthreads();
  for (size_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const size_t kt = tile / ctiles, col = (tile - kt * ctiles) * kCflThreads + threadIdx.x;
    const int k0 = (int)kt * kL;
    const bool in = col < nxy;
    const T scale = zs ? (in ? z_top - zs[col] : (T)1) : z_top;
    const float fscale = trunc_signed(scale);
    const bool deep = !(fabsf(fscale) < 1e30f);
    if (in && k0 == 0) {
      T dz = fmin(dext[0] * scale, dext[1] * scale);
      if (dz < (T)1) dz = (T)1;
      mdz = fmin(mdz, dz);
    }
    T qu[kL], qv[kL], qw[kL];
    const size_t e0 = (size_t)k0 * nxy + col;
#pragma unroll
    for (int m = 0; m < kL; ++m) {
      const size_t e = e0 + m * nxy;
      const bool on = in && k0 + m < nz;
      qu[m] = on ? u[e] : (T)0;
      qv[m] = on ? v[e] : (T)0;
      qw[m] = on ? w[e] : (T)0;
    }
    float ec[kL], es[kL], tc = 0.f, ts = 0.f;
#pragma unroll
    for (int m = 0; m < kL; ++m) {
      const int k = k0 + m < nz ? k0 + m : nz - 1;
      const float fu = trunc_abs(qu[m]), fv = trunc_abs(qv[m]), fw = trunc_abs(qw[m]);
      const float some = (fu + fv + fw > 0.f) ? 1e-36f : 0.f;  // products below 2^-126 count as that much
      const float fzeta = trunc_signed(dzeta[k]);
      float fdz = fzeta * fscale;
      if (fdz < 1.f) fdz = 1.f;
      ec[m] = bdt * (fu * bdx + fv * bdy + fw * __frcp_rn(fdz)) + some;
      if (deep || !(fabsf(fzeta) < 1e30f) || fdz > 3e38f) ec[m] = __int_as_float(0x7f800000);  // no bound
      es[m] = up * (fu * fu + fv * fv + fw * fw) + some;
      tc = fmaxf(tc, ec[m]);
      ts = fmaxf(ts, es[m]);
    }
    if (plain) {
      const unsigned wc = __reduce_max_sync(0xffffffffu, __float_as_uint(tc));
      const unsigned ws = __reduce_max_sync(0xffffffffu, __float_as_uint(ts));
      if ((threadIdx.x & 31) == 0) {
        atomicMax(&seen[par][0], wc);
        atomicMax(&seen[par][1], ws);
      }
    }
    __syncthreads();
    // (another warp may raise best meanwhile: any value read is a maximum already reached)
    const float bc = round_down(from_order(sh.best[0])), bs = round_down(from_order(sh.best[1]));
    const float mc = __uint_as_float(seen[par][0]), ms = __uint_as_float(seen[par][1]);
    // under these a cell cannot be the tile's maximum (no such limit where a bound is tiny or not finite)
    const float lc = (mc > cfloor && mc < 3e38f) ? mc * 0.99995f : 0.f, ls = (ms > 1e-30f && ms < 3e38f) ? ms * 0.99995f : 0.f;
    if (threadIdx.x < 2) seen[par ^ 1][threadIdx.x] = 0u;
    if constexpr (sizeof(T) == 4) {  // evaluation is cheap
#pragma unroll
      for (int m = 0; m < kL; ++m) {
        const int k = k0 + m;
        const T uu = qu[m], vv = qv[m], ww = qw[m];
        if (in && k < nz && (!plain || (!(ec[m] <= bc) && !(ec[m] < lc)))) {
          T dz = dzeta[k] * scale;
          if (dz < (T)1) dz = (T)1;
          const T c = dt * (fabs(uu) / dx + fabs(vv) / dy + fabs(ww) / dz);
          if (c > from_order(sh.best[0])) atomicMax(&sh.best[0], order_bits(c));
        }
        if (in && k < nz && (!plain || (!(es[m] <= bs) && !(es[m] < ls)))) {
          const T s2 = uu * uu + vv * vv + ww * ww;
          if (s2 > from_order(sh.best[1])) atomicMax(&sh.best[1], order_bits(s2));
        }
      }
    } else {
      // the few cells that are left are read again: kept, they would take the registers of a block an SM
      unsigned left = 0u;
#pragma unroll
      for (int m = 0; m < kL; ++m)
        if (in && k0 + m < nz) {
          if (!plain || (!(ec[m] <= bc) && !(ec[m] < lc))) left |= 1u << m;
          if (!plain || (!(es[m] <= bs) && !(es[m] < ls))) left |= 0x10000u << m;
        }
      while (left) {
        const int m = (__ffs(left) - 1) & 15;
        const size_t e = e0 + m * nxy;
        const T au = fabs(u[e]), av = fabs(v[e]), aw = fabs(w[e]);
        const auto bu = order_bits(au), bv = order_bits(av), bw = order_bits(aw);
        if (left >> m & 1u) {
          T dz = dzeta[k0 + m] * scale;
          if (dz < (T)1) dz = (T)1;
          const auto bz = order_bits(dz);
          const T b = from_order(sh.best[0]);
          bool go = true;
          if (plain) {
            go = bu > sh.top_c[0][tid] || bv > sh.top_c[1][tid] || bw > sh.top_c[2][tid] ||
                 (bz < sh.top_c[3][tid] && bw != 0);
            if (go && b > (T)1e-250) {  // (what underflows in the products is nothing beside such a best)
              const T rdz = (T)(fmaxf(__frcp_rn(trunc_signed(dz)), 3e-39f) * 1.000001f);  // 1/dz or more
              go = !((aw * rdz + (av * sh.inv_dy + au * sh.inv_dx)) * sh.up_dt <= b);
            }
          }
          if (go) {
            const T c = dt * (au / dx + av / dy + aw / dz);
            if (c >= b) {
              sh.top_c[0][tid] = bu, sh.top_c[1][tid] = bv, sh.top_c[2][tid] = bw, sh.top_c[3][tid] = bz;
              if (c > b) atomicMax(&sh.best[0], order_bits(c));
            }
          }
        }
        if ((left >> m & 0x10000u) && (bu > sh.top_s[0][tid] || bv > sh.top_s[1][tid] || bw > sh.top_s[2][tid])) {
          const T s2 = au * au + av * av + aw * aw, b = from_order(sh.best[1]);
          if (s2 >= b) {
            sh.top_s[0][tid] = bu, sh.top_s[1][tid] = bv, sh.top_s[2][tid] = bw;
            if (s2 > b) atomicMax(&sh.best[1], order_bits(s2));
          }
        }
        left &= ~(0x10001u << m);
      }
    }
    par ^= 1;
    __syncthreads();  // seen[par] is clear, best is settled
  }
  T worst = tid == 0 ? from_order(sh.best[0]) : (T)0, mw2 = tid == 0 ? from_order(sh.best[1]) : (T)0;
  max3_block(worst, mw2, mdz);
  if (threadIdx.x == 0) {
    partials[3 * blockIdx.x] = worst;
    partials[3 * blockIdx.x + 1] = sqrt(mw2);
    partials[3 * blockIdx.x + 2] = mdz;
  }
}
// The same with every cell evaluated, a grid-stride loop, for grids that the tiles
// are not worth their barriers on.
template <typename T>
__global__ void k_cfl_cells(const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ w,
                              const T* __restrict__ dzeta, const T* __restrict__ zs, int nx, int ny, int nz, T dx, T dy,
                              T z_top, T dt, T* __restrict__ partials) {
  const size_t n = (size_t)nx * ny * nz, nxy = (size_t)nx * ny;  // (no negative dimension reaches here)
  // the largest squared speed, one square root at the end: a correctly
  // rounded square root is monotone, so the maximum of the roots is the root
  // of the maximum, bit for bit
  T worst = 0, mw2 = 0, mdz = (T)1e30;
  const size_t S = (size_t)gridDim.x * blockDim.x;
  size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e < n) {
    // the cell's level and column, stepped along with e (no division per cell)
    size_t k = e / nxy, col = e - k * nxy;
    const size_t sk = S / nxy, sc = S - sk * nxy;
    for (; e < n; e += S) {
      const T uu = u[e], vv = v[e], ww = w[e];
      const T scale = zs ? (z_top - zs[col]) : z_top;
      T dz = dzeta[k] * scale;
      if (dz < (T)1) dz = (T)1;
      mdz = fmin(mdz, dz);
      mw2 = fmax(mw2, uu * uu + vv * vv + ww * ww);
      worst = fmax(worst, dt * (fabs(uu) / dx + fabs(vv) / dy + fabs(ww) / dz));
      col += sc;
      k += sk;
      if (col >= nxy) {
        col -= nxy;
        ++k;
      }
    }
  }
  T mw = sqrt(mw2);
  max3_block(worst, mw, mdz);
  if (threadIdx.x == 0) {
    partials[3 * blockIdx.x] = worst;
    partials[3 * blockIdx.x + 1] = mw;
    partials[3 * blockIdx.x + 2] = mdz;
  }
}

template <typename T>
__global__ void k_cfl_final(const T* __restrict__ partials, int nb, T* __restrict__ out3) {
  T a = 0, b = 0, c = (T)1e30;
  for (int e = threadIdx.x; e < nb; e += blockDim.x) {
    a = fmax(a, partials[3 * e]);
    b = fmax(b, partials[3 * e + 1]);
    c = fmin(c, partials[3 * e + 2]);
  }
  max3_block(a, b, c);
  if (threadIdx.x == 0) {
    out3[0] = a;
    out3[1] = b;
    out3[2] = (c > (T)1e29) ? (T)0 : c;
  }
}

// flux advection (c_kernels.c:209-286). Every face flux is computed once: a
// warp is 32 consecutive columns, whose west fluxes serve the 31 cells between
// them (the neighbour's by shuffle); a block's nine rows of south fluxes serve
// eight rows of cells through shared memory; a thread marches up the levels
// and keeps its lower face's flux. With the cell's two quotients from one reciprocal
// that is about 41 FP64 operations, the bound (384 x 384 x 60 674 us, the pipe 86 %
// busy), where one thread per cell with its six faces spent 70 and three index
// divisions (1180 us). The halves of the two means are exact
// powers of two and are applied once. The upper face's flux stands in its
// difference unrounded (fluxes nearly cancel, and their rounding is most of the
// result's), as one face of each pair did in the kernel before.
// x < 1 and x > 1e-12 on the integer pipe (a NaN x, of either sign, is not below
// one; a NaN rho makes the fluxes NaN whatever the divisor)
__device__ __forceinline__ bool below_one(double x) {
  const int h = __double2hiint(x);
  return h < 0x3ff00000 && (unsigned)h <= 0xfff00000u;
}
__device__ __forceinline__ bool below_one(float x) { return x < 1.f; }
__device__ __forceinline__ bool above_floor(double x) { return __double_as_longlong(x) > __double_as_longlong(1e-12); }
__device__ __forceinline__ bool above_floor(float x) { return x > 1e-12f; }
// (h + z / dz) / r with both quotients rounded as divisions round: one reciprocal
// of dz r gives those of dz and r, and each quotient is corrected by its residual
// (eight FP64 operations less than two divisions)
__device__ __forceinline__ double flux_quotient(double h, double z, double dz, double r) {
  const double den = dz * r, i = 1.0 / den;
  const double x = quotient(h + quotient(z, dz, r * i), r, dz * i);
  return ordinary(den, 0x03d00000u, 0x7fc00000u) && ordinary(x, 0u, 0x7ff00000u) ? x : (h + z / dz) / r;
}
__device__ __forceinline__ float flux_quotient(float h, float z, float dz, float r) { return (h + z / dz) / r; }
constexpr int kFluxRows = 8, kFluxCols = 31;
template <typename T>
__global__ void __launch_bounds__(32 * (kFluxRows + 1)) k_flux_adv(
    const T* __restrict__ q, const T* __restrict__ rho, const T* __restrict__ u, const T* __restrict__ v,
    const T* __restrict__ w, const T* __restrict__ dzeta, const T* __restrict__ zs, int nx, int ny, int nz, T dx, T dy,
    T z_top, T* __restrict__ dqdt, int xtiles, int kz) {
  __shared__ T sy[2][kFluxRows + 1][32];
  const size_t nxy = (size_t)nx * ny;
  const int lane = threadIdx.x, row = threadIdx.y;
  const int i0 = (int)(blockIdx.x % (unsigned)xtiles) * kFluxCols, j0 = (int)(blockIdx.x / (unsigned)xtiles) * kFluxRows;
  const int k0 = blockIdx.y * kz, k1 = k0 + kz < nz ? k0 + kz : nz;
  const int i = (i0 + lane) % nx, j = (j0 + row) % ny;  // periodic; the columns and rows past the grid wrap onto it
  const int im = i > 0 ? i - 1 : nx - 1, js = j > 0 ? j - 1 : ny - 1;
  const bool cells = row < kFluxRows;  // the last row only has south fluxes
  const bool mine = cells && lane < kFluxCols && i0 + lane < nx && j0 + row < ny;
  const size_t c = (size_t)j * nx + i, cs = (size_t)js * nx + i, cw = (size_t)j * nx + im;
  const T ax = (T)0.25 * ((T)1 / dx), ay = (T)0.25 * ((T)1 / dy);
  const T scale = zs ? (z_top - zs[c]) : z_top;
  size_t o = (size_t)k0 * nxy;
  T qc = q[o + c], rc = rho[o + c], fb = 0;
  if (cells && k0 > 0) fb = w[o + c] * (rho[o - nxy + c] + rc) * (q[o - nxy + c] + qc);
  for (int k = k0; k < k1; ++k, o += nxy) {
    const T fs = v[o + c] * (rho[o + cs] + rc) * (q[o + cs] + qc);
    sy[k & 1][row][lane] = fs;
    T qt = 0, rt = 0, mt = 0, fw = 0, fe = 0;
    if (k + 1 < nz) {
      qt = q[o + nxy + c];
      rt = rho[o + nxy + c];
    }
    if (cells) {
      if (k + 1 < nz) mt = w[o + nxy + c] * (rc + rt);
      T qw = __shfl_up_sync(0xffffffffu, qc, 1), rw = __shfl_up_sync(0xffffffffu, rc, 1);
      if (lane == 0) {
        qw = q[o + cw];
        rw = rho[o + cw];
      }
      fw = u[o + c] * (rw + rc) * (qw + qc);
      fe = __shfl_down_sync(0xffffffffu, fw, 1);
    }
    __syncthreads();  // (the buffer of two levels ago: every thread read it before the barrier in between)
    const T qm = qc + qt;
    if (mine) {
      T dz = dzeta[k] * scale;
      if (below_one(dz)) dz = (T)1;
      const T rr = above_floor(rc) ? rc : (T)1e-12;
      const T h = (fe - fw) * ax + (sy[k & 1][row + 1][lane] - fs) * ay;
      const T z = (k > 0 && k + 1 < nz) ? (T)0.25 * fma(mt, qm, -fb) : (T)0;
      dqdt[o + c] = -flux_quotient(h, z, dz, rr);
    }
    qc = qt;
    rc = rt;
    fb = mt * qm;
  }
}

// The same, one thread per cell with its six faces, for grids that fill the
// tiles badly (flux_tiles below).
template <typename T>
__global__ void k_flux_cell(const T* __restrict__ q, const T* __restrict__ rho, const T* __restrict__ u,
                           const T* __restrict__ v, const T* __restrict__ w, const T* __restrict__ dzeta,
                           const T* __restrict__ zs, int nx, int ny, int nz, T dx, T dy, T z_top, T* __restrict__ dqdt) {
  const size_t nxy = (size_t)nx * ny, n = nxy * nz;
  const T inv_dx = (T)1 / dx, inv_dy = (T)1 / dy, hf = (T)0.5;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(idx / nxy);
    const int j = (int)((idx / nx) % ny);
    const int i = (int)(idx % nx);
    const size_t base_k = (size_t)k * nxy;
    const T scale = zs ? (z_top - zs[(size_t)j * nx + i]) : z_top;
    T dz = dzeta[k] * scale;
    if (dz < (T)1) dz = (T)1;
    const size_t c = idx;
    const size_t e = base_k + (size_t)j * nx + (size_t)((i + 1) % nx);
    const size_t ws = base_k + (size_t)j * nx + (size_t)((i + nx - 1) % nx);
    const T fxE = u[e] * (hf * (rho[c] + rho[e])) * (hf * (q[c] + q[e]));
    const T fxW = u[c] * (hf * (rho[ws] + rho[c])) * (hf * (q[ws] + q[c]));
    const size_t nn = base_k + (size_t)((j + 1) % ny) * nx + (size_t)i;
    const size_t ss = base_k + (size_t)((j + ny - 1) % ny) * nx + (size_t)i;
    const T fyN = v[nn] * (hf * (rho[c] + rho[nn])) * (hf * (q[c] + q[nn]));
    const T fyS = v[c] * (hf * (rho[ss] + rho[c])) * (hf * (q[ss] + q[c]));
    T fzT = 0, fzB = 0;
    if (k > 0 && k + 1 < nz) {
      const size_t t = c + nxy, b = c - nxy;
      fzT = w[t] * (hf * (rho[c] + rho[t])) * (hf * (q[c] + q[t]));
      fzB = w[c] * (hf * (rho[b] + rho[c])) * (hf * (q[b] + q[c]));
    }
    const T div = (fxE - fxW) * inv_dx + (fyN - fyS) * inv_dy + (fzT - fzB) / dz;
    const T rr = (rho[idx] > (T)1e-12) ? rho[idx] : (T)1e-12;
    dqdt[idx] = -div / rr;
  }
}

// ---- allocation-free batched Thomas ------------------------------------
// Some callers of this library may not allocate device memory at all: a host
// model whose own allocator has reserved the device's memory and forbids any
// other allocation, or a time-critical step loop in which a cudaMalloc or
// cudaFree (both can synchronise the whole device) is not acceptable. For
// them, vibe_tridiagonal_solve_batched_f64_dev_noalloc keeps its Thomas
// workspace (the modified super-diagonal, n doubles per system) in this
// fixed device array instead of the allocated scratch buffer. The array is
// sized here, once, and every GPU that loads the library holds it until the
// process exits; only columns too tall for the on-chip sweep use it, with the
// one-thread-per-system sweep (k_thomas_batched). It sweeps for every n, also
// where the allocating _dev form runs the warp-per-system solver: there the
// two agree to rounding, and this form's singular test is the sweep's
// exact-zero pivot.
constexpr size_t kNoAllocThomasDoubles = (size_t)1 << 18;  // 2 MiB: n * n_sys <= 262144
static __device__ __align__(256) double g_noalloc_thomas_work[kNoAllocThomasDoubles];
// Device address of that array per device. Host code only sees a host-side
// stand-in for the symbol; the address a kernel may use comes from
// cudaGetSymbolAddress, called with the device current, on the first call per
// device, and is kept for the life of the process: a process that resets a
// device (cudaDeviceReset) loads the module into a new context there, and
// must not call this entry point on that device afterwards.
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[64] = {};

constexpr int kRedThreads = 256;
constexpr int kNeuBlocks = 608, kCflBlocks = 608;  // 4 x 152 SMs

// ---- entry points, one template per ABI function: T = double (the
// reference's *_f64 names) or float (the *_f32 twins its header reserves,
// c_kernels.h:15-16). The _dev forms take their scratch from the calling
// thread's DevScratch; the host forms stage everything through one HostCall
// (cabi_host.cuh) and allocate nothing once the thread's buffers are large
// enough. ----
using vgb_cabi::DevScratch;
using vgb_cabi::HostCall;

// The staged sweep runs whenever its columns fit in shared memory and n is at
// most kTallN, or the systems are many enough that it is done before the
// warp-per-system solver would be. A wave of the sweep (32 systems a block, as
// many blocks an SM as their columns leave room for) takes 0.73 us a row in
// FP64 and 0.25 in FP32; the other is bound by latency for few systems and by
// its traffic for many. Measured, sweep against solver: FP64 1000 x 129 94 and
// 154 us, 256 x 300 212 and 121, 1000 x 380 267 and 223, 4864 x 380 268 and 854;
// FP32 1000 x 129 33 and 23, 4864 x 129 34 and 50, 1000 x 760 170 and 74, 4864 x 760
// 170 and 446.
constexpr size_t kSweepSmem = 200 * 1024;
constexpr int kSweepSystems = 256;
template <typename T>
bool thomas_sweeps(int n, int n_sys) {
  const size_t sm = Sweep<T>::smem(n);
  if (sm > kSweepSmem) return false;
  if (n <= kTallN) return true;
  if (n_sys < kSweepSystems) return false;
  const bool d = sizeof(T) == 8;
  const long blocks = (n_sys + 31L) / 32, wave = 152L * (long)(227 * 1024 / (sm + 1024));
  const double sweep = (double)((blocks + wave - 1) / wave) * n * (d ? 0.73 : 0.25);
  const double latency = d ? 73.0 + 0.16 * n : 13.0 + 0.045 * n;
  const double each = d ? 0.10 + 1.9e-4 * n : (4.5e-5 + 7e-8 * n) * n;
  return sweep <= std::max(latency, 0.4 * latency + each * n_sys);
}
template <typename T>
size_t thomas_work(int n, int n_sys) {
  return thomas_sweeps<T>(n, n_sys) ? 0 : (size_t)n * (size_t)n_sys * 3;
}
template <typename T>
int thomas_sweep_launch(const T* a, const T* b, const T* c, const T* d, int n, int n_sys, T* x, int* status,
                        cudaStream_t st) {
  const size_t sm = Sweep<T>::smem(n);
  if (sm > 48 * 1024 && !device_ok(cudaFuncSetAttribute(k_thomas_sweep<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)kSweepSmem),
                                   "thomas shared memory"))
    return VIBE_C_ERR_DEVICE;
  k_thomas_sweep<T><<<(n_sys + 31) / 32, 32, sm, st>>>(a, b, c, d, n, n_sys, x, status);
  return device_ok(cudaGetLastError(), "thomas launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

template <typename T>
int thomas_launch(const T* a, const T* b, const T* c, const T* d, int n, int n_sys, T* x, T* work, int* status,
                  cudaStream_t st) {
  if (thomas_sweeps<T>(n, n_sys)) return thomas_sweep_launch<T>(a, b, c, d, n, n_sys, x, status, st);
  k_thomas_tall<T><<<(n_sys + kTallWarps - 1) / kTallWarps, 32 * kTallWarps, 0, st>>>(a, b, c, d, n, n_sys, x, work,
                                                                                     status);
  return device_ok(cudaGetLastError(), "thomas launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

template <typename T>
int thomas_batched_dev(const T* a, const T* b, const T* c, const T* d, int n, int n_sys, T* x, int* status,
                       vibe_stream_t stream) {
  if (n <= 0 || n_sys < 0 || b == nullptr || d == nullptr || x == nullptr) return VIBE_C_ERR_BAD_ARG;
  if (n_sys == 0) return VIBE_C_OK;
  if (thomas_sweeps<T>(n, n_sys)) return thomas_sweep_launch<T>(a, b, c, d, n, n_sys, x, status, (cudaStream_t)stream);
  DevScratch w(thomas_work<T>(n, n_sys) * sizeof(T), (cudaStream_t)stream);
  if (!w.get()) return VIBE_C_ERR_DEVICE;
  int rc = thomas_launch<T>(a, b, c, d, n, n_sys, x, (T*)w.get(), status, (cudaStream_t)stream);
  if (!w.release() && rc == VIBE_C_OK) rc = VIBE_C_ERR_DEVICE;
  return rc;
}

template <typename T>
int thomas_batched_host(const T* a, const T* b, const T* c, const T* d, int n, int n_sys, T* x) {
  if (n <= 0 || n_sys < 0 || b == nullptr || d == nullptr || x == nullptr) return VIBE_C_ERR_BAD_ARG;
  if (n_sys == 0) return VIBE_C_OK;
  const size_t e = sizeof(T), nn = (size_t)n * n_sys, no = (size_t)(n - 1) * n_sys;
  HostCall hc;
  const int ia = hc.add(a, no * e, HostCall::kIn), ib = hc.add(b, nn * e, HostCall::kIn);
  const int ic = hc.add(c, no * e, HostCall::kIn), id = hc.add(d, nn * e, HostCall::kIn);
  // x comes back through the staging buffer and is copied out only for the
  // systems that solved: a failed system's x stays as it was, as in the
  // reference, which returns before it writes x (c_kernels.c:26,34,40)
  const int ix = hc.add(nullptr, nn * e, HostCall::kOut);
  const int is = hc.add(nullptr, (size_t)n_sys * sizeof(int), HostCall::kOut);
  const int iw = hc.add(nullptr, thomas_work<T>(n, n_sys) * e, HostCall::kScratch);
  if (!hc.commit()) return VIBE_C_ERR_DEVICE;
  int rc = thomas_launch<T>(hc.dev<T>(ia), hc.dev<T>(ib), hc.dev<T>(ic), hc.dev<T>(id), n, n_sys, hc.dev<T>(ix),
                            hc.dev<T>(iw), hc.dev<int>(is), hc.stream());
  if (!hc.finish()) return VIBE_C_ERR_DEVICE;
  if (rc) return rc;
  const int* sv = (const int*)hc.host(is);
  const T* xv = (const T*)hc.host(ix);
  for (int q = 0; q < n_sys; ++q) {
    if (sv[q] == VIBE_C_OK)
      std::memcpy(x + (size_t)q * n, xv + (size_t)q * n, (size_t)n * e);
    else if (rc == VIBE_C_OK)
      rc = sv[q];
  }
  return rc;
}

template <typename T>
int weno_batched_dev(const T* q, size_t n, T* q_left, T* q_right, vibe_stream_t stream) {
  if (!q || !q_left || !q_right) return VIBE_C_ERR_BAD_ARG;
  if (n == 0) return VIBE_C_OK;
  const int blocks = (int)((n + 255) / 256 < 65535 ? (n + 255) / 256 : 65535);
  k_weno_batched<T><<<blocks, 256, 0, (cudaStream_t)stream>>>(q, n, q_left, q_right);
  return device_ok(cudaGetLastError(), "weno launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

template <typename T>
void weno_host(T qm2, T qm1, T q0, T q1, T q2, T* q_left, T* q_right) {
  if (q_left == nullptr || q_right == nullptr) return;
  const T q[5] = {qm2, qm1, q0, q1, q2};
  const size_t e = sizeof(T);
  HostCall hc;
  const int iq = hc.add(q, 5 * e, HostCall::kIn), il = hc.add(q_left, e, HostCall::kOut),
            ir = hc.add(q_right, e, HostCall::kOut);
  bool ok = hc.commit();
  ok = ok && weno_batched_dev<T>(hc.dev<T>(iq), 1, hc.dev<T>(il), hc.dev<T>(ir), (vibe_stream_t)hc.stream()) ==
                 VIBE_C_OK;
  ok = hc.finish() && ok;
  if (!ok) *q_left = *q_right = (T)NAN;
}

template <typename T>
T bilinear_host(const T* f, int halo, int nsx, int nsy, int nz, T xi, T yj, int k) {
  if (f == nullptr || nz <= 0) return (T)0;
  if (halo < 0 || nsx < halo + 1 || nsy < halo + 1) {  // the clamped point would lie outside the plane
    g_cerr = "bilinear: halo < 0 or a plane narrower than halo + 1";
    return (T)NAN;
  }
  if (k < 0) k = 0;
  if (k >= nz) k = nz - 1;
  const size_t plane = (size_t)nsx * nsy, e = sizeof(T);
  T r = (T)NAN;
  HostCall hc;
  const int ip = hc.add(f + (size_t)(k + halo) * plane, plane * e, HostCall::kIn), io = hc.add(&r, e, HostCall::kOut);
  bool ok = hc.commit();
  if (ok) {
    k_bilinear<T><<<1, 1, 0, hc.stream()>>>(hc.dev<T>(ip), halo, nsx, nsy, xi, yj, hc.dev<T>(io));
    ok = device_ok(cudaGetLastError(), "bilinear launch");
  }
  ok = hc.finish() && ok;
  return ok ? r : (T)NAN;
}

// From this many cells on the tiled scan is the faster one whatever the winds: FP64 by
// the divisions it saves (97 x 65 x 33, white noise 16 us against 30, nearly uniform 31 and
// 30; 40 x 30 x 20 14.6 and 16.8, 18.7 and 16.7), FP32 by memory (384 x 384 x 60 43 to 76
// against 78 to 109; 300 x 300 x 48 25 to 40 and 25 to 39, nearly uniform 31 and 25).
template <typename T>
constexpr size_t kCflCells = sizeof(T) == 8 ? (size_t)1 << 16 : (size_t)1 << 23;

template <typename T>
int cfl_launch(const T* u, const T* v, const T* w, const T* dzeta, const T* zs, int nx, int ny, int nz, T dx, T dy,
               T z_top, T dt, T* out3, T* part, cudaStream_t st) {
  const size_t ctiles = ((size_t)nx * ny + kCflThreads - 1) / kCflThreads;
  size_t tiles = ctiles * (((size_t)nz + kCflLevels - 1) / kCflLevels);
  int nb = (int)(tiles < 1 ? 1 : tiles < (size_t)kCflBlocks ? tiles : (size_t)kCflBlocks);
  if ((size_t)nx * ny * nz < kCflCells<T>) {
    nb = kCflBlocks / 2;
    k_cfl_cells<T><<<nb, kRedThreads, 0, st>>>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, part);
  } else if (sizeof(T) == 8 && tiles <= kCflBlocks / 2) {
    tiles = ctiles * (((size_t)nz + kCflLevels / 2 - 1) / (kCflLevels / 2));
    nb = (int)(tiles < (size_t)kCflBlocks ? tiles : (size_t)kCflBlocks);
    k_cfl_partial<T, kCflLevels / 2><<<nb, kCflThreads, 0, st>>>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, tiles, part);
  } else {
    k_cfl_partial<T, kCflLevels><<<nb, kCflThreads, 0, st>>>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, tiles, part);
  }
  k_cfl_final<T><<<1, kRedThreads, 0, st>>>(part, nb, out3);
  return device_ok(cudaGetLastError(), "cfl launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

template <typename T>
int cfl_dev(const T* u, const T* v, const T* w, const T* dzeta, const T* zs, int nx, int ny, int nz, T dx, T dy,
            T z_top, T dt, T* out3, vibe_stream_t stream) {
  if (!u || !v || !w || !dzeta || !out3 || nx < 0 || ny < 0 || nz < 0) return VIBE_C_ERR_BAD_ARG;
  DevScratch part((size_t)3 * kCflBlocks * sizeof(T), (cudaStream_t)stream);
  if (!part.get()) return VIBE_C_ERR_DEVICE;
  int rc = cfl_launch<T>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, out3, (T*)part.get(),
                         (cudaStream_t)stream);
  if (!part.release() && rc == VIBE_C_OK) rc = VIBE_C_ERR_DEVICE;
  return rc;
}

template <typename T>
T cfl_host(const T* u, const T* v, const T* w, const T* dzeta, const T* zs, int nx, int ny, int nz, T dx, T dy, T z_top,
           T dt, T* max_wind_out, T* min_dz_out) {
  if (u == nullptr || v == nullptr || w == nullptr || dzeta == nullptr) return (T)0;
  if (nx <= 0 || ny <= 0 || nz <= 0) {  // no cells: the reference's loops run zero times
    if (max_wind_out) *max_wind_out = (T)0;
    if (min_dz_out) *min_dz_out = (T)0;
    return (T)0;
  }
  const size_t e = sizeof(T);
  const size_t n = (size_t)nx * ny * nz, nzp = (size_t)nz, nxy = (size_t)nx * ny;
  T r[3] = {(T)NAN, (T)NAN, (T)NAN};
  HostCall hc;
  const int iu = hc.add(u, n * e, HostCall::kIn), iv = hc.add(v, n * e, HostCall::kIn),
            iw = hc.add(w, n * e, HostCall::kIn), iz = hc.add(dzeta, nzp * e, HostCall::kIn),
            izs = hc.add(zs, zs ? nxy * e : 0, HostCall::kIn), io = hc.add(r, 3 * e, HostCall::kOut),
            ip = hc.add(nullptr, (size_t)3 * kCflBlocks * e, HostCall::kScratch);
  bool ok = hc.commit();
  ok = ok && cfl_launch<T>(hc.dev<T>(iu), hc.dev<T>(iv), hc.dev<T>(iw), hc.dev<T>(iz), hc.dev<T>(izs), nx, ny, nz, dx,
                           dy, z_top, dt, hc.dev<T>(io), hc.dev<T>(ip), hc.stream()) == VIBE_C_OK;
  ok = hc.finish() && ok;
  if (!ok) return (T)NAN;
  if (max_wind_out) *max_wind_out = r[1];
  if (min_dz_out) *min_dz_out = r[2];
  return r[0];
}

template <typename T>
int neu_launch(const T* x, size_t n, T* out, T* part, cudaStream_t st) {
  // blocks of at least 2048 elements (8 a thread), at most kNeuBlocks
  const size_t want = (n + 2047) / 2048;
  const int nb = (int)(want < 1 ? 1 : want < (size_t)kNeuBlocks ? want : (size_t)kNeuBlocks);
  const size_t chunk = (n + nb - 1) / nb;
  k_neu_partial<T><<<nb, kNeuThreads, 0, st>>>(x, n, chunk > 0 ? chunk : 1, part);
  k_neu_final<T><<<1, kRedThreads, 0, st>>>(part, nb, out);
  return device_ok(cudaGetLastError(), "neumaier launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

template <typename T>
int neu_dev(const T* x, size_t n, T* out, vibe_stream_t stream) {
  if (!x || !out) return VIBE_C_ERR_BAD_ARG;
  DevScratch part((size_t)2 * kNeuBlocks * sizeof(T), (cudaStream_t)stream);
  if (!part.get()) return VIBE_C_ERR_DEVICE;
  int rc = neu_launch<T>(x, n, out, (T*)part.get(), (cudaStream_t)stream);
  if (!part.release() && rc == VIBE_C_OK) rc = VIBE_C_ERR_DEVICE;
  return rc;
}

template <typename T>
T neu_host(const T* x, size_t n) {
  if (x == nullptr) return (T)0;
  const size_t e = sizeof(T);
  T r = (T)NAN;
  HostCall hc;
  const int ix = hc.add(x, n * e, HostCall::kIn), io = hc.add(&r, e, HostCall::kOut),
            ip = hc.add(nullptr, (size_t)2 * kNeuBlocks * e, HostCall::kScratch);
  bool ok = hc.commit();
  ok = ok && neu_launch<T>(hc.dev<T>(ix), n, hc.dev<T>(io), hc.dev<T>(ip), hc.stream()) == VIBE_C_OK;
  ok = hc.finish() && ok;
  return ok ? r : (T)NAN;
}

// The tiled kernel where it is the faster one. FP64: it takes 75 ps a cell of its
// tiles, the cells beyond the grid included, and no less than 15 us (at least
// four levels a block in turn); a thread per cell takes 7 us and 130 ps a cell.
// Tiles against cells: 48 x 48 x 20 15.0 and 14.7 us, 96 x 96 x 10 14.9 and 19.0,
// 16 x 512 x 60 (half of each tile used) 82 and 70, 1 x 1000 x 40 97 and 15. FP32, bound by memory:
// 16 x 512 x 60 10.8 and 10.6, 3 x 4096 x 40 31 and 11, 384 x 384 x 60 82 and 117.
template <typename T>
bool flux_tiles(size_t tiles, int nz, size_t cells) {
  const size_t padded = tiles * kFluxCols * kFluxRows * nz;
  if (sizeof(T) == 4) return padded <= 2 * cells;
  return std::max(15.0, 7.5e-5 * (double)padded) <= 7.0 + 1.3e-4 * (double)cells;
}

template <typename T>
int flux_dev(const T* q, const T* rho, const T* u, const T* v, const T* w, const T* dzeta, const T* zs, int nx, int ny,
             int nz, T dx, T dy, T z_top, T* dqdt, vibe_stream_t stream) {
  if (!q || !rho || !u || !v || !w || !dzeta || !dqdt || nx < 0 || ny < 0 || nz < 0) return VIBE_C_ERR_BAD_ARG;
  const size_t n = (size_t)nx * ny * nz;
  if (n == 0) return VIBE_C_OK;
  // level chunks for about 24 blocks an SM, so that the last wave weighs little,
  // of at least 4 levels (a chunk computes its first lower face again)
  const int xt = (nx + kFluxCols - 1) / kFluxCols;
  const size_t tiles = (size_t)xt * ((ny + kFluxRows - 1) / kFluxRows);
  if (!flux_tiles<T>(tiles, nz, n)) {
    const int blocks = (int)((n + 255) / 256 < 65535 ? (n + 255) / 256 : 65535);
    k_flux_cell<T><<<blocks, 256, 0, (cudaStream_t)stream>>>(q, rho, u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dqdt);
    return device_ok(cudaGetLastError(), "flux advection launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
  }
  const int want = tiles >= 3648 ? 1 : (int)(3648 / tiles);
  int kz = (nz + want - 1) / want;
  if (kz < 4) kz = 4;
  if (kz < (nz + 65534) / 65535) kz = (nz + 65534) / 65535;
  k_flux_adv<T><<<dim3((unsigned)tiles, (nz + kz - 1) / kz), dim3(32, kFluxRows + 1), 0, (cudaStream_t)stream>>>(
      q, rho, u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dqdt, xt, kz);
  return device_ok(cudaGetLastError(), "flux advection launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

template <typename T>
void flux_host(const T* q, const T* rho, const T* u, const T* v, const T* w, const T* dzeta, const T* zs, int nx, int ny,
               int nz, T dx, T dy, T z_top, T* dqdt) {
  if (q == nullptr || rho == nullptr || u == nullptr || v == nullptr || w == nullptr || dzeta == nullptr ||
      dqdt == nullptr)
    return;
  if (nx <= 0 || ny <= 0 || nz <= 0) return;  // no cells: the reference's loops run zero times
  const size_t n = (size_t)nx * ny * nz, e = sizeof(T);
  HostCall hc;
  const int iq = hc.add(q, n * e, HostCall::kIn), ir = hc.add(rho, n * e, HostCall::kIn),
            iu = hc.add(u, n * e, HostCall::kIn), iv = hc.add(v, n * e, HostCall::kIn),
            iw = hc.add(w, n * e, HostCall::kIn), iz = hc.add(dzeta, (size_t)nz * e, HostCall::kIn),
            izs = hc.add(zs, zs ? (size_t)nx * ny * e : 0, HostCall::kIn), io = hc.add(dqdt, n * e, HostCall::kOut);
  bool ok = hc.commit();
  ok = ok && flux_dev<T>(hc.dev<T>(iq), hc.dev<T>(ir), hc.dev<T>(iu), hc.dev<T>(iv), hc.dev<T>(iw), hc.dev<T>(iz),
                         hc.dev<T>(izs), nx, ny, nz, dx, dy, z_top, hc.dev<T>(io), (vibe_stream_t)hc.stream()) ==
                 VIBE_C_OK;
  hc.finish();
}

}  // namespace

// ---- vgb_cabi: the call machinery declared in cabi_host.cuh ----
namespace vgb_cabi {

void set_error(const char* what, cudaError_t e) { device_ok(e, what); }
unsigned long long allocations() { return g_allocs.load(); }

HostCall::HostCall() {
  Ctx* c = ctx();
  ctx_ = c;
  ok_ = c != nullptr;
}

int HostCall::add(const void* h, size_t bytes, Kind kind) {
  Arg a{h, bytes, 0, kind, (kind == kIn || kind == kInOut) && h == nullptr};
  args_.push_back(a);
  return (int)args_.size() - 1;
}

cudaStream_t HostCall::stream() const { return ctx_ ? static_cast<Ctx*>(ctx_)->st : nullptr; }

// Layout in the device buffer: [inputs | in-outs | outputs | scratch]; the
// pinned buffer mirrors the first three regions. One copy moves
// [0, end of in-outs) to the device, one copy moves [in-outs, outputs) back.
bool HostCall::commit() {
  if (!ok_) return false;
  Ctx* c = static_cast<Ctx*>(ctx_);
  size_t off = 0;
  for (int k = kIn; k <= kScratch; ++k) {
    if (k == kInOut) d2h_beg_ = off;
    for (auto& a : args_)
      if (a.kind == k && !a.absent) {
        a.off = off;
        off = align256(off + a.bytes);
      }
    if (k == kInOut) h2d_end_ = off;
    if (k == kOut) d2h_end_ = off;
  }
  const size_t total = off > 0 ? off : 256;
  if (c->dbuf_n < total) {
    if (c->dbuf) cudaFree(c->dbuf);
    c->dbuf = nullptr;
    const size_t n = grown(c->dbuf_n, total);
    c->dbuf_n = 0;
    ++g_allocs;
    if (!device_ok(cudaMalloc(&c->dbuf, n), "cudaMalloc (staging)")) return ok_ = false;
    c->dbuf_n = n;
  }
  if (c->pin_n < d2h_end_) {
    if (c->pin) cudaFreeHost(c->pin);
    c->pin = nullptr;
    const size_t n = grown(c->pin_n, d2h_end_);
    c->pin_n = 0;
    ++g_allocs;
    if (!device_ok(cudaMallocHost(&c->pin, n), "cudaMallocHost (staging)")) return ok_ = false;
    c->pin_n = n;
  }
  base_ = c->dbuf;
  for (const auto& a : args_)
    if ((a.kind == kIn || a.kind == kInOut) && !a.absent && a.bytes) std::memcpy(c->pin + a.off, a.h, a.bytes);
  if (h2d_end_ && !device_ok(cudaMemcpyAsync(c->dbuf, c->pin, h2d_end_, cudaMemcpyHostToDevice, c->st), "H2D"))
    return ok_ = false;
  return true;
}

bool HostCall::finish() {
  if (!ctx_) return false;
  Ctx* c = static_cast<Ctx*>(ctx_);
  bool good = ok_;
  if (good && d2h_end_ > d2h_beg_)
    good = device_ok(cudaMemcpyAsync(c->pin + d2h_beg_, c->dbuf + d2h_beg_, d2h_end_ - d2h_beg_,
                                     cudaMemcpyDeviceToHost, c->st),
                     "D2H");
  // always wait: the staging buffers must be idle before the thread's next call
  good = device_ok(cudaStreamSynchronize(c->st), "sync") && good;
  if (good)
    for (const auto& a : args_)
      if ((a.kind == kInOut || a.kind == kOut) && a.h && a.bytes)
        std::memcpy(const_cast<void*>(a.h), c->pin + a.off, a.bytes);
  return ok_ = good;
}

const void* HostCall::host(int id) const {
  return ctx_ ? static_cast<Ctx*>(ctx_)->pin + args_[id].off : nullptr;
}

DevScratch::DevScratch(size_t bytes, cudaStream_t stream) : s_(stream) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (!device_ok(cudaStreamIsCapturing(stream, &cs), "cudaStreamIsCapturing")) return;
  if (cs != cudaStreamCaptureStatusNone) {  // inside a capture: graph-owned, stream-ordered memory
    graph_ = true;
    if (!device_ok(cudaMallocAsync(&p_, bytes > 0 ? bytes : 256, stream), "cudaMallocAsync (captured scratch)"))
      p_ = nullptr;
    return;
  }
  Ctx* c = ctx();
  if (!c) return;
  if (c->scr_n < bytes) {
    // the old buffer goes once its last user has finished
    if (c->has_last && !device_ok(cudaEventSynchronize(c->last), "scratch wait")) return;
    if (c->scr) cudaFree(c->scr);
    c->scr = nullptr;
    const size_t n = grown(c->scr_n, bytes);
    c->scr_n = 0;
    ++g_allocs;
    if (!device_ok(cudaMalloc(&c->scr, n), "cudaMalloc (scratch)")) return;
    c->scr_n = n;
  }
  // after the previous user of this thread's scratch, whatever its stream
  if (c->has_last && !device_ok(cudaStreamWaitEvent(stream, c->last, 0), "scratch order")) return;
  p_ = c->scr;
}

bool DevScratch::release() {
  if (released_) return p_ != nullptr;
  released_ = true;
  if (!p_) return false;
  if (graph_) return device_ok(cudaFreeAsync(p_, s_), "cudaFreeAsync (captured scratch)");
  Ctx* c = ctx();
  if (!c) return false;
  if (!device_ok(cudaEventRecord(c->last, s_), "scratch record")) return false;
  c->has_last = true;
  return true;
}

DevScratch::~DevScratch() {
  if (!released_) release();
}

}  // namespace vgb_cabi

extern "C" {

const char* vibe_c_last_error(void) { return g_cerr.c_str(); }

unsigned long long vibe_c_allocations(void) { return vgb_cabi::allocations(); }

// ---- FP64: the reference's names ----
int vibe_tridiagonal_solve_batched_f64_dev(const double* a, const double* b, const double* c, const double* d, int n,
                                           int n_sys, double* x, int* status, vibe_stream_t stream) {
  return thomas_batched_dev<double>(a, b, c, d, n, n_sys, x, status, stream);
}

int vibe_tridiagonal_solve_batched_f64_dev_noalloc(const double* a, const double* b, const double* c,
                                                   const double* d, int n, int n_sys, double* x, int* status,
                                                   vibe_stream_t stream) {
  if (n <= 0 || n_sys < 0 || b == nullptr || d == nullptr || x == nullptr) return VIBE_C_ERR_BAD_ARG;
  if ((size_t)n * (size_t)n_sys > kNoAllocThomasDoubles) {
    g_cerr = "vibe_tridiagonal_solve_batched_f64_dev_noalloc: n * n_sys = " + std::to_string((size_t)n * n_sys) +
             " exceeds the fixed workspace of " + std::to_string(kNoAllocThomasDoubles) + " doubles";
    return VIBE_C_ERR_BAD_ARG;
  }
  if (n_sys == 0) return VIBE_C_OK;
  const int dev = cur_dev();
  if (dev < 0 || dev >= 64) { g_cerr = "device ordinal out of range"; return VIBE_C_ERR_DEVICE; }
  double* work = nullptr;
  {
    // set-up on the first call per device, of any size (a later call may be
    // captured): resolve the array's device address
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
      void* p = nullptr;
      if (!device_ok(cudaGetSymbolAddress(&p, g_noalloc_thomas_work), "cudaGetSymbolAddress")) return VIBE_C_ERR_DEVICE;
      g_noalloc_ptr[dev] = (double*)p;
    }
    work = g_noalloc_ptr[dev];
  }
  if (Sweep<double>::smem(n) <= kSweepSmem)  // on chip: the workspace is not needed
    return thomas_sweep_launch<double>(a, b, c, d, n, n_sys, x, status, (cudaStream_t)stream);
  // the workspace needs no clearing: every system writes cp[k] before it reads it
  k_thomas_batched<double><<<(n_sys + 127) / 128, 128, 0, (cudaStream_t)stream>>>(a, b, c, d, n, n_sys, x, work,
                                                                                 status);
  return device_ok(cudaGetLastError(), "thomas (no-alloc) launch") ? VIBE_C_OK : VIBE_C_ERR_DEVICE;
}

int vibe_tridiagonal_solve_batched_f64(const double* a, const double* b, const double* c, const double* d, int n,
                                       int n_sys, double* x) {
  return thomas_batched_host<double>(a, b, c, d, n, n_sys, x);
}

int vibe_tridiagonal_solve_f64(const double* a, const double* b, const double* c, const double* d, int n, double* x,
                               double* ws) {
  if (n <= 0 || b == nullptr || d == nullptr || x == nullptr || ws == nullptr) return VIBE_C_ERR_BAD_ARG;
  return thomas_batched_host<double>(a, b, c, d, n, 1, x);
}

int vibe_weno5_reconstruct_batched_f64_dev(const double* q, size_t n, double* q_left, double* q_right,
                                           vibe_stream_t stream) {
  return weno_batched_dev<double>(q, n, q_left, q_right, stream);
}

void vibe_weno5_reconstruct_f64(double qm2, double qm1, double q0, double q1, double q2, double* q_left,
                                double* q_right) {
  weno_host<double>(qm2, qm1, q0, q1, q2, q_left, q_right);
}

double vibe_bilinear_f64(const double* f, int halo, int nsx, int nsy, int nz, double xi, double yj, int k) {
  return bilinear_host<double>(f, halo, nsx, nsy, nz, xi, yj, k);
}

int vibe_cfl_scan_f64_dev(const double* u, const double* v, const double* w, const double* dzeta, const double* zs,
                          int nx, int ny, int nz, double dx, double dy, double z_top, double dt, double* out3,
                          vibe_stream_t stream) {
  return cfl_dev<double>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, out3, stream);
}

double vibe_cfl_scan_f64(const double* u, const double* v, const double* w, const double* dzeta, const double* zs,
                         int nx, int ny, int nz, double dx, double dy, double z_top, double dt, double* max_wind_out,
                         double* min_dz_out) {
  return cfl_host<double>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, max_wind_out, min_dz_out);
}

int vibe_neumaier_sum_f64_dev(const double* x, size_t n, double* out, vibe_stream_t stream) {
  return neu_dev<double>(x, n, out, stream);
}

double vibe_neumaier_sum_f64(const double* x, size_t n) { return neu_host<double>(x, n); }

int vibe_advect_scalar_flux_f64_dev(const double* q, const double* rho, const double* u, const double* v,
                                    const double* w, const double* dzeta, const double* zs, int nx, int ny, int nz,
                                    double dx, double dy, double z_top, double* dqdt, vibe_stream_t stream) {
  return flux_dev<double>(q, rho, u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dqdt, stream);
}

void vibe_advect_scalar_flux_f64(const double* q, const double* rho, const double* u, const double* v, const double* w,
                                 const double* dzeta, const double* zs, int nx, int ny, int nz, double dx, double dy,
                                 double z_top, double* dqdt) {
  flux_host<double>(q, rho, u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dqdt);
}

// ---- FP32 twins ----
int vibe_tridiagonal_solve_f32(const float* a, const float* b, const float* c, const float* d, int n, float* x,
                               float* ws) {
  if (n <= 0 || b == nullptr || d == nullptr || x == nullptr || ws == nullptr) return VIBE_C_ERR_BAD_ARG;
  return thomas_batched_host<float>(a, b, c, d, n, 1, x);
}
int vibe_tridiagonal_solve_batched_f32(const float* a, const float* b, const float* c, const float* d, int n,
                                       int n_sys, float* x) {
  return thomas_batched_host<float>(a, b, c, d, n, n_sys, x);
}
int vibe_tridiagonal_solve_batched_f32_dev(const float* a, const float* b, const float* c, const float* d, int n,
                                           int n_sys, float* x, int* status, vibe_stream_t stream) {
  return thomas_batched_dev<float>(a, b, c, d, n, n_sys, x, status, stream);
}
void vibe_weno5_reconstruct_f32(float qm2, float qm1, float q0, float q1, float q2, float* q_left, float* q_right) {
  weno_host<float>(qm2, qm1, q0, q1, q2, q_left, q_right);
}
int vibe_weno5_reconstruct_batched_f32_dev(const float* q, size_t n, float* q_left, float* q_right,
                                           vibe_stream_t stream) {
  return weno_batched_dev<float>(q, n, q_left, q_right, stream);
}
float vibe_bilinear_f32(const float* f, int halo, int nsx, int nsy, int nz, float xi, float yj, int k) {
  return bilinear_host<float>(f, halo, nsx, nsy, nz, xi, yj, k);
}
float vibe_cfl_scan_f32(const float* u, const float* v, const float* w, const float* dzeta, const float* zs, int nx,
                        int ny, int nz, float dx, float dy, float z_top, float dt, float* max_wind_out,
                        float* min_dz_out) {
  return cfl_host<float>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, max_wind_out, min_dz_out);
}
int vibe_cfl_scan_f32_dev(const float* u, const float* v, const float* w, const float* dzeta, const float* zs, int nx,
                          int ny, int nz, float dx, float dy, float z_top, float dt, float* out3, vibe_stream_t stream) {
  return cfl_dev<float>(u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dt, out3, stream);
}
float vibe_neumaier_sum_f32(const float* x, size_t n) { return neu_host<float>(x, n); }
int vibe_neumaier_sum_f32_dev(const float* x, size_t n, float* out, vibe_stream_t stream) {
  return neu_dev<float>(x, n, out, stream);
}
void vibe_advect_scalar_flux_f32(const float* q, const float* rho, const float* u, const float* v, const float* w,
                                 const float* dzeta, const float* zs, int nx, int ny, int nz, float dx, float dy,
                                 float z_top, float* dqdt) {
  flux_host<float>(q, rho, u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dqdt);
}
int vibe_advect_scalar_flux_f32_dev(const float* q, const float* rho, const float* u, const float* v, const float* w,
                                    const float* dzeta, const float* zs, int nx, int ny, int nz, float dx, float dy,
                                    float z_top, float* dqdt, vibe_stream_t stream) {
  return flux_dev<float>(q, rho, u, v, w, dzeta, zs, nx, ny, nz, dx, dy, z_top, dqdt, stream);
}

}  // extern "C"
