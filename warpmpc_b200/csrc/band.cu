// Band form of the persistent ADMM iterations (sm_100a); tables in band.cuh.
//
// One CTA walks 32-instance tiles (lane = instance).  The chain warp runs the
// serial part of both sweeps over the chain; a producer warp streams the chain's
// L into a shared-memory ring; the other warps, the item warps, do everything
// that needs no order: per iteration, in the B phase (beside the backward sweep)
// each subtree of the head is solved as soon as the chain rows it reads are
// final, its indices take their ADMM update and its root's next forward result
// is formed; in the F phase (beside the next forward sweep) each chain row takes
// its ADMM update and subtracts its head entries from its next right-hand side.
// Only chain rows and root results stay in shared memory; head entries of L are
// read once per sweep direction, the chain's entries are stored once and read by
// both sweeps.
//
// What bounds it: the chain's latency and the items' shared-memory loads, about
// alike.  Per column the forward sweep's updates of the window are independent
// of one another, the backward sweep's sum is a serial chain of additions (the
// reference's order starts with the row solved last): alone on an SM a 16-row
// column takes 82 and 99 cycles, a third of the launch's time per column.  HBM is
// behind (0.66 of the copy rate with a tile on every SM; 65,536 instances of the
// 30-step quadrotor class: 3.27 MB per tile and iteration, 26 ms at the copy rate).
// ADMM of 25 iterations, this form against the streaming form: 2.68 against 5.37
// ms for one instance, 40.0 against 58.8 ms for 65,536; 1.07 against 2.15 ms for 97 of the 50-step
// cartpole class.  Measured and left: all items' copies from one producer warp
// (a bulk copy costs it some 500 cycles with its handshakes: 3.2 ms at one
// instance, 46.6 ms at 65,536), L loaded two columns ahead (3.4 ms: its
// registers are the item warps'), 9, 12 or (with spilled registers) 15 item warps
// for the 16-row window (3.07, 2.72, 3.48 ms); a second CTA per SM for the 50-step
// cartpole class with rings of little more than an item (16,384 instances, two
// solves, 9.7 ms against 9.3).
//
// Arithmetic is the reference's operation order (warp_backend.py:176-218,
// solver.py:806-820), every product and sum rounded separately.  Padding
// entries are L = 0: where they stand for a row outside the column they add
// (+-0) to a sum, which changes no value; an instance whose iterate has
// overflowed may turn an infinity into a NaN there (its status is NONFINITE
// either way).
#include <algorithm>
#include <type_traits>
#include <vector>

#include "band.cuh"
#include "common.cuh"
#include "osqp.cuh"

namespace wmpc {

namespace {

constexpr int kMaxBandJobs = 6;
constexpr uint64_t kBandWaitNs = 2000000000ull;

struct BandJob {
  BandPlan bp;
  float* stream;
  float* pres;
  int* iters;
  const float* rho_b;
  const int* rho_count;
  int max_iter, batch, check_every, m;
  float chg_eps, sigma, alpha, oma;
};

struct BandArgs {
  BandJob job[kMaxBandJobs];
  int tile_end[kMaxBandJobs];
  int n_jobs, warps, stages;  // item warps, chain stages
  int vrows, yrows, t4, n_chunks, n_items, chunk_bytes, ring_bytes, maxima_sets;
  int* error;
  unsigned long long wait_limit_ns;
};

static_assert(sizeof(BandArgs) <= 4000, "launch arguments exceed the kernel parameter space");

// Bounded waits that read the clock only once they have polled for a while
// (a read of the global timer takes longer than most of these waits).
// After limit_ns, or when another warp gave up, they return false.  kSpins
// polls in a row, then one every kSleep ns: the chain warp spins, the producers
// (which share its scheduler and are a stage ahead) do not.
template <int kSpins = 16, int kSleep = 20, typename Done>
__device__ __forceinline__ bool band_poll(Done done, const volatile int* abort, uint64_t limit_ns) {
  for (int i = 0; i < kSpins; ++i)
    if (done()) return true;
  uint64_t start = 0;
  for (uint32_t i = 0;; ++i) {
    __nanosleep(kSleep);
    if (done()) return true;
    if ((i & 31u) == 0) {
      const uint64_t now = global_timer_ns();
      if (i == 0) start = now;
      if ((abort && *abort) || now - start > limit_ns) return false;
    }
  }
}

template <int kSpins = 16, int kSleep = 20>
__device__ __forceinline__ bool band_wait_count(const unsigned* ctr, unsigned target, const volatile int* abort,
                                                uint64_t limit_ns) {
  return band_poll<kSpins, kSleep>([&] { return ld_acquire_cta(ctr) >= target; }, abort, limit_ns);
}

template <int kSpins = 16, int kSleep = 20>
__device__ __forceinline__ bool band_wait_full(uint64_t* bar, uint32_t parity, const volatile int* abort,
                                               uint64_t limit_ns) {
  return band_poll<kSpins, kSleep>([&] { return mbar_try_wait(bar, parity); }, abort, limit_ns);
}

__device__ __forceinline__ int band_job_of(const BandArgs& a, int g) {
  int c = 0;
  while (c + 1 < a.n_jobs && g >= a.tile_end[c]) ++c;
  return c;
}

// This lane's instance's rho by row class where its rho adapted (the rule of
// the rho update), else the records' values.
struct BandRho {
  bool on;
  float est;
};

struct BandUpd {
  float sigma, alpha, oma;
  bool frozen;
  BandRho rho;
  float chg, pres;
};

template <bool kRho>
__device__ __forceinline__ void band_rho(const BandUpd& u, int kind, float& rho, float& rinv) {
  if constexpr (kRho) {
    if (u.rho.on) {
      const int cls = (kind >> 1) - 1;
      rho = cls < 0 ? 1e-6f : (cls > 0 ? 1e3f * u.rho.est : u.rho.est);
      rinv = 1.0f / rho;
    }
  }
}

// The right-hand side of an index from its iterate (it) and parameters (par),
// both staged: sigma x - q, or z - y / rho.
template <bool kRho>
__device__ __forceinline__ float band_rhs(const BandUpd& u, int kind, float rinv, const unsigned char* it,
                                          const unsigned char* par, int lane) {
  if (kind & 1) {
    const float2 s = reinterpret_cast<const float2*>(it)[lane];
    float rho = 0.0f;
    band_rho<kRho>(u, kind, rho, rinv);
    return s.x - rinv * s.y;
  }
  return u.sigma * reinterpret_cast<const float*>(it)[lane] - reinterpret_cast<const float*>(par)[lane];
}

// ADMM update of one index given its KKT solution xs (solver.py:806-820); the
// new iterate goes to HBM, the next right-hand side is returned.  kTrack: the
// scaled primal residual follows the iterates exactly (A x~ = z~ from the KKT
// solve: e' = (z_relaxed - z') + (1 - alpha) e), and a frozen lane keeps its state.
// c: {rho, 1/rho, unscale, residual offset}; gs: the iterate's place in HBM, ge:
// the tile's residuals.
template <bool kTrack, bool kRho>
__device__ __forceinline__ float band_update(BandUpd& u, int kind, float xs, const float4& c, const unsigned char* it,
                                             const unsigned char* par, float* gs, float* ge, int lane) {
  if (kind & 1) {
    const float2 s = reinterpret_cast<const float2*>(it)[lane];
    const float2 b = reinterpret_cast<const float2*>(par)[lane];
    float rho = c.x, rinv = c.y;
    band_rho<kRho>(u, kind, rho, rinv);
    const float rz = s.x - rinv * s.y;
    const float zt = rz + rinv * xs;
    const float zr = u.alpha * zt + u.oma * s.x;
    float zn = zr + rinv * s.y;
    zn = (zn < b.x) ? b.x : zn;
    zn = (zn > b.y) ? b.y : zn;
    float yn = s.y + rho * (zr - zn);
    if constexpr (kTrack) {
      ge += __float_as_int(c.w);
      const float e = ge[lane];
      const float en = u.frozen ? e : (zr - zn) + u.oma * e;
      zn = u.frozen ? s.x : zn;
      yn = u.frozen ? s.y : yn;
      ge[lane] = en;
      u.pres = fmaxf(u.pres, fabsf(en) * c.z);
      u.chg = fmaxf(u.chg, fmaxf(fabsf(zn - s.x), fabsf(yn - s.y)) * c.z);
    }
    reinterpret_cast<float2*>(gs)[lane] = make_float2(zn, yn);
    return zn - rinv * yn;
  }
  const float x = reinterpret_cast<const float*>(it)[lane];
  float xn = u.alpha * xs + u.oma * x;
  if constexpr (kTrack) {
    xn = u.frozen ? x : xn;
    u.chg = fmaxf(u.chg, fabsf(xn - x) * c.z);
  }
  gs[lane] = xn;
  return u.sigma * xn - reinterpret_cast<const float*>(par)[lane];
}

// ---------------------------------------------------------------------------
// chain
// ---------------------------------------------------------------------------

// Columns per turn of the sweeps' inner loops (alone on an SM: 4 columns 82
// forward and 99 backward cycles per column with a 16-row window, 2 columns 88
// and 128).
constexpr int kTurn = 4;

__device__ __forceinline__ int comp4(const int4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// One column's window units (lst: this lane's 16 bytes of the chunk's first
// unit); the last one is zero where the column does not have it.
template <int MU>
__device__ __forceinline__ void chain_load(const unsigned char* lst, int word, float4 (&L)[MU]) {
  const unsigned char* p = lst + (word >> 1) * 512;
#pragma unroll
  for (int j = 0; j < MU - 1; ++j) L[j] = *reinterpret_cast<const float4*>(p + j * 512);
  L[MU - 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (word & 1) L[MU - 1] = *reinterpret_cast<const float4*>(p + (MU - 1) * 512);
}

// Forward over one chunk: column t's result y_t = A[0] is subtracted from the
// rows of its window (A: rows t .. t + 4 MU + kTurn - 1 of a turn), rows past it
// in shared memory, before they enter the window.  v: this lane's column of the
// work vector at row t0.
template <int MU, bool kFar>
__device__ __forceinline__ void chain_forward(float (&A)[4 * MU + kTurn], const unsigned char* stage, float* v,
                                              float* v0, const int* words, int cols, const int4* far, int n_far,
                                              int lane) {
  const unsigned char* lst = stage + lane * 16;
  float4 L[2][MU];
  int4 w = *reinterpret_cast<const int4*>(words);
  int f = 0;
  chain_load<MU>(lst, w.x, L[0]);
#pragma unroll 1
  for (int t = 0; t < cols; t += kTurn) {
    // (past the end: not used)
    const int4 wn = *reinterpret_cast<const int4*>(words + (t + kTurn < cols ? t + kTurn : 0));
#pragma unroll
    for (int p = 0; p < kTurn; ++p) {
      chain_load<MU>(lst, p < kTurn - 1 ? comp4(w, p + 1) : wn.x, L[(p + 1) & 1]);
      A[4 * MU + p] = v[(4 * MU + p) * 32];
      const float y = A[p];
#pragma unroll
      for (int j = 0; j < MU; ++j) {
        const float4 l = L[p & 1][j];
        A[p + 1 + 4 * j] = A[p + 1 + 4 * j] - l.x * y;
        A[p + 2 + 4 * j] = A[p + 2 + 4 * j] - l.y * y;
        A[p + 3 + 4 * j] = A[p + 3 + 4 * j] - l.z * y;
        A[p + 4 + 4 * j] = A[p + 4 + 4 * j] - l.w * y;
      }
      if constexpr (kFar) {
        for (; f < n_far && __ldg(far + f).x == t + p; ++f) {
          const int4 e = __ldg(far + f);
          float* q = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(v0) + e.y);
          *q = *q - *reinterpret_cast<const float*>(lst + e.z) * y;
        }
      }
    }
#pragma unroll
    for (int p = 0; p < kTurn; ++p) v[p * 32] = A[p];
#pragma unroll
    for (int i = 0; i < 4 * MU; ++i) A[i] = A[i + kTurn];
    w = wn;
    v += 32 * kTurn;
  }
}

// Backward over one chunk (W: rows t + kTurn .. t + 4 MU + kTurn - 1 of the turn
// at t): x_t = y_t D^-1_t - (0 + L x of the column's rows, ascending).
template <int MU, bool kFar>
__device__ __forceinline__ void chain_backward(float (&W)[4 * MU], const unsigned char* stage, int unit_bytes, float* v,
                                               const float* v0, const int* words, int cols, const int4* far, int n_far,
                                               int lane) {
  const unsigned char* lst = stage + lane * 16;
  const float* d = reinterpret_cast<const float*>(stage + unit_bytes) + lane;
  float4 L[2][MU];
  int4 w = *reinterpret_cast<const int4*>(words + cols - kTurn);
  int f1 = n_far;
  chain_load<MU>(lst, w.w, L[1]);
#pragma unroll 1
  for (int t = cols - kTurn; t >= 0; t -= kTurn) {
    const int4 wn = *reinterpret_cast<const int4*>(words + (t > 0 ? t - kTurn : 0));
    float* vt = v + t * 32;
    float X[kTurn], yd[kTurn];
#pragma unroll
    for (int p = 0; p < kTurn; ++p) yd[p] = vt[p * 32] * d[(t + p) * 32];
#pragma unroll
    for (int p = kTurn - 1; p >= 0; --p) {
      chain_load<MU>(lst, p > 0 ? comp4(w, p - 1) : wn.w, L[(p + 1) & 1]);
      float corr = 0.0f;
#pragma unroll
      for (int j = 0; j < MU; ++j) {
        const float4 l = L[p & 1][j];
        const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = p + 1 + 4 * j + e;  // row t + i
          corr = corr + lv[e] * (i < kTurn ? X[i < kTurn ? i : 0] : W[i < kTurn ? 0 : i - kTurn]);
        }
      }
      if constexpr (kFar) {
        int f0 = f1;
        while (f0 > 0 && __ldg(far + f0 - 1).x == t + p) --f0;
        for (int f = f0; f < f1; ++f) {
          const int4 e = __ldg(far + f);
          corr = corr + *reinterpret_cast<const float*>(lst + e.z) *
                            *reinterpret_cast<const float*>(reinterpret_cast<const unsigned char*>(v0) + e.y);
        }
        f1 = f0;
      }
      X[p] = yd[p] - corr;
      vt[p * 32] = X[p];
    }
#pragma unroll
    for (int i = 4 * MU - 1; i >= kTurn; --i) W[i] = W[i - kTurn];
#pragma unroll
    for (int p = 0; p < kTurn; ++p) W[p] = X[p];
    w = wn;
  }
}

// ---------------------------------------------------------------------------
// items
// ---------------------------------------------------------------------------

// sum (kAdd) or difference of init and the products of an item's units with the
// values its record points to (vec: this lane's column), in entry order; two
// units at a time, every load before the additions.
template <bool kAdd>
__device__ __forceinline__ float band_dot(float sum, int units, const int4* rows, const unsigned char* lu,
                                          const unsigned char* vec) {
  for (int e = 0; e < units; e += 2) {
    const bool two = e + 1 < units;
    const int4 r0 = rows[e], r1 = two ? rows[e + 1] : r0;
    const float4 l0 = *reinterpret_cast<const float4*>(lu + e * 512);
    float4 l1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (two) l1 = *reinterpret_cast<const float4*>(lu + e * 512 + 512);
    auto at = [&](int o) { return *reinterpret_cast<const float*>(vec + o); };
    const float x0 = at(r0.x), x1 = at(r0.y), x2 = at(r0.z), x3 = at(r0.w);
    float x4 = at(r1.x), x5 = at(r1.y), x6 = at(r1.z), x7 = at(r1.w);
    if (kAdd) {
      sum = sum + l0.x * x0;
      sum = sum + l0.y * x1;
      sum = sum + l0.z * x2;
      sum = sum + l0.w * x3;
    } else {
      sum = sum - l0.x * x0;
      sum = sum - l0.y * x1;
      sum = sum - l0.z * x2;
      sum = sum - l0.w * x3;
    }
    if (two) {
      if (kAdd) {
        sum = sum + l1.x * x4;
        sum = sum + l1.y * x5;
        sum = sum + l1.z * x6;
        sum = sum + l1.w * x7;
      } else {
        sum = sum - l1.x * x4;
        sum = sum - l1.y * x5;
        sum = sum - l1.z * x6;
        sum = sum - l1.w * x7;
      }
    }
  }
  return sum;
}

}  // namespace

// Shared memory: V [band_vrows][32] chain rows (right-hand side -> forward
// result -> solution, in place), zero rows, the pre-chain's solution |
// YR [n_yr + 1][32] the roots' and the pre-chain's forward results | chain
// ring | the item warps' rings | column words, chunk descriptors, item words |
// per-warp maxima (checks) | barriers | counters.
// (The producer keeps its table in shared memory: an arrival on a barrier waits
// for the loads before it, so a descriptor read ahead from global memory would
// cost its whole latency per copy.)
// Counters, all monotone over the launch: chain_done (chunks the backward
// sweeps finished), b_done (B phases finished, once per item warp), f_done
// (chain rows finished in F phases, per item warp), pre_b / pre_f (phases in
// which the pre-chain is solved / its right-hand sides are formed).  Waits: a
// B item for the chunks it reads, at least one; an F item for every B item (b_done)
// and the whole backward sweep; items that read pre-chain values for item warp 0,
// which does them first; a forward chunk for the F items of its rows and of
// the rows it adds to.  A backward sweep follows the whole forward sweep, so B
// items never overlap the F items of the phase before.
// Items belong to a warp for the whole solve: it writes their iterates with
// ordinary stores and copies them back itself an iteration later.
// Warps: 0 the chain, 4 its producer (on the same scheduler: 65,536 quadrotor
// instances 39.7 ms, with warp 1 in its place 41.0), the rest items.  (As many
// items as the registers allow: with two or three warps left idle so that the
// chain's scheduler issues for it alone, all cases took 2 to 7 % longer.)
// kWide: the launch has a class with a 16-row window, whose chain code needs 128
// registers.
constexpr int kProducerWarp = 4;

template <bool kTrack, bool kRho, bool kWide>
__global__ void __launch_bounds__(kWide ? 512 : 640, 1) band_admm_kernel(const __grid_constant__ BandArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, K = a.warps;
  float* V = reinterpret_cast<float*>(smem);
  float* YR = V + (size_t)a.vrows * 32;
  unsigned char* ring = reinterpret_cast<unsigned char*>(YR + (size_t)a.yrows * 32);
  unsigned char* stages = ring + (size_t)a.stages * a.chunk_bytes;
  int* colw = reinterpret_cast<int*>(stages + (size_t)K * a.ring_bytes);
  int4* chunkw = reinterpret_cast<int4*>(reinterpret_cast<unsigned char*>(colw) + (a.t4 * 4 + 15) / 16 * 16);
  int2* pchunk = reinterpret_cast<int2*>(chunkw + a.n_chunks);  // the chain producer's {offset, bytes | columns << 24}
  unsigned* itemw = reinterpret_cast<unsigned*>(pchunk + a.n_chunks);
  float* maxima = reinterpret_cast<float*>(itemw + (K * a.n_items + 1) / 2 * 2);  // [maxima_sets][K][2][32]
  uint64_t* cfull = reinterpret_cast<uint64_t*>(maxima + a.maxima_sets * K * 64);
  uint64_t* cempty = cfull + a.stages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(cempty + a.stages);
  unsigned* chain_done = reinterpret_cast<unsigned*>(cempty + a.stages) + 1;
  unsigned* b_done = chain_done + 1;
  unsigned* pre_b = chain_done + 2;
  unsigned* pre_f = chain_done + 3;
  // tiles (of this CTA) before this one are over; [stages] tile ordinal of a stage's copy; [K]
  volatile int* skip_to = reinterpret_cast<volatile int*>(chain_done + 4);
  volatile int* tag = reinterpret_cast<volatile int*>(chain_done + 5);
  unsigned* f_done = chain_done + 5 + a.stages;
  const int total = a.tile_end[a.n_jobs - 1];
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * a.stages; ++s) mbar_init(cfull + s, 1);
    *abort_flag = 0;
    *chain_done = 0;
    *b_done = 0;
    *pre_b = 0;
    *pre_f = 0;
    *skip_to = 0;
    for (int w = 0; w < K; ++w) f_done[w] = 0;
    fence_mbarrier_init();
  }
  __syncthreads();
  bool ok = true;
  // chain rows of the phases counted so far, per item warp (lane w: warp w's
  // share), and the rows of the current phase known to be done
  unsigned f_base = 0;
  int f_ready = 0;
  auto f_share = [&](int rows, int w) { return w < K && rows > w ? (unsigned)((rows - w + K - 1) / K) : 0u; };
  auto wait_f = [&](int need) -> bool {  // until the first `need` rows of the phase are done
    if (f_ready >= need) return true;
    const unsigned* ctr = f_done + (lane < K ? lane : 0);
    return band_poll(
        [&] {
          const int next = lane < K ? lane + (int)(ld_acquire_cta(ctr) - f_base) * K : 0x7fffffff;
          f_ready = __reduce_min_sync(0xffffffffu, next);
          return f_ready >= need;
        },
        abort_flag, a.wait_limit_ns);
  };
  auto next_phase = [&](int rows) {
    f_base += f_share(rows, lane);
    f_ready = 0;
  };
  // what a lane's termination decisions are made of: its largest iterate
  // change and primal residual over the iteration, over all item warps
  bool frozen = false;
  int frozen_at = 0;
  auto maxima_of = [&](int it) { return maxima + (a.maxima_sets > 1 ? (it & 1) * K * 64 : 0); };
  auto decide = [&](const BandJob& J, int it) -> bool {
    const float* all = maxima_of(it);
    float chg = 0.0f, pres = 0.0f;
    for (int w = 0; w < K; ++w) {
      chg = fmaxf(chg, all[w * 64 + lane]);
      pres = fmaxf(pres, all[w * 64 + 32 + lane]);
    }
    if (!frozen && chg <= J.chg_eps && pres <= J.chg_eps) {
      frozen = true;
      frozen_at = it;
    }
    return __all_sync(0xffffffffu, frozen);
  };
  auto check_at = [&](const BandJob& J, int it) {
    return kTrack && J.check_every > 0 && it > 0 && it % J.check_every == 0 && it < J.max_iter;
  };

  if (warp == 0) {
    // ------------------------------ chain ------------------------------
    int stage = 0, have = -1, ordinal = 0;
    uint32_t phase = 0;
    unsigned done = 0;
    auto used = [&]() {  // the current stage has been read
      __syncwarp();
      if (lane == 0) mbar_arrive(cempty + stage);
      if (++stage == a.stages) {
        stage = 0;
        phase ^= 1u;
      }
    };
    for (int g = blockIdx.x; g < total && ok; g += gridDim.x) {
      const int c = band_job_of(a, g);
      const BandJob& J = a.job[c];
      const BandPlan& bp = J.bp;
      if (J.max_iter <= 0) continue;
      ++ordinal;
      if (have != c) {  // the class's tables
        for (int i = lane; i < bp.T4; i += 32) colw[i] = __ldg(bp.col_word + i);
        for (int i = lane; i < bp.n_chunks; i += 32) chunkw[i] = __ldg(bp.chunk + i);
        __syncwarp();
        have = c;
      }
      frozen = false;
      float* v = V + lane;
      const int n_chunks = bp.n_chunks, cc = bp.chunk_cols;
      bool stop = false;
      // both sweeps of every iteration; MU: the class's window units
      auto sweeps = [&](auto units) {
        constexpr int MU = decltype(units)::value;
        for (int it = 0; it < J.max_iter; ++it) {
          {
            float A[4 * MU + kTurn];
            for (int ch = 0; ch < n_chunks; ++ch) {
              const int4 cd = chunkw[ch];
              if (!wait_f(cd.w) || !band_wait_full(cfull + stage, phase, abort_flag, a.wait_limit_ns)) {
                ok = false;
                return;
              }
              if (ch == 0) {
#pragma unroll
                for (int i = 0; i < 4 * MU; ++i) A[i] = v[i * 32];
              }
              const unsigned char* st = ring + (size_t)stage * a.chunk_bytes;
              const int* words = colw + ch * cc;
              const int n_far = cd.z >> 8;
              if (n_far == 0)
                chain_forward<MU, false>(A, st, v + ch * cc * 32, v, words, cd.z, nullptr, 0, lane);
              else
                chain_forward<MU, true>(A, st, v + ch * cc * 32, v, words, cd.z & 255, bp.far + __ldg(bp.far_ptr + ch),
                                        n_far, lane);
              used();
            }
          }
          next_phase(bp.T);
          if (check_at(J, it) && decide(J, it)) {  // (it iterations are complete once their F items are)
            stop = true;
            return;
          }
          float W[4 * MU];
#pragma unroll
          for (int i = 0; i < 4 * MU; ++i) W[i] = 0.0f;
          for (int ch = n_chunks - 1; ch >= 0; --ch) {
            const int4 cd = chunkw[ch];
            if (!band_wait_full(cfull + stage, phase, abort_flag, a.wait_limit_ns)) {
              ok = false;
              return;
            }
            const unsigned char* st = ring + (size_t)stage * a.chunk_bytes;
            const int* words = colw + ch * cc;
            const int n_far = cd.z >> 8;
            if (n_far == 0)
              chain_backward<MU, false>(W, st, cd.y, v + ch * cc * 32, v, words, cd.z, nullptr, 0, lane);
            else
              chain_backward<MU, true>(W, st, cd.y, v + ch * cc * 32, v, words, cd.z & 255,
                                       bp.far + __ldg(bp.far_ptr + ch), n_far, lane);
            ++done;
            used();
            if (lane == 0) st_release_cta(chain_done, done);
          }
        }
      };
      if constexpr (kWide) {
        if (bp.units == 2)
          sweeps(std::integral_constant<int, 2>{});
        else
          sweeps(std::integral_constant<int, 4>{});
      } else {
        sweeps(std::integral_constant<int, 2>{});
      }
      if (!ok) break;
      if (stop) {
        // leave the tile: the producer moves on to the next one, the copies it
        // made for this one's remaining sweeps are dropped, and one count past
        // the sweeps' tells the item warps that the work vector is free
        if (lane == 0) *skip_to = ordinal + 1;
        ++done;
        __syncwarp();
        if (lane == 0) st_release_cta(chain_done, done);
        for (;;) {
          if (!band_wait_full(cfull + stage, phase, abort_flag, a.wait_limit_ns)) {
            ok = false;
            break;
          }
          if (tag[stage] > ordinal) break;
          used();
        }
      } else {
        next_phase(bp.T);  // the last iteration's F items (updates only)
      }
    }
    if (!ok && lane == 0) *abort_flag = 1;
  } else if (warp == kProducerWarp) {
    // -------------------------- chain producer --------------------------
    uint32_t issued = 0;
    int stage = 0, ordinal = 0, have = -1;
    uint32_t phase = 1;  // (a fresh barrier's previous phase counts as complete)
    // the next stage, free; tagged
    auto acquire = [&](int t) -> bool {
      if (!band_wait_full<1, 150>(cempty + stage, phase, abort_flag, a.wait_limit_ns)) return false;
      if (lane == 0) tag[stage] = t;
      return true;
    };
    auto next = [&]() {
      ++issued;
      if (++stage == a.stages) {
        stage = 0;
        phase ^= 1u;
      }
    };
    for (int g = blockIdx.x; g < total && ok; g += gridDim.x) {
      const int c = band_job_of(a, g);
      const BandJob& J = a.job[c];
      if (J.max_iter <= 0) continue;
      ++ordinal;
      const int n = J.bp.n_chunks, max_iter = J.max_iter;
      if (have != c) {
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
          const int4 d = __ldg(J.bp.chunk + i);
          pchunk[i] = make_int2(d.x, d.y | (d.z & 255) << 24);
        }
        __syncwarp();
        have = c;
      }
      const float* base = J.stream + (size_t)(g - (c ? a.tile_end[c - 1] : 0)) * J.bp.blen;
      bool skipped = false;
      for (int it = 0; it < max_iter && ok && !skipped; ++it)
        for (int k = 0; k < 2 * n; ++k) {  // forward, then backward
          const int2 d = pchunk[k < n ? k : 2 * n - 1 - k];
          if (!acquire(ordinal)) {
            ok = false;
            break;
          }
          if (kTrack && *skip_to > ordinal) {
            skipped = true;
            break;
          }
          const uint32_t bytes = (uint32_t)(d.y & 0xffffff) + (k < n ? 0u : ((uint32_t)d.y >> 24) * 128u);
          if (lane == 0) {
            mbar_arrive_expect_tx(cfull + stage, bytes);
            bulk_g2s(ring + (size_t)stage * a.chunk_bytes, base + d.x, bytes, cfull + stage);
          }
          next();
        }
    }
    // a stage without a copy ends the sequence (a tile that stops early looks for what follows it)
    const uint32_t copies = issued;
    const int last_stage = stage;
    if (kTrack && ok && acquire(0x7fffffff) && lane == 0) mbar_arrive(cfull + last_stage);
    if (!ok && lane == 0) *abort_flag = 1;
    // the last copies have landed before the CTA may leave (bounded)
    for (uint32_t s = 0; s < (uint32_t)a.stages && s < copies; ++s) {
      const uint32_t last = s + (uint32_t)a.stages * ((copies - 1 - s) / (uint32_t)a.stages);
      if (!(kTrack && ok && (int)s == last_stage))
        band_wait_full(cfull + s, (last / (uint32_t)a.stages) & 1u, nullptr, kBandWaitNs);
    }
  } else {
    // ------------------------------ items ------------------------------
    const int iw = warp - 1 - (warp > kProducerWarp);
    int have = -1;
    unsigned chunks = 0, phases = 0;  // chain chunks and B phases of the phases gone by
    unsigned chain_seen = 0;          // counter as last read
    unsigned char* mine = stages + (size_t)iw * a.ring_bytes;
    unsigned* words = itemw + iw * a.n_items;  // this warp's items of an iteration, B then F
    auto seen = [&](const unsigned* ctr, unsigned& last, unsigned target) -> bool {
      if (last >= target) return true;
      return band_poll<2, 100>([&] { return (last = ld_acquire_cta(ctr)) >= target; }, abort_flag, a.wait_limit_ns);
    };
    for (int g = blockIdx.x; g < total && ok; g += gridDim.x) {
      const int c = band_job_of(a, g);
      const BandJob& J = a.job[c];
      const BandPlan& bp = J.bp;
      const int tile = g - (c ? a.tile_end[c - 1] : 0);
      float* stream = J.stream + (size_t)tile * bp.blen;
      float* pres = kTrack ? J.pres + (size_t)tile * J.m * 32 : nullptr;
      frozen = false;
      frozen_at = 0;
      int it_run = J.max_iter > 0 ? J.max_iter : 0;
      if (J.max_iter > 0) {
        BandUpd u{J.sigma, J.alpha, J.oma, false, {false, 0.0f}, 0.0f, 0.0f};
        if constexpr (kRho) {
          const int b = tile * 32 + lane, bb = b < J.batch ? b : J.batch - 1;
          u.rho.on = J.rho_count[bb] > 0;
          u.rho.est = J.rho_b[bb];
        }
        // this warp's items: every K-th subtree and chain row; item warp 0
        // has the pre-chain's columns and rows before them
        const int n_pre = iw == 0 ? bp.n_pre : 0;
        const int mb = n_pre + (bp.nb > iw ? (bp.nb - iw + K - 1) / K : 0);
        const int mf = n_pre + (bp.T > iw ? (bp.T - iw + K - 1) / K : 0);
        const int per_it = mb + mf;
        // the items of an iteration in this warp's order, copied ahead as far as
        // they fit into its ring; each lies there in one piece (at the end of the
        // one before or, where it would not fit, at the start).  An item's copy
        // follows its release in the iteration before.
        if (have != c) {
          __syncwarp();
          for (int i = lane; i < per_it; i += 32) {
            const int first = i < mb ? 0 : bp.n_pre + bp.nb, j = i < mb ? i : i - mb;
            words[i] = (unsigned)__ldg(bp.item + first + (j < n_pre ? j : bp.n_pre + iw + (j - n_pre) * K));
          }
          __syncwarp();
          have = c;
        }
        const int depth = per_it < kBandAhead ? per_it : kBandAhead;
        const bool fence = band_item_fence(mb, mf);
        int next_i = 0, next_it = 0;                // the next one to copy
        int head = 0, tail = 0, flying = 0, size = 0;  // the oldest one and its size, the end of the newest, how many
        bool wrapped = false;                       // the newest lies before the oldest
        const unsigned char* rec = mine;            // the current item
        auto fill = [&]() {
          while (flying < depth && next_it <= J.max_iter) {
            const unsigned w = words[next_i];
            const int bytes = (int)(w >> 22) * 128;
            int at = tail;
            if (wrapped) {
              if (at + bytes > head) break;
            } else if (at + bytes > a.ring_bytes) {
              if (bytes > head) break;
              at = 0;
              wrapped = true;
            }
            const float* src = stream + (size_t)(w & 0x3fffffu) * 32 + lane * 4;
            unsigned char* dst = mine + at + lane * 16;
            for (int k = lane * 16; k < bytes; k += 512) {
              cp_async16(dst, src);
              dst += 512;
              src += 128;
            }
            cp_async_commit();
            tail = at + bytes;
            ++flying;
            if (++next_i == per_it) {
              next_i = 0;
              ++next_it;
            }
          }
        };
        fill();
        static_assert(kBandAhead == 4, "take() counts copies in flight up to four");
        auto take = [&](int i) {
          size = (int)(words[i] >> 22) * 128;
          if (head + size > a.ring_bytes) {
            head = 0;
            wrapped = false;
          }
          if (flying >= 4) cp_async_wait_group<3>();
          else if (flying == 3) cp_async_wait_group<2>();
          else if (flying == 2) cp_async_wait_group<1>();
          else cp_async_wait_group<0>();
          __syncwarp();
          rec = mine + head;
        };
        auto release = [&]() {
          if (fence) __threadfence_block();  // (as publish() below)
          __syncwarp();
          head += size;
          if (--flying == 0) {
            head = tail = 0;
            wrapped = false;
          }
          fill();
        };
        // a phase's stores ordered before the copies that read them back
        auto publish = [&]() {
          __threadfence_block();
          __syncwarp();
        };
        bool stop = false;
        for (int it = 0; it <= J.max_iter && ok; ++it) {
          // ---- B phase ----
          if (it > 0) {
            if (check_at(J, it - 1)) {
              if (!wait_f(bp.T)) {
                ok = false;
                break;
              }
              stop = decide(J, it - 1);
              u.frozen = frozen;
            }
            next_phase(bp.T);
            if (stop) {
              it_run = it - 1;
              break;
            }
          }
          if (kTrack) u.chg = u.pres = 0.0f;
          if (it == 0 && iw == 0) YR[(size_t)bp.n_yr * 32 + lane] = 0.0f;
          for (int j = 0; j < mb; ++j) {
            take(j);
            const int4 h = *reinterpret_cast<const int4*>(rec);
            if (it > 0 &&
                (!seen(chain_done, chain_seen, chunks + (h.z & (kBandUsesPre - 1))) ||
                 ((h.z & kBandUsesPre) && !band_wait_count(pre_b, phases + 1, abort_flag, a.wait_limit_ns)))) {
              ok = false;
              break;
            }
            const int units = h.x & 15, nc = (h.x >> 4) & 15;
            const unsigned char* blk = rec + ((unsigned)h.x >> 27) * 128;
            const unsigned char* q = blk + units * 512;
            unsigned char* vl = reinterpret_cast<unsigned char*>(V + lane);
            float* yr = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(YR + lane) + h.y);
            float xr = 0.0f;
            if (it > 0)
              xr = *yr * reinterpret_cast<const float*>(q)[lane] -
                   band_dot<true>(0.0f, units, reinterpret_cast<const int4*>(rec) + kBandRecB / 4, blk + lane * 16, vl);
            if (j < n_pre) {  // a pre-chain column: solved only, its row's update is an F item
              if (it > 0) *reinterpret_cast<float*>(vl + h.w) = xr;
              release();
              if (j == n_pre - 1 && lane == 0) st_release_cta(pre_b, phases + 1);
              continue;
            }
            float rhs = 0.0f;
            float* gs = stream + h.w;  // the same place in HBM
            // the children's L entries: the last slots
            const float4 lc = *reinterpret_cast<const float4*>(q - 512 + lane * 16);
            for (int e = 0; e <= nc; ++e) {  // the root, then its children
              const int kind = (h.x >> (8 + 4 * e)) & 15;
              const int w = (kind & 1) ? 64 : 32;
              const float4 k = reinterpret_cast<const float4*>(rec)[1 + e];
              const unsigned char *par = q + 128, *it_p = par + w * 4;
              const float l = e == 1 ? lc.w : lc.z;
              float xs = xr, r = 0.0f;
              if (e > 0 || it == 0) r = band_rhs<kRho>(u, kind, k.y, it_p, par, lane);
              if (e > 0) {
                const float cc = 0.0f + l * xr;
                xs = r * reinterpret_cast<const float*>(q)[lane] - cc;
              }
              if (it > 0)
                r = band_update<kTrack, kRho>(u, kind, xs, k, it_p, par, gs + 32 + w, pres, lane);
              rhs = e > 0 ? rhs - l * r : r;
              gs += 32 + 2 * w;
              q = it_p + w * 4;
            }
            *yr = rhs;
            release();
          }
          if (!ok) break;
          if (it > 0) chunks += (unsigned)bp.n_chunks;
          ++phases;
          // (not before the first iteration: after a tile that stopped early a warp may
          // still be reading that set)
          if (kTrack && mf == 0 && it > 0) {
            float* m = maxima_of(it) + iw * 64;
            m[lane] = u.chg;
            m[32 + lane] = u.pres;
          }
          publish();
          if (lane == 0) atomicAdd(b_done, 1u);
          // ---- F phase: every B item and the whole backward sweep are done ----
          if (!band_wait_count<2, 60>(b_done, phases * (unsigned)K, abort_flag, a.wait_limit_ns) ||
              !band_wait_count<2, 60>(chain_done, chunks, abort_flag, a.wait_limit_ns)) {
            ok = false;
            break;
          }
          if (it == 0 && iw == 0)  // the window's overhang and the zero row
            for (int i = bp.T; i <= band_vzero(bp.T4, bp.units); ++i) V[(size_t)i * 32 + lane] = 0.0f;
          unsigned rows_done = f_done[iw];
          for (int j = 0; j < mf; ++j) {
            take(mb + j);
            const int4 h = *reinterpret_cast<const int4*>(rec);
            if (j >= n_pre && (h.x & kBandUsesPre) && !band_wait_count(pre_f, phases, abort_flag, a.wait_limit_ns)) {
              ok = false;
              break;
            }
            const int units = h.x & 255, kind = (h.x >> 8) & 15, w = (kind & 1) ? 64 : 32;
            const unsigned char* blk = rec + ((unsigned)h.x >> 27) * 128;
            const unsigned char *par = blk + units * 512, *it_p = par + w * 4;
            float* vr = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(V + lane) + h.y);
            const float4 k = reinterpret_cast<const float4*>(rec)[1];
            float acc;
            if (it > 0)
              acc = band_update<kTrack, kRho>(u, kind, *vr, k, it_p, par, stream + h.w + w, pres, lane);
            else
              acc = band_rhs<kRho>(u, kind, k.y, it_p, par, lane);
            if (it < J.max_iter) {
              unsigned char* yl = reinterpret_cast<unsigned char*>(YR + lane);
              acc = band_dot<false>(acc, units, reinterpret_cast<const int4*>(rec) + kBandRecF / 4, blk + lane * 16, yl);
              if (h.z >= 0)  // a pre-chain row: its forward result
                *reinterpret_cast<float*>(yl + h.z) = acc;
              else
                *vr = acc;
            }
            if (kTrack && j == mf - 1) {  // published with the phase's last row
              float* m = maxima_of(it) + iw * 64;
              m[lane] = u.chg;
              m[32 + lane] = u.pres;
            }
            release();
            if (j >= n_pre) {
              ++rows_done;
              if (lane == 0) st_release_cta(f_done + iw, rows_done);
            } else if (j == n_pre - 1 && lane == 0) {
              st_release_cta(pre_f, phases);
            }
          }
          if (!ok) break;
          publish();
        }
        if (!ok) break;
        if (stop) {
          // the chain warp has left the tile (one count past its sweeps')
          if (!band_wait_count(chain_done, ++chunks, abort_flag, a.wait_limit_ns)) {
            ok = false;
            break;
          }
        } else {
          next_phase(bp.T);
        }
      }
      // A tile that stopped early has copies in flight: every lane's have landed before
      // any lane's for the next tile go to the same bytes.
      cp_async_wait_group<0>();
      __syncwarp();
      if (iw == 0 && J.iters && tile * 32 + lane < J.batch) J.iters[tile * 32 + lane] = frozen ? frozen_at : it_run;
    }
    if (!ok && lane == 0) *abort_flag = 1;
    cp_async_wait_group<0>();  // (no copy outlives the CTA)
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.error, 1);
}

// ---------------------------------------------------------------------------
// state layout conversions: symbolic-major (KKT row, instance) <-> tile records
// ---------------------------------------------------------------------------

// form: the scaled primal residual A x - z of a warm start whose termination
// is checked (a cold start's is 0; without checks nothing reads it).
__global__ void band_state_in_kernel(BandPlan bp, Osqp o, const float* __restrict__ aT, long long lda, int sba,
                                     bool track, bool form, const float* __restrict__ x, const float* __restrict__ z,
                                     const float* __restrict__ y, const float* __restrict__ qs,
                                     const float* __restrict__ ls, const float* __restrict__ us,
                                     float* __restrict__ stream, float* __restrict__ pres, int batch, int n_tiles) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_tiles * 32) return;
  const int bb = b < batch ? b : batch - 1;  // padding lanes solve a copy of the last instance
  const int tile = b >> 5, lane = b & 31;
  for (int k = blockIdx.y; k < bp.n; k += gridDim.y) {
    float* it = stream + (size_t)tile * bp.blen + __ldg(bp.iter_off + k);
    float* pa = stream + (size_t)tile * bp.blen + __ldg(bp.param_off + k);
    if (k < bp.n_prim) {
      it[lane] = x[(size_t)k * batch + bb];
      pa[lane] = qs[(size_t)k * batch + bb];
      continue;
    }
    const int r = k - bp.n_prim;
    const float zr = z[(size_t)r * batch + bb];
    reinterpret_cast<float2*>(it)[lane] = make_float2(zr, y[(size_t)r * batch + bb]);
    reinterpret_cast<float2*>(pa)[lane] = make_float2(ls[(size_t)r * batch + bb], us[(size_t)r * batch + bb]);
    if (!track) continue;
    float e = 0.0f;
    if (form) {
      float ax = 0.0f;
      const int e0 = __ldg(o.a_row_ptr + r), e1 = __ldg(o.a_row_ptr + r + 1);
      for (int t = e0; t < e1; ++t) {
        const int j = __ldg(o.a_row_ent + t);
        ax = ax + (aT[(long long)j * lda + (long long)bb * sba] * __ldg(o.a_scale + j)) *
                      x[(size_t)__ldg(o.a_cols + j) * batch + bb];
      }
      e = ax - zr;
    }
    pres[((size_t)tile * o.m + r) * 32 + lane] = e;
  }
}

// The records and item offsets, the same for every tile.
__global__ void band_records_kernel(BandPlan bp, float* __restrict__ stream) {
  float* t = stream + (size_t)blockIdx.x * bp.blen;
  for (int i = blockIdx.y * blockDim.y + threadIdx.y; i < bp.n_rows; i += gridDim.y * blockDim.y)
    t[__ldg(bp.rec_off + i) + threadIdx.x] = __int_as_float(__ldg(bp.rec + i * 32 + threadIdx.x));
}

__global__ void band_state_out_kernel(BandPlan bp, const float* __restrict__ stream, float* __restrict__ x,
                                      float* __restrict__ z, float* __restrict__ y, int batch) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  const int tile = b >> 5, lane = b & 31;
  for (int k = blockIdx.y; k < bp.n; k += gridDim.y) {
    const float* it = stream + (size_t)tile * bp.blen + __ldg(bp.iter_off + k);
    if (k < bp.n_prim) {
      x[(size_t)k * batch + b] = it[lane];
    } else {
      const float2 v = reinterpret_cast<const float2*>(it)[lane];
      z[(size_t)(k - bp.n_prim) * batch + b] = v.x;
      y[(size_t)(k - bp.n_prim) * batch + b] = v.y;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

size_t band_workspace_floats(const BandPlan& bp, int batch) {
  const size_t tiles = (size_t)(batch + 31) / 32;
  return tiles * ((size_t)bp.blen + 32 * (size_t)(bp.n - bp.n_prim)) + 64;
}

BandWork band_work(const BandPlan& bp, int batch, float* work) {
  const size_t tiles = (size_t)(batch + 31) / 32;
  return BandWork{work, work + tiles * bp.blen, (int)tiles};
}

int band_state_in(const BandPlan& bp, const Osqp& o, const float* aT, long long lda, int sba, bool track, bool warm,
                  const float* x, const float* z, const float* y, const float* qs, const float* ls, const float* us,
                  const BandWork& w, int batch, cudaStream_t s) {
  dim3 grid(ceil_div((long long)w.tiles * 32, 128), bp.n < 1024 ? bp.n : 1024);
  band_state_in_kernel<<<grid, 128, 0, s>>>(bp, o, aT, lda, sba, track, warm && track, x, z, y, qs, ls, us, w.stream,
                                            w.pres, batch, w.tiles);
  WMPC_LAUNCH_CHECK();
  band_records_kernel<<<dim3(w.tiles, 8), dim3(32, 8), 0, s>>>(bp, w.stream);
  WMPC_LAUNCH_CHECK();
  return WMPC_OK;
}

int band_state_out(const BandPlan& bp, const BandWork& w, float* x, float* z, float* y, int batch, cudaStream_t s) {
  dim3 grid(ceil_div(batch, 128), bp.n < 1024 ? bp.n : 1024);
  band_state_out_kernel<<<grid, 128, 0, s>>>(bp, w.stream, x, z, y, batch);
  WMPC_LAUNCH_CHECK();
  return WMPC_OK;
}

namespace {

// A launch's sizes over its classes, and its shared memory.
struct BandSizes {
  int vrows = 0, yrows = 0, t4 = 0, n_chunks = 0, chunk = 0, item = 0, rows = 1 << 30;  // rows: the shortest chain's
  bool wide = false;
  std::vector<const BandPlan*> plans;
  void add(const BandPlan& bp) {
    vrows = std::max(vrows, band_vrows(bp.T4, bp.units, bp.n_pre));
    yrows = std::max(yrows, bp.n_yr + 1);
    t4 = std::max(t4, bp.T4);
    n_chunks = std::max(n_chunks, bp.n_chunks);
    chunk = std::max(chunk, bp.chunk_bytes);
    item = std::max(item, bp.item_bytes);
    rows = std::min(rows, bp.T);
    wide = wide || bp.units > 2;
    plans.push_back(&bp);
  }
  int warps() const { return wide ? kBandWideWarps : kBandWarps; }
  int items(int w) const {  // the longest list of a warp
    int v = 0;
    for (const BandPlan* p : plans) v = std::max(v, band_items(p->n_pre, p->nb, p->T, w));
    return v;
  }
  size_t bytes(int w, int ring) const {
    return band_smem_bytes(vrows, yrows, t4, n_chunks, items(w), chunk, ring, w, kBandStages,
                           band_maxima_sets(rows, w));
  }
};

}  // namespace

bool band_fits(const BandPlan* const* plans, int n) {
  BandSizes z;
  for (int i = 0; i < n; ++i) z.add(*plans[i]);
  return n <= kMaxBandJobs && z.bytes(z.warps(), z.item) <= (size_t)kMaxSmemBytes;
}

// One launch over every class's tiles, the costliest class first.
int band_run(const BandJobDesc* jobs, int n_jobs, int* error, int num_sms, cudaStream_t s) {
  if (n_jobs < 1 || n_jobs > kMaxBandJobs)
    return fail(WMPC_ERR_INVALID_ARGUMENT, "1 to %d classes per launch", kMaxBandJobs);
  bool track = false, rho = false;
  int order[kMaxBandJobs], limit = jobs[0].ctas_limit, total = 0;
  double cost[kMaxBandJobs];
  BandSizes z;
  for (int i = 0; i < n_jobs; ++i) {
    z.add(jobs[i].bp);
    track = track || jobs[i].check_every > 0;
    rho = rho || jobs[i].rho_b != nullptr;
    limit = std::min(limit, jobs[i].ctas_limit);
    order[i] = i;
    cost[i] = (double)(jobs[i].max_iter + 1) * jobs[i].bp.blen;
    total += jobs[i].n_tiles;
  }
  if (rho && (track || n_jobs > 1))
    return fail(WMPC_ERR_UNSUPPORTED, "per-instance rho runs one class with fixed iterations");
  if (total == 0) return WMPC_OK;
  std::sort(order, order + n_jobs, [&](int x, int y) { return cost[x] > cost[y]; });
  int dev = 0, sm_bytes = 0, reserved = 0;
  WMPC_CUDA_TRY(cudaGetDevice(&dev));
  WMPC_CUDA_TRY(cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  WMPC_CUDA_TRY(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
  // Two CTAs (two chains) per SM where there are more tiles than SMs and both
  // fit with 8 item warps each (10 warps in all: the registers allow 20 per
  // SM), else one.
  BandArgs a{};
  int ctas = 1;
  size_t room = (size_t)kMaxSmemBytes;
  a.warps = z.warps();
  if (!z.wide && limit >= 2 && total > num_sms && z.bytes(8, 2 * z.item) <= (size_t)(sm_bytes / 2 - reserved)) {
    ctas = 2;
    a.warps = 8;
    room = (size_t)(sm_bytes / 2 - reserved);
  }
  const size_t least = z.bytes(a.warps, z.item);
  if (least > room) return fail(WMPC_ERR_UNSUPPORTED, "these classes do not fit one launch's shared memory");
  a.stages = kBandStages;
  a.vrows = z.vrows;
  a.yrows = z.yrows;
  a.t4 = z.t4;
  a.n_chunks = z.n_chunks;
  a.n_items = z.items(a.warps);
  a.chunk_bytes = z.chunk;
  a.maxima_sets = band_maxima_sets(z.rows, a.warps);
  a.ring_bytes = std::min(16384, z.item + (int)((room - least) / a.warps) / 128 * 128);
  const size_t smem = z.bytes(a.warps, a.ring_bytes);
  int end = 0;
  for (int k = 0; k < n_jobs; ++k) {
    const BandJobDesc& d = jobs[order[k]];
    end += d.n_tiles;
    a.tile_end[k] = end;
    a.job[k] = BandJob{d.bp, d.stream, d.pres, d.iters, d.rho_b, d.rho_count, d.max_iter, d.batch,
                       d.check_every, d.bp.n - d.bp.n_prim, d.chg_eps, d.sigma, d.alpha, d.one_minus_alpha};
  }
  a.n_jobs = n_jobs;
  a.error = error;
  a.wait_limit_ns = kBandWaitNs;
  if (const char* v = getenv("WMPC_STREAM_WAIT_LIMIT_NS")) {
    const long long ns = atoll(v);
    if (ns > 0) a.wait_limit_ns = (unsigned long long)ns;
  }
  auto kernel = z.wide ? (track ? band_admm_kernel<true, false, true>
                              : rho ? band_admm_kernel<false, true, true> : band_admm_kernel<false, false, true>)
                     : (track ? band_admm_kernel<true, false, false>
                              : rho ? band_admm_kernel<false, true, false> : band_admm_kernel<false, false, false>);
  WMPC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  WMPC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared));
  const int grid = total < ctas * num_sms ? total : ctas * num_sms;
  profile_mark_begin(s);
  kernel<<<grid, 32 * (a.warps + 2), smem, s>>>(a);
  profile_mark_end(s);
  record_stream_launch(3, ctas, grid, (int)smem);
  WMPC_LAUNCH_CHECK();
  return WMPC_OK;
}

}  // namespace wmpc
