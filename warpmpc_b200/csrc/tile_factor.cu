// Factorization of 32-instance tiles, one CTA per tile (sm_100a); the program it
// runs is described in tile_factor.cuh.
#include <climits>

#include "osqp.cuh"
#include "tile_factor.cuh"

namespace wmpc {

namespace {

constexpr unsigned kAll = 0xffffffffu;

// a slot by its byte offset (lane4: this lane's 4 bytes)
__device__ __forceinline__ float& at(unsigned char* smem, unsigned off) { return *reinterpret_cast<float*>(smem + off); }
__device__ __forceinline__ unsigned low(unsigned w, unsigned lane4) { return (w & kTfF) | lane4; }
__device__ __forceinline__ unsigned high(unsigned w, unsigned lane4) { return ((w >> 11) & kTfF) | lane4; }

// 4 updates: slot -= (y' dinv) val, to distinct slots (the rows of one column)
struct Upd4 {
  unsigned ay[4];
  float y[4], l[4];
  __device__ __forceinline__ void load(unsigned char* smem, const int4& w, unsigned lane4) {
    const unsigned u[4] = {(unsigned)w.x, (unsigned)w.y, (unsigned)w.z, (unsigned)w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ay[i] = low(u[i], lane4);
      y[i] = at(smem, ay[i]);
      l[i] = at(smem, high(u[i], lane4));
    }
  }
  __device__ __forceinline__ void store(unsigned char* smem, float dinv, float val) {
#pragma unroll
    for (int i = 0; i < 4; ++i) at(smem, ay[i]) = y[i] - (l[i] * dinv) * val;
  }
};

}  // namespace

struct TileFactorOut {
  float *b, *f, *d;      // L (backward and forward place), D^-1
  long long tile_b, tile_f, tile_d;  // floats per tile
  float* dd;             // D itself (planes only), or null
  long long ld;          // planes: [index][ld] with one column per instance; 0: stream layout
};

// What bounds it: instructions on the tick's longest warp (a step takes some 75,
// an update 9; 1.7 million warp instructions per tile of the 30-step quadrotor
// class, issued at 0.39 per cycle and scheduler), not memory.  One tile of that
// class: 0.58 ms, where one warp per tile with L re-read from memory took 4.97
// ms; 65,536 instances 5.16 ms against 8.17; 97 of the 50-step cartpole class
// 0.29 against 1.64; 65,536 of the 10-step small class (4 states) 0.49 against 0.53; 5000
// of the 40-step nonlinear quadrotor QP 2.03 against 7.73.
template <bool kPlanes>
__global__ void __launch_bounds__(32 * kTfWarps, 2)
tile_factor_kernel(TileFactor tf, TileFactorOut out, const float* __restrict__ src_p, long long ldp, int sbp, int np,
                   const float* __restrict__ src_a, long long lda, int sba, int na, const float* __restrict__ src_r,
                   long long ldr, const int* __restrict__ pad_b, int n_pad_b, const int* __restrict__ pad_f,
                   int n_pad_f, int* __restrict__ status, int n_tiles, int batch, const int* __restrict__ only) {
  extern __shared__ __align__(128) unsigned char tf_smem[];
  __shared__ unsigned bad_lanes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lane4 = lane * 4;
  int4* ring = reinterpret_cast<int4*>(tf_smem + (size_t)tf.slots * 128) + warp * 128;
  const int4* list = tf.prog + __ldg(tf.warp_off + warp);
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int b = tile * 32 + lane, bb = b < batch ? b : batch - 1;  // padding lanes factor a copy of the last instance
    if (only != nullptr && !__syncthreads_or(b < batch && only[bb] != 0)) continue;
    if (threadIdx.x == 0) bad_lanes = 0;
    const float* pin = src_p + (long long)bb * sbp;
    const float* ain = src_a + (long long)bb * sba;
    const float* rin = src_r + (src_r ? bb : 0);
    const bool write = !kPlanes || (b < batch && (only == nullptr || only[b] != 0));
    float* Lu = kPlanes ? out.b + b : out.b + (size_t)tile * out.tile_b + lane * 4;
    float* F = kPlanes ? nullptr : out.f + (size_t)tile * out.tile_f + lane * 4;
    float* Ld = kPlanes ? out.d + b : out.d + (size_t)tile * out.tile_d + lane;
    const long long ld = kPlanes ? out.ld : 1;
    bool bad = false;
    // the list: the current piece is in the ring, three more are under way.
    // (Asynchronous copies: a load into a register would be waited for at the
    // next barrier.)
    int piece = 0, tick = 0, entered[3] = {0, 0, 0};  // ticks in which the last pieces were entered
    auto fetch = [&](int q) { cp_async16(ring + (q & 3) * 32 + lane, list + q * 32 + lane); };
    for (int q = 0; q < 4; ++q) fetch(q);
    cp_async_commit();
    cp_async_wait_group<0>();
    __syncwarp();
    const int4* w = ring;
    auto end_tick = [&]() {
      cp_async_commit();
      __syncthreads();
      ++tick;
    };
    auto finish = [&](unsigned slot, float dk, int doff) {
      const float di = 1.0f / dk;
      at(tf_smem, slot) = di;
      bad |= !(di != 0.0f) || !isfinite(di);
      if (write) {
        Ld[doff * ld] = di;
        if (kPlanes && out.dd) out.dd[b + doff * ld] = dk;
      }
    };
    for (;;) {
      const int4 h = *w++;
      const int kind = h.x & 7;
      int cnt = (h.x >> 5) & 63;
      if (kind == kTfStep) {
        const unsigned x = (unsigned)h.x, y = (unsigned)h.y;
        const float val = at(tf_smem, low(y, lane4)), dinv = at(tf_smem, high(y, lane4));
        const unsigned dslot = ((x >> 14) & kTfF) | lane4;
        float dk = at(tf_smem, dslot);
        const float lval = val * dinv;
        dk = dk - val * lval;
        if (x & 16) {
          finish(dslot, dk, w->x);
          ++w;
        } else {
          at(tf_smem, dslot) = dk;
        }
        if (write) {
          Lu[h.z * ld] = lval;
          if (!kPlanes) {
            float* f = h.w >= 0 ? F + h.w : Lu + (-1 - h.w);
            *f = lval;
          }
        }
        Upd4 p, q;
#pragma unroll 1
        for (; cnt >= 2; cnt -= 2) {
          p.load(tf_smem, w[0], lane4);
          q.load(tf_smem, w[1], lane4);
          w += 2;
          p.store(tf_smem, dinv, val);
          q.store(tf_smem, dinv, val);
        }
        if (cnt) {
          p.load(tf_smem, *w++, lane4);
          p.store(tf_smem, dinv, val);
        }
      } else if (kind == kTfInputs) {
        cp_async_wait_group<kTfDelay - 1>();
#pragma unroll 1
        for (; cnt > 0; --cnt) {
          const int4 e = *w++;
          float& s = at(tf_smem, low((unsigned)e.x, lane4));
          s = s * __int_as_float(e.y) + __int_as_float(e.z);
        }
      } else if (kind == kTfZeros) {
#pragma unroll 1
        for (; cnt > 0; --cnt) {
          const int4 e = *w++;
          at(tf_smem, low((unsigned)e.x, lane4)) = 0.0f;
          at(tf_smem, low((unsigned)e.y, lane4)) = 0.0f;
          at(tf_smem, low((unsigned)e.z, lane4)) = 0.0f;
          at(tf_smem, low((unsigned)e.w, lane4)) = 0.0f;
        }
      } else if (kind == kTfConsts) {
#pragma unroll 1
        for (; cnt > 0; --cnt) {
          const int4 e = *w++;
          at(tf_smem, low((unsigned)e.x, lane4)) = __int_as_float(e.y);
          at(tf_smem, low((unsigned)e.z, lane4)) = __int_as_float(e.w);
        }
      } else if (kind == kTfPivot) {
        const unsigned s = low((unsigned)h.y, lane4);
        finish(s, at(tf_smem, s), h.z);
      } else if (kind == kTfLoad) {
        const float* base = h.y == 0 ? pin : h.y == 1 ? ain : rin;
        const long long ld_in = h.y == 0 ? ldp : h.y == 1 ? lda : ldr;
#pragma unroll 1
        for (; cnt > 0; --cnt) {
          const int4 e = *w++;
          const unsigned u[4] = {(unsigned)e.x, (unsigned)e.y, (unsigned)e.z, (unsigned)e.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            cp_async4(tf_smem + (((u[i] >> 13) & kTfF) | lane4), base + (u[i] & 0xfffffu) * ld_in);
        }
      } else if (kind == kTfTicks) {
        for (int i = 0; i < h.y; ++i) end_tick();
      } else {
        if (h.y) break;
        // the next piece was asked for when the last but two was entered
        if (tf_piece_wait(tick - entered[2]) == kTfDelay - 1) cp_async_wait_group<kTfDelay - 1>();
        else cp_async_wait_all();
        __syncwarp();
        fetch(piece + 4);
        ++piece;
        entered[2] = entered[1];
        entered[1] = entered[0];
        entered[0] = tick;
        w = ring + (piece & 3) * 32;
      }
      if (h.x & 8) end_tick();
    }
    cp_async_wait_group<0>();
    if (!kPlanes) {
      for (int i = warp; i < n_pad_b; i += kTfWarps) Lu[__ldg(pad_b + i)] = 0.0f;
      for (int i = warp; i < n_pad_f; i += kTfWarps) F[__ldg(pad_f + i)] = 0.0f;
    }
    const unsigned mine = __ballot_sync(kAll, bad);
    if (mine && lane == 0) atomicOr(&bad_lanes, mine);
    __syncthreads();
    if (status && warp == 0 && write) status[b] = (bad_lanes >> lane & 1u) ? WMPC_STATUS_ZERO_PIVOT : 0;
    __syncthreads();
  }
}

static int tile_factor_launch(int slots, int n_tiles, int num_sms, int* grid, size_t* smem) {
  *smem = tile_factor_smem(slots);
  int dev = 0, sm_bytes = 0, reserved = 0;
  WMPC_CUDA_TRY(cudaGetDevice(&dev));
  WMPC_CUDA_TRY(cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  WMPC_CUDA_TRY(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
  const int most = num_sms * (2 * (*smem + reserved + 1024) <= (size_t)sm_bytes ? 2 : 1);
  *grid = n_tiles < most ? n_tiles : most;
  return WMPC_OK;
}

int tile_factor_stream(const TileFactor& tf, const StreamPlan& sp, const TileFactorInputs& in, float* bstream,
                       float* fstream, int* status, int batch, int num_sms, const int* only, cudaStream_t s) {
  const int n_tiles = (batch + 31) / 32;
  int grid = 0;
  size_t smem = 0;
  if (int rc = tile_factor_launch(tf.slots, n_tiles, num_sms, &grid, &smem)) return rc;
  auto kernel = tile_factor_kernel<false>;
  WMPC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const TileFactorOut out{bstream, fstream, bstream, sp.blen, sp.flen, sp.blen, nullptr, 0};
  profile_mark_begin(s, kProfileFactor);
  kernel<<<grid, 32 * kTfWarps, smem, s>>>(tf, out, in.p, in.ldp, in.sbp, in.np, in.a, in.lda, in.sba, in.na, in.r,
                                           in.ldr, sp.pad_boff, sp.n_pad_b, sp.pad_foff, sp.n_pad_f, status, n_tiles,
                                           batch, only);
  profile_mark_end(s, kProfileFactor);
  WMPC_LAUNCH_CHECK();
  return WMPC_OK;
}

int tile_factor_planes(const TileFactor& tf, const float* values, long long ld, int sb, float* lx, float* d,
                       float* dinv, int batch, int num_sms, const int* only, cudaStream_t s) {
  const int n_tiles = (batch + 31) / 32;
  const TileFactorOut out{lx, nullptr, dinv, 0, 0, 0, d, batch};
  int grid = 0;
  size_t smem = 0;
  auto kernel = tile_factor_kernel<true>;
  if (int rc = tile_factor_launch(tf.slots, n_tiles, num_sms, &grid, &smem)) return rc;
  WMPC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  profile_mark_begin(s, kProfileFactor);
  kernel<<<grid, 32 * kTfWarps, smem, s>>>(tf, out, values, ld, sb, INT_MAX, values, 0, 0, 0, nullptr, 0, nullptr, 0,
                                           nullptr, 0, nullptr, n_tiles, batch, only);
  profile_mark_end(s, kProfileFactor);
  WMPC_LAUNCH_CHECK();
  return WMPC_OK;
}

}  // namespace wmpc
