// Single-token decoding: one persistent kernel runs a whole step of the network.
//
// What bounds it: every weight is read once per token (2 bytes each), and a layer is a chain of five
// dependent phases (LN+QKV, attention, projection, LN+c_fc, c_proj), each of which needs the whole
// output of the one before. One CTA per SM owns a contiguous run of output rows of every matrix; its
// producer warp streams those rows through a shared-memory ring with 1-D bulk copies in the fixed
// order of the phases, so weights of the next phases (of the next layer, too) keep arriving while the
// consumers wait for each other: the waits hide behind the copies for large models and are what remains
// for small ones.
//
// A weight tile is up to 16 rows; a ring slot takes it whole (one bulk copy: the rows are contiguous in
// memory) or, where rows are long, some of its columns (a copy for each row), and the biases of its rows
// and the weights of the LayerNorms travel in the ring as well, so that no phase waits for a load of its
// own. 15 consumer warps split the columns; each takes 64 at a time from 16-byte shared-memory reads and
// feeds four
// mma.m16n8k16 (rows x up to 8 sequences): a batch costs the same reads as one sequence. The columns
// inside such a step are dealt to the lanes in the same permuted order for weights and activations, which
// a sum over columns does not see. Neighbouring rows start on the same bank; the lanes of odd rows read
// the second half of their 64 columns first, so that the two rows of a quarter warp never collide.
//
// Between the phases the CTAs exchange activations without barriers or fences: two bf16 values travel in
// one 8-byte word together with the number of their phase (the "epoch"), and a reader polls the data
// itself until the epochs are the ones it needs. A buffer is written again one layer later, and by then
// every CTA has handed over results that it could only compute after it had read the old contents: each of
// the phases QKV, projection, c_fc and c_proj waits for rows of every CTA (the grid is chosen so that each
// CTA owns rows of every matrix), and the attention phase waits for all of QKV through its heads.
// Against a grid barrier with plain stores this leaves out the release fence, the counter's and the data's
// round trips.
//
// Activations keep the roundings of the batched kernels (bf16 after every LayerNorm, projection and
// residual addition), sums are fp32; attention probabilities stay fp32.
//
// All waits are bounded. A CTA that gives up records the status and runs on without waiting (no index
// depends on data, and the control flow of its warps stays uniform); its producer stops issuing and
// waits, bounded, for the copies in flight.
#include <atomic>
#include "../common/launch.cuh"
#include "../common/ptx.cuh"
#include "decode.h"

namespace z2h {
namespace {

constexpr int kWarps = 15;                   // consumer warps: with the producer's 512 threads, 128 registers each
constexpr int kConsumers = kWarps * 32;
constexpr int kEpochsPerLayer = 5;
constexpr int kThreads = kConsumers + 32;    // + the producer warp
constexpr int kTileRows = 16;
constexpr int kRowPad = 64;                  // bytes between the activations of two sequences
constexpr int kMaxSlots = 12;
constexpr int kSmemLimit = 227 * 1024;
constexpr int kMaxItems = 8;                 // (sequence, head, key range)s of one CTA
constexpr int kMaxSplits = 8;                // key ranges of one (sequence, head)
constexpr int kPartFloats = 68;              // m, l, padding, o[64]
constexpr int kMaxChunk = 1024;              // columns of a slot, at 16 rows
constexpr int kBiasBytes = 128;              // behind the weights of a slot
constexpr int kKeysPerLane = 4;               // keys whose loads a lane has in flight together
constexpr int kKeysPerRound = kWarps * 4 * kKeysPerLane;

struct Params {
  DecodeArgs a;
  int slots, slot_bytes, xs_stride, splits;  // a slot: slot_bytes of weights, kBiasBytes of biases
  // exchange buffers, 8 bytes a unit: two bf16 values (or one fp32) and the epoch
  uint64_t *resid, *mid, *att, *act, *qkv;  // [batch][C / 2], act: 4C / 2, qkv: 3C / 2
  uint64_t* part;                           // [batch][heads][splits][kPartFloats]
};

// How a matrix of n rows and K columns is cut for the ring: tiles of `rows` rows, `cols` columns a slot.
struct Cut {
  int rows, cols;
};
__host__ __device__ inline Cut cut_matrix(int slot_bytes, int n, int K, int grid) {
  Cut c;
  const int own = ((n + 1) / 2 + grid - 1) / grid * 2;  // most rows of a CTA
  c.rows = own < kTileRows ? own : kTileRows;
  const int fit = slot_bytes / (c.rows * 2) / 64, units = K / 64, parts = (units + fit - 1) / fit;
  c.cols = (units + parts - 1) / parts * 64;
  return c;
}

// What a CTA does, worked out once per launch: integer divisions inside the phases cost more than their
// arithmetic.
enum Matrix : int { kQkv, kProj, kFc, kFc2, kHead, kMatrices };
struct Share {
  int r0, r1;      // its rows of a matrix, a run that starts on an even row
  int rows, cols;  // tile
};
struct Item {
  int b, h, k0, k1, index;  // sequence, head, keys
};

struct Smem {
  Share share[kMatrices];
  Item items[kMaxItems];
  int num_items;
  uint64_t full[kMaxSlots], empty[kMaxSlots];
  float red[2][kWarps][kTileRows * 8];
  float att[kWarps][kPartFloats];
  float stream[kTileRows][8];  // residual stream of the rows this CTA owns in the matrices with C rows
  int abort_flag;
};

__device__ __forceinline__ void consumer_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory");
}
__device__ __forceinline__ uint4 ld_cg(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }

__device__ void plan(const Params& p, Smem* sm, int t) {
  if (t < kMatrices) {
    const int C = p.a.C, n = t == kQkv ? 3 * C : t == kFc ? 4 * C : t == kHead ? p.a.vocab : C;
    const long long pairs = (n + 1) / 2;
    const Cut cut = cut_matrix(p.slot_bytes, n, t == kFc2 ? 4 * C : C, gridDim.x);
    sm->share[t] = {(int)(pairs * blockIdx.x / gridDim.x) * 2, min(n, (int)(pairs * (blockIdx.x + 1) / gridDim.x) * 2),
                    cut.rows, cut.cols};
  }
  const int S = p.splits, total = p.a.batch * p.a.heads * S, keys = p.a.pos + 1;
  if (t < kMaxItems) {
    const int i = blockIdx.x + t * gridDim.x, part = i % S, bh = i / S;
    if (i < total)
      sm->items[t] = {bh / p.a.heads, bh % p.a.heads, (int)((long long)keys * part / S), (int)((long long)keys * (part + 1) / S), i};
  }
  if (t == 0) sm->num_items = blockIdx.x < total ? (total - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
}

// ---- exchange ----------------------------------------------------------------------------------
// A maximum that the L2 takes (epochs only grow, and the newer one wins): it shows earlier than a plain store
// on a line that other SMs are polling (one token: 124M model 230 -> 206 us, 1.5B for four sequences 1.65 ->
// 1.50 ms).
__device__ __forceinline__ void put(uint64_t* p, uint32_t value, uint32_t epoch) {
  asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(p), "l"((uint64_t)epoch << 32 | value) : "memory");
}
struct Units2 {
  uint64_t a, b;
  __device__ __forceinline__ bool ready(uint32_t epoch) const {
    return (uint32_t)(a >> 32) == epoch && (uint32_t)(b >> 32) == epoch;
  }
  __device__ __forceinline__ uint2 values() const { return make_uint2((uint32_t)a, (uint32_t)b); }
};
__device__ __forceinline__ Units2 look(const uint64_t* p) {  // 16-byte aligned
  Units2 u;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u.a), "=l"(u.b) : "l"(p) : "memory");
  return u;
}
// n <= N double units, the i-th at at(i): all are polled together until all are there, so that a wait
// costs one round trip after the last of them has arrived and not one for each.
template <int N, typename At>
__device__ __forceinline__ void gather(const Params& p, Smem* sm, int n, At at, uint32_t epoch, uint2 (&out)[N]) {
  Units2 u[N];
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (true) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < n) u[i] = look(at(i));
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < n) ok = ok && u[i].ready(epoch);
    if (ok) break;
    if ((++spins & 63u) == 0u) {
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (*(volatile int*)&sm->abort_flag != 0) break;
      if (now - t0 > Z2H_WAIT_BUDGET_NS) {
        if (p.a.status != nullptr) atomicCAS(p.a.status, 0, (int)kTimeoutLocal);
        *(volatile int*)&sm->abort_flag = 1;
        break;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < n) out[i] = u[i].values();
}

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- producer (a warp) --------------------------------------------------------------------------
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  __device__ void advance(int slots) {
    if (++slot == slots) { slot = 0; phase ^= 1; }
  }
};

struct Producer {
  const Params& p;
  Smem* sm;
  uint8_t* ring;
  Ring st;
  long long issued = 0;
  const __nv_bfloat16* w;

  // lane 0 has the slot's transaction count armed on return
  __device__ __noinline__ bool open(uint32_t bytes) {
    const bool ok = mbar_wait_bounded(&sm->empty[st.slot], st.phase ^ 1, &sm->abort_flag, p.a.status, kTimeoutEmpty);
    if (!__all_sync(0xffffffffu, ok)) return false;
    if ((threadIdx.x & 31) == 0) mbar_arrive_expect_tx(&sm->full[st.slot], bytes);
    __syncwarp();
    return true;
  }
  __device__ void close() {
    ++issued;
    st.advance(p.slots);
  }
  __device__ uint8_t* at() const { return ring + (size_t)st.slot * (p.slot_bytes + kBiasBytes); }

  // bias < 0: none
  __device__ bool matrix(int which, long long offset, long long bias, int K) {
    const Share own = sm->share[which];
    const int lane = threadIdx.x & 31;
    for (int r = own.r0; r < own.r1; r += own.rows) {
      const int rows = min(own.rows, own.r1 - r);
      for (int k = 0; k < K; k += own.cols) {
        const uint32_t row_bytes = (uint32_t)min(own.cols, K - k) * 2;
        // the 16-byte groups that hold this tile's biases (the buffer's tensors are padded to 64 elements)
        const long long b0 = (bias + r) & ~7ll;
        const uint32_t bias_bytes = bias < 0 || k > 0 ? 0 : (uint32_t)(((bias + r + rows + 7) & ~7ll) - b0) * 2;
        if (!open(row_bytes * rows + bias_bytes)) return false;
        const __nv_bfloat16* src = w + offset + (long long)r * K + k;
        if (own.cols >= K) {
          if (lane == 0) bulk_load_1d(at(), src, row_bytes * rows, &sm->full[st.slot]);
        } else if (lane < rows) {
          bulk_load_1d(at() + lane * row_bytes, src + (long long)lane * K, row_bytes, &sm->full[st.slot]);
        }
        if (lane == 31 && bias_bytes != 0) bulk_load_1d(at() + p.slot_bytes, w + b0, bias_bytes, &sm->full[st.slot]);
        close();
      }
    }
    return true;
  }
  // weight and bias (< 0: none) of a LayerNorm
  __device__ bool norm(long long weight, long long bias) {
    const uint32_t bytes = (uint32_t)p.a.C * 2;
    if (!open(bias < 0 ? bytes : 2 * bytes)) return false;
    if ((threadIdx.x & 31) == 0) {
      bulk_load_1d(at(), w + weight, bytes, &sm->full[st.slot]);
      if (bias >= 0) bulk_load_1d(at() + bytes, w + bias, bytes, &sm->full[st.slot]);
    }
    close();
    return true;
  }
};

// ---- consumers ---------------------------------------------------------------------------------
// y[row][b] = sum_k W[row][k] xs[b][k] (+ bias) over the rows this CTA owns. done(row, b, y, mine) is called
// by the 128 threads that hold the 16 x 8 results of a tile (four whole warps; `mine`: the row and the
// sequence exist). `bias`: where the biases lie in the packed buffer, < 0: there are none.
template <typename Done>
__device__ __forceinline__ void matvec(const Params& p, Smem* sm, const uint8_t* ring, const uint8_t* xs, Ring& st,
                                       int& buf, int which, int K, long long bias, Done done) {
  const Share own = sm->share[which];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int in_tile = (int)threadIdx.x >> 3, b = threadIdx.x & 7;
  const bool live = g < p.a.batch, odd = (g & 1) != 0;
  const uint8_t* xrow = xs + (live ? g : 0) * p.xs_stride + t * 16;
  const int first = odd ? 64 : 0, second = 64 - first;  // bytes: which half of the 64 columns comes first
  for (int r = own.r0; r < own.r1; r += own.rows) {
    const int rows = min(own.rows, own.r1 - r), row = r + in_tile;
    const bool mine = in_tile < rows && b < p.a.batch;
    float acc[4][4] = {}, add = 0.f;  // four chains: a step's products do not wait for each other
    for (int k = 0; k < K; k += own.cols) {
      const int n = min(own.cols, K - k);
      mbar_wait_bounded(&sm->full[st.slot], st.phase, &sm->abort_flag, p.a.status, kTimeoutFull);
      const uint8_t* slot = ring + (size_t)st.slot * (p.slot_bytes + kBiasBytes);
      if (k == 0 && bias >= 0 && mine)
        add = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(slot + p.slot_bytes)[((bias + r) & 7) + in_tile]);
      // rows that the tile does not have read its first one; nobody takes their sums
      const uint8_t* w0 = slot + t * 16 + (g < rows ? g : 0) * n * 2;
      const uint8_t* w1 = slot + t * 16 + (g + 8 < rows ? g + 8 : 0) * n * 2;
#pragma unroll 1
      for (int s = warp; s < n / 64; s += kWarps) {
        const uint4 a0f = *reinterpret_cast<const uint4*>(w0 + s * 128 + first);
        const uint4 a1f = *reinterpret_cast<const uint4*>(w1 + s * 128 + first);
        const uint4 a0s = *reinterpret_cast<const uint4*>(w0 + s * 128 + second);
        const uint4 a1s = *reinterpret_cast<const uint4*>(w1 + s * 128 + second);
        uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
        if (live) {
          x0 = *reinterpret_cast<const uint4*>(xrow + k * 2 + s * 128);
          x1 = *reinterpret_cast<const uint4*>(xrow + k * 2 + s * 128 + 64);
        }
        const uint4 a0 = odd ? a0s : a0f, a1 = odd ? a1s : a1f, c0 = odd ? a0f : a0s, c1 = odd ? a1f : a1s;
        mma_16816(acc[0], a0.x, a1.x, a0.y, a1.y, x0.x, x0.y);
        mma_16816(acc[1], a0.z, a1.z, a0.w, a1.w, x0.z, x0.w);
        mma_16816(acc[2], c0.x, c1.x, c0.y, c1.y, x1.x, x1.y);
        mma_16816(acc[3], c0.z, c1.z, c0.w, c1.w, x1.z, x1.w);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->empty[st.slot]);
      st.advance(p.slots);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[0][i] += acc[1][i] + (acc[2][i] + acc[3][i]);
    float* red = sm->red[buf][warp];
    *reinterpret_cast<float2*>(red + g * 8 + 2 * t) = make_float2(acc[0][0], acc[0][1]);
    *reinterpret_cast<float2*>(red + (g + 8) * 8 + 2 * t) = make_float2(acc[0][2], acc[0][3]);
    consumer_sync();
    if (threadIdx.x < kTileRows * 8) {
      float y = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) y += sm->red[buf][w][threadIdx.x];
      done(row, b, y + add, mine);
    }
    buf ^= 1;  // the next tile writes the other half; this one is rewritten two barriers on
  }
}
// Rows 2i and 2i + 1 of a sequence (lanes 8 apart) leave as one unit.
__device__ __forceinline__ void put_pair(uint64_t* dst, int n_rows, int row, int b, __nv_bfloat16 v, bool mine,
                                         uint32_t epoch) {
  const uint32_t low = __bfloat16_as_ushort(v), high = __shfl_down_sync(0xffffffffu, low, 8);
  if (mine && (row & 1) == 0) put(dst + (long long)b * (n_rows / 2) + row / 2, low | high << 16, epoch);
}

__device__ __forceinline__ long long token_of(const Params& p, int b) {
  long long tok = p.a.tokens[b * p.a.token_stride];
  if (tok < 0 || tok >= p.a.vocab) {  // clamped and reported, as the batched embedding does
    if (p.a.status != nullptr) atomicCAS(p.a.status, 0, (int)kBadArgument);
    tok = tok < 0 ? 0 : p.a.vocab - 1;
  }
  return tok;
}

__device__ __forceinline__ uint4 embed8(const Params& p, const __nv_bfloat16* W, long long tok, int c) {
  const uint4 e = *reinterpret_cast<const uint4*>(W + p.a.lay.wte + tok * p.a.C + c);
  const uint4 q = *reinterpret_cast<const uint4*>(W + p.a.lay.wpe + (long long)p.a.pos * p.a.C + c);
  uint4 o;
  const uint32_t *a = &e.x, *b = &q.x;
  uint32_t* w = &o.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = unpack_bf16x2(a[j]), y = unpack_bf16x2(b[j]);
    w[j] = pack_bf16x2(x.x + y.x, x.y + y.y);
  }
  return o;
}

// xs[b] = src[b], K columns
__device__ __forceinline__ void copy_rows(const Params& p, Smem* sm, uint8_t* xs, const uint64_t* src, int K,
                                       uint32_t epoch) {
  const int per_row = K / 4, total = p.a.batch * per_row;
  constexpr int kFlight = 4;
  for (int i0 = threadIdx.x; i0 < total; i0 += kFlight * kConsumers) {
    uint2 v[kFlight];
    const int n = min(kFlight, (total - i0 + kConsumers - 1) / kConsumers);
    gather(p, sm, n, [&](int j) { return src + 2ll * (i0 + j * kConsumers); }, epoch, v);
#pragma unroll
    for (int j = 0; j < kFlight; ++j)
      if (j < n) {
        int c = i0 + j * kConsumers, b = 0;
        for (; c >= per_row; c -= per_row) ++b;
        *reinterpret_cast<uint2*>(xs + b * p.xs_stride + c * 8) = v[j];
      }
  }
  consumer_sync();
}

// xs[b] = LayerNorm(xs[b]), warp b takes row b; the LayerNorm's parameters are the ring's next slot.
__device__ __forceinline__ void layer_norm_rows(const Params& p, Smem* sm, const uint8_t* ring, uint8_t* xs,
                                                const Ring& st, bool has_bias) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, C = p.a.C;
  if (warp < p.a.batch) {
    uint8_t* row = xs + warp * p.xs_stride;
    float sum = 0.f, sq = 0.f;
#pragma unroll 1
    for (int c = lane * 8; c < C; c += 256) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + c * 2);
      const uint32_t* u = &v.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(u[j]);
        sum += f.x + f.y;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / C;
#pragma unroll 1
    for (int c = lane * 8; c < C; c += 256) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + c * 2);
      const uint32_t* u = &v.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(u[j]);
        sq += (f.x - mean) * (f.x - mean) + (f.y - mean) * (f.y - mean);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rstd = rsqrtf(sq / C + 1e-5f);
    mbar_wait_bounded(&sm->full[st.slot], st.phase, &sm->abort_flag, p.a.status, kTimeoutFull);
    const uint8_t* norm = ring + (size_t)st.slot * (p.slot_bytes + kBiasBytes);
#pragma unroll 1
    for (int c = lane * 8; c < C; c += 256) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + c * 2);
      const uint4 wv = *reinterpret_cast<const uint4*>(norm + c * 2);
      const uint4 bv = has_bias ? *reinterpret_cast<const uint4*>(norm + C * 2 + c * 2) : make_uint4(0, 0, 0, 0);
      const uint32_t *u = &v.x, *ww = &wv.x, *bb = &bv.x;
      uint4 o;
      uint32_t* ow = &o.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(u[j]), a = unpack_bf16x2(ww[j]), d = unpack_bf16x2(bb[j]);
        ow[j] = pack_bf16x2((f.x - mean) * rstd * a.x + d.x, (f.y - mean) * rstd * a.y + d.y);
      }
      *reinterpret_cast<uint4*>(row + c * 2) = o;
    }
    __syncwarp();
  }
  if (lane == 0) mbar_arrive(&sm->empty[st.slot]);
  consumer_sync();
}

// The larger one, NaN if one is NaN (fmaxf drops it, and a warp or a key range of NaNs alone would then look
// like one without keys).
__device__ __forceinline__ float max_nan(float a, float b) {
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  return m;
}

// One (sequence, head, key range): keys are dealt to the warps four at a time (8 lanes per key, 16
// bytes each), 16 per warp and round, with all key and value loads of a round in flight together.
__device__ __forceinline__ void attend(const Params& p, Smem* sm, int layer, uint32_t in_epoch, uint32_t out_epoch) {
  const int C = p.a.C, S = p.splits;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, oct = lane & 7;
  const long long plane = (long long)p.a.batch * p.a.max_len * C;
  const __nv_bfloat16* kv = reinterpret_cast<const __nv_bfloat16*>(p.a.kv) + 2 * layer * plane;
  for (int turn = 0; turn < sm->num_items; ++turn) {
    const Item it = sm->items[turn];
    const int b = it.b, h = it.h, k0 = it.k0, k1 = it.k1;
    const __nv_bfloat16* kb = kv + (long long)b * p.a.max_len * C + h * 64 + oct * 8;
    const __nv_bfloat16* vb = kb + plane;
    // the new token's query, key and value for this lane's eight columns, as this step's QKV phase left them
    const uint64_t* fresh = p.qkv + (long long)b * (3 * C / 2) + h * 32 + oct * 4;
    // the first round's cached keys and values do not wait for this step
    uint4 kk[kKeysPerLane], vv[kKeysPerLane];
    auto load_round = [&](int base) {
#pragma unroll
      for (int i = 0; i < kKeysPerLane; ++i) {
        const int key = base + i * (kWarps * 4) + warp * 4 + grp;
        kk[i] = vv[i] = make_uint4(0, 0, 0, 0);
        if (key < k1 && key != p.a.pos) {
          kk[i] = ld_cg(kb + (long long)key * C);
          vv[i] = ld_cg(vb + (long long)key * C);
        }
      }
    };
    load_round(k0);
    uint2 got[6] = {};
    gather(p, sm, 6, [&](int j) { return fresh + (j >> 1) * (C / 2) + (j & 1) * 2; }, in_epoch, got);
    const uint4 new_k = make_uint4(got[2].x, got[2].y, got[3].x, got[3].y);
    const uint4 new_v = make_uint4(got[4].x, got[4].y, got[5].x, got[5].y);
    float q[8];
    {
      const uint32_t w[4] = {got[0].x, got[0].y, got[1].x, got[1].y};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]);
        q[2 * j] = f.x * (0.125f * 1.4426950408889634f);  // 1/sqrt(64), exponentials in base 2
        q[2 * j + 1] = f.y * (0.125f * 1.4426950408889634f);
      }
    }
    float m = -INFINITY, l = 0.f, o[8] = {};
    for (int base = k0; base < k1; base += kKeysPerRound) {
      if (base > k0) load_round(base);
#pragma unroll
      for (int i = 0; i < kKeysPerLane; ++i)
        if (base + i * (kWarps * 4) + warp * 4 + grp == p.a.pos) {
          kk[i] = new_k;
          vv[i] = new_v;
        }
      float sc[kKeysPerLane], mr = -INFINITY;
#pragma unroll
      for (int i = 0; i < kKeysPerLane; ++i) {
        const uint32_t* w = &kk[i].x;
        float d = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(w[j]);
          d = fmaf(f.x, q[2 * j], fmaf(f.y, q[2 * j + 1], d));
        }
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        d += __shfl_xor_sync(0xffffffffu, d, 4);
        sc[i] = base + i * (kWarps * 4) + warp * 4 + grp < k1 ? d : -INFINITY;
        mr = max_nan(mr, sc[i]);
      }
      mr = max_nan(mr, __shfl_xor_sync(0xffffffffu, mr, 8));
      mr = max_nan(mr, __shfl_xor_sync(0xffffffffu, mr, 16));
      if (!(mr == -INFINITY)) {  // warp-uniform: this warp has keys in the round (or a NaN, which l and o take on)
        const float mn = max_nan(m, mr), keep = ex2_fast(m - mn);
        m = mn;
        l *= keep;
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] *= keep;
#pragma unroll
        for (int i = 0; i < kKeysPerLane; ++i) {
          const float e = ex2_fast(sc[i] - m);
          l += e;
          const uint32_t* w = &vv[i].x;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(w[j]);
            o[2 * j] = fmaf(e, f.x, o[2 * j]);
            o[2 * j + 1] = fmaf(e, f.y, o[2 * j + 1]);
          }
        }
      }
    }
#pragma unroll
    for (int x = 8; x <= 16; x <<= 1) {
      l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] += __shfl_xor_sync(0xffffffffu, o[j], x);
    }
    if (grp == 0) {
      float* d = sm->att[warp];
      if (oct == 0) { d[0] = m; d[1] = l; }
#pragma unroll
      for (int j = 0; j < 8; ++j) d[4 + oct * 8 + j] = o[j];
    }
    consumer_sync();
    if (threadIdx.x < 64) {
      float M = -INFINITY, Lsum = 0.f, O = 0.f;
#pragma unroll 5
      for (int w = 0; w < kWarps; ++w) M = fmaxf(M, sm->att[w][0]);
#pragma unroll 5
      for (int w = 0; w < kWarps; ++w) {
        const float mw = sm->att[w][0], f = mw > -INFINITY ? ex2_fast(mw - M) : 0.f;
        Lsum += sm->att[w][1] * f;
        O += sm->att[w][4 + threadIdx.x] * f;
      }
      if (S == 1) {
        const uint32_t low = __bfloat16_as_ushort(__float2bfloat16(O / Lsum));
        const uint32_t high = __shfl_down_sync(0xffffffffu, low, 1);
        if ((threadIdx.x & 1) == 0)
          put(p.att + (long long)b * (C / 2) + h * 32 + threadIdx.x / 2, low | high << 16, out_epoch);
      } else {
        uint64_t* d = p.part + (long long)it.index * kPartFloats;
        if (threadIdx.x == 0) {
          put(d, __float_as_uint(M), out_epoch);
          put(d + 1, __float_as_uint(Lsum), out_epoch);
        }
        put(d + 4 + threadIdx.x, __float_as_uint(O), out_epoch);
      }
    }
    consumer_sync();
  }
}

// xs[b] = attention output, folded from the key ranges' parts
__device__ __forceinline__ void fold_attention(const Params& p, Smem* sm, uint8_t* xs, uint32_t epoch) {
  const int S = p.splits, quads = p.a.C / 4;
  for (int i = threadIdx.x; i < p.a.batch * quads; i += kConsumers) {
    int b = 0, c = i;
    for (; c >= quads; c -= quads) ++b;
    c *= 4;
    const uint64_t* d = p.part + ((long long)b * p.a.heads + c / 64) * S * kPartFloats;
    float m = -INFINITY, l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < S; ++s, d += kPartFloats) {  // (m, l), then the four columns
      uint2 v[3];
      gather(p, sm, 3, [&](int j) { return d + (j == 0 ? 0 : 2 + 2 * j + c % 64); }, epoch, v);
      const float ms = __uint_as_float(v[0].x);
      if (ms > -INFINITY) {
        const float mn = fmaxf(m, ms), f = ex2_fast(m - mn), g = ex2_fast(ms - mn);
        m = mn;
        l = l * f + __uint_as_float(v[0].y) * g;
        o.x = o.x * f + __uint_as_float(v[1].x) * g;
        o.y = o.y * f + __uint_as_float(v[1].y) * g;
        o.z = o.z * f + __uint_as_float(v[2].x) * g;
        o.w = o.w * f + __uint_as_float(v[2].y) * g;
      } else {
        l += __uint_as_float(v[0].y);  // 0, or NaN from keys of NaN
      }
    }
    *reinterpret_cast<uint2*>(xs + b * p.xs_stride + c * 2) =
        make_uint2(pack_bf16x2(o.x / l, o.y / l), pack_bf16x2(o.z / l, o.w / l));
  }
  consumer_sync();
}

// One loop over the phases of all layers with a single instance of each piece of code: laid out phase by
// phase, the same code took 330 us for one token of the 124M model instead of 230 and 2.4 ms instead of 1.65 for
// one of the 1.5B model in four sequences. The bounded waits are inlined all the same.
__device__ __forceinline__ void consume(const Params& p, Smem* sm, const uint8_t* ring, uint8_t* xs) {
  const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(p.a.weights);
  const DecodeLayout& lay = p.a.lay;
  const int C = p.a.C;
  const long long plane = (long long)p.a.batch * p.a.max_len * C;
  Ring st;
  int buf = 0;
  // The matrices with C rows give every CTA the same rows each time: it keeps their values of the residual
  // stream for the next addition to it.
  const int own0 = sm->share[kProj].r0;
  {
    const int row = own0 + (threadIdx.x >> 3), b = threadIdx.x & 7;
    if (threadIdx.x < kTileRows * 8 && row < sm->share[kProj].r1 && b < p.a.batch) {
      const long long tok = token_of(p, b);
      sm->stream[row - own0][b] = __bfloat162float(__float2bfloat16(
          __bfloat162float(W[lay.wte + tok * C + row]) + __bfloat162float(W[lay.wpe + (long long)p.a.pos * C + row])));
    }
  }
  if (int b = threadIdx.x >> 5; b < p.a.batch) {  // the tokens' embeddings
    const long long tok = token_of(p, b);
    for (int c = (threadIdx.x & 31) * 8; c < C; c += 256)
      *reinterpret_cast<uint4*>(xs + b * p.xs_stride + c * 2) = embed8(p, W, tok, c);
  }
  consumer_sync();
  uint32_t epoch = p.a.epoch_base;  // of the phase's input
  int which = kQkv, layer = 0;
  while (true) {
    // ---- input into xs
    const int K = which == kFc2 ? 4 * C : C;
    if (which == kProj) {
      attend(p, sm, layer, epoch, epoch + 1);
      ++epoch;
    }
    if (which == kProj && p.splits > 1) {
      fold_attention(p, sm, xs, epoch);
    } else if (layer > 0 || which != kQkv) {
      copy_rows(p, sm, xs, which == kProj ? p.att : which == kFc ? p.mid : which == kFc2 ? p.act : p.resid, K, epoch);
    }
    if (which == kQkv || which == kFc || which == kHead) {
      layer_norm_rows(p, sm, ring, xs, st, which == kQkv ? lay.o_ln1_b >= 0 : which == kFc ? lay.o_ln2_b >= 0 : lay.lnf_b >= 0);
      st.advance(p.slots);
    }
    // ---- product
    const long long o_bias = which == kQkv ? lay.o_b_qkv : which == kProj ? lay.o_b_proj : which == kFc ? lay.o_b_fc : lay.o_b_fc2;
    const long long bias = which == kHead ? -1 : lay.layer0 + layer * lay.layer_stride + o_bias;
    ++epoch;
    matvec(p, sm, ring, xs, st, buf, which, K, bias, [&](int r, int b, float y, bool mine) {
      if (which == kHead) {
        if (mine) p.a.logits[(long long)b * p.a.vocab + r] = __bfloat162float(__float2bfloat16(y));
        return;
      }
      if (which == kFc) y = gelu_tanh(y);
      float* stream = nullptr;
      if (which == kProj || which == kFc2) {
        stream = &sm->stream[mine ? r - own0 : 0][b];
        y += *stream;
      }
      const __nv_bfloat16 v = __float2bfloat16(y);
      if (stream != nullptr && mine) *stream = __bfloat162float(v);
      if (which == kQkv) {
        put_pair(p.qkv, 3 * C, r, b, v, mine, epoch);
        if (mine && r >= C) {  // for the steps to come; this one's attention reads the exchange
          const int part = r >= 2 * C, c = r - (part + 1) * C;
          reinterpret_cast<__nv_bfloat16*>(p.a.kv)[(2 * layer + part) * plane +
                                                   ((long long)b * p.a.max_len + p.a.pos) * C + c] = v;
        }
      } else {
        const int rows = which == kFc ? 4 * C : C;
        put_pair(which == kProj ? p.mid : which == kFc ? p.act : p.resid, rows, r, b, v, mine, epoch);
      }
    });
    // ---- next phase
    if (which == kHead) return;
    if (which == kFc2) {
      ++layer;
      if (layer == p.a.layers && p.a.logits == nullptr) return;
      which = layer == p.a.layers ? kHead : kQkv;
    } else {
      ++which;
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1) decode_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(128) uint8_t dyn[];
  __shared__ Smem sm;
  uint8_t* xs = dyn + (size_t)p.slots * (p.slot_bytes + kBiasBytes);
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.slots; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], kWarps);
    }
    sm.abort_flag = 0;
    fence_mbar_init();
  }
  plan(p, &sm, threadIdx.x);
  __syncthreads();
  if (threadIdx.x < kConsumers) {
    consume(p, &sm, dyn, xs);
    return;
  }
  Producer prod{p, &sm, dyn};
  prod.w = reinterpret_cast<const __nv_bfloat16*>(p.a.weights);
  const DecodeLayout& lay = p.a.lay;
  const int C = p.a.C;
  bool ok = true;
  const int phases = 4 * p.a.layers + (p.a.logits != nullptr);
  for (int i = 0; ok && i < phases; ++i) {  // the consumers' order; one instance of each piece of code here, too
    const int layer = i >> 2, which = layer == p.a.layers ? kHead : i & 3;
    const long long base = lay.layer0 + layer * lay.layer_stride;
    if (which == kQkv || which == kFc || which == kHead) {
      const long long w = which == kQkv ? lay.o_ln1_w : lay.o_ln2_w, b = which == kQkv ? lay.o_ln1_b : lay.o_ln2_b;
      ok = which == kHead ? prod.norm(lay.lnf_w, lay.lnf_b) : prod.norm(base + w, b < 0 ? -1 : base + b);
      if (!ok) break;
    }
    const long long w = which == kQkv ? lay.o_qkv : which == kProj ? lay.o_proj : which == kFc ? lay.o_fc : lay.o_fc2;
    const long long b = which == kQkv ? lay.o_b_qkv : which == kProj ? lay.o_b_proj : which == kFc ? lay.o_b_fc : lay.o_b_fc2;
    ok = prod.matrix(which, which == kHead ? lay.wte : base + w, which == kHead ? -1 : base + b, which == kFc2 ? 4 * C : C);
  }
  const long long issued = prod.issued;
  // the copies in flight land before this CTA's shared memory goes away; a phase that is already past
  // answers at once, and a wait that another role abandoned must not cut this one short
  const long long last = issued < p.slots ? issued : p.slots;
  volatile int never = 0;
  for (long long i = 0; i < last; ++i) {
    const int slot = (int)((issued - 1 - i) % p.slots);
    const uint32_t phase = (uint32_t)((issued - 1 - i) / p.slots) & 1u;
    mbar_wait_bounded(&sm.full[slot], phase, &never, p.a.status, kTimeoutFull);
  }
}

int xs_stride_for(int C) { return 4 * C * 2 + kRowPad; }
// The ring: slots of 16 rows of C columns, or of an even share of them where C is above kMaxChunk.
int slot_bytes_for(int batch, int C, int* slots) {
  const int parts = (C + kMaxChunk - 1) / kMaxChunk, cols = (C / 64 + parts - 1) / parts * 64;
  const int bytes = kTileRows * cols * 2;
  const int n = (kSmemLimit - (int)sizeof(Smem) - 128 - batch * xs_stride_for(C)) / (bytes + kBiasBytes);
  *slots = n > kMaxSlots ? kMaxSlots : n;
  return bytes;
}
long long align256(long long n) { return (n + 255) / 256 * 256; }

}  // namespace

long long decode_scratch_bytes(int batch, int C, int heads) {
  return align256((long long)batch * C * 4) * 3 + align256((long long)batch * 4 * C * 4) +
         align256((long long)batch * 3 * C * 4) + align256((long long)batch * heads * kMaxSplits * kPartFloats * 8);
}

// Every CTA owns rows of every matrix, and at most one tile of those with C rows.
static int decode_grid(int C) {
  const int sms = sm_count_current_device(), pairs = C / 2;
  return sms < pairs ? sms : pairs;
}

unsigned int decode_epochs(int batch, int C, int layers) {
  if (batch < 1 || batch > kDecodeMaxBatch || C < 64 || C % 64 || C > 2048 || layers < 1) return 0;
  int slots = 0;
  slot_bytes_for(batch, C, &slots);
  if (slots < 2) return 0;
  const int grid = decode_grid(C), pairs = C / 2;
  if (2 * ((pairs + grid - 1) / grid) > kTileRows || batch * (C / 64) > kMaxItems * grid) return 0;
  return (unsigned int)(kEpochsPerLayer * layers);
}

int decode_step(const DecodeArgs& a, cudaStream_t stream) {
  if (decode_epochs(a.batch, a.C, a.layers) == 0 || a.heads * 64 != a.C || a.pos < 0 ||
      a.pos >= a.max_len || a.vocab < 1 || a.epoch_base == 0 || a.weights == nullptr || a.kv == nullptr || a.scratch == nullptr ||
      a.tokens == nullptr)
    return 1;
  Params p;
  p.a = a;
  p.slot_bytes = slot_bytes_for(a.batch, a.C, &p.slots);
  p.xs_stride = xs_stride_for(a.C);
  const int grid = decode_grid(a.C);
  // Key ranges per (sequence, head): as many as there are idle SMs, none shorter than half a round.
  const int room = grid / (a.batch * a.heads), want = (a.pos + 1 + kKeysPerRound / 2 - 1) / (kKeysPerRound / 2);
  p.splits = room < want ? room : want;
  if (p.splits > kMaxSplits) p.splits = kMaxSplits;
  if (p.splits < 1) p.splits = 1;
  if (a.batch * a.heads * p.splits > kMaxItems * grid) return 1;
  uint8_t* s = reinterpret_cast<uint8_t*>(a.scratch);
  auto take = [&s](long long units) {
    uint64_t* r = reinterpret_cast<uint64_t*>(s);
    s += align256(units * 8);
    return r;
  };
  const long long pairs = (long long)a.batch * a.C / 2;
  p.resid = take(pairs);
  p.mid = take(pairs);
  p.att = take(pairs);
  p.act = take(4 * pairs);
  p.qkv = take(3 * pairs);
  p.part = take((long long)a.batch * a.heads * p.splits * kPartFloats);
  const size_t smem = (size_t)p.slots * (p.slot_bytes + kBiasBytes) + (size_t)a.batch * p.xs_stride;
  static std::atomic<unsigned long long> seen{0};
  if (first_use_on_current_device(seen) &&
      cudaFuncSetAttribute(decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kSmemLimit - (int)sizeof(Smem) - 128) != cudaSuccess)
    return 3;
  void* args[] = {&p};
  return cudaLaunchCooperativeKernel((const void*)decode_kernel, dim3(grid), dim3(kThreads), args, smem, stream) ==
                 cudaSuccess ? 0 : 3;
}

// -------------------------------------------------------------------------------------------------
// Packing: fp32 or bf16 parameters into one bf16 buffer, and keys / values out of a batched QKV
// -------------------------------------------------------------------------------------------------
namespace {

constexpr int kPackEntries = 128;   // tensors per launch: the table travels as a kernel argument
constexpr int kPackChunk = 8192;    // elements of one CTA's piece

struct PackTable {
  const void* src[kPackEntries];
  long long dst[kPackEntries];     // element offset, multiple of 8
  long long n[kPackEntries];       // multiple of 8
  int first_chunk[kPackEntries + 1];
  int count;
};

// bound by memory: 6 bytes per fp32 parameter; one launch for 128 tensors instead of a cast for each
__global__ void __launch_bounds__(256) pack_kernel(const __grid_constant__ PackTable t, __nv_bfloat16* dst, int src_fp32) {
  for (int c = blockIdx.x; c < t.first_chunk[t.count]; c += gridDim.x) {
    int lo = 0, hi = t.count;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (t.first_chunk[mid] <= c) lo = mid; else hi = mid;
    }
    const long long at = (long long)(c - t.first_chunk[lo]) * kPackChunk;
    const int n = (int)min((long long)kPackChunk, t.n[lo] - at);
    uint4* d = reinterpret_cast<uint4*>(dst + t.dst[lo] + at);
    if (src_fp32) {
      const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(t.src[lo]) + at);
#pragma unroll 4
      for (int i = threadIdx.x; i < n / 8; i += 256) {
        const float4 a = s[2 * i], b = s[2 * i + 1];
        d[i] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
      }
    } else {
      const uint4* s = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(t.src[lo]) + at);
#pragma unroll 4
      for (int i = threadIdx.x; i < n / 8; i += 256) d[i] = s[i];
    }
  }
}

// qkv [batch][len][3C] -> one layer's kv [2][batch][max_len][C], positions 0 .. len-1
__global__ void __launch_bounds__(256) kv_from_qkv_kernel(const __nv_bfloat16* qkv, __nv_bfloat16* kv, int batch,
                                                          int len, int max_len, int C) {
  const int vecs = C / 8;
  const long long total = (long long)batch * len * 2 * vecs;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int c = (int)(i % vecs) * 8, part = (int)(i / vecs % 2);
    const long long row = i / (2 * vecs), b = row / len, t = row - b * len;
    *reinterpret_cast<uint4*>(kv + ((part * (long long)batch + b) * max_len + t) * C + c) =
        *reinterpret_cast<const uint4*>(qkv + row * 3 * C + (part + 1) * C + c);
  }
}

}  // namespace

int pack_bf16(const void* const* src, const long long* dst, const long long* n, int count, int src_fp32, void* out,
              cudaStream_t stream) {
  for (int i0 = 0; i0 < count; i0 += kPackEntries) {
    PackTable t;
    t.count = count - i0 < kPackEntries ? count - i0 : kPackEntries;
    t.first_chunk[0] = 0;
    for (int i = 0; i < t.count; ++i) {
      t.src[i] = src[i0 + i];
      t.dst[i] = dst[i0 + i];
      t.n[i] = n[i0 + i];
      if ((reinterpret_cast<uintptr_t>(t.src[i]) & 15) || t.dst[i] % 8 || t.n[i] % 8 || t.n[i] < 0) return 1;
      t.first_chunk[i + 1] = t.first_chunk[i] + (int)((t.n[i] + kPackChunk - 1) / kPackChunk);
    }
    const int chunks = t.first_chunk[t.count], most = 8 * sm_count_current_device();
    if (chunks == 0) continue;
    pack_kernel<<<chunks < most ? chunks : most, 256, 0, stream>>>(t, reinterpret_cast<__nv_bfloat16*>(out), src_fp32);
    if (cudaGetLastError() != cudaSuccess) return 3;
  }
  return 0;
}

int kv_from_qkv(const void* qkv, void* kv, int batch, int len, int max_len, int C, cudaStream_t stream) {
  if (batch < 1 || len < 1 || len > max_len || C % 8) return 1;
  const long long work = ((long long)batch * len * 2 * (C / 8) + 255) / 256;
  const int most = 8 * sm_count_current_device();
  kv_from_qkv_kernel<<<work < most ? (int)work : most, 256, 0, stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(qkv), reinterpret_cast<__nv_bfloat16*>(kv), batch, len, max_len, C);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace z2h

extern "C" {
long long z2h_decode_scratch_bytes(int batch, int C, int heads) { return z2h::decode_scratch_bytes(batch, C, heads); }
unsigned int z2h_decode_epochs(int batch, int C, int layers) { return z2h::decode_epochs(batch, C, layers); }
// `layout`: the 18 offsets of DecodeLayout in their order
int z2h_decode_step(const long long* layout, const void* weights, void* kv, const long long* tokens,
                    long long token_stride, float* logits, void* scratch, unsigned int epoch_base, int batch, int C,
                    int heads, int layers, int vocab, int pos, int max_len, int* status, void* stream) {
  z2h::DecodeArgs a;
  const long long* o = layout;
  a.lay = {o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7], o[8], o[9], o[10], o[11], o[12], o[13], o[14], o[15], o[16], o[17]};
  a.weights = weights; a.kv = kv; a.tokens = tokens; a.token_stride = token_stride; a.logits = logits;
  a.scratch = scratch; a.epoch_base = epoch_base; a.batch = batch; a.C = C; a.heads = heads; a.layers = layers;
  a.vocab = vocab; a.pos = pos; a.max_len = max_len; a.status = status;
  return z2h::decode_step(a, (cudaStream_t)stream);
}
int z2h_pack_bf16(const void* const* src, const long long* dst, const long long* n, int count, int src_fp32, void* out,
                  void* stream) {
  return z2h::pack_bf16(src, dst, n, count, src_fp32, out, (cudaStream_t)stream);
}
int z2h_kv_from_qkv(const void* qkv, void* kv, int batch, int len, int max_len, int C, void* stream) {
  return z2h::kv_from_qkv(qkv, kv, batch, len, max_len, C, (cudaStream_t)stream);
}
}
