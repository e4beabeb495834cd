// Fused Fourier layer of the FNO surrogate (width 32, 16 x 16 modes) on the
// 5th-generation tensor cores.
//
// A layer v' = act(K(v) + W v + b) reads its activations once and writes them
// once: one kernel evaluates the inverse x-transform and the channel map of a
// row tile as one product, applies bias and GELU, and takes the next layer's
// truncated forward x-transform of the result while it is still on the chip.
// (As separate GEMMs the layer moved the activations five times.)
//
// Activations live pixel-major, v[b][g0][x][32 channels] (128 bytes a pixel), the
// eight 16-byte pieces of pixel x at positions piece ^ (x & 7): a tile of
// consecutive pixels then IS the tensor core's 128-byte-swizzled K-major
// operand, so a plain bulk copy brings it in and another takes it out.  The
// inverse p-transform writes its rows (32 channels x 32 mode parts per g0) in
// the same form.
//
// One CTA per SM keeps the constants of one 128-pixel x tile in shared memory
// (inverse and forward DFT tiles, channel matrix) and walks the rows (b, g0) in
// two slots of four warps, each with its own buffers, barriers and TMEM
// columns, so one slot's tensor-core products overlap the other's GELUs:
//
//   D1[x][o] = sum_k AA[k][x] Gx[o][k]  +  sum_c v[x][c] W[o][c]     128 x 32, K = 32 + 32
//   v'       = act(D1 + b)                                           registers
//   D2[k][o] = sum_x CS[x][k] v'[x][o]                               64 x 32, K = 128
//
// All products are TF32 split (a_hi b_hi + a_hi b_lo + a_lo b_hi, D2 also
// a_lo b_lo).  An MMA's time is that of reading its operands from shared memory
// (128 bytes a cycle), so the high and low parts are stacked: a_hi meets b_hi and
// b_lo in one 64-column product, and D2 stacks CS_hi over CS_lo along its rows
// too.  The tensor core's FP32 accumulation truncates; at most eight MMAs add
// into one accumulator and the pieces are summed in registers.  D2 covers one x
// tile; the p-transform adds the tiles up.
// The last layer's kernel evaluates the projection instead of D2: hidden =
// Q1 v' (128 wide), out = Q2 GELU(hidden + c1) + c2, nothing but `out` written.
// The lift of the inputs is the same kernel without D1.
//
// Measured, 16 instances at 512^2: inference 10.58 -> 3.53 ms.  A layer takes about
// 3000 cycles a tile (two slots), 1200 of them the tensor core's operand reads
// (1700 with one product per split term); the rest is one slot's chain of
// waits, TMEM reads, GELUs and shared-memory stores with two warps per scheduler
// to cover it.  MMAs are issued by an elected lane of a warp-uniform branch.
//
// Every mbarrier wait is bounded; on expiry the CTA records FW_FNO_TIMEOUT and
// returns with its remaining tiles unwritten.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include "fno_act.cuh"
#include "fno_umma.cuh"
#include "fw_internal.h"
#include "tma.cuh"

namespace fw {
namespace fnol {

namespace cg = cooperative_groups;

constexpr int LC = 32;        // channels
constexpr int LK = 32;        // x-mode parts: 16 cosine, 16 sine
constexpr int LX = 128;       // pixels of a tile
constexpr int LM = 17;        // |p-modes|: 0 .. 16
constexpr int PROJ = 128;     // hidden width of the projection
constexpr int kMaxParams = 14;
constexpr long long kLayerPolls = 1LL << 20;

enum { LAYER_LIFT = 0, LAYER_MID = 1, LAYER_LAST = 2 };

// byte offsets of the shared-memory buffers (each on 1024 bytes: the swizzle's period)
constexpr uint32_t S_AAH = 0, S_AAL = 16384, S_CS = 32768, S_WH = 65536, S_WL = 69632, S_SLOT = 73728;
// per slot: V twice; VL: low parts of v, then (with the 16 KiB after it) v' transposed, four chunks of 32 high and 32
// low rows, or the high and low parts of v' for the projection; G: high rows, then low rows
constexpr uint32_t T_V = 0, T_VL = 32768, T_B2L = 49152, T_G = 65536, T_BYTES = 73728;
constexpr uint32_t S_BYTES = S_SLOT + 2 * T_BYTES;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t D1_COL = 0, D2_COL = 128, SLOT_COLS = 256;  // 2 x 64 columns each; D2 also the 128-wide hidden layer

struct LayerArgs {
  const float* vin;    // [rows][G1][32], swizzled
  const float* gx;     // [rows][32 o][32 k], swizzled
  const float* AA;     // 32 x G1
  const float* CS;     // G1 x 32
  const float* W;      // 32 x 32 (o, c)
  const float* bias;   // 32
  const float* par;    // LIFT: rows / G0 x NP inputs; W is then 32 x (NP + 2): inputs, x, p
  int NP, G0;
  const float *xs, *ps;  // LIFT: the coordinates
  int* status;
  float* vout;         // swizzled
  float* fx;           // [tile][rows][32 o][32 k]
  const float *Q1, *c1, *Q2, *c2;  // LAST
  float* out;          // LAST: [rows][G1]
  int rows, G1, tiles, act;  // act: 0 none, 1 GELU, 2 times GELU'(aux)
  const float* aux;     // channel-major [b][32][G0][G1], as vcm; LIFT: v' is read from it instead
  float* vcm;           // MID: optional copy of v'
};

// float index of element (row, k) of a 128-byte-row, 128-byte-swizzled tile
__device__ __forceinline__ int sw(int row, int k) { return row * 32 + ((((k >> 2) ^ row) & 7) << 2) + (k & 3); }

// K-major, 128-byte swizzle, 1024 bytes between 8-row groups
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<uint64_t>(dst)),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_store_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_store_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

template <int MODE>
__global__ void __launch_bounds__(256, 1) fno_layer_kernel(LayerArgs a) {
  using namespace umma;
  extern __shared__ __align__(128) unsigned char sm_dyn[];
  __shared__ __align__(8) uint64_t bars[2][5];  // per slot: [0], [1] loads of v into buffer 0, 1; [2] D1 done; [3] D2 / hidden done; [4] load of G
  __shared__ uint32_t tmem_base;
  __shared__ float s_bias[LC], s_c1[PROJ], s_q2[PROJ], s_row[2][LC];
  unsigned char* sm = sm_dyn + ((1024u - (smem_u32(sm_dyn) & 1023u)) & 1023u);
  const int tid = threadIdx.x, st = tid & 127, lane = tid & 31;
  const int uw = __shfl_sync(0xffffffffu, tid >> 5, 0), slot = uw >> 2, warp = uw & 3;  // warp-uniform
  const int tile = blockIdx.x % a.tiles, x0 = tile * LX;
  const int nx = min(LX, a.G1 - x0);
  const int ncta = (gridDim.x - tile + a.tiles - 1) / a.tiles;  // CTAs of this x tile
  const int stride = 2 * ncta;
  const bool next = MODE != LAYER_LAST && a.fx != nullptr;  // v' goes on: pixel-major copy and x-transform

  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < 2; ++s)
      for (int i = 0; i < 5; ++i) mbar_init(&bars[s][i], 1);
    mbar_fence_init();
  }
  float* AAh = reinterpret_cast<float*>(sm + S_AAH);
  float* AAl = reinterpret_cast<float*>(sm + S_AAL);
  float* CSs = reinterpret_cast<float*>(sm + S_CS);
  float* Wh = reinterpret_cast<float*>(sm + S_WH);
  float* Wl = reinterpret_cast<float*>(sm + S_WL);  // right after the high rows
  if (MODE != LAYER_LIFT) {
    for (int i = tid; i < LX * LK; i += 256) {
      const int k = i >> 7, x = i & 127;
      float h, l;
      split_tf32(x < nx ? __ldg(a.AA + (size_t)k * a.G1 + x0 + x) : 0.f, h, l);
      AAh[sw(x, k)] = h;
      AAl[sw(x, k)] = l;
    }
    for (int i = tid; i < LC * LC; i += 256) {
      float h, l;
      split_tf32(__ldg(a.W + i), h, l);
      Wh[sw(i >> 5, i & 31)] = h;
      Wl[sw(i >> 5, i & 31)] = l;
    }
  }
  if (next) {
    // 4 chunks of 32 pixels: rows 0-31 the modes' high parts, 32-63 the low parts
    for (int i = tid; i < LX * LK; i += 256) {
      const int x = i >> 5, k = i & 31;
      float h, l;
      split_tf32(x < nx ? __ldg(a.CS + (size_t)(x0 + x) * LK + k) : 0.f, h, l);
      CSs[(x >> 5) * 2048 + sw(k, x & 31)] = h;
      CSs[(x >> 5) * 2048 + sw(32 + k, x & 31)] = l;
    }
  } else if (MODE == LAYER_LAST) {
    for (int i = tid; i < PROJ * LC; i += 256) {
      float h, l;
      split_tf32(__ldg(a.Q1 + i), h, l);
      CSs[sw(i >> 5, i & 31)] = h;
      CSs[4096 + sw(i >> 5, i & 31)] = l;
    }
    if (tid < PROJ) {
      s_c1[tid] = __ldg(a.c1 + tid);
      s_q2[tid] = __ldg(a.Q2 + tid);
    }
  }
  if (tid < LC) s_bias[tid] = a.bias != nullptr ? __ldg(a.bias + tid) : 0.f;
  float* s_w0 = AAh;  // LIFT: the input weights, input-major, in the unused DFT tile
  if (MODE == LAYER_LIFT && a.aux == nullptr)
    for (int i = tid; i < LC * (a.NP + 2); i += 256) s_w0[(i % (a.NP + 2)) * LC + i / (a.NP + 2)] = __ldg(a.W + i);
  unsigned char* mine = sm + S_SLOT + slot * T_BYTES;
  // pixels past the row's end are never loaded: keep their buffer rows finite
  for (int i = st; i < (int)(T_VL / 16); i += 128) reinterpret_cast<float4*>(mine + T_V)[i] = make_float4(0, 0, 0, 0);
  proxy_fence_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base + slot * SLOT_COLS;
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
  float* Vl = reinterpret_cast<float*>(mine + T_VL);    // low parts of v, then high parts of v' transposed
  float* B2l = reinterpret_cast<float*>(mine + T_B2L);  // low parts of v' transposed (or of v' for the projection)
  float* G = reinterpret_cast<float*>(mine + T_G);
  const uint32_t aVl = smem_u32(Vl), aB2l = smem_u32(B2l), aG = smem_u32(G);
  const uint32_t aAAh = smem_u32(AAh), aAAl = smem_u32(AAl), aCS = smem_u32(CSs), aW = smem_u32(Wh);
  uint64_t* bar = bars[slot];
  const uint32_t vbytes = (uint32_t)nx * LC * 4;
  const size_t chs = (size_t)a.G0 * a.G1;                     // channel stride of the channel-major arrays
  auto cm_base = [&](int r) {                                 // this thread's pixel of row r, channel 0
    const int b = r / a.G0;
    return ((size_t)b * LC * a.G0 + (r - b * a.G0)) * a.G1 + x0 + st;
  };
  auto slot_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + slot) : "memory"); };
  // a wait of this thread ran out.  The slot's threads decide on it together, at
  // their barrier: a flag in memory, set by a later wait while a slower thread still
  // reads it for the earlier one, would part them
  bool bad = false;
  auto slot_any = [&](bool v) {  // slot_sync that returns whether any thread of the slot brought v
    uint32_t r;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(1 + slot)
        : "memory");
    return r != 0;
  };
  auto load_v = [&](int r, int buf) {  // one thread of the slot
    mbar_arrive_expect_tx(&bar[buf], vbytes);
    bulk_load(mine + T_V + buf * 16384, a.vin + ((size_t)r * a.G1 + x0) * LC, vbytes, &bar[buf]);
  };
  auto load_g = [&](int r) {
    mbar_arrive_expect_tx(&bar[4], LC * LK * 4);
    bulk_load(mine + T_G, a.gx + (size_t)r * LC * LK, LC * LK * 4, &bar[4]);
  };
  // D += A B^T over one 32-wide chunk, three products
  auto mma3 = [&](uint32_t d, uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, uint32_t id) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      umma_tf32(d, desc_sw128(ah + 32 * q), desc_sw128(bh + 32 * q), id, q > 0);
      umma_tf32(d, desc_sw128(ah + 32 * q), desc_sw128(bl + 32 * q), id, 1u);
      umma_tf32(d, desc_sw128(al + 32 * q), desc_sw128(bh + 32 * q), id, 1u);
    }
  };
  uint32_t ph_ld = 0, ph1 = 0, ph2 = 0, ph_g = 0;  // ph_ld: bit b = parity of load barrier b
  bool d2_pending = false, ok = true;
  int prev = 0;
  // D2 (or the hidden layer) complete: its operands' buffers may be written again
  auto wait_d2 = [&] {
    if (!mbar_wait_bounded(&bar[3], ph2, kLayerPolls)) bad = true;
    ph2 ^= 1u;
    tc_fence_after();
  };
  // store the transform of row `prev`: its high and low mode parts sit 32 TMEM rows apart
  auto store_d2 = [&] {
    float s[LC];
    float t[64];
    tmem_ld64(trow + D2_COL, t);
#pragma unroll
    for (int i = 0; i < LC; ++i) s[i] = t[i] + t[32 + i];
    tmem_ld64(trow + D2_COL + 64, t);
#pragma unroll
    for (int i = 0; i < LC; ++i) s[i] = (s[i] + t[i]) + t[32 + i];
    const int k = (warp & 1) * 16 + lane;  // lanes 0 .. 15 hold rows 16 warp + lane
    if (warp >= 2 && lane < 16) {
#pragma unroll
      for (int o = 0; o < LC; ++o) B2l[o * LK + k] = s[o];
    }
    tc_fence_before();
    slot_sync();
    if (warp < 2 && lane < 16) {
      float* f = a.fx + ((size_t)tile * a.rows + prev) * (LC * LK) + k;
#pragma unroll
      for (int o = 0; o < LC; ++o) f[o * LK] = s[o] + B2l[o * LK + k];
    }
    slot_sync();
  };

  int buf = 0;
  int r = (int)(blockIdx.x / a.tiles) * 2 + slot;
  if (MODE != LAYER_LIFT && r < a.rows && warp == 0 && elect_lane()) {
    load_v(r, 0);
    load_g(r);
  }
  for (; r < a.rows; r += stride) {
    float* V = reinterpret_cast<float*>(mine + T_V + buf * 16384);
    const bool d2_prev = d2_pending;
    if (d2_prev) wait_d2();
    d2_pending = false;
    float v[LC];
    if (MODE != LAYER_LIFT) {
      if (!mbar_wait_bounded(&bar[buf], (ph_ld >> buf) & 1u, kLayerPolls)) bad = true;
      ph_ld ^= 1u << buf;
      if (!mbar_wait_bounded(&bar[4], ph_g, kLayerPolls)) bad = true;
      ph_g ^= 1u;
      // split in place: high parts stay, low parts beside them
      float4 w[10];  // all loads first
#pragma unroll
      for (int i = 0; i < 10; ++i)
        w[i] = i < 8 ? reinterpret_cast<float4*>(V)[st + i * 128] : reinterpret_cast<float4*>(G)[st + (i - 8) * 128];
#pragma unroll
      for (int i = 0; i < 10; ++i) {
        float4 l;
        split_tf32(w[i].x, w[i].x, l.x);
        split_tf32(w[i].y, w[i].y, l.y);
        split_tf32(w[i].z, w[i].z, l.z);
        split_tf32(w[i].w, w[i].w, l.w);
        reinterpret_cast<float4*>(i < 8 ? V : G - 1024 * 4)[st + i * 128] = w[i];
        reinterpret_cast<float4*>(i < 8 ? Vl : G - 1024 * 4 + 1024)[st + i * 128] = l;
      }
      proxy_fence_smem();
      tc_fence_before();
      ok = !slot_any(bad);
      tc_fence_after();
      if (!ok) break;
      const int nr = r + stride;
      if (warp == 0 && elect_lane()) {
        const uint32_t id2 = instr_desc(2 * LC), id = instr_desc(LC), aV = smem_u32(V);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t d = tmem + D1_COL, o = 32 * q;
          umma_tf32(d, desc_sw128(aAAh + o), desc_sw128(aG + o), id2, q > 0);
          umma_tf32(d + 64, desc_sw128(aV + o), desc_sw128(aW + o), id2, q > 0);
          umma_tf32(d, desc_sw128(aAAl + o), desc_sw128(aG + o), id, 1u);
          umma_tf32(d + 64, desc_sw128(aVl + o), desc_sw128(aW + o), id, 1u);
        }
        umma_commit(&bar[2]);
        if (nr < a.rows) {
          bulk_store_read_done();  // the other buffer's outgoing copy has been read
          load_v(nr, buf ^ 1);
        }
      }
      if (MODE == LAYER_MID && d2_prev) store_d2();  // while D1 is computed
      if (!mbar_wait_bounded(&bar[2], ph1, kLayerPolls)) bad = true;
      ph1 ^= 1u;
      tc_fence_after();
      if (nr < a.rows && warp == 0 && elect_lane()) load_g(nr);
      float t[64];
      tmem_ld64(trow + D1_COL, t);
#pragma unroll
      for (int i = 0; i < LC; ++i) v[i] = t[i] + t[32 + i];
      tmem_ld64(trow + D1_COL + 64, t);
#pragma unroll
      for (int i = 0; i < LC; ++i) v[i] = v[i] + (t[i] + t[32 + i]) + s_bias[i];
      if (a.act == 1) {
#pragma unroll
        for (int i = 0; i < LC; i += 2) gelu2(v[i], v[i + 1]);
      } else if (MODE == LAYER_MID && a.act == 2) {
        const float* p = a.aux + cm_base(r);
#pragma unroll
        for (int h = 0; h < LC; h += 16) {
          float x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = st < nx ? __ldg(p + (h + i) * chs) : 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) v[h + i] *= gelu_d_tail(x[i]);
        }
      }
    } else {
      if (d2_prev) store_d2();
      if (warp == 0 && elect_lane()) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the buffers alternate
      if (a.aux == nullptr && warp == 1) {  // the row's constant part, a channel per lane
        const int b = r / a.G0;
        float c = s_bias[lane] + s_w0[(a.NP + 1) * LC + lane] * __ldg(a.ps + (r - b * a.G0));
        for (int q = 0; q < a.NP; ++q) c += s_w0[q * LC + lane] * __ldg(a.par + (size_t)b * a.NP + q);
        s_row[slot][lane] = c;
      }
      slot_sync();  // the outgoing copy of this buffer has been read
      if (a.aux != nullptr) {
        const float* p = a.aux + cm_base(r);
#pragma unroll
        for (int i = 0; i < LC; ++i) v[i] = st < nx ? __ldg(p + i * chs) : 0.f;
      } else {
        const float x = st < nx ? __ldg(a.xs + x0 + st) : 0.f;
#pragma unroll
        for (int i = 0; i < LC; ++i) v[i] = s_row[slot][i] + s_w0[a.NP * LC + i] * x;
      }
    }
    if (st >= nx) {
#pragma unroll
      for (int i = 0; i < LC; ++i) v[i] = 0.f;
    }
    if (MODE == LAYER_MID && a.vcm != nullptr && st < nx) {
      float* p = a.vcm + cm_base(r);
#pragma unroll
      for (int i = 0; i < LC; ++i) p[i * chs] = v[i];
    }
    if (MODE != LAYER_LAST && !next) {  // nothing on the chip follows
      buf ^= 1;
      continue;
    }
    if (MODE != LAYER_LAST) {
      // v' as a pixel row for the outgoing copy, and transposed (channel rows
      // of 32 pixels per warp), split, for the x-transform
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float4*>(V + sw(st, 4 * j)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
#pragma unroll
      for (int o = 0; o < LC; ++o) {
        float h, l;
        split_tf32(v[o], h, l);
        Vl[warp * 2048 + sw(o, lane)] = h;
        Vl[warp * 2048 + 1024 + sw(o, lane)] = l;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float4 h, l;
        split_tf32(v[4 * j], h.x, l.x);
        split_tf32(v[4 * j + 1], h.y, l.y);
        split_tf32(v[4 * j + 2], h.z, l.z);
        split_tf32(v[4 * j + 3], h.w, l.w);
        *reinterpret_cast<float4*>(Vl + sw(st, 4 * j)) = h;
        *reinterpret_cast<float4*>(B2l + sw(st, 4 * j)) = l;
      }
    }
    proxy_fence_smem();
    tc_fence_before();
    ok = !slot_any(bad);
    tc_fence_after();
    if (!ok) break;
    if (warp == 0 && elect_lane()) {
      if (MODE != LAYER_LAST) {
        const uint32_t id = (instr_desc(2 * LC) & ~(0x1Fu << 24)) | (4u << 24);  // M = 64
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
          for (int c = 0; c < 2; ++c) {  // pixels 64 c + 8 q .. : neighbouring products have accumulators of their own
            const uint32_t o = 8192 * (2 * c + (q >> 2)) + 32 * (q & 3);
            umma_tf32(tmem + D2_COL + c * 64, desc_sw128(aCS + o), desc_sw128(aVl + o), id, q > 0);
          }
      } else {
        mma3(tmem + D2_COL, aVl, aB2l, aCS, aCS + 16384, instr_desc(PROJ));
      }
      umma_commit(&bar[3]);
      if (MODE != LAYER_LAST) bulk_store(a.vout + ((size_t)r * a.G1 + x0) * LC, V, vbytes);
    }
    d2_pending = true;
    prev = r;
    if (MODE == LAYER_LAST) {
      wait_d2();
      d2_pending = false;
      float sum = 0.f;
#pragma unroll 1
      for (int cb = 0; cb < PROJ / 64; ++cb) {
        float t[64];
        tmem_ld64(trow + D2_COL + cb * 64, t);
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          float h0 = t[i] + s_c1[cb * 64 + i], h1 = t[i + 1] + s_c1[cb * 64 + i + 1];
          gelu2(h0, h1);
          sum += s_q2[cb * 64 + i] * h0;
          sum += s_q2[cb * 64 + i + 1] * h1;
        }
      }
      if (st < nx) a.out[(size_t)r * a.G1 + x0 + st] = sum + __ldg(a.c2);
    }
    buf ^= 1;
  }
  if (ok && d2_pending) {
    wait_d2();
    store_d2();
    d2_pending = false;
  }
  if (bad) atomicCAS(a.status, 0, FW_FNO_TIMEOUT);
  if (warp == 0) {
    const bool drain = !ok || __any_sync(0xffffffffu, bad);
    if (drain && elect_lane()) {
      // products and copies still in flight: once more, bounded, before the buffers are released
      mbar_wait_bounded(&bar[2], ph1, kLayerPolls >> 8);
      if (d2_pending) mbar_wait_bounded(&bar[3], ph2, kLayerPolls >> 8);
      for (int i = 0; i < 2; ++i) mbar_wait_bounded(&bar[i], (ph_ld >> i) & 1u, kLayerPolls >> 8);
      mbar_wait_bounded(&bar[4], ph_g, kLayerPolls >> 8);
    }
  }
  if (warp == 0 && elect_lane()) bulk_store_done();
  tc_fence_before();
  __syncthreads();
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// ---------------------------------------------------------------------------
// Truncated p-transforms, FP32 FMAs.  Modes +m and -m share their cosines and
// sines: with C_m = sum_p cos F and S_m = sum_p sin F, the coefficient at +-m is
// C_m -+ i S_m (17 values of m instead of 32 modes: half the multiply-adds).
// The tables (cosines, sines) sit in shared memory and are read by broadcast;
// a thread owns one x-mode (complex) and every eighth row p.  Four CTAs (a
// cluster) share a channel's rows and add their sums through distributed
// shared memory: one CTA per channel left most of the chip waiting on its loads.
constexpr int kPdftSplit = 4;
// TILES: x tiles to add up (0: the argument's number), known so that their loads go out together
template <int TILES>
__global__ void __cluster_dims__(1, 1, kPdftSplit) __launch_bounds__(128) fno_pdft_kernel(int rows, int G0, int tiles, const float* __restrict__ fx,
                                                       const float* __restrict__ Dpv, float* __restrict__ F2) {
  extern __shared__ __align__(16) float tabs[];  // [rows of this CTA][2 LM]
  cg::cluster_group cl = cg::this_cluster();
  const int o = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int per = (G0 + kPdftSplit - 1) / kPdftSplit, p0 = blockIdx.z * per, np = max(0, min(per, G0 - p0));
  for (int i = tid; i < LM * np; i += 128) {
    const int m = i / np, p = i - m * np;
    const float2 cs = __ldg(reinterpret_cast<const float2*>(Dpv + (size_t)m * 2 * G0 + 2 * (p0 + p)));
    tabs[p * 2 * LM + 2 * m] = cs.x;
    tabs[p * 2 * LM + 2 * m + 1] = m == 16 ? -cs.y : cs.y;  // row 16 of the matrix is mode -16
  }
  __syncthreads();
  const int kx = tid & 15, pg = tid >> 4;
  float2 C[LM], S[LM];
#pragma unroll
  for (int m = 0; m < LM; ++m) C[m] = S[m] = make_float2(0.f, 0.f);
  const size_t ts = (size_t)rows * (LC * LK);
  const float* f = fx + ((size_t)b * G0 + p0) * (LC * LK) + o * LK + kx;
#pragma unroll 2
  for (int p = pg; p < np; p += 8) {
    const float* q = f + (size_t)p * (LC * LK);
    float re = __ldg(q), im = __ldg(q + 16);
    if constexpr (TILES > 0) {
#pragma unroll
      for (int t = 1; t < TILES; ++t) {
        re += __ldg(q + t * ts);
        im += __ldg(q + t * ts + 16);
      }
    } else {
      for (int t = 1; t < tiles; ++t) {
        re += __ldg(q + t * ts);
        im += __ldg(q + t * ts + 16);
      }
    }
    const float2* tp = reinterpret_cast<const float2*>(tabs + p * 2 * LM);
#pragma unroll
    for (int m = 0; m < LM; ++m) {
      const float2 cs = tp[m];
      C[m].x += cs.x * re;
      C[m].y += cs.x * im;
      S[m].x += cs.y * re;
      S[m].y += cs.y * im;
    }
  }
  // sum the eight row groups: pairs of groups share a warp, then through shared memory
#pragma unroll
  for (int m = 0; m < LM; ++m) {
    C[m].x += __shfl_xor_sync(0xffffffffu, C[m].x, 16);
    C[m].y += __shfl_xor_sync(0xffffffffu, C[m].y, 16);
    S[m].x += __shfl_xor_sync(0xffffffffu, S[m].x, 16);
    S[m].y += __shfl_xor_sync(0xffffffffu, S[m].y, 16);
  }
  __syncthreads();  // the tables are no longer read
  float4* red = reinterpret_cast<float4*>(tabs);  // [4 warps][LM][16]
  if ((tid & 16) == 0)
#pragma unroll
    for (int m = 0; m < LM; ++m) red[((tid >> 5) * LM + m) * 16 + kx] = make_float4(C[m].x, C[m].y, S[m].x, S[m].y);
  __syncthreads();
  cl.sync();
  float* out = F2 + ((size_t)b * LC + o) * (2 * 32 * 16);
  for (int i = blockIdx.z * 128 + tid; i < LM * 16; i += 128 * kPdftSplit) {
    const int m = i >> 4, k = i & 15;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < kPdftSplit; ++c) {
      const float4* rc = cl.map_shared_rank(red, c);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float4 t = rc[w * LM * 16 + i];
        s.x += t.x;
        s.y += t.y;
        s.z += t.z;
        s.w += t.w;
      }
    }
    // (c - i s)(re + i im): +m at row m; -m (m >= 1) at row 32 - m
    if (m < 16) {
      out[m * 16 + k] = s.x + s.w;
      out[512 + m * 16 + k] = s.y - s.z;
    }
    if (m > 0) {
      out[(32 - m) * 16 + k] = s.x - s.w;
      out[512 + (32 - m) * 16 + k] = s.y + s.z;
    }
  }
  cl.sync();  // no CTA leaves while its sums are read
}

// gx[b][p][o][k] (swizzled rows) = sum over the 32 p-modes of O2[b][o][2][32 x 16].
__global__ void __launch_bounds__(128) fno_pidft_kernel(int G0, const float* __restrict__ O2,
                                                        const float* __restrict__ Dpiv, float* __restrict__ gx) {
  extern __shared__ float tabs[];  // [p of this block][2 LM]
  const int o = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int per = (G0 + gridDim.z - 1) / gridDim.z, p0 = blockIdx.z * per, np = min(per, G0 - p0);
  for (int i = tid; i < LM * np; i += 128) {
    const int p = i / LM, m = i - p * LM;
    const float* d = Dpiv + (size_t)(2 * (p0 + p)) * 64 + m;
    tabs[p * 2 * LM + 2 * m] = __ldg(d);
    const float s = __ldg(d + 64);
    tabs[p * 2 * LM + 2 * m + 1] = m == 16 ? -s : s;
  }
  const int kx = tid & 15, pg = tid >> 4;
  const float* in = O2 + ((size_t)b * LC + o) * (2 * 32 * 16) + kx;
  float2 A[LM], D[LM];  // sums and differences of the coefficients at +m and -m
#pragma unroll
  for (int m = 0; m < LM; ++m) {
    const float2 hi = m < 16 ? make_float2(__ldg(in + m * 16), __ldg(in + 512 + m * 16)) : make_float2(0.f, 0.f);
    const float2 lo = m > 0 ? make_float2(__ldg(in + (32 - m) * 16), __ldg(in + 512 + (32 - m) * 16)) : make_float2(0.f, 0.f);
    A[m] = make_float2(hi.x + lo.x, hi.y + lo.y);
    D[m] = make_float2(hi.x - lo.x, hi.y - lo.y);
  }
  __syncthreads();
  for (int p = pg; p < np; p += 8) {
    const float2* tp = reinterpret_cast<const float2*>(tabs + p * 2 * LM);
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int m = 0; m < LM; ++m) {
      const float2 cs = tp[m];
      re += cs.x * A[m].x - cs.y * D[m].y;
      im += cs.x * A[m].y + cs.y * D[m].x;
    }
    float* g = gx + ((size_t)b * G0 + p0 + p) * (LC * LK);
    g[sw(o, kx)] = re;
    g[sw(o, 16 + kx)] = im;
  }
}

// ---------------------------------------------------------------------------
// Surrogate output: harmonic baseline + its peak x network, normalised.  The
// baseline exp(-c (H - min H)), H = p^2/2 + w^2 (x - x_e)^2/2 with its minimum over the
// grid (a well centred far outside the box would underflow everywhere), is a
// product of two Gaussians, so its sum and its peak come from two vectors per
// sample; one pass adds and sums (FP64), a second scales.
__device__ __forceinline__ double block_reduce(double v, double* red, bool max_) {
  for (int o = 16; o > 0; o >>= 1) {
    const double u = __shfl_xor_sync(0xffffffffu, v, o);
    v = max_ ? fmax(v, u) : v + u;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); ++i) v = max_ ? fmax(v, red[i]) : v + red[i];
  return v;
}

__global__ void __launch_bounds__(256) fno_thermal_kernel(int G0, int G1, const double* __restrict__ wc, const double* __restrict__ xs,
                                                          const double* __restrict__ ps, double x_e, float* out,
                                                          double* __restrict__ part) {
  extern __shared__ double gs[];  // [G1] x Gaussian, [rows of this block] p Gaussian
  __shared__ double red[8];
  const int b = blockIdx.y, tid = threadIdx.x;
  const double w = wc[2 * b], c = wc[2 * b + 1];
  const int per = (G0 + gridDim.x - 1) / gridDim.x, p0 = blockIdx.x * per, np = max(0, min(per, G0 - p0));
  double sx = 0, mx = 0, sp = 0, mp = 0, ex = -INFINITY, ep = -INFINITY;  // ex, ep: less the minima of the two exponents
  for (int i = tid; i < G1; i += 256) {
    const double d = w * (xs[i] - x_e), e = 0.5 * d * d;
    gs[i] = e;
    ex = fmax(ex, -e);
  }
  for (int i = tid; i < G0; i += 256) ep = fmax(ep, -0.5 * ps[i] * ps[i]);
  ex = block_reduce(ex, red, true);
  ep = block_reduce(ep, red, true);
  for (int i = tid; i < G1; i += 256) {
    const double g = exp(-c * (gs[i] + ex));
    gs[i] = g;
    sx += g;
    mx = fmax(mx, g);
  }
  for (int i = tid; i < G0; i += 256) {
    const double g = exp(-c * (0.5 * ps[i] * ps[i] + ep));
    if (i >= p0 && i < p0 + np) gs[G1 + i - p0] = g;
    sp += g;
    mp = fmax(mp, g);
  }
  sx = block_reduce(sx, red, false);
  mx = block_reduce(mx, red, true);
  sp = block_reduce(sp, red, false);
  mp = block_reduce(mp, red, true);
  const double inv = 1.0 / (sx * sp);
  const float peak = (float)(mx * mp * inv);
  double s = 0;
  float* o = out + ((size_t)b * G0 + p0) * G1;
  for (int p = 0; p < np; ++p) {
    const double gp = gs[G1 + p] * inv;
    for (int x = tid; x < G1; x += 256) {
      const float v = (float)(gs[x] * gp) + peak * o[(size_t)p * G1 + x];
      o[(size_t)p * G1 + x] = v;
      s += (double)v;
    }
  }
  s = block_reduce(s, red, false);
  if (tid == 0) part[(size_t)b * gridDim.x + blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) fno_scale_kernel(long long n, int nparts, const double* __restrict__ part, double dxdp,
                                                        float* out) {
  const int b = blockIdx.y;
  double s = 0;
  for (int i = 0; i < nparts; ++i) s += part[(size_t)b * nparts + i];
  const float f = (float)(s * dxdp);
  float* o = out + (size_t)b * n;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) o[i] = o[i] / f;
}

template <int MODE> cudaError_t launch_layer(const LayerArgs& a, cudaStream_t st) {
  static PerDeviceOnce attr;
  cudaError_t e = set_smem_once(attr, fno_layer_kernel<MODE>, S_BYTES + 1024);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long want = (long long)a.tiles * ((a.rows + 1) / 2);
  int grid = (int)(want < sms ? want : sms);
  if (grid < a.tiles) grid = a.tiles;
  fno_layer_kernel<MODE><<<grid, 256, S_BYTES + 1024, st>>>(a);
  return cudaGetLastError();
}

constexpr int kMaxG0 = 1024;  // p-transform tables in shared memory: 136 bytes per row of a CTA

int check_dims(int B, int G0, int G1, const char* who) {
  if (B <= 0 || B > 65535 || G0 < 32 || G0 > kMaxG0 || G1 < 32 || G1 > 65536 || G1 % 4 != 0)
    return fail(FW_EINVAL, std::string(who) + ": needs 1 <= B <= 65535, 32 <= G0 <= 1024, G1 >= 32 a multiple of 4");
  return FW_OK;
}
bool on16(const void* p) { return p != nullptr && ((uintptr_t)p & 15u) == 0; }
}  // namespace fnol
}  // namespace fw

using namespace fw;
using namespace fw::fnol;

extern "C" int fw_fno_layer(int mode, int B, int G0, int G1, const float* vin, const float* gx, const float* AA,
                            const float* CS, const float* W, const float* bias, int act, int NP, const float* par,
                            const float* xs, const float* ps, const float* Q1, const float* c1, const float* Q2, const float* c2,
                            float* vout, float* fx, float* out, const float* aux, float* vcm, void* stream) {
  if (int rc = check_dims(B, G0, G1, "fw_fno_layer")) return rc;
  if (mode < LAYER_LIFT || mode > LAYER_LAST) return fail(FW_EINVAL, "fw_fno_layer: mode must be 0, 1 or 2");
  const bool copy = mode == LAYER_LIFT && aux != nullptr;
  if (!copy && (W == nullptr || (bias == nullptr && mode != LAYER_MID)))
    return fail(FW_EINVAL, "fw_fno_layer: NULL weights");
  if (mode == LAYER_LIFT && (NP < 0 || NP > kMaxParams)) return fail(FW_EINVAL, "fw_fno_layer: NP must be in [0, 14]");
  if (act < 0 || act > 2 || (act == 2 && (mode != LAYER_MID || aux == nullptr)))
    return fail(FW_EINVAL, "fw_fno_layer: act must be 0, 1 or (mode 1, with aux) 2");
  if (mode == LAYER_LIFT ? (!copy && ((NP > 0 && par == nullptr) || xs == nullptr || ps == nullptr))
                         : (!on16(vin) || !on16(gx) || AA == nullptr))
    return fail(FW_EINVAL, "fw_fno_layer: NULL input, or activations off 16 bytes");
  if (mode == LAYER_LAST ? (Q1 == nullptr || c1 == nullptr || Q2 == nullptr || c2 == nullptr || out == nullptr)
      : fx == nullptr    ? (mode != LAYER_MID || vcm == nullptr || vout != nullptr)
                         : (!on16(vout) || CS == nullptr))
    return fail(FW_EINVAL, "fw_fno_layer: NULL output, or activations off 16 bytes");
  if (vcm != nullptr && mode != LAYER_MID) return fail(FW_EINVAL, "fw_fno_layer: vcm is mode 1's");
  LayerArgs a{};
  a.vin = vin, a.gx = gx, a.AA = AA, a.CS = CS, a.W = W, a.bias = bias, a.act = act;
  a.NP = NP, a.par = par, a.xs = xs, a.ps = ps, a.G0 = G0;
  if (int rc = fno_status_ptr(&a.status)) return rc;
  a.vout = vout, a.fx = fx, a.Q1 = Q1, a.c1 = c1, a.Q2 = Q2, a.c2 = c2, a.out = out;
  a.aux = aux, a.vcm = vcm;
  a.rows = B * G0, a.G1 = G1, a.tiles = (G1 + LX - 1) / LX;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = mode == LAYER_LIFT  ? launch_layer<LAYER_LIFT>(a, st)
                  : mode == LAYER_MID ? launch_layer<LAYER_MID>(a, st)
                                      : launch_layer<LAYER_LAST>(a, st);
  count_launch(1);
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_layer");
}

extern "C" int fw_fno_pdft(int B, int G0, int G1, const float* fx, const float* Dpv, float* F2, void* stream) {
  if (int rc = check_dims(B, G0, G1, "fw_fno_pdft")) return rc;
  if (fx == nullptr || Dpv == nullptr || F2 == nullptr) return fail(FW_EINVAL, "fw_fno_pdft: NULL argument");
  if (((uintptr_t)Dpv & 7u) != 0) return fail(FW_EINVAL, "fw_fno_pdft: Dpv must start on 8 bytes");
  const size_t tab = (size_t)((G0 + kPdftSplit - 1) / kPdftSplit) * 2 * LM * 4, red = 4 * LM * 16 * 16;
  const size_t smem = tab > red ? tab : red;  // at most 34 KiB (G0 = 1024)
  const int tiles = (G1 + LX - 1) / LX;
  auto kern = tiles == 1 ? fno_pdft_kernel<1> : tiles == 2 ? fno_pdft_kernel<2> : tiles == 3 ? fno_pdft_kernel<3>
            : tiles == 4 ? fno_pdft_kernel<4> : fno_pdft_kernel<0>;
  kern<<<dim3(LC, B, kPdftSplit), 128, smem, static_cast<cudaStream_t>(stream)>>>(B * G0, G0, tiles, fx, Dpv, F2);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_pdft");
}

extern "C" int fw_fno_pidft(int B, int G0, const float* O2, const float* Dpiv, float* gx, void* stream) {
  if (int rc = check_dims(B, G0, 32, "fw_fno_pidft")) return rc;
  if (O2 == nullptr || Dpiv == nullptr || gx == nullptr) return fail(FW_EINVAL, "fw_fno_pidft: NULL argument");
  const int nz = G0 >= 256 ? 4 : 1;
  const size_t smem = (size_t)((G0 + nz - 1) / nz) * 2 * LM * 4;
  fno_pidft_kernel<<<dim3(LC, B, nz), 128, smem, static_cast<cudaStream_t>(stream)>>>(G0, O2, Dpiv, gx);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_pidft");
}

extern "C" int fw_fno_thermal(int B, int G0, int G1, const double* wc, const double* xs, const double* ps, double x_e,
                              double dxdp, float* out, double* work, void* stream) {
  if (B <= 0 || B > 65535 || G0 <= 0 || G1 <= 0 || G1 > 16384 || G0 > (1 << 20))
    return fail(FW_EINVAL, "fw_fno_thermal: bad size");
  if (wc == nullptr || xs == nullptr || ps == nullptr || out == nullptr || work == nullptr)
    return fail(FW_EINVAL, "fw_fno_thermal: NULL argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int nb = 64, per = (G0 + nb - 1) / nb;
  const size_t smem = (size_t)(G1 + per) * sizeof(double);
  static PerDeviceOnce attr;
  cudaError_t e = set_smem_once(attr, fno_thermal_kernel, 200 << 10);
  if (e != cudaSuccess) return cuda_fail(e, "fw_fno_thermal");
  if (smem > (size_t)(200 << 10)) return fail(FW_EINVAL, "fw_fno_thermal: grid too large");
  fno_thermal_kernel<<<dim3(nb, B), 256, smem, st>>>(G0, G1, wc, xs, ps, x_e, out, work);
  fno_scale_kernel<<<dim3(64, B), 256, 0, st>>>((long long)G0 * G1, nb, work, dxdp, out);
  count_launch(2);
  e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_thermal");
}
