// The surrogate network's whole forward pass (n_in <= 64 -> w -> w -> w -> out_pad, w = 128 or
// 256, SiLU on the hidden layers) in one persistent tcgen05 kernel: a 128-row tile's activations never leave
// the SM between layers.
//
// One CTA per SM (704 threads, 22 warps), looping over 128-row tiles.  Several tiles are in flight
// per CTA, in slots: three for the narrow network with up to 160 outputs, else two (fused_plan).
// Each slot owns a 128 x w BF16 activation buffer in shared memory (16 KB K-chunks in the
// 128-byte-swizzled K-major layout the MMA reads) and an FP32 accumulator in tensor memory.  The
// units of work -- (slot, layer) -- run in the order (0,L1) (1,L1) .. (0,L2) (1,L2) .., so the
// tensor cores work on one slot while the epilogue warps drain another:
//   warp 0, lane 0  TMA producer: a tile's BF16 input rows (128 x 64; the narrow network's slots
//                   have input buffers of their own, so the next tile's are fetched early), and
//                   the weights, 128 output rows x 64 K at a time, through a ring of four 16 KB
//                   stages (the same for every tile and L2-resident; a layer of the narrow
//                   network is loaded once for all slots)
//   warp 1          MMA issuer: per stage four K = 16 tcgen05.mma (M = 128, N = 128 or the
//                   output layer's remainder) from the slot's activation chunk and the stage into
//                   the slot's accumulator; tcgen05.commit frees the stage, and after a unit's
//                   last stage signals the epilogue ("acc full")
//   warps 2-17      epilogue, two groups of eight: warp w reads accumulator lanes 32 (w % 4) .. + 31
//                   (one row per thread) and half of the columns; hidden layers: + bias, SiLU,
//                   BF16, written straight into the slot's activation buffer (the next layer's A
//                   operand, same swizzle); output layer: + bias, rows through the slot's buffer
//                   and a TMA store to global memory.  Then "epi done": the accumulator is
//                   drained and the buffer holds the next layer's input.
//   warps 18-21     loaders, with FP32 input rows instead of BF16 ones: rounded into the slot's
//                   input buffer by ordinary stores
//
// What bounds it (118,016 rows, w = 128, clock64 marks): per 64-wide K stage the issuer needs about
// 480 cycles where the MMAs compute for 256, and the output layer's units take 5,000 to 6,000 cycles.
// Counters name no saturated unit (tensor pipe 14 % of the elapsed cycles, LSU part of the l1tex data
// pipe 42 %, issue 37 %, MUFU 16 %), but do not show the MMAs' operand reads: that these (8 KB per K =
// 16 step, what shared memory delivers while it computes) and the epilogue's stores compete is inferred.  65.7 us before: issue from a lane == 0 branch (230 cycles per MMA),
// two slots, one epilogue group, output rows stored one row per lane (7,000 to 9,000 cycles per
// tile); 36.4 us now, w = 256 100.5 -> 69.0 us.  With FP32 rows in and out (souffle_mlp_forward)
// a packing and an unpacking kernel, 41 and 47 us, went too: 168 -> 55.7 us per call.
// SiLU(z) = z sigma(z) = h + h tanh(h), h = z / 2: one tanh.approx (a single MUFU operation,
// relative error below 2^-10) per element instead of an exponential and a division; the result
// is rounded to BF16 (2^-9) right after.  Every wait is bounded (umma.cuh); a timeout sets the
// caller's error bit and a shared abort flag that makes the other roles leave their loops.
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "gemm.cuh"
#include "umma.cuh"

namespace souffle {

namespace {

constexpr int kFRows = 128;                   // tile rows = MMA M
constexpr int kFK = 64;                       // K per chunk / stage (128 bytes of BF16)
constexpr int kFWidth = 256;                  // largest hidden width (bias slots are sized for it)
constexpr int kFChunk = kFRows * kFK * 2;     // 16 KB: one K-chunk of a tile, or one weight stage
constexpr int kFMaxStages = 6, kFMaxSlots = 3;
constexpr int kFEpiWarps = 8, kFEpiGroups = 2, kFLoadWarps = 4;  // epilogue warps per unit, units at a time
constexpr int kFThreads = 32 * (2 + kFEpiGroups * kFEpiWarps + kFLoadWarps);
constexpr int kFOutBuf = 32 * 128;             // 32 output rows of 128 bytes on their way out, per warp
constexpr int kFMaxOut = 256;
constexpr int kFBias = 3 * kFWidth + kFMaxOut;  // hidden half-biases, then the output bias
// barriers: full[kFMaxStages], empty[kFMaxStages], then per slot x_full, acc_full[2] (even and odd
// layers), epi_done, x_free, then drain
constexpr int kFBars = 2 * kFMaxStages + 5 * kFMaxSlots + 1;

// Tiles in flight per CTA (slots), weight stages and accumulator columns per slot.  The narrow
// network fits three tiles on chip (three 32 KB buffers, three times 160 of the 512 accumulator
// columns for up to 160 outputs); the wide one, or more outputs, two.
struct FusedPlan {
  int slots, stages, acc_cols, act_bytes, x_bytes, smem;
  bool shared;  // a layer's weight stages serve every slot before they are released
};
__host__ __device__ constexpr FusedPlan fused_plan(int width, int out_pad) {
  FusedPlan p{};
  p.slots = width == 128 && out_pad <= 160 ? 3 : 2;
  p.acc_cols = p.slots == 3 ? 160 : kFWidth;
  p.act_bytes = width / kFK * kFChunk;
  p.x_bytes = width == 128 ? kFChunk : 0;  // narrow network: input buffers of their own, else chunk 0 of the slot's
  p.stages = 4;
  p.shared = width == 128;  // a layer is at most four stages; the wide one's eight do not fit
  p.smem = 1024 + p.slots * (p.act_bytes + p.x_bytes) + p.stages * kFChunk + kFBias * 4 + kFBars * 8 + 16;
  return p;
}
static_assert(kFEpiWarps * kFOutBuf <= fused_plan(128, 160).act_bytes, "output rows leave through the slot's buffer");
static_assert(fused_plan(128, 160).smem <= 232448 && fused_plan(256, 256).smem <= 232448, "fits one CTA per SM");

struct FusedArgs {
  int m_cap;            // rows of the input / output buffers
  const int* m_dyn;     // live rows (device), or null = m_cap
  int n_in;             // <= 64
  int width;            // hidden width: 128 or 256
  int out_pad;          // output columns computed and stored (multiple of 16, <= 256)
  const float* bias[4];  // [256] x 3, [out_pad]
  const float* x32;     // [m_cap][n_in] FP32 input rows, or null: BF16 rows by TMA
  bool out_bf16;        // output rows (tensor map) in BF16, else FP32
  unsigned int* err;
  unsigned int err_bit;
};

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t pack2_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// bounded wait that also gives up when another role has aborted
__device__ __forceinline__ bool fwait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (unsigned i = 0; i < kMaxPolls; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 63u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// output columns of the layer: stage parts of up to 128 rows (the last may be narrower)
__device__ __forceinline__ int layer_n(int l, int out_pad, int width) { return l == 3 ? out_pad : width; }
__device__ __forceinline__ int layer_k_chunks(int l, int n_in, int width) {
  return l == 0 ? (n_in + kFK - 1) / kFK : width / kFK;
}

}  // namespace

__global__ void __launch_bounds__(kFThreads, 1)
    k_mlp_fused(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw0,
                const __grid_constant__ CUtensorMap tw1, const __grid_constant__ CUtensorMap tw2,
                const __grid_constant__ CUtensorMap tw3, const __grid_constant__ CUtensorMap ty, FusedArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int s_abort;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const FusedPlan plan = fused_plan(a.width, a.out_pad);
  const int nslots = plan.slots, nstages = plan.stages;
  const uint32_t act_bytes = (uint32_t)plan.act_bytes, acc_cols = (uint32_t)plan.acc_cols;
  const uint32_t act0 = base;                               // slot buffers: act0 + s * act_bytes
  const uint32_t ring = base + nslots * act_bytes;          // stage g: ring + g * kFChunk
  const uint32_t xbufs = ring + nstages * kFChunk;
  const uint32_t xbuf0 = plan.x_bytes ? xbufs : act0;       // slot s's input: xbuf0 + s * x_bytes
  const uint32_t x_bytes = plan.x_bytes ? (uint32_t)plan.x_bytes : act_bytes;
  const uint32_t bias_s = xbufs + nslots * plan.x_bytes;    // float [kFBias]
  const uint32_t bars = bias_s + kFBias * 4;
  const uint32_t full0 = bars, empty0 = bars + 8 * kFMaxStages;
  const uint32_t xfull0 = bars + 16 * kFMaxStages, accfull0 = xfull0 + 8 * kFMaxSlots,
                 epidone0 = accfull0 + 16 * kFMaxSlots, xfree0 = epidone0 + 8 * kFMaxSlots,
                 drain = xfree0 + 8 * kFMaxSlots;
  const uint32_t tmem_slot = drain + 8;
  float* s_bias = reinterpret_cast<float*>(smem_raw + (bias_s - raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - raw));
  volatile int* abort_flag = &s_abort;
  // (warp-wide reductions give the compiler values that it knows to be the same in every lane)
  const int warp = (int)__reduce_max_sync(0xffffffffu, threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int m_rows = (int)__reduce_max_sync(0xffffffffu, (unsigned)(a.m_dyn ? max(0, min(a.m_cap, *a.m_dyn)) : a.m_cap));
  const int tiles = (m_rows + kFRows - 1) / kFRows;
  if ((int)blockIdx.x >= tiles) return;  // uniform over the CTA, before any allocation
  // this CTA's tiles: blockIdx.x + i gridDim.x, tile i in slot i % nslots, group i / nslots
  const int my_tiles = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int groups = (my_tiles + nslots - 1) / nslots;

  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < nstages; s++) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int s = 0; s < nslots; s++) {
      mbar_init(xfull0 + 8 * s, a.x32 ? kFLoadWarps : 1);
      mbar_init(accfull0 + 16 * s, 1);
      mbar_init(accfull0 + 16 * s + 8, 1);
      mbar_init(epidone0 + 8 * s, kFEpiWarps);
      mbar_init(xfree0 + 8 * s, plan.x_bytes ? 1 : kFEpiWarps);
    }
    mbar_init(drain, 1);
    mbar_fence_init();
  }
  if (threadIdx.x == 32) {
    tma_prefetch_map(&tx);
    tma_prefetch_map(&tw0);
    tma_prefetch_map(&tw1);
    tma_prefetch_map(&tw2);
    tma_prefetch_map(&tw3);
    tma_prefetch_map(&ty);
  }
  // biases: half of each hidden bias (SiLU works on z / 2), the output bias as it is
  for (int t = threadIdx.x; t < kFBias; t += blockDim.x) {
    float v = 0.f;
    if (t < 3 * kFWidth) {
      if (t % kFWidth < a.width) v = 0.5f * a.bias[t / kFWidth][t % kFWidth];
    }
    else if (t - 3 * kFWidth < a.out_pad) v = a.bias[3][t - 3 * kFWidth];
    s_bias[t] = v;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_ptr;
  const CUtensorMap* wmap[4] = {&tw0, &tw1, &tw2, &tw3};

  if (warp == 0) {
    if (lane == 0) {
      // ---- producer
      int g = 0;          // weight stages issued
      int xs[kFMaxSlots] = {0, 0, 0};  // inputs loaded per slot
      bool ok = true;
      for (int p = 0; p < groups && ok; p++) {
        for (int l = 0; l < 4 && ok; l++) {
          for (int s = 0; s < nslots && ok; s++) {
            const int i = nslots * p + s;
            if (i >= my_tiles) continue;
            if (l == 0 && !a.x32) {
              // the slot's previous tile has finished its output layer (its MMAs read the buffer)
              if (xs[s] > 0 && !fwait(xfree0 + 8 * s, (uint32_t)(xs[s] - 1) & 1u, abort_flag)) {
                ok = false;
                break;
              }
              const int tile = (int)blockIdx.x + i * (int)gridDim.x;
              mbar_expect_tx(xfull0 + 8 * s, kFChunk);
              tma_load_2d(xbuf0 + s * x_bytes, &tx, 0, tile * kFRows, xfull0 + 8 * s);
              xs[s]++;
            }
            if (plan.shared && s > 0) continue;
            const int nk = layer_k_chunks(l, a.n_in, a.width), parts = (layer_n(l, a.out_pad, a.width) + 127) / 128;
            for (int kc = 0; kc < nk && ok; kc++) {
              for (int part = 0; part < parts; part++, g++) {
                const int st = g % nstages;
                const uint32_t use = (uint32_t)(g / nstages);
                if (use > 0 && !fwait(empty0 + 8 * st, (use - 1) & 1u, abort_flag)) {
                  ok = false;
                  break;
                }
                mbar_expect_tx(full0 + 8 * st, kFChunk);
                tma_load_2d(ring + st * kFChunk, wmap[l], kc * kFK, part * 128, full0 + 8 * st);
              }
            }
          }
        }
      }
      // every copy started here has landed before the CTA can leave
      for (int q = (g > nstages ? g - nstages : 0); q < g; q++)
        if (!mbar_wait(full0 + 8 * (q % nstages), (uint32_t)(q / nstages) & 1u)) ok = false;
      for (int s = 0; s < nslots; s++)
        if (xs[s] > 0 && !mbar_wait(xfull0 + 8 * s, (uint32_t)(xs[s] - 1) & 1u)) ok = false;
      if (!ok) {
        *abort_flag = 1;
        atomicOr(a.err, a.err_bit);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the whole warp walks the units, one elected lane issues.  No branch
    // depends on a wait's outcome, so the walk stays uniform; after a failed wait (the abort
    // flag makes the later ones give up at once) it only runs out on data that nobody uses.
    int st = 0;            // next weight stage and the parity of its full barrier
    uint32_t st_par = 0;
    uint32_t epi_par = 1;  // of the slots' epi_done barriers (four units per tile: the same for all)
    bool ok = true;
    for (int p = 0; p < groups; p++) {
      const int active = min(nslots, my_tiles - nslots * p);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        const int st_layer = st;
        const uint32_t par_layer = st_par;
        const int n = layer_n(l, a.out_pad, a.width);
        const int nk = layer_k_chunks(l, a.n_in, a.width), parts = (n + 127) / 128;
        for (int s = 0; s < active; s++) {
          if (plan.shared) {
            st = st_layer;
            st_par = par_layer;
          }
          const bool loaded = plan.shared && s > 0;  // the first slot has waited for these stages
          const bool release = !plan.shared || s == active - 1;
          // the slot's previous unit has been drained by the epilogue (and, from the second
          // layer on, its output is this unit's input)
          if (p + l > 0) ok &= fwait(epidone0 + 8 * s, epi_par, abort_flag);
          if (l == 0) ok &= fwait(xfull0 + 8 * s, (uint32_t)p & 1u, abort_flag);
          tc_fence_after();
          const uint32_t acc = tmem + (uint32_t)s * acc_cols;
          const uint32_t abuf = l == 0 ? xbuf0 + s * x_bytes : act0 + s * act_bytes;
          for (int kc = 0; kc < nk; kc++) {
            for (int part = 0; part < parts; part++) {
              if (!loaded) {
                ok &= fwait(full0 + 8 * st, st_par, abort_flag);
                tc_fence_after();
              }
              const uint32_t idesc = umma_idesc_bf16(kFRows, min(128, n - 128 * part));
              const uint64_t ad = sw128_kmajor_desc(abuf + kc * kFChunk);
              const uint64_t bd = sw128_kmajor_desc(ring + st * kFChunk);
              const uint32_t d = acc + (uint32_t)(128 * part);
              if (elect_one()) {
#pragma unroll
                for (int j = 0; j < kFK / 16; j++) umma_bf16(d, ad + 2 * j, bd + 2 * j, idesc, (kc | j) != 0 ? 1u : 0u);
                if (release) umma_commit(empty0 + 8 * st);
              }
              __syncwarp();
              if (++st == nstages) {
                st = 0;
                st_par ^= 1u;
              }
            }
          }
          if (elect_one()) {
            umma_commit(accfull0 + 16 * s + 8 * (l & 1));
            if (l == 0 && plan.x_bytes) umma_commit(xfree0 + 8 * s);
          }
          __syncwarp();
        }
        epi_par ^= 1u;
      }
    }
    if (!warp_agrees(ok)) {
      // MMAs issued before the failure may still be running: drain them (bounded) before the
      // tensor memory is released
      if (elect_one()) {
        atomicOr(a.err, a.err_bit);
        umma_commit(drain);
      }
      mbar_wait(drain, 0);
    }
  } else if (warp < 2 + kFEpiGroups * kFEpiWarps) {
    // ---- epilogue
    // Units alternate between the two groups of eight warps by (layer + slot), so one group's
    // loads, MUFU and hand-off latencies overlap the other's.  For a slot a group then sees
    // either the even or the odd layers, and each kind has a barrier of its own: a parity wait
    // can tell two successive phases apart, not every second one.
    const int q = warp & 3, half = ((warp - 2) & 7) >> 2, grp = (warp - 2) >> 3;
    const int r_local = q * 32 + lane;  // tile row = accumulator lane
    bool ok = true;
    for (int p = 0; p < groups && ok; p++) {
      for (int l = 0; l < 4 && ok; l++) {
        for (int s = 0; s < nslots && ok; s++) {
          const int i = nslots * p + s;
          if (i >= my_tiles) continue;
          if (((l + s) & 1) != grp) continue;
          if (!warp_agrees(fwait(accfull0 + 16 * s + 8 * (l & 1), (uint32_t)(l >> 1) & 1u, abort_flag))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t t_row = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)s * acc_cols;
          if (l < 3) {
            // hidden layer: columns [half w/2, (half + 1) w/2) -> SiLU -> BF16 into the buffer
            const float* hb = s_bias + l * kFWidth;
            const uint32_t abuf = act0 + s * act_bytes;
            const uint32_t rsw = (uint32_t)(r_local & 7);
#pragma unroll 1
            for (int c0 = half * (a.width >> 1); c0 < (half + 1) * (a.width >> 1); c0 += 32) {
              float v[32];
              tmem_ld32(t_row + (uint32_t)c0, v);
              // K-chunk c0 / 64, 16-byte units (c0 % 64) / 8 .. + 3, swizzled by the row
              const uint32_t rowaddr = abuf + (uint32_t)(c0 >> 6) * kFChunk + (uint32_t)r_local * 128u;
              const uint32_t u0 = (uint32_t)((c0 & 63) >> 3);
#pragma unroll
              for (int k = 0; k < 4; k++) {
                uint32_t pk[4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                  const int e = 8 * k + 4 * j;
                  const float4 b = *reinterpret_cast<const float4*>(hb + c0 + e);
                  const float h0 = fmaf(v[e], 0.5f, b.x), h1 = fmaf(v[e + 1], 0.5f, b.y);
                  const float h2 = fmaf(v[e + 2], 0.5f, b.z), h3 = fmaf(v[e + 3], 0.5f, b.w);
                  pk[2 * j] = pack2_bf16(fmaf(h0, tanh_approx(h0), h0), fmaf(h1, tanh_approx(h1), h1));
                  pk[2 * j + 1] = pack2_bf16(fmaf(h2, tanh_approx(h2), h2), fmaf(h3, tanh_approx(h3), h3));
                }
                st_shared_v4(rowaddr + (((u0 + k) ^ rsw) << 4), pk[0], pk[1], pk[2], pk[3]);
              }
            }
            fence_proxy_async_smem();
          } else {
            // output layer: + bias -> rows in global memory.  A thread holds one row, and storing
            // straight from registers would touch 32 lines per instruction (7,000 to 9,000
            // cycles per tile).  The slot's buffer is free -- the output layer's MMAs have read
            // it -- so each warp puts its 32 rows there 128 bytes at a time (the two halves of
            // the warps alternate; 128-byte swizzle) and a TMA store takes them out.
            const int row0 = ((int)blockIdx.x + i * (int)gridDim.x) * kFRows + q * 32;
            const float* ob = s_bias + 3 * kFWidth;
            const uint32_t buf = act0 + s * act_bytes + (uint32_t)((warp - 2) & 7) * kFOutBuf;
            const uint32_t wr = buf + (uint32_t)lane * 128u, wsw = (uint32_t)lane & 7u;
            const int cw = a.out_bf16 ? 64 : 32;  // columns of 128 bytes
#pragma unroll 1
            for (int c0 = half * cw; c0 < a.out_pad; c0 += 2 * cw) {
              if (c0 != half * cw) {
                if (lane == 0) bulk_wait_read();
                __syncwarp();
              }
              if (a.out_bf16) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                  const int cc = c0 + 32 * h;
                  if (cc >= a.out_pad) break;
                  float v[32];
                  tmem_ld32(t_row + (uint32_t)cc, v);
#pragma unroll
                  for (int u = 0; u < 4; u++) {
                    const float4 b0 = *reinterpret_cast<const float4*>(ob + cc + 8 * u);
                    const float4 b1 = *reinterpret_cast<const float4*>(ob + cc + 8 * u + 4);
                    st_shared_v4(wr + (((uint32_t)(4 * h + u) ^ wsw) << 4), pack2_bf16(v[8 * u] + b0.x, v[8 * u + 1] + b0.y),
                                 pack2_bf16(v[8 * u + 2] + b0.z, v[8 * u + 3] + b0.w),
                                 pack2_bf16(v[8 * u + 4] + b1.x, v[8 * u + 5] + b1.y),
                                 pack2_bf16(v[8 * u + 6] + b1.z, v[8 * u + 7] + b1.w));
                  }
                }
              } else {
                float v[32];
                tmem_ld32(t_row + (uint32_t)c0, v);
#pragma unroll
                for (int u = 0; u < 8; u++) {
                  const float4 b = *reinterpret_cast<const float4*>(ob + c0 + 4 * u);
                  st_shared_v4(wr + (((uint32_t)u ^ wsw) << 4), __float_as_uint(v[4 * u] + b.x), __float_as_uint(v[4 * u + 1] + b.y),
                               __float_as_uint(v[4 * u + 2] + b.z), __float_as_uint(v[4 * u + 3] + b.w));
                }
              }
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0 && row0 < m_rows) tma_store_2d(&ty, buf, c0, row0);
            }
          }
          // this warp has read its part of the accumulator and written its part of the buffer
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (l == 3) bulk_wait_read();  // the slot's buffer may be written again
            mbar_arrive(epidone0 + 8 * s);
            if (l == 3 && !plan.x_bytes) mbar_arrive(xfree0 + 8 * s);  // ... by the next tile's input
          }
        }
      }
    }
    if (!ok) atomicOr(a.err, a.err_bit);
  } else if (a.x32) {
    // ---- loaders (FP32 input): a tile's rows, rounded to BF16, into chunk 0 of its slot's buffer
    // in the layout the TMA box would have, zero beyond n_in and the last row.  Each warp takes 32
    // rows; a lane holds 16 bytes of BF16 (8 columns) of row 4 k + lane / 8 at a time.
    const int w = warp - 2 - kFEpiGroups * kFEpiWarps;
    const int u = lane & 7, c = 8 * u;
    const bool vec = (reinterpret_cast<uintptr_t>(a.x32) & 15) == 0;  // n_in is a multiple of 8
    bool ok = true;
    for (int i = 0; i < my_tiles && ok; i++) {
      const int s = i % nslots, use = i / nslots;
      const int row0 = ((int)blockIdx.x + i * (int)gridDim.x) * kFRows + 32 * w;
      float4 v[8][2];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int row = row0 + 4 * k + (lane >> 3);
        v[k][0] = v[k][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < m_rows && c < a.n_in) {
          const float* p = a.x32 + (size_t)row * a.n_in + c;
          if (vec) {
            v[k][0] = __ldg(reinterpret_cast<const float4*>(p));
            v[k][1] = __ldg(reinterpret_cast<const float4*>(p + 4));
          } else {
            v[k][0] = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
            v[k][1] = make_float4(__ldg(p + 4), __ldg(p + 5), __ldg(p + 6), __ldg(p + 7));
          }
        }
      }
      // the slot's previous tile has finished its output layer (its MMAs read the buffer)
      if (use > 0 && !warp_agrees(fwait(xfree0 + 8 * s, (uint32_t)(use - 1) & 1u, abort_flag))) {
        ok = false;
        break;
      }
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint32_t r = (uint32_t)(32 * w + 4 * k + (lane >> 3));
        st_shared_v4(xbuf0 + s * x_bytes + r * 128u + (((uint32_t)u ^ (r & 7u)) << 4),
                     pack2_bf16(v[k][0].x, v[k][0].y), pack2_bf16(v[k][0].z, v[k][0].w),
                     pack2_bf16(v[k][1].x, v[k][1].y), pack2_bf16(v[k][1].z, v[k][1].w));
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(xfull0 + 8 * s);
    }
    if (!ok) atomicOr(a.err, a.err_bit);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 fused_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// [rows][cols] BF16 (or FP32), row stride ld elements; box 128 bytes of columns x 128 rows (or 32
// for the output's stores), 128-byte swizzle
bool fused_map(CUtensorMap* m, const void* p, int rows, int cols, int ld, bool fp32 = false, int box_rows = kFRows) {
  auto fn = fused_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * (fp32 ? 4 : 2)};
  cuuint32_t box[2] = {(cuuint32_t)(fp32 ? 32 : kFK), (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  return fn(m, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool mlp_fused_supported(int n_in, int width, int out_pad) {
  return n_in >= 8 && n_in <= kFK && n_in % 8 == 0 && (width == 128 || width == kFWidth) && out_pad >= 16 &&
         out_pad <= kFMaxOut && out_pad % 16 == 0;
}

cudaError_t mlp_forward_fused(const __nv_bfloat16* x, int ldx, int m_cap, const int* m_dyn, int n_in, int width,
                              const __nv_bfloat16* const w[4], const int ldw[4], int out_pad, const float* const bias[4],
                              float* y, int ldy, unsigned int* err, unsigned int err_bit, cudaStream_t st,
                              __nv_bfloat16* yb, const float* x32, int n_store) {
  if (n_store <= 0) n_store = out_pad;
  if (!mlp_fused_supported(n_in, width, out_pad) || m_cap < 1 || !x || !(y || yb) || !err || ldx < n_in || ldx % 8 ||
      n_store > out_pad || ldy < n_store || ldy % (yb ? 8 : 4) ||
      (reinterpret_cast<uintptr_t>(yb ? (const void*)yb : (const void*)y) & 15) ||
      (reinterpret_cast<uintptr_t>(x) & 15) || ldw[0] < n_in || ldw[1] < width || ldw[2] < width || ldw[3] < width)
    return cudaErrorInvalidValue;
  for (int l = 0; l < 4; l++)
    if (!w[l] || !bias[l] || ldw[l] % 8 || (reinterpret_cast<uintptr_t>(w[l]) & 15)) return cudaErrorInvalidValue;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_mlp_fused, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                std::max(fused_plan(128, 160).smem, fused_plan(256, 256).smem));
  });
  if (attr != cudaSuccess) return attr;
  CUtensorMap tx, ty, tw[4];
  if (!fused_map(&ty, yb ? (const void*)yb : (const void*)y, m_cap, n_store, ldy, !yb, 32) || !fused_map(&tx, x, m_cap, n_in, ldx) || !fused_map(&tw[0], w[0], width, n_in, ldw[0]) ||
      !fused_map(&tw[1], w[1], width, width, ldw[1]) || !fused_map(&tw[2], w[2], width, width, ldw[2]) ||
      !fused_map(&tw[3], w[3], out_pad, width, ldw[3]))
    return cudaErrorInvalidValue;
  static int sms = 0;
  static std::once_flag once_sm;
  std::call_once(once_sm, [] {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      sms = 0;
  });
  FusedArgs a;
  a.m_cap = m_cap;
  a.m_dyn = m_dyn;
  a.n_in = n_in;
  a.width = width;
  a.out_pad = out_pad;
  for (int l = 0; l < 4; l++) a.bias[l] = bias[l];
  a.x32 = x32;
  a.out_bf16 = yb != nullptr;
  a.err = err;
  a.err_bit = err_bit;
  // one CTA per SM, each looping over tiles; CTAs beyond the live tiles leave at once
  const long long tiles = ((long long)m_cap + kFRows - 1) / kFRows;
  const int gx = (int)std::min<long long>(tiles, sms > 0 ? sms : 148);
  k_mlp_fused<<<gx, kFThreads, fused_plan(width, out_pad).smem, st>>>(tx, tw[0], tw[1], tw[2], tw[3], ty, a);
  return cudaGetLastError();
}

}  // namespace souffle
