// gfx_mt.cu -- bank of 4096 MT607 Mersenne Twisters (w = 32, n = 19, m = 9, r = 1,
// tempering shifts 12/7/15/18), restated from the published Mersenne Twister
// recurrence (Matsumoto & Nishimura 1998) with per-generator parameters
// (matrix_a, mask_b, mask_c) read from the twister-parameter file.
//
// Call semantics reproduce the reference bank (MersenneTwister.cu:142-229,
// 236-323) bit for bit:
//   * output j of twister r goes to out[r + 4096*j], as ((float)x + 1) / 2^32;
//   * every call restarts at ring slot 0 of the saved 19-word state, and saves
//     the state and seed = state[0] at the end;
//   * initialized == 0 re-seeds the state from seed with the MT init recurrence;
//   * gaussian fields: Box-Muller on the pairs (2k, 2k+1) of each twister's outputs,
//     applied in the generator before the outputs are stored.
// This translation unit is compiled with -prec-sqrt=false -prec-div=false,
// the flags of the reference build, so the Box-Muller arithmetic matches it.
#include "gfx_internal.h"

namespace gfx {

namespace {
constexpr uint32_t kUMask = 0xFFFFFFFEu;
constexpr uint32_t kLMask = 0x1u;
constexpr float kInv2p32 = 2.3283064365386963e-10f;  // 2^-32, exact
}  // namespace

__device__ __forceinline__ void box_muller(float u1, float u2, float& g1, float& g2) {
  const float PIf = 3.14159265358979f;
  const float r = sqrtf(-2.0f * logf(u1));
  const float phi = 2 * PIf * u2;
  g1 = r * __cosf(phi);
  g2 = r * __sinf(phi);
}

// A twister's outputs are x_19, x_20, .. of the sequence x_{n+19} = x_{n+9} ^ f(x_n, x_{n+1})
// that starts from its 19 saved words; x_m belongs to ring slot m mod 19.  Ten outputs depend
// on none of each other, so ten lanes make ten a step: lane p holds the last two words with
// index p mod 10, has x_{n+9} itself and gets x_n and x_{n+1} from the next two lanes, two
// shuffles a step.  A warp has three twisters.  (One warp a twister, 19 outputs in two
// dependent half-steps of four shuffles, kept a third of the lanes busy: 87 us for an update
// of 4M gaussians and 16M uniforms, launches and wait included, against 54 us.)
// A block has 27 twisters, 152 blocks, one for each SM.  Its first nine warps put kTileRows
// outputs of each into shared memory while the others write the tile before them, a row a
// warp, and form the Box-Muller pairs (2k, 2k+1) of each twister.  (32 twisters a block, for
// whole 128-byte rows, keep 128 SMs busy: 43 instead of 29 us for the uniforms; 11 or 15
// writers instead of 7: no faster.)
constexpr int kTwistersPerWarp = 3;
constexpr int kMTWarps = 9;
constexpr int kMTWriters = 7;
constexpr int kTwistersPerBlock = kTwistersPerWarp * kMTWarps;
constexpr int kStepOutputs = 10;
constexpr int kTileRows = 16 * kStepOutputs;  // even: pairs never straddle a tile
constexpr int kTileCols = kTwistersPerBlock + 2;  // and a column for lanes without a twister

// the recurrence from words n, n + 1 and n + 9 (the product in place of a selection runs
// beside the logic operations, which bound the kernel)
__device__ __forceinline__ uint32_t mt_step(uint32_t mti, uint32_t mti1, uint32_t mtm, uint32_t A) {
  const uint32_t x = (mti & kUMask) | (mti1 & kLMask);
  return mtm ^ (x >> 1) ^ ((mti1 & kLMask) * A);
}

__device__ __forceinline__ float mt_temper(uint32_t x, uint32_t B, uint32_t C) {
  x ^= (x >> 12);
  x ^= (x << 7) & B;
  x ^= (x << 15) & C;
  x ^= (x >> 18);
  return ((float)x + 1.0f) * kInv2p32;
}

// rows of a tile of cnt outputs -> out[row * kMTCount + twister], a warp a row
template <bool GAUSS>
__device__ __forceinline__ void mt_write(const float (*tile)[kTileCols], float* out, int cnt,
                                         int ncol, int w) {
  const int lane = threadIdx.x & 31;
  if (lane >= ncol) return;
  if (GAUSS) {
    // an unpaired last output (odd nper) is not written, as in the sequential form
#pragma unroll 4
    for (int pr = w; 2 * pr + 1 < cnt; pr += kMTWriters) {
      float g1, g2;
      box_muller(tile[2 * pr][lane], tile[2 * pr + 1][lane], g1, g2);
      out[(size_t)(2 * pr) * kMTCount + lane] = g1;
      out[(size_t)(2 * pr + 1) * kMTCount + lane] = g2;
    }
  } else {
#pragma unroll 8
    for (int row = w; row < cnt; row += kMTWriters)
      out[(size_t)row * kMTCount + lane] = tile[row][lane];
  }
}

// init_MT (initialized 0) or update_MT (1): nper_g gaussians, then nper_u uniforms of every
// twister, each a call of the reference's generator (from ring slot 0 of the saved state, or
// from the seed).  A twister's two calls follow each other in its own warp, so one launch
// makes both fields.
__global__ void __launch_bounds__((kMTWarps + kMTWriters) * 32)
    mt_fields_kernel(MTBank bank, float* __restrict__ gauss, int nper_g,
                     float* __restrict__ unif, int nper_u, int initialized) {
  __shared__ float tile[2][kTileRows][kTileCols];
  const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int r0 = blockIdx.x * kTwistersPerBlock;
  const int ncol = min(kTwistersPerBlock, kMTCount - r0);
  const int tiles_g = (nper_g + kTileRows - 1) / kTileRows;
  const int ntiles = tiles_g + (nper_u + kTileRows - 1) / kTileRows;
  if (w >= kMTWarps) {
    for (int t = 0; t <= ntiles; t++) {
      const int u = t - 1;  // written while tile t is made
      if (t && u < tiles_g)
        mt_write<true>(tile[u & 1], gauss + (size_t)u * kTileRows * kMTCount + r0,
                       min(kTileRows, nper_g - u * kTileRows), ncol, w - kMTWarps);
      else if (t)
        mt_write<false>(tile[u & 1], unif + (size_t)(u - tiles_g) * kTileRows * kMTCount + r0,
                        min(kTileRows, nper_u - (u - tiles_g) * kTileRows), ncol, w - kMTWarps);
      if (t < ntiles) __syncthreads();  // tile t is there, and tile t - 1 may be overwritten
    }
    return;
  }
  const int g = lane / kStepOutputs, p = lane - g * kStepOutputs;  // lanes 30, 31: g = 3
  const int col = w * kTwistersPerWarp + g;
  const bool mine = g < kTwistersPerWarp && col < ncol;
  const int r = r0 + (mine ? col : 0);
  const int k = p == 9 ? 0 : p + 1;  // this lane's output of a step
  const int src1 = lane - p + k, src2 = lane - p + (k == 9 ? 0 : k + 1);
  const uint32_t past1 = p == 9 ? ~0u : 0u, past2 = p == 9 || p == 0 ? ~0u : 0u;
  const uint32_t A = bank.a[r], B = bank.b[r], C = bank.c[r];
  int t = 0;
#pragma unroll 1
  for (int call = 0; call < 2; call++) {
    const int nper = call ? nper_u : nper_g;
    // words x_p and x_{10+p}; lane 9, which makes the step's first word, x_9 as its newer one
    uint32_t older = 0, newer = 0;
    if (!initialized) {
      uint32_t v = bank.seed[r];
      for (int i = 0; i < kMTN; i++) {
        if (i) v = 1812433253u * (v ^ (v >> 30)) + (uint32_t)i;
        if (i == p) older = v;
        if (i == p + 10) newer = v;
      }
    } else {
      older = bank.status[p * kMTCount + r];
      if (p < 9) newer = bank.status[(10 + p) * kMTCount + r];
    }
    if (p == 9) newer = older;
    __syncwarp();  // read before any lane saves the next state
    // the next word of this lane.  The words 18 and 19 back are the next lanes' older ones,
    // but for the lanes past the step's end, whose last word is their newer one
    auto step = [&]() {
      const uint32_t x19 = __shfl_sync(0xffffffffu, (newer & past1) | (older & ~past1), src1);
      const uint32_t x18 = __shfl_sync(0xffffffffu, (newer & past2) | (older & ~past2), src2);
      return mt_step(x19, x18, newer, A);
    };
    int done = 0;  // outputs of whole steps
    uint32_t last = 0;
    for (int o = 0; o < nper; o += kTileRows, t++) {
      const int cnt = min(kTileRows, nper - o);
      float* to = &tile[t & 1][k][mine ? col : kTwistersPerBlock];
      auto whole = [&](int j) {
        const uint32_t x = step();
        older = newer;
        newer = x;
        to[j * kTileCols] = mt_temper(x, B, C);
      };
      int j = 0;
      if (cnt == kTileRows) {
#pragma unroll
        for (int i = 0; i < kTileRows; i += kStepOutputs) whole(i);
        j = kTileRows;
      } else {
#pragma unroll 1
        for (; j + kStepOutputs <= cnt; j += kStepOutputs) whole(j);
      }
      done += j;
      if (j < cnt) {  // the last outputs, fewer than ten
        last = step();
        if (j + k < cnt) to[j * kTileCols] = mt_temper(last, B, C);
      }
      __syncthreads();
    }
    // the 19 words after the last output, by ring slot
    const int rem = nper - done;  // outputs of the last, partial step
    auto save = [&](int m, uint32_t v) {
      const int slot = m % kMTN;
      bank.status[slot * kMTCount + r] = v;
      if (slot == 0) bank.seed[r] = v;
    };
    const int m = done + 9 + k;  // the newer word's index
    if (mine) {
      if (p < 9 && p >= rem) save(m - 10, older);
      save(m, newer);
      if (k < rem) save(m + 10, last);
    }
    __syncwarp();  // the state is read by other lanes of the warp
  }
}

void launch_mt_fields(const MTBank& bank, float* gauss, int nper_g, float* unif, int nper_u,
                      int initialized, cudaStream_t s) {
  const int grid = (kMTCount + kTwistersPerBlock - 1) / kTwistersPerBlock;
  mt_fields_kernel<<<grid, (kMTWarps + kMTWriters) * 32, 0, s>>>(bank, gauss, nper_g, unif,
                                                                 nper_u, initialized);
}

}  // namespace gfx
