// fp32 3x3 convolution (stride 1, pad 1, group 1) of any layout and any image size on the CUDA cores: what the tensor-core kernels
// do not take -- NCHW tensors between operators that keep the reference's layout, channel counts and image sizes that do not tile.
//
// One thread per output with its window from global memory (the general kernel) spends its time on loads and indexes. Here a block owns
// 16 rows x 16 or 32 columns of one image and 16 output channels; the haloed input tile comes four channels at a time by asynchronous copies,
// the next four under these, and the block's weights of all channels stay in shared memory. A thread owns eight outputs below one
// another and eight channels; the lanes of a warp are 16 neighbouring columns x two groups of channels, so that each weight (a 16-byte
// broadcast) feeds 16 packed FMAs and a warp stores whole lines of a 16-channel NHWC tensor. Every output is one chain of FMAs, two
// channels at a time (each product and sum is rounded as the scalar ones are).
// 1024 images of 16 x 16: 8 -> 16 channels 89 -> 28 us, 16 -> 16 164 -> 46; 256 x 64 -> 64 at 56 x 56 8369 -> 1795 (12.6 of the 37 TMAC/s of the
// FMA units: the copies, the duplicated inputs of the packed FMAs and 12 warps an SM); a Session of a residual block on 1024 images 477 -> 291.
#include "contract.cuh"

namespace sofie {
namespace {

constexpr int kDcRows = 16, kDcChunk = 4, kDcOut = 16, kDcHalo = kDcRows + 2;
__host__ __device__ constexpr int dc_pitch(int groups) { return 16 * groups + 8; } // image columns x0 - 4 ... x0 + 16 * groups + 3
__host__ __device__ constexpr int dc_tile_floats(int groups) { return kDcChunk * kDcHalo * dc_pitch(groups); }

__device__ __forceinline__ size_t dc_weight_index(const ConvGeom &g, int oc, int c, int rt)
{
   return g.w_packed ? ((size_t)oc * 9 + rt) * g.C + c : ((size_t)oc * g.C + c) * 9 + rt;
}

// GROUPS of 16 columns; VEC: NCHW rows of whole 16-byte words.
template <int POOL, int GROUPS, bool VEC>
__global__ void __launch_bounds__(64 * GROUPS, 6 / GROUPS)
conv3x3_direct_f32_kernel(ConvGeom g, const float *__restrict__ X, const float *__restrict__ Wt, const float *__restrict__ bias, float *__restrict__ Y,
                          long long num_tiles, int tiles_x, int tiles_y, int chunks)
{
   constexpr int THREADS = 64 * GROUPS, PITCH = dc_pitch(GROUPS);
   extern __shared__ __align__(16) float smem[];
   float *tiles = smem;                                   // two tiles [channel][row][column]
   float *s_w = smem + 2 * dc_tile_floats(GROUPS);        // [channel][tap][16]
   __shared__ float s_bias[kDcOut];
   griddep_launch_dependents();
   griddep_wait(X, Wt, bias);
   const int tid = threadIdx.x, oc_base = blockIdx.y * kDcOut;
   for (int i = tid; i < chunks * kDcChunk * 9 * kDcOut; i += THREADS) {
      const int o = i % kDcOut, rt = i / kDcOut % 9, c = i / (9 * kDcOut);
      const bool in = c < g.C && oc_base + o < g.Cout;
      // (waited for with the first tile)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(s_w + i)), "l"(in ? Wt + dc_weight_index(g, oc_base + o, c, rt) : Wt), "r"(in ? 4 : 0)
                   : "memory");
   }
   if (tid < kDcOut) s_bias[tid] = oc_base + tid < g.Cout && bias ? __ldg(bias + oc_base + tid) : 0.f;
   auto origin = [&](long long id, int &n, int &h0, int &w0) {
      w0 = (int)(id % tiles_x) * 16 * GROUPS;
      const long long t = id / tiles_x;
      h0 = (int)(t % tiles_y) * kDcRows;
      n = (int)(t / tiles_y);
   };
   auto copy = [&](long long id, int c0, int buf) {
      if (id < num_tiles) {
         int n, h0, w0;
         origin(id, n, h0, w0);
         float *tile = tiles + buf * dc_tile_floats(GROUPS);
         if constexpr (VEC) {
            constexpr int WORDS = PITCH / 4;
            for (int i = tid; i < kDcChunk * kDcHalo * WORDS; i += THREADS) {
               const int c = i / (kDcHalo * WORDS), r = i / WORDS % kDcHalo, w = i % WORDS;
               const int ih = h0 - 1 + r, iw = w0 - 4 + 4 * w;
               const bool in = c0 + c < g.C && ih >= 0 && ih < g.H && iw >= 0 && iw < g.W;
               const float *src = in ? X + (((size_t)n * g.C + c0 + c) * g.H + ih) * g.W + iw : X;
               asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(tile + 4 * i)), "l"(src), "r"(in ? 16 : 0) : "memory");
            }
         } else {
            constexpr int COLS = 16 * GROUPS + 2;
            for (int i = tid; i < kDcChunk * kDcHalo * COLS; i += THREADS) {
               // the index that is contiguous in memory runs fastest
               const int c = g.x_nhwc ? i % kDcChunk : i / (kDcHalo * COLS), p = g.x_nhwc ? i / kDcChunk : i % (kDcHalo * COLS);
               const int r = p / COLS, col = p % COLS, ih = h0 - 1 + r, iw = w0 - 1 + col;
               const bool in = c0 + c < g.C && ih >= 0 && ih < g.H && iw >= 0 && iw < g.W;
               const size_t at = g.x_nhwc ? (((size_t)n * g.H + ih) * g.W + iw) * g.C + c0 + c : (((size_t)n * g.C + c0 + c) * g.H + ih) * g.W + iw;
               asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(tile + (c * kDcHalo + r) * PITCH + 3 + col)),
                            "l"(in ? X + at : X), "r"(in ? 4 : 0)
                            : "memory");
            }
         }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
   };
   // this thread's channels, column and first row in the tile
   const int oc_local = (tid & 1) * 8, oc = oc_base + oc_local, col = (tid >> 5) % GROUPS * 16 + ((tid & 31) >> 1), row0 = (tid >> 5) / GROUPS * 8;
   copy(blockIdx.x, 0, 0);
   int buf = 0;
   for (long long id = blockIdx.x; id < num_tiles; id += gridDim.x) {
      int n, h0, w0;
      origin(id, n, h0, w0);
      const int oh0 = h0 + row0, ow = w0 + col;
      const bool inside = oh0 < g.oH && w0 + (col & ~15) < g.oW; // something of this warp lies in the image
      uint64_t acc2[8][4]; // two neighbouring channels each
#pragma unroll
      for (int q = 0; q < 8; q++)
#pragma unroll
         for (int o = 0; o < 4; o++) acc2[q][o] = 0;
      for (int chunk = 0; chunk < chunks; chunk++, buf ^= 1) {
         __syncthreads(); // the tile before this one is no longer read: its buffer is the next one's
         if (chunk + 1 < chunks) copy(id, (chunk + 1) * kDcChunk, buf ^ 1);
         else copy(id + gridDim.x, 0, buf ^ 1);
         asm volatile("cp.async.wait_group 1;" ::: "memory");
         __syncthreads();
         if (!inside) continue;
         const float *in = tiles + buf * dc_tile_floats(GROUPS) + row0 * PITCH + col + 3;
         const float *w = s_w + chunk * kDcChunk * 9 * kDcOut + oc_local;
#pragma unroll 1
         for (int c = 0; c < kDcChunk; c++, in += kDcHalo * PITCH, w += 9 * kDcOut) {
            uint64_t win[10][3]; // the inputs under the eight outputs, each twice
#pragma unroll
            for (int r = 0; r < 10; r++)
#pragma unroll
               for (int t = 0; t < 3; t++) {
                  const float v = in[r * PITCH + t];
                  win[r][t] = pack_f32x2(v, v);
               }
#pragma unroll
            for (int rt = 0; rt < 9; rt++)
#pragma unroll
               for (int o4 = 0; o4 < 2; o4++) {
                  const ulonglong2 wv = *reinterpret_cast<const ulonglong2 *>(w + rt * kDcOut + 4 * o4);
#pragma unroll
                  for (int q = 0; q < 8; q++) {
                     acc2[q][2 * o4] = fma_f32x2(win[q + rt / 3][rt % 3], wv.x, acc2[q][2 * o4]);
                     acc2[q][2 * o4 + 1] = fma_f32x2(win[q + rt / 3][rt % 3], wv.y, acc2[q][2 * o4 + 1]);
                  }
               }
         }
      }
      if (!inside) continue;
      float acc[8][8];
#pragma unroll
      for (int q = 0; q < 8; q++)
#pragma unroll
         for (int o = 0; o < 4; o++) {
            unpack_f32x2(acc2[q][o], acc[q][2 * o], acc[q][2 * o + 1]);
#pragma unroll
            for (int e = 2 * o; e < 2 * o + 2; e++) {
               const float x = acc[q][e] + s_bias[oc_local + e];
               acc[q][e] = g.relu ? relu_ref(x) : x;
            }
         }
      auto store_pixel = [&](const float *v, int ph, int pw) {
         if (ph >= g.pH || pw >= g.pW || oc >= g.Cout) return;
         if (g.y_nhwc) {
            float *y = Y + (((size_t)n * g.pH + ph) * g.pW + pw) * g.Cout + oc;
            if (oc + 8 <= g.Cout && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
               *reinterpret_cast<float4 *>(y) = make_float4(v[0], v[1], v[2], v[3]);
               *reinterpret_cast<float4 *>(y + 4) = make_float4(v[4], v[5], v[6], v[7]);
            } else {
#pragma unroll
               for (int o = 0; o < 8; o++)
                  if (oc + o < g.Cout) y[o] = v[o];
            }
         } else {
#pragma unroll
            for (int o = 0; o < 8; o++)
               if (oc + o < g.Cout) Y[(((size_t)n * g.Cout + oc + o) * g.pH + ph) * g.pW + pw] = v[o];
         }
      };
      if constexpr (POOL == 2) {
         // The pixel beside is in lane ^ 2; of a pair of lanes the even column keeps the upper two windows, the odd one the lower two. The
         // maximum is that of the comparisons v > best from the window's first pixel on: a NaN counts there and is passed over elsewhere.
         const bool second = col & 1;
#pragma unroll
         for (int h = 0; h < 2; h++) {
            float best[8];
#pragma unroll
            for (int o = 0; o < 8; o++) {
               auto column = [&](float upper, float lower) { return second ? fmaxf(upper, lower) : (lower > upper ? lower : upper); };
               const float first = column(acc[2 * h][o], acc[2 * h + 1][o]), later = column(acc[2 * h + 4][o], acc[2 * h + 5][o]);
               const float got = __shfl_xor_sync(0xffffffffu, second ? first : later, 2), mine = second ? later : first;
               const float left = second ? got : mine, right = second ? mine : got;
               best[o] = right > left ? right : left;
            }
            store_pixel(best, (oh0 >> 1) + (second ? 2 : 0) + h, ow >> 1);
         }
      } else {
#pragma unroll
         for (int q = 0; q < 8; q++) store_pixel(acc[q], oh0 + q, ow);
      }
   }
}

template <int POOL, int GROUPS, bool VEC>
int launch_direct(cudaStream_t s, const ConvGeom &g, const float *X, const float *W, const float *bias, float *Y, int chunks)
{
   const int tiles_x = ceil_div(g.oW, 16 * GROUPS), tiles_y = ceil_div(g.oH, kDcRows), groups_y = ceil_div(g.Cout, kDcOut);
   const long long num_tiles = (long long)g.N * tiles_x * tiles_y;
   const int smem = (2 * dc_tile_floats(GROUPS) + chunks * kDcChunk * 9 * kDcOut) * (int)sizeof(float);
   auto kern = conv3x3_direct_f32_kernel<POOL, GROUPS, VEC>;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), smem));
   const long long cap = ceil_div(kNumSMs * (6 / GROUPS), groups_y);
   const long long blocks = num_tiles < cap ? num_tiles : cap;
   SOFIE_CUDA_TRY(launch_dependent(kern, dim3((unsigned)blocks, groups_y), dim3(64 * GROUPS), smem, s, g, X, W, bias, Y, num_tiles, tiles_x, tiles_y, chunks));
   SOFIE_LAUNCH_CHECK("conv3x3_direct_f32_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

// ---- few tiles: the input channels of a tile shared out between the block's warps ------------------------------------------------
// The kernel above walks a tile's channels one after the other in two warps: one image of 16 x 16 takes as long as 800 do (8 -> 16 channels 11.8 us,
// 16 -> 16 17.5), most of it round trips. Here a block of eight warps owns 4 RH rows x 16 columns x 16 output channels; a warp takes four of the
// rows and every (8 / RH)-th channel, a thread four outputs below one another x eight channels, and the sums of the 8 / RH warps meet in shared memory.
// All of up to 32 channels' inputs and weights are one round trip of asynchronous copies. Chains are shorter than the other kernel's, sums no less exact.
constexpr int kDsThreads = 256, kDsChunk = 32, kDsPitch = 24, kDsWPitch = 20; // 20: a warp's weights in four banks apart, 16 bytes aligned
__host__ __device__ constexpr int ds_channel(int RH) { return (4 * RH + 2) * kDsPitch + 4; } // + 4: neighbouring channels start in other banks
__host__ __device__ constexpr int ds_out(int RH) { return 4 * RH * 16 + 2; }
__host__ __device__ constexpr int ds_partial(int RH) { return kDcOut * ds_out(RH); }

template <int POOL, int RH, bool VEC>
__global__ void __launch_bounds__(kDsThreads, 2)
conv3x3_split_f32_kernel(ConvGeom g, const float *__restrict__ X, const float *__restrict__ Wt, const float *__restrict__ bias, float *__restrict__ Y, FastDiv tiles_x,
                         FastDiv tiles_y, int chunk)
{
   constexpr int KS = 8 / RH, ROWS = 4 * RH + 2, CST = ds_channel(RH), OST = ds_out(RH);
   extern __shared__ __align__(16) float smem[];
   float *tile = smem;                 // [channel][row][column], from column w0 - 4 on
   float *s_w = smem + chunk * CST;    // [channel][tap][16], rows of kDsWPitch
   float *partial = smem;              // [sharer][output channel][row][column], where the inputs and weights were
   __shared__ float s_bias[kDcOut];
   griddep_launch_dependents();
   griddep_wait(X, Wt, bias);
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, oc_base = blockIdx.y * kDcOut, outs = min(kDcOut, g.Cout - oc_base);
   if (tid < kDcOut) s_bias[tid] = tid < outs && bias ? __ldg(bias + oc_base + tid) : 0.f;
   uint32_t tx, ty;
   const uint32_t n = tiles_y.divmod(tiles_x.divmod(blockIdx.x, tx), ty);
   const int h0 = (int)ty * 4 * RH, w0 = (int)tx * 16;
   const int col = lane >> 1, oc_local = (lane & 1) * 8, half = warp / KS, sharer = warp % KS;
   uint64_t acc2[4][4]; // two neighbouring channels each
#pragma unroll
   for (int q = 0; q < 4; q++)
#pragma unroll
      for (int o = 0; o < 4; o++) acc2[q][o] = 0;
   for (int c0 = 0; c0 < g.C; c0 += chunk) {
      const int ck = min(chunk, g.C - c0);
      if (c0) __syncthreads(); // the chunk before this one is no longer read
      auto copy4 = [](float *dst, const float *src, int bytes) {
         asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
      };
      if constexpr (VEC) {
         constexpr int WORDS = kDsPitch / 4;
         for (int i = tid; i < ck * ROWS * WORDS; i += kDsThreads) {
            const int c = i / (ROWS * WORDS), p = i % (ROWS * WORDS), r = p / WORDS, w = p % WORDS;
            const int ih = h0 - 1 + r, iw = w0 - 4 + 4 * w;
            const bool in = ih >= 0 && ih < g.H && iw >= 0 && iw < g.W;
            const float *src = in ? X + (((size_t)n * g.C + c0 + c) * g.H + ih) * g.W + iw : X;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(tile + c * CST + 4 * p)), "l"(src), "r"(in ? 16 : 0) : "memory");
         }
      } else {
         constexpr int COLS = 18;
         for (int i = tid; i < ck * ROWS * COLS; i += kDsThreads) {
            // the index that is contiguous in memory runs fastest
            const int c = g.x_nhwc ? i % ck : i / (ROWS * COLS), p = g.x_nhwc ? i / ck : i % (ROWS * COLS);
            const int r = p / COLS, k = p % COLS, ih = h0 - 1 + r, iw = w0 - 1 + k;
            const bool in = ih >= 0 && ih < g.H && iw >= 0 && iw < g.W;
            const size_t at = g.x_nhwc ? (((size_t)n * g.H + ih) * g.W + iw) * g.C + c0 + c : (((size_t)n * g.C + c0 + c) * g.H + ih) * g.W + iw;
            copy4(tile + c * CST + r * kDsPitch + 3 + k, in ? X + at : X, in ? 4 : 0);
         }
      }
      // a filter's weights of these channels are consecutive in memory, tap by tap or channel by channel
      for (int i = tid; i < kDcOut * ck * 9; i += kDsThreads) {
         const int o = i / (ck * 9), e = i - o * (ck * 9);
         const int c = g.w_packed ? e % ck : e / 9, rt = g.w_packed ? e / ck : e % 9;
         copy4(s_w + (c * 9 + rt) * kDsWPitch + o, o < outs ? Wt + dc_weight_index(g, oc_base + o, c0 + c, rt) : Wt, o < outs ? 4 : 0);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      const float *in = tile + half * 4 * kDsPitch + col + 3;
#pragma unroll 1
      for (int c = sharer; c < ck; c += KS) {
         uint64_t win[6][3]; // the inputs under the four outputs, each twice
#pragma unroll
         for (int r = 0; r < 6; r++)
#pragma unroll
            for (int t = 0; t < 3; t++) {
               const float v = in[c * CST + r * kDsPitch + t];
               win[r][t] = pack_f32x2(v, v);
            }
         const float *w = s_w + c * 9 * kDsWPitch + oc_local;
#pragma unroll
         for (int rt = 0; rt < 9; rt++)
#pragma unroll
            for (int o4 = 0; o4 < 2; o4++) {
               const ulonglong2 wv = *reinterpret_cast<const ulonglong2 *>(w + rt * kDsWPitch + 4 * o4);
#pragma unroll
               for (int q = 0; q < 4; q++) {
                  acc2[q][2 * o4] = fma_f32x2(win[q + rt / 3][rt % 3], wv.x, acc2[q][2 * o4]);
                  acc2[q][2 * o4 + 1] = fma_f32x2(win[q + rt / 3][rt % 3], wv.y, acc2[q][2 * o4 + 1]);
               }
            }
      }
   }
   __syncthreads(); // inputs and weights are no longer read
   {
      float *p = partial + sharer * ds_partial(RH) + oc_local * OST + half * 64 + col;
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
         for (int o = 0; o < 4; o++) {
            float a, b;
            unpack_f32x2(acc2[q][o], a, b);
            p[2 * o * OST + q * 16] = a;
            p[(2 * o + 1) * OST + q * 16] = b;
         }
   }
   __syncthreads();
   // one output of the convolution
   auto output = [&](int o, int row, int column) {
      const float *p = partial + o * OST + row * 16 + column;
      float v = p[0];
#pragma unroll
      for (int k = 1; k < KS; k++) v += p[k * ds_partial(RH)];
      v += s_bias[o];
      return g.relu ? relu_ref(v) : v;
   };
   constexpr int SIDE = POOL == 2 ? 2 : 1, PR = 4 * RH / SIDE, PC = 16 / SIDE;
   for (int i = tid; i < PR * PC * kDcOut; i += kDsThreads) {
      // threads along what is contiguous in Y
      const int o = g.y_nhwc ? i % kDcOut : i / (PR * PC), p = g.y_nhwc ? i / kDcOut : i % (PR * PC);
      const int pr = p / PC, pc = p % PC, ph = h0 / SIDE + pr, pw = w0 / SIDE + pc;
      if (o >= outs || ph >= g.pH || pw >= g.pW) continue;
      float v = output(o, SIDE * pr, SIDE * pc);
      if constexpr (POOL == 2) {
         // the comparisons v > best from the window's first pixel on: a NaN counts there and is passed over elsewhere
#pragma unroll
         for (int k = 1; k < 4; k++) {
            const float u = output(o, 2 * pr + k / 2, 2 * pc + k % 2);
            v = u > v ? u : v;
         }
      }
      Y[g.y_nhwc ? (((size_t)n * g.pH + ph) * g.pW + pw) * g.Cout + oc_base + o : (((size_t)n * g.Cout + oc_base + o) * g.pH + ph) * g.pW + pw] = v;
   }
}

// -1 when the grid would not hold the tiles
template <int POOL, int RH, bool VEC>
int launch_split(cudaStream_t s, const ConvGeom &g, const float *X, const float *W, const float *bias, float *Y)
{
   const int tiles_x = ceil_div(g.oW, 16), tiles_y = ceil_div(g.oH, 4 * RH), chunk = g.C < kDsChunk ? g.C : kDsChunk;
   const long long tiles = (long long)g.N * tiles_x * tiles_y;
   if (tiles >= 1ll << 31) return -1;
   const int staged = chunk * (ds_channel(RH) + 9 * kDsWPitch), sums = 8 / RH * ds_partial(RH), smem = (staged > sums ? staged : sums) * (int)sizeof(float);
   auto kern = conv3x3_split_f32_kernel<POOL, RH, VEC>;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), smem));
   SOFIE_CUDA_TRY(launch_dependent(kern, dim3((unsigned)tiles, ceil_div(g.Cout, kDcOut)), dim3(kDsThreads), smem, s, g, X, W, bias, Y, FastDiv(tiles_x), FastDiv(tiles_y), chunk));
   SOFIE_LAUNCH_CHECK("conv3x3_split_f32_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

} // namespace

// 3x3 / stride 1 / pad 1 / group 1 with at most 128 input channels (their weights for 16 outputs are 72 KB): -1 for any other shape.
int launch_conv2d_f32_direct3x3(cudaStream_t s, const ConvGeom &g, const float *X, const float *W, const float *bias, float *Y)
{
   if (!(g.kH == 3 && g.kW == 3 && g.pad_h == 1 && g.pad_w == 1 && g.sh == 1 && g.sw == 1 && g.dh == 1 && g.dw == 1 && g.group == 1)) return -1;
   if (g.C > 128 || (g.pool != 0 && g.pool != 2) || g.N < 1 || ceil_div(g.Cout, kDcOut) > 65535) return -1;
   const int chunks = ceil_div(g.C, kDcChunk);
   const bool vec = !g.x_nhwc && g.W % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0, wide = g.oW > 16;
   // Images that fill less than a quarter of the large tiles stay with one thread per output: 1000 x 32 -> 32 at 7 x 7 141 us against 190 here, at 8 x 8
   // (24 channels, NHWC) 145 against 136. So do those that fill less than 0.6 of them where it is faster by the time in us that either takes, fitted
   // to 200 calls of 1 to 1024 images (to 14 and 12 %; three of them are 6 to 16 % slower here all the same): few channels, whose time here is copies and indexes (32 x 5 -> 61 at 43 x 9 14.0 us against 22.3;
   // 133 x 15 -> 103 at 65 x 6 212 against 248).
   const long long groups = ceil_div(g.Cout, kDcOut), tiles = (long long)ceil_div(g.oH, kDcRows) * ceil_div(g.oW, wide ? 32 : 16), area = kDcRows * (wide ? 32 : 16);
   const long long outputs = (long long)g.oH * g.oW;
   const double positions = 1e-6 * g.N * outputs, units = (double)g.N * tiles * groups * (wide ? 2 : 1);
   // images of one row: a third of the taps lie on them (447 x 84 -> 39 at 1 x 7 90 us, 144 with shared channels, which were estimated faster without this factor)
   const double inside = g.oH > 1 ? 1.0 : (g.oW > 1 ? 0.65 : 0.5);
   const double general = 1.9 + inside * (1.69 * g.C + positions * 25 * groups * g.C) + positions * 2.6 * g.Cout;
   const double sparse = 2.5 + chunks * (vec ? 3.5 : 4.7) + 1e-3 * units * (chunks * (vec ? 5.1 : 8.1) + 4.8);
   const bool filled = 5 * outputs >= 3 * tiles * area;
   const bool large = 4 * outputs >= tiles * area && (filled || 1.05 * general > sparse);
   // Shared channels take what is estimated faster that way by a twentieth: the first block of an SM costs its round trips, each further one its work.
   // (us, by channels; 8 RH = 1, 2, 4; 16 -> 16 channels of 16 x 16, 1 / 128 / 512 / 1024 images: 4.9 / 12.0 / 38 / 74, 5.8 / 8.6 / 27 / 51, 8.2 / 11.7 / 24 / 41, large tiles 19.6 / 20.2 / 34 / 44.)
   double best = large ? (filled ? (vec ? 1.0 : 1.1) * (2.5 + 4.3 * chunks + (units > kNumSMs ? units / kNumSMs - 1 : 0) * 0.29 * g.C) : sparse) : general;
   best *= 0.95;
   int share = 0;
   for (int i = 0; i < 3; i++) {
      static const double first[3] = {0.17, 0.235, 0.35}, more[3] = {0.145, 0.21, 0.35}, fixed[3] = {0.5, 0.7, 0.8};
      const double blocks = (double)g.N * ceil_div(g.oH, 4 << i) * ceil_div(g.oW, 16) * groups;
      const double time = (vec ? 1.0 : 1.25) * (2.4 + first[i] * g.C + (blocks > kNumSMs ? blocks / kNumSMs - 1 : 0) * (fixed[i] + more[i] * g.C));
      if (time < best) best = time, share = 1 << i;
   }
#define SOFIE_SPLIT(P, R) rc = vec ? launch_split<P, R, true>(s, g, X, W, bias, Y) : launch_split<P, R, false>(s, g, X, W, bias, Y)
   int rc = -1;
   if (g.pool == 2) {
      if (share == 1) SOFIE_SPLIT(2, 1);
      if (share == 2) SOFIE_SPLIT(2, 2);
      if (share == 4) SOFIE_SPLIT(2, 4);
   } else {
      if (share == 1) SOFIE_SPLIT(0, 1);
      if (share == 2) SOFIE_SPLIT(0, 2);
      if (share == 4) SOFIE_SPLIT(0, 4);
   }
#undef SOFIE_SPLIT
   if (rc >= 0 || !large) return rc;
#define SOFIE_DIRECT(P, G) return vec ? launch_direct<P, G, true>(s, g, X, W, bias, Y, chunks) : launch_direct<P, G, false>(s, g, X, W, bias, Y, chunks)
   if (g.pool == 2) {
      if (wide) SOFIE_DIRECT(2, 2);
      SOFIE_DIRECT(2, 1);
   }
   if (wide) SOFIE_DIRECT(0, 2);
   SOFIE_DIRECT(0, 1);
#undef SOFIE_DIRECT
}

} // namespace sofie
