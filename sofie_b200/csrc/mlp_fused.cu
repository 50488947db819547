// Fused multi-layer perceptron for small layers: Y = L_{n-1}(... L_0(X)), L_l(x) = act(x W_l^T + b_l),
// all layer widths <= 256 and all weights together small enough for shared memory. One launch
// replaces one GEMM launch per layer: at these sizes (C1: 64 -> 128 -> 128 -> 10, 104 KB of
// weights, 52 kFLOP per sample) a layer is far too small to fill the GPU and its time is launch
// latency plus the round trip of its activations through memory. A block keeps every layer's
// weights in shared memory and walks tiles of ROWS batch rows; activations never leave the SM.
//   weights     [n][ld], ld = K rounded up to 4, plus a pad that makes ld / 4 odd: the rows that the
//               column subgroups of a warp read start 16 bytes apart in the banks
//   activations [row][ld], same padding rule: the rows of a quarter warp hit distinct banks
//   thread      (warp w, lane): batch row lane % ROWS, columns q + CSTEP j with q = w * SUB + lane / ROWS;
//               per four k one 16-byte load of its row and one 16-byte load per column
//   ROWS        32, 16 or 8: the largest that still gives every SM a tile, so that a small batch
//               spreads over the whole GPU (each block stages the weights from L2 either way)
// A kernel of its own for eight rows (K split over a warp's quarters, 512 threads, two more shuffles and barriers of twice the warps) was
// slower at every size: 64 -> 128 -> 128 -> 10 9.2 us instead of 8.25 for one row and 9.6 instead of 8.6 for 1024, back to back; 14.3
// instead of 12.3 after an L2 flush.
// Staging uses 16-byte asynchronous copies (all of a block's weight bytes in flight at once) when
// the layout allows it: [N][K] weights, K a multiple of 4, 16-byte aligned pointers. The input
// tile of the next batch rows is fetched while the layers after the first run.
// fp32 FMA throughout (K <= 256 per layer, accumulation in order of k).
#include "common.cuh"
#include "contract.cuh"

namespace sofie {
namespace {

constexpr int kMlpThreads = 256;

struct MlpParams {
   sofie_mlp_desc d;
   const float *W[SOFIE_MLP_MAX_LAYERS];
   const float *B[SOFIE_MLP_MAX_LAYERS];
   int w_off[SOFIE_MLP_MAX_LAYERS]; // offset of layer l's [Np][w_ld] weights in shared memory, in floats
   int w_ld[SOFIE_MLP_MAX_LAYERS];
   int b_off[SOFIE_MLP_MAX_LAYERS]; // offset of its Np biases
   int x_off, x_ld;                 // input tile [ROWS][x_ld]
   int act_off[2], act_ld;          // the two activation buffers [ROWS][act_ld]
   int w_vec[SOFIE_MLP_MAX_LAYERS]; // layer's weights can be staged with 16-byte copies
   int x_vec;
};

inline int padded_ld(int k) { return sofie_mlp_padded_ld(k); }

__device__ __forceinline__ void cp_async16(float *dst_smem, const float *src, bool valid)
{
   const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
   const int bytes = valid ? 16 : 0; // 0 source bytes: the 16 destination bytes are zero-filled
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst_smem, const float *src)
{
   const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
   asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// wait until at most `n` of the most recently committed groups are still in flight (the count is an immediate)
__device__ __forceinline__ void cp_async_wait_pending(int n)
{
   switch (n) {
   case 0: asm volatile("cp.async.wait_group 0;\n" ::: "memory"); break;
   case 1: asm volatile("cp.async.wait_group 1;\n" ::: "memory"); break;
   case 2: asm volatile("cp.async.wait_group 2;\n" ::: "memory"); break;
   case 3: asm volatile("cp.async.wait_group 3;\n" ::: "memory"); break;
   case 4: asm volatile("cp.async.wait_group 4;\n" ::: "memory"); break;
   case 5: asm volatile("cp.async.wait_group 5;\n" ::: "memory"); break;
   case 6: asm volatile("cp.async.wait_group 6;\n" ::: "memory"); break;
   case 7: asm volatile("cp.async.wait_group 7;\n" ::: "memory"); break;
   default: asm volatile("cp.async.wait_group 8;\n" ::: "memory"); break;
   }
}

// Rows of `kq` 16-byte pieces walked by the whole block without a division per piece: the thread's piece
// index advances by the block size, that is by (step_n rows, step_c pieces) with one carry.
struct PieceWalker {
   int n, c, step_n, step_c, kq;
   __device__ __forceinline__ PieceWalker(int tid, int kq_) : kq(kq_)
   {
      n = tid / kq;
      c = tid - n * kq;
      step_n = kMlpThreads / kq;
      step_c = kMlpThreads - step_n * kq;
   }
   __device__ __forceinline__ void next()
   {
      n += step_n;
      c += step_c;
      if (c >= kq) {
         c -= kq;
         n++;
      }
   }
};

template <int ROWS>
__device__ __forceinline__ void load_x_tile(const MlpParams &p, const float *__restrict__ X, float *sm, int tile, int tid)
{
   const int K0 = p.d.dims[0], M = p.d.M, m0 = tile * ROWS;
   float *xin = sm + p.x_off;
   if (p.x_vec) {
      for (PieceWalker it(tid, K0 >> 2); it.n < ROWS; it.next()) {
         const bool ok = m0 + it.n < M;
         cp_async16(xin + it.n * p.x_ld + 4 * it.c, X + (size_t)(ok ? m0 + it.n : 0) * K0 + 4 * it.c, ok);
      }
   } else {
      const int K0p = (K0 + 3) & ~3;
      for (int i = tid; i < ROWS * K0p; i += kMlpThreads) {
         const int r = i / K0p, k = i - r * K0p;
         xin[r * p.x_ld + k] = (m0 + r < M && k < K0) ? __ldg(X + (size_t)(m0 + r) * K0 + k) : 0.f;
      }
   }
}

// One layer for one thread: batch row `arow`, columns q + CSTEP j for j < J, J = NB * 32 / CSTEP known at compile time
// (NB = the layer's width in units of 32 columns).
template <int ROWS, int NB>
__device__ __forceinline__ void mlp_layer(const float *__restrict__ arow, const float *__restrict__ wrow, const float *__restrict__ bs,
                                          float *__restrict__ nxt, int Kp, int ldw, int N4, int q, bool relu)
{
   constexpr int CSTEP = 8 * (32 / ROWS);
   constexpr int J = NB * 32 / CSTEP;
   float acc[J];
#pragma unroll
   for (int j = 0; j < J; j++) acc[j] = 0.f;
#pragma unroll 2
   for (int k = 0; k < Kp; k += 4) {
      const float4 a = *reinterpret_cast<const float4 *>(arow + k);
#pragma unroll
      for (int j = 0; j < J; j++) {
         const float4 wv = *reinterpret_cast<const float4 *>(wrow + j * CSTEP * ldw + k);
         acc[j] = fmaf(a.x, wv.x, acc[j]);
         acc[j] = fmaf(a.y, wv.y, acc[j]);
         acc[j] = fmaf(a.z, wv.z, acc[j]);
         acc[j] = fmaf(a.w, wv.w, acc[j]);
      }
   }
#pragma unroll
   for (int j = 0; j < J; j++) {
      const int n = q + CSTEP * j;
      if (n < N4) {
         const float v = acc[j] + bs[n];
         nxt[n] = relu ? relu_ref(v) : v;
      }
   }
}

template <int ROWS>
__global__ void __launch_bounds__(kMlpThreads, 1)
mlp_fused_f32_kernel(MlpParams p, const float *__restrict__ X, float *__restrict__ Y)
{
   constexpr int SUB = 32 / ROWS;  // column subgroups of a warp; two columns of one thread are 8 * SUB apart
   extern __shared__ __align__(16) float sm[];
   const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
   const int r = lane % ROWS, q = w * SUB + lane / ROWS;
   const int L = p.d.layers, M = p.d.M;
   const int tiles = (M + ROWS - 1) / ROWS;
   // ---- the first input tile, then weights and biases, once per block
   // Copy groups in order: [input tile + layer 0], [layer 1], ..., [layer L-1]; layer l of the first tile
   // starts as soon as its own group has landed while the later layers' weights are still arriving.
   load_x_tile<ROWS>(p, X, sm, blockIdx.x, tid);
   for (int l = 0; l < L; l++) {
      const int K = p.d.dims[l], N = p.d.dims[l + 1], Np = (N + 31) & ~31, ld = p.w_ld[l];
      float *wt = sm + p.w_off[l];
      const float *Wg = p.W[l];
      if (p.w_vec[l]) {
         for (PieceWalker it(tid, K >> 2); it.n < N; it.next()) cp_async16(wt + it.n * ld + 4 * it.c, Wg + (size_t)it.n * K + 4 * it.c, true);
         for (int i = tid; i < (Np - N) * ld; i += kMlpThreads) wt[N * ld + i] = 0.f; // columns past N contribute nothing
      } else if (p.d.w_is_nk[l]) {
         const int Kp = (K + 3) & ~3;
         for (int i = tid; i < Np * Kp; i += kMlpThreads) {
            const int n = i / Kp, k = i - n * Kp;
            wt[n * ld + k] = (n < N && k < K) ? __ldg(Wg + (size_t)n * K + k) : 0.f;
         }
      } else {
         // global [K][N] -> shared [n][k]: consecutive threads take consecutive n, reads coalesced
         const int Kp = (K + 3) & ~3;
         for (int i = tid; i < Np * Kp; i += kMlpThreads) {
            const int k = i / Np, n = i - k * Np;
            wt[n * ld + k] = (n < N && k < K) ? __ldg(Wg + (size_t)k * N + n) : 0.f;
         }
      }
      float *bs = sm + p.b_off[l];
      for (int n = tid; n < Np; n += kMlpThreads) {
         if (n < N && p.B[l])
            cp_async4(bs + n, p.B[l] + n);
         else
            bs[n] = 0.f;
      }
      cp_async_commit();
   }
   bool first = true;
   for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int m0 = tile * ROWS;
      if (!first) {
         cp_async_wait_all();
         __syncthreads(); // this tile's input has landed; the previous tile's buffers are free
      }
      for (int l = 0; l < L; l++) {
         if (first) {
            // groups still allowed in flight: the later layers' and, behind layer 0, the next tile's input
            cp_async_wait_pending(L - 1 - l + (l > 0 ? 1 : 0));
            __syncthreads();
         }
         const int K = p.d.dims[l], N = p.d.dims[l + 1], Kp = (K + 3) & ~3;
         const int ldw = p.w_ld[l], lda = l == 0 ? p.x_ld : p.act_ld;
         const float *arow = sm + (l == 0 ? p.x_off : p.act_off[(l - 1) & 1]) + r * lda;
         const float *wrow = sm + p.w_off[l] + q * ldw;
         const float *bs = sm + p.b_off[l];
         const bool relu = p.d.relu[l] != 0;
         const int N4 = (N + 3) & ~3; // the next layer reads k up to its K rounded to 4: columns N .. N4 are written as zeros
         float *nxt = sm + p.act_off[l & 1] + r * p.act_ld;
         switch (((N + 31) & ~31) >> 5) { // the column count is a compile-time constant inside: no predicated-off work
         case 1: mlp_layer<ROWS, 1>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         case 2: mlp_layer<ROWS, 2>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         case 3: mlp_layer<ROWS, 3>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         case 4: mlp_layer<ROWS, 4>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         case 5: mlp_layer<ROWS, 5>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         case 6: mlp_layer<ROWS, 6>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         case 7: mlp_layer<ROWS, 7>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         default: mlp_layer<ROWS, 8>(arow, wrow, bs, nxt, Kp, ldw, N4, q, relu); break;
         }
         __syncthreads(); // the next layer (or the copy-out) reads what every warp wrote
         if (l == 0) {
            if (tile + (int)gridDim.x < tiles) load_x_tile<ROWS>(p, X, sm, tile + gridDim.x, tid); // the input buffer is free
            cp_async_commit(); // committed even when empty: the group count above does not depend on the tile
         }
      }
      first = false;
      {
         // the tile's rows are one contiguous piece of Y
         const int N = p.d.dims[L];
         const float *out = sm + p.act_off[(L - 1) & 1];
         const int rows = M - m0 < ROWS ? M - m0 : ROWS;
         float *Yt = Y + (size_t)m0 * N;
         for (int i = tid; i < rows * N; i += kMlpThreads) {
            const int rr = i / N, n = i - rr * N;
            Yt[i] = out[rr * p.act_ld + n];
         }
      }
   }
   cp_async_wait_all();
}

template <int ROWS>
int launch_mlp(cudaStream_t stream, MlpParams &p, int floats, int maxact, const float *X, float *Y)
{
   p.x_off = floats;
   p.x_ld = padded_ld(p.d.dims[0]);
   floats += ROWS * p.x_ld;
   p.act_ld = padded_ld(maxact);
   p.act_off[0] = floats;
   p.act_off[1] = floats + ROWS * p.act_ld;
   floats += 2 * ROWS * p.act_ld;
   const size_t smem = (size_t)floats * sizeof(float);
   const int tiles = (p.d.M + ROWS - 1) / ROWS, blocks = tiles < kNumSMs ? tiles : kNumSMs;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(mlp_fused_f32_kernel<ROWS>), (int)smem));
   mlp_fused_f32_kernel<ROWS><<<blocks, kMlpThreads, smem, stream>>>(p, X, Y);
   SOFIE_LAUNCH_CHECK("mlp_fused_f32_kernel");
   return SOFIE_CUDA_OK;
}

// ---- few rows: the weights in registers ---------------------------------------------------------------------------
// With a row or two a block each weight is used once or twice: staging them in shared memory is half of such a call. Here S lanes share an output's sum and a thread
// holds its pieces of the weights of all (up to three) layers in registers, asked for at once and beside the inputs, which come the longest way (across PCIe where a Session
// leaves them in host memory); what remains of a layer is its sum, two to five shuffles and a barrier. What bounds it: the launch and two round trips, then the
// weights' way out of L2. 64 -> 128 -> 128 -> 10, launch and wait, inputs and results in host memory: 1 row 17.4 -> 14.5 us, 128 20.4 -> 18.0, 256 21.6 -> 19.4; a Session on 1 / 64 / 128 /
// 256 rows 22.1 -> 18.1, 23.8 -> 22.2, 30.7 -> 23.7, 32.5 -> 27.8. From three rows a block on it is no faster (400 rows 35.2 both, 592 35.2 against 37.4: its reads of the rows).
// A cluster of 2, 4 or 8 blocks that shares the outputs and writes them to each other's shared memory saves one to two us of a row's and loses from 64 rows on.
constexpr int kRegThreads = 512, kRegPieces = 8, kRegRows = 2;
struct RegParams {
   int M, rows, ld;
   int K[3], N[3], S[3], pieces[3], relu[3];
   const float *W[3], *B[3];
};

template <int NL>
__global__ void __launch_bounds__(kRegThreads, 1) mlp_registers_f32_kernel(RegParams p, const float *__restrict__ X, float *__restrict__ Y)
{
   extern __shared__ __align__(16) float sm[]; // the inputs of every layer, [row][ld], zeros behind them
   const int tid = threadIdx.x, m0 = blockIdx.x * p.rows, rows = min(p.rows, p.M - m0), L4 = p.ld >> 2;
   for (int i = tid; i < rows * L4; i += kRegThreads) {
      const int r = i / L4, k = 4 * (i - r * L4);
      const bool in = k < p.K[0];
      cp_async16(sm + r * p.ld + k, X + (size_t)(m0 + r) * p.K[0] + (in ? k : 0), in);
   }
   float4 w[NL][kRegPieces];
   float b[NL];
#pragma unroll
   for (int l = 0; l < NL; l++) {
      const int S = p.S[l], n = tid / S;
      const bool ok = n < p.N[l];
      const float4 *row = reinterpret_cast<const float4 *>(p.W[l] + (size_t)(ok ? n : 0) * p.K[l]);
      b[l] = ok && p.B[l] ? __ldg(p.B[l] + n) : 0.f;
#pragma unroll
      for (int i = 0; i < kRegPieces; i++) {
         const int k = (tid & (S - 1)) + S * i;
         w[l][i] = ok && 4 * k < p.K[l] ? __ldg(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
   }
   for (int i = tid; i < (NL - 1) * p.rows * p.ld; i += kRegThreads) sm[p.rows * p.ld + i] = 0.f;
   cp_async_wait_all();
   __syncthreads();
#pragma unroll
   for (int l = 0; l < NL; l++) {
      const int S = p.S[l], s = tid & (S - 1), n = tid / S, pieces = p.pieces[l], N = p.N[l];
      const float *in = sm + l * p.rows * p.ld + 4 * s;
      if ((tid & ~31) / S < N) // some output of this warp
         for (int r = 0; r < rows; r++) {
            float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kRegPieces; i++)
               if (i < pieces) {
                  const float4 x = *reinterpret_cast<const float4 *>(in + r * p.ld + 4 * S * i);
                  c.x = fmaf(x.x, w[l][i].x, c.x);
                  c.y = fmaf(x.y, w[l][i].y, c.y);
                  c.z = fmaf(x.z, w[l][i].z, c.z);
                  c.w = fmaf(x.w, w[l][i].w, c.w);
               }
            float v = (c.x + c.y) + (c.z + c.w);
            for (int d = 1; d < S; d *= 2) v += __shfl_xor_sync(0xffffffffu, v, d);
            v += b[l];
            if (p.relu[l]) v = relu_ref(v);
            if (s == 0 && n < N) {
               if (l + 1 < NL) sm[((l + 1) * p.rows + r) * p.ld + n] = v;
               else Y[(size_t)(m0 + r) * N + n] = v;
            }
         }
      if (l + 1 < NL) __syncthreads();
   }
}

// -1 for more rows or layers, and for weights that are not read in 16-byte pieces or of which a thread would hold more than kRegPieces a layer
int launch_mlp_registers(cudaStream_t stream, const MlpParams &m, const float *X, float *Y)
{
   const sofie_mlp_desc &d = m.d;
   if (d.layers > 3 || d.M > kRegRows * kNumSMs || !m.x_vec) return -1;
   RegParams p = {};
   p.M = d.M;
   p.rows = ceil_div(d.M, kNumSMs);
   for (int l = 0; l < d.layers; l++) {
      int S = 32;
      while (S > 1 && S * d.dims[l + 1] > kRegThreads) S >>= 1;
      p.K[l] = d.dims[l], p.N[l] = d.dims[l + 1], p.S[l] = S, p.pieces[l] = ceil_div(ceil_div(d.dims[l], 4), S), p.relu[l] = d.relu[l];
      p.W[l] = m.W[l], p.B[l] = m.B[l];
      if (!m.w_vec[l] || S * p.N[l] > kRegThreads || p.pieces[l] > kRegPieces) return -1;
      if (p.ld < 4 * S * p.pieces[l]) p.ld = 4 * S * p.pieces[l];
   }
   const size_t smem = (size_t)d.layers * p.rows * p.ld * sizeof(float); // at most 3 x 2 x 256 floats
   const int blocks = ceil_div(d.M, p.rows);
   if (d.layers == 1) mlp_registers_f32_kernel<1><<<blocks, kRegThreads, smem, stream>>>(p, X, Y);
   else if (d.layers == 2) mlp_registers_f32_kernel<2><<<blocks, kRegThreads, smem, stream>>>(p, X, Y);
   else mlp_registers_f32_kernel<3><<<blocks, kRegThreads, smem, stream>>>(p, X, Y);
   SOFIE_LAUNCH_CHECK("mlp_registers_f32_kernel");
   return SOFIE_CUDA_OK;
}

} // namespace
} // namespace sofie

using namespace sofie;

extern "C" size_t sofie_cuda_mlp_f32_smem(const sofie_mlp_desc *d)
{
   if (!d || d->layers < 1 || d->layers > SOFIE_MLP_MAX_LAYERS) return 0;
   return sofie_mlp_smem_bytes(d);
}

extern "C" int sofie_cuda_mlp_f32(void *stream, const sofie_mlp_desc *d, const float *X, const float *const *W, const float *const *B, float *Y)
{
   SOFIE_REQUIRE(d != nullptr, "NULL descriptor");
   SOFIE_REQUIRE(d->layers >= 1 && d->layers <= SOFIE_MLP_MAX_LAYERS, "1 to %d layers", SOFIE_MLP_MAX_LAYERS);
   SOFIE_REQUIRE(d->M >= 0, "negative batch");
   SOFIE_REQUIRE(W != nullptr, "NULL weight table");
   MlpParams p = {};
   p.d = *d;
   int floats = 0, maxact = 0;
   for (int l = 0; l <= d->layers; l++) {
      SOFIE_REQUIRE(d->dims[l] >= 1, "layer width must be positive");
      if (d->dims[l] > SOFIE_MLP_MAX_WIDTH)
         return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "the fused MLP takes layer widths up to %d, got %d", SOFIE_MLP_MAX_WIDTH, d->dims[l]);
      if (l >= 1 && d->dims[l] > maxact) maxact = d->dims[l];
   }
   for (int l = 0; l < d->layers; l++) {
      SOFIE_REQUIRE(W[l] != nullptr, "NULL weights of layer %d", l);
      const int K = d->dims[l], Np = (d->dims[l + 1] + 31) & ~31;
      p.W[l] = W[l];
      p.B[l] = B ? B[l] : nullptr;
      p.w_vec[l] = d->w_is_nk[l] && K % 4 == 0 && (reinterpret_cast<uintptr_t>(W[l]) & 15) == 0;
      p.w_ld[l] = padded_ld(K);
      p.w_off[l] = floats;
      floats += Np * p.w_ld[l];
      p.b_off[l] = floats;
      floats += Np;
   }
   p.x_vec = d->dims[0] % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
   // the size test assumes the largest tile, so that it does not depend on the batch
   const size_t worst = sofie_mlp_smem_bytes(d);
   if (worst > SOFIE_MLP_MAX_SMEM)
      return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "the fused MLP needs %zu bytes of shared memory for these layers (limit %d)", worst, SOFIE_MLP_MAX_SMEM);
   if (d->M == 0) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(X && Y, "NULL tensor");
   cudaStream_t s = as_stream(stream);
   // The tensor-core chain (umma_mlp.cu) runs when the caller forces that engine. It is not the default: measured on
   // B200 for 64 -> 128 -> 128 -> 10 it takes 42 us at 1024 rows (this file's FMA kernel: 17 us, on 128 SMs instead of 8)
   // and 311 us at 2^18 rows (one tensor-core GEMM launch per layer: 193 us) -- every CTA re-reads and re-splits all the
   // weights for each 128-row slab, and those reads from L2 and their shared-memory writes, not the MMAs, set its time.
   if (forced_engine() == SOFIE_ENGINE_TCGEN05) {
      const int rc = launch_mlp_f32_umma(s, d, X, W, B, Y);
      if (rc >= 0) return rc;
      return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "these layer widths are not served by the tensor-core chain");
   }
   set_last_engine(SOFIE_ENGINE_SIMT);
   const int few = launch_mlp_registers(s, p, X, Y);
   if (few >= 0) return few;
   int rows = 32;
   while (rows > 8 && (d->M + rows - 1) / rows < kNumSMs) rows >>= 1;
   if (rows == 32) return launch_mlp<32>(s, p, floats, maxact, X, Y);
   if (rows == 16) return launch_mlp<16>(s, p, floats, maxact, X, Y);
   return launch_mlp<8>(s, p, floats, maxact, X, Y);
}
