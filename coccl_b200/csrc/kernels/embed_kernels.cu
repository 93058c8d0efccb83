// Gradient of the word and position embeddings, summed in fp32 straight into the parameters' gradient buffers.
//
// PyTorch's embedding backward builds a dense bf16 gradient of the whole table (50304 x 4096: 412 MB), which then had to be
// cast to fp32 and added to the gradient buffer: 1.4 ms a micro-batch for 4096 tokens. Only the rows of the tokens at hand
// change, so here the work is one read of the output gradient and one read-modify-write of those rows (167 MB, 26 us to
// copy): 38 us, with 9 us for the order of the tokens and 15 us for the positions. Rows are summed in a fixed order,
// whatever the launch: the result does not depend on scheduling.
#include "dependent_launch.h"
#include "launch_count.h"
#include "common.cuh"
#include "train_api.h"

namespace coccl {

using bf16 = __nv_bfloat16;
constexpr int kEmbThreads = 256;
constexpr int kEmbLanes = 128;     // threads side by side on the columns of a row, eight values each
constexpr int kEmbCols = kEmbLanes * 8;

// A token's place: its stable rank when the ids are sorted (smaller ids first, then earlier tokens), its place in the run of
// equal ids and the run's length. places[rank] = {token, place in the run, length of the run, id (-1: not one of a table)}.
// A warp per token compares its id with all others (T^2 comparisons in all). The counters of embedRowsKernel are zeroed on the way.
__global__ void __launch_bounds__(256) embedOrderKernel(const long* ids, int4* places, unsigned* counters, int nCounters, int T) {
  releaseNext();
  awaitPrevious();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < nCounters; i += gridDim.x * 256) counters[i] = 0u;
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  // The low words: valid ids have no others. Behind awaitPrevious(), as loadOrdered is, and a plain dereference costs more here too
  // (16384 ids: 97.3 us with their sums, 87.2 with this and with __ldg).
  auto idOf = [&](int i) {
    int low;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(low) : "l"(ids + i));
    return low;
  };
  const int id = idOf(t), strip = t & ~31;
  int rank = 0, earlier = 0, equal = 0;
#pragma unroll 4
  for (int i = lane; i < strip; i += 32) {   // tokens before the strip of t: an equal id comes first
    const int o = idOf(i);
    rank += o <= id ? 1 : 0;
    earlier += o == id ? 1 : 0;
  }
  if (strip + lane < T) {
    const int o = idOf(strip + lane);
    const bool e = o == id, before = e && strip + lane < t;
    rank += o < id || before ? 1 : 0;
    earlier += before ? 1 : 0;
    equal += e && !before ? 1 : 0;
  }
#pragma unroll 4
  for (int i = strip + 32 + lane; i < T; i += 32) {
    const int o = idOf(i);
    rank += o < id ? 1 : 0;
    equal += o == id ? 1 : 0;
  }
  equal += earlier;
  for (int s = 16; s > 0; s >>= 1) {
    rank += __shfl_xor_sync(0xffffffffu, rank, s);
    equal += __shfl_xor_sync(0xffffffffu, equal, s);
    earlier += __shfl_xor_sync(0xffffffffu, earlier, s);
  }
  if (lane == 0) places[rank] = make_int4(t, earlier, equal, (ids[t] >> 31) == 0 ? id : -1);
}

// grad[id] += sum over the tokens with that id of dy[token]. A run of equal ids is cut into pieces of kEmbPiece tokens; one CTA
// takes a piece (it starts at the piece's first place; the CTAs of the other places leave at once) and a block of 1024 columns.
// Its two halves take every other token of the piece, four rows in flight each, and meet in shared memory. A run of one piece
// goes straight to the table. The pieces of a longer one (padding, a token that fills the batch) leave their sums in `parts`, and
// the CTA that finds all of them there, whichever it is, adds them up in order: the result does not depend on scheduling.
// One CTA for a whole run summed 16384 equal ids in 1.5 ms (512 wide) and 2.4 ms (4096 wide), in pieces they take 45 and 97 us.
// 40 registers keep six CTAs on an SM, which is what ids that differ need (50304 x 4096, 4096 of them: 38 us, 50 with 51 registers).
// No dependent launch: most CTAs leave after one look at their place, and the two instructions of such a launch cost each of them more
// than the early start gains (4096 x 4096, equal ids: 39.0 us with them, 33.2 without; 512 x 512: 4.9 and 4.8).
//
// parts: a row per window of kEmbPiece places and kind of piece (first of its run or not). Two pieces of one kind, both of long
// runs, never start in the same window: later pieces of a run are kEmbPiece apart, a run's later piece and the next run's lie
// further apart, and so do the first pieces of two long runs.
constexpr int kEmbPiece = 64;
__global__ void __launch_bounds__(kEmbThreads, 6) embedRowsKernel(const bf16* dy, const int4* places, float* parts,
                                                               unsigned* counters, float* grad, int T, int H, long vocab) {
  __shared__ float other[kEmbLanes][9];
  __shared__ bool last;
  const int i0 = blockIdx.x;
  const int4 me = places[i0];
  if (me.y % kEmbPiece != 0) return;
  const long id = me.w;
  if (id < 0 || id >= vocab) return;   // the lookup of the forward pass has refused such ids
  const int half = threadIdx.x / kEmbLanes, lane = threadIdx.x % kEmbLanes;
  const int col = blockIdx.y * kEmbCols + lane * 8;
  const int end = i0 + min(kEmbPiece, me.z - me.y);   // at most T
  float acc[8];
  auto clear = [&]() {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  };
  // the other half's sums, then this half's own: the sum in acc of the first half
  auto meet = [&]() {
    if (half == 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) other[lane][j] = acc[j];
    }
    __syncthreads();
    if (half == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += other[lane][j];
    }
  };
  float* g = grad + id * H + col;
  const bool whole = me.z <= kEmbPiece, writes = half == 0 && col < H;
  auto addToTable = [&]() {
    float v[8];
    Vec8<float>::load(g, 8, true, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += acc[j];
    Vec8<float>::store(g, 8, true, v);
  };
  clear();
  if (col < H) {
    for (int i = i0 + half; i < end; i += 8) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = i + 2 * u;
        raw[u] = k < end ? loadOrdered(dy + (long)places[k].x * H + col) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i + 2 * u >= end) continue;
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * j] += __uint_as_float(w[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
        }
      }
    }
  }
  meet();
  if (whole) {
    if (writes) addToTable();
    return;
  }
  const int first = i0 - me.y, pieces = (me.z + kEmbPiece - 1) / kEmbPiece;
  auto part = [&](int p) { return parts + (2L * ((first + p * kEmbPiece) / kEmbPiece) + (p > 0 ? 1 : 0)) * H + col; };
  if (writes) Vec8<float>::store(part(me.y / kEmbPiece), 8, true, acc);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicAdd(counters + (long)blockIdx.y * ((T + kEmbPiece - 1) / kEmbPiece) + first / kEmbPiece, 1u) == (unsigned)pieces - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  clear();
  if (col < H) {
    for (int p = half; p < pieces; p += 4) {   // two rows in flight: more would cost the rest of the kernel registers
      float4 a[2], b[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (p + 2 * u >= pieces) continue;
        a[u] = __ldcg(reinterpret_cast<const float4*>(part(p + 2 * u)));       // other CTAs wrote them
        b[u] = __ldcg(reinterpret_cast<const float4*>(part(p + 2 * u)) + 1);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (p + 2 * u >= pieces) continue;
        acc[0] += a[u].x; acc[1] += a[u].y; acc[2] += a[u].z; acc[3] += a[u].w;
        acc[4] += b[u].x; acc[5] += b[u].y; acc[6] += b[u].z; acc[7] += b[u].w;
      }
    }
  }
  meet();
  if (writes) addToTable();
}

// grad[s] += sum over the batch of dy[b][s], for the `seq` positions of dy [batch][seq][H]
__global__ void __launch_bounds__(256) embedPositionsKernel(const bf16* dy, float* grad, int batch, long n) {
  releaseNext();
  awaitPrevious();
  const long i = ((long)blockIdx.x * 256 + threadIdx.x) * 8;   // n = seq * H, a multiple of 8
  if (i >= n) return;
  float acc[8], v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  for (int b = 0; b < batch; ++b) {
    Vec8<bf16>::load(dy + (long)b * n + i, 8, true, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += v[j];
  }
  Vec8<float>::load(grad + i, 8, true, v);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] += acc[j];
  Vec8<float>::store(grad + i, 8, true, v);
}

}  // namespace coccl

using namespace coccl;

// Scratch: places, then the parts of long runs, then a counter per window and block of columns.
struct EmbedScratch {
  long windows, colBlocks, partsAt, countersAt, bytes;
  EmbedScratch(int T, int H) : windows(((long)T + kEmbPiece - 1) / kEmbPiece), colBlocks((H + kEmbCols - 1) / kEmbCols) {
    partsAt = 16L * T;
    countersAt = partsAt + (T > kEmbPiece ? 2 * windows * H * 4 : 0);   // no run is longer than a piece
    bytes = countersAt + windows * colBlocks * 4;
  }
};
extern "C" long cocclkEmbedScratchBytes(int T, int H) { return T > 0 && H > 0 ? EmbedScratch(T, H).bytes : 0; }

extern "C" int cocclkEmbedBwd(const void* dy, const long* ids, void* scratch, float* grad, int T, int H, long vocab, cudaStream_t s) {
  if (T <= 0 || H <= 0 || H % 8) return -1;
  const EmbedScratch L(T, H);
  char* b = (char*)scratch;
  int4* places = (int4*)b;
  unsigned* counters = (unsigned*)(b + L.countersAt);
  launchAfter(embedOrderKernel, (T + 7) / 8, 256, 0, s, ids, places, counters, (int)(L.windows * L.colBlocks), T);
  embedRowsKernel<<<dim3((unsigned)T, (unsigned)L.colBlocks), kEmbThreads, 0, s>>>((const bf16*)dy, places, (float*)(b + L.partsAt), counters,
                                                                            grad, T, H, vocab);
  cocclkCountLaunches(2);
  return (int)cudaGetLastError();
}

extern "C" int cocclkEmbedPositionsBwd(const void* dy, float* grad, int batch, int seq, int H, cudaStream_t s) {
  if (batch <= 0 || seq <= 0 || H <= 0 || H % 8) return -1;
  const long n = (long)seq * H;
  launchAfter(embedPositionsKernel, (unsigned)((n / 8 + 255) / 256), 256, 0, s, (const bf16*)dy, grad, batch, n);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}
