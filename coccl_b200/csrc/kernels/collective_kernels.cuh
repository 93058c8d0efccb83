// Fused compressed collectives: ONE persistent launch per collective that
// encodes, moves the encoded bytes with direct stores into the peers' receive
// slots over NVLink, signals per-slice flags, and decodes (with reduction and,
// for the two-shot all-reduce, re-encoding) on the receiving side.
//
// What the reference does with host-side stage lists — Compress -> AllToAll ->
// DecompressReduce for ReduceScatter one-shot
// (extensions/primitives/coccl_reducescatter.cc:12-29), Compress -> AllGather
// -> Decompress (coccl_allgather.cc:12-22), Compress -> AllToAll -> Decompress
// (coccl_alltoall.cc:12-21), Compress -> AllGather -> DecompressReduce for
// AllReduce one-shot and Compress -> A2A -> DecompReduceComp -> AllGather ->
// Decompress for two-shot (coccl_allreduce.cc:12-53) — is here three device
// phases of one kernel; `pipeline.depth` becomes the slice granularity.
//
// Work decomposition: a chunk (the elements one rank owns / sends to one peer)
// is cut into slices of `sliceTiles` tiles of 8192 elements. One CTA owns one
// (peer, slice) item at a time; finishing it publishes flag[src][slice]=epoch
// on the receiver with release semantics. Encode items never wait, so every
// wait in a later phase depends only on work that cannot itself block.
// All waits are bounded by a globaltimer deadline and report through the
// status word instead of trapping.
//
// `rankBase`/blockIdx.y let one cooperative launch play all ranks on a single
// GPU (every pointer then refers to local memory); production launches use
// gridDim.y == 1 and peer-mapped pointers.
#pragma once
#include "codecs.cuh"
#include "tile_io.cuh"

namespace coccl {

enum CollOp : int {
  kOpReduceScatter = 0, kOpAllGather = 1, kOpAllToAll = 2, kOpAllReduceOneShot = 3, kOpAllReduceTwoShot = 4,
  // All-gather of DELTAS (the reference's subAdd AllGather, sdp4bit/quantization/sub_quantize.cu:176-262 and
  // dequantize_add.cu:145-275): `out` holds the result of the previous call on every rank, a rank encodes
  // in - out[own chunk] and every rank adds the decoded deltas to all chunks of `out`. Every rank performs the same
  // arithmetic on the same bytes, so the copies of `out` stay identical. The first call must fill `out` exactly.
  kOpAllGatherDelta = 5
};

constexpr int kMaxSlices = 4096;  // per source rank and region

struct CollArgs {
  int op;
  int nRanks;
  int rankBase;
  int dtype;
  long count;            // elements per chunk (AR one-shot: the whole vector; AR two-shot: count/nRanks)
  int sliceTiles;
  unsigned int epoch;
  unsigned long long timeoutNs;
  CodecCfg codec;
  long slotBytes;        // distance between per-source slots inside a region
  long regionBOffset;    // byte offset of region B (two-shot all-reduce)
  const void* in[kMaxRanks];
  void* out[kMaxRanks];
  uint8_t* ws[kMaxRanks];          // workspace of every rank as mapped here (parity offset applied)
  unsigned int* flags[kMaxRanks];  // [2 regions][kMaxRanks sources][kMaxSlices]
  StatusWord* status[kMaxRanks];
  unsigned long long* trace[kMaxRanks];  // optional phase timestamps, 4 per CTA
};

constexpr int kTraceMaxCtas = 2048;
__device__ __forceinline__ void tracePhase(unsigned long long* tr, int phase) {
  if (tr != nullptr && threadIdx.x == 0 && blockIdx.x < kTraceMaxCtas) tr[blockIdx.x * 4 + phase] = globalTimerNs();
}

__device__ __forceinline__ unsigned int* flagPtr(unsigned int* base, int region, int src, int slice) {
  return base + ((long)region * kMaxRanks + src) * kMaxSlices + slice;
}

// Stages of raw values: for codecs that are bound by instructions the next tile's are on their way to shared memory while this one
// is encoded, except for fp32, where the loads alone take 0.95 of the copy rate with four CTAs an SM and a second stage leaves
// room for three (4 bits, groups of 128, 8 x 8 Mi: fp32 48.1 us with one stage, 52.9 with two; bf16 38.5 and 35.6; 8 bits in
// groups of 8, bound by stores: bf16 63.7 and 84.3; 4 bits in groups of 8: 53.9 and 71.7).
template <typename T, class Codec>
constexpr int kEncodeStages = sizeof(T) == 2 && Codec::kEncodeAhead ? 2 : 1;

// Encode the tiles [t0, t1) of one source chunk and store the result into the nDst chunk buffers dst(0), dst(1), ... With DELTA
// what is sent is the change since the previous result, `prev`.
template <typename T, class Codec, bool DELTA, class Dst>
__device__ __forceinline__ void encodeTiles(const T* src, const ChunkLayout& L, const CodecCfg& c, long t0, long t1,
                                            int nDst, Dst dst, TileStage<T>* stage, float* sm,
                                            uint64_t rngBase, const T* prev) {
  constexpr int S = DELTA ? 1 : kEncodeStages<T, Codec>;
  auto start = [&](const T* chunk, long t, int s) {
    const long e0 = t * kTileElems, left = L.count - e0;
    if (t < t1) TileIO<T, false>::template bring<S == 2>(chunk + e0, left, e0 == 0, TileIO<T, false>::fast(chunk + e0, left), stage[s]);
    if (S == 2) commitCopies();
  };
  auto take = [&](const T* chunk, long t, int s, float (&v)[32]) {
    const long e0 = t * kTileElems, left = L.count - e0;
    TileIO<T, false>::take(chunk + e0, left, e0 == 0, TileIO<T, false>::fast(chunk + e0, left), stage[s], v);
  };
  int s = 0;
  __syncwarp();   // the stages are not in use any more
  if (S == 2) start(src, t0, 0);
  for (long t = t0; t < t1; ++t, s ^= S - 1) {
    const long e = t * kTileElems + (long)threadIdx.x * kElemsPerThread;
    float v[32];
    __syncwarp();
    start(src, S == 2 ? t + 1 : t, S == 2 ? s ^ 1 : 0);
    if (S == 2) waitCopies<1>();
    take(src, t, s, v);
    if constexpr (DELTA) {
      float pv[32];
      __syncwarp();
      start(prev, t, 0);
      take(prev, t, 0, pv);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] -= pv[i];
    }
    const typename Codec::Enc enc = Codec::encode(v, c, true, sm, rngBase + (uint64_t)e, TileIO<T, false>::window(stage[s]));
    if (!COCCL_CHUNK_RANGE_OK(Codec, L, c, e, 1)) continue;
    for (int d = 0; d < nDst; ++d) Codec::store(enc, dst(d), L, c, e);
  }
}

// A CTA takes its items in batches: one barrier and one system-wide fence publish a whole batch, one barrier follows the
// waits for a whole batch, and inside a batch the warps run free. An item on its own costs about 3 us in the two (8 ranks
// emulated, 16 Mi bf16, two-shot: one tile an item 738 us, six tiles 307 us for the same work; batched 381 and 293 us), so
// batches grow with the items a CTA has; one with less than four keeps single items, because a batch delays the receivers.
// That is the case of ranks that share a GPU. A rank alone on its GPU has about one item a CTA (the slices are cut so) until a
// slice has its most tiles: batches then need some 170 million elements a rank, or a limit on the CTAs.
constexpr int kMaxBatch = 4;
__device__ __forceinline__ int batchOf(int items) {
  const int each = (items + (int)gridDim.x - 1) / (int)gridDim.x;
  return each >= 8 ? kMaxBatch : (each >= 4 ? 2 : 1);
}

// Publish n flags (n <= 32) after every thread of the CTA has finished its stores; addr(i) is the i-th flag.
template <class Addr>
__device__ __forceinline__ void publish(int n, Addr addr, unsigned int epoch) {
  __syncthreads();
  if (threadIdx.x < n) {
    __threadfence_system();
    stReleaseSys(addr(threadIdx.x), epoch);
  }
}

// Wait for n flags (n <= 32). Returns false for the whole CTA on timeout; item(i) names the i-th flag in the report.
template <class Addr, class Item>
__device__ __forceinline__ bool waitAll(int n, Addr addr, Item item, unsigned int epoch, unsigned long long timeoutNs,
                                        StatusWord* st, int phase, bool skip) {
  bool ok = true;
  if (!skip && threadIdx.x < n) {
    ok = waitFlag(addr(threadIdx.x), epoch, timeoutNs);
    if (!ok) reportTimeout(st, phase, item(threadIdx.x).x, item(threadIdx.x).y);
  }
  return __syncthreads_and(ok ? 1 : 0) != 0;
}
static_assert(kMaxBatch * kMaxRanks <= 32, "a batch's flags are handled by one warp");

// Decode the tiles [t0, t1) of one encoded chunk into dst. With ADD they are added to what dst holds.
template <typename T, class Codec, bool ADD>
__device__ __forceinline__ void decodeTiles(const uint8_t* enc, T* dst, const ChunkLayout& L, const CodecCfg& c, long t0, long t1,
                                            bool aligned, TileStage<T>& stage, float* sm) {
  auto put = [&](long t, float (&acc)[32]) {
    const long e0 = t * kTileElems, left = L.count - e0;
    const bool fast = TileIO<T, false>::fast(dst + e0, left);
    Codec::finish(acc, c, TileIO<T, false>::window(stage));
    if constexpr (ADD) {
      float pv[32];
      TileIO<T, false>::load(dst, L.count, e0, fast, stage, pv);
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] += pv[i];
    }
    TileIO<T, false>::storeTile(dst + e0, left, fast, stage, acc);
  };
  const long lane = (long)threadIdx.x * kElemsPerThread;
  if constexpr (HasDirectSums<Codec>::value) {
    typename Codec::Ahead r = Codec::ahead(enc, L, c, t0 * kTileElems + lane);
    for (long t = t0; t < t1; ++t) {
      float acc[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0.f;
      Codec::addAhead(r, c, Codec::finishScale(c), acc);
      if (t + 1 < t1) r = Codec::ahead(enc, L, c, (t + 1) * kTileElems + lane);
      put(t, acc);
    }
  } else {
    for (long t = t0; t < t1; ++t) {
      float acc[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0.f;
      decodeSum<Codec>(enc, 0, 1, L, c, t * kTileElems + lane, Codec::finishScale(c), acc, sm, aligned, true);
      put(t, acc);
    }
  }
}

// What a collective does after its encoded chunks have arrived; one kernel each, so that none carries another's code and registers.
enum CollForm : int { kFormGather = 0, kFormGatherDelta = 1, kFormReduce = 2, kFormTwoShot = 3 };
inline CollForm collForm(int op) {
  switch (op) {
    case kOpReduceScatter: case kOpAllReduceOneShot: return kFormReduce;
    case kOpAllReduceTwoShot: return kFormTwoShot;
    case kOpAllGatherDelta: return kFormGatherDelta;
    default: return kFormGather;
  }
}

// The delta form holds a second run of values: with a codec that needs most of the registers itself, one CTA an SM fewer (TACO, 8 x 1 Mi
// fp32: 215 us with three, 164 with two).
template <class Codec, int FORM>
constexpr int kFusedBlocks = FORM == kFormGatherDelta && Codec::kExchanges ? 2 : Codec::kMinBlocks;
template <typename T, class Codec, int FORM>
__global__ void __launch_bounds__(kTileThreads, kFusedBlocks<Codec, FORM>) fusedCollectiveKernel(const __grid_constant__ CollArgs a) {
  __shared__ TileStage<T> stage[FORM == kFormGatherDelta ? 1 : kEncodeStages<T, Codec>];
  __shared__ __align__(16) float sm[Codec::kSmemFloats];
  Codec::initShared(sm);
  __syncthreads();

  const int N = a.nRanks;
  const int rank = a.rankBase + blockIdx.y;
  const CodecCfg c = a.codec;
  const ChunkLayout L = makeChunkLayout(c, a.count, 16);
  const long tiles = (a.count + kTileElems - 1) / kTileElems;
  const int slices = (int)((tiles + a.sliceTiles - 1) / a.sliceTiles);   // at most kMaxSlices
  const T* in = reinterpret_cast<const T*>(a.in[rank]);
  T* out = reinterpret_cast<T*>(a.out[rank]);
  uint8_t* myWs = a.ws[rank];
  unsigned int* myFlags = a.flags[rank];
  StatusWord* st = a.status[rank];
  unsigned long long* tr = a.trace[rank];
  tracePhase(tr, 0);
  // The slot geometry comes from the host: a chunk that does not fit its slot, or a second region that overlaps the
  // first, would make ranks write over each other's data. Checked in every build, before anything is touched.
  if (L.stride > a.slotBytes || (a.op == kOpAllReduceTwoShot && a.regionBOffset < (long)N * a.slotBytes)) {
    if (threadIdx.x == 0) reportTimeout(st, 0xB, rank, 0);
    return;
  }
  bool failed = false;
  const bool perPeer = (a.op == kOpReduceScatter || a.op == kOpAllToAll || a.op == kOpAllReduceTwoShot);

  // the d-th peer of this rank (d < N; every rank starts at its neighbour), and the one an item in peer order refers to
  auto peerAt = [&](int d) { const int p = rank + 1 + d; return p >= N ? p - N : p; };
  auto peer = [&](int item) { return peerAt(item % N); };
  // ---------------- phase 1: encode + push ----------------
  {
    const int items = perPeer ? slices * N : slices;
    const int nDst = perPeer ? 1 : N, B = batchOf(items);
    for (int it0 = blockIdx.x; it0 < items; it0 += B * (int)gridDim.x) {
      int nb = 0;
      for (; nb < B && it0 + nb * (int)gridDim.x < items; ++nb) {
        const int it = it0 + nb * (int)gridDim.x;
        const int s = perPeer ? it / N : it;
        const int p = peer(it);   // perPeer only
        const long t0 = (long)s * a.sliceTiles;
        const long t1 = min(tiles, t0 + (long)a.sliceTiles);
        encodeTiles<T, Codec, FORM == kFormGatherDelta>(perPeer ? in + (long)p * a.count : in, L, c, t0, t1, nDst,
                              [&](int d) { return a.ws[perPeer ? p : peerAt(d)] + (long)rank * a.slotBytes; }, stage, sm,
                              (uint64_t)(perPeer ? rank * N + p : rank) << 40,
                              out + (long)rank * a.count);
      }
      publish(nb * nDst, [&](int i) {
        const int it = it0 + i / nDst * (int)gridDim.x;
        return flagPtr(a.flags[perPeer ? peer(it) : peerAt(i % nDst)], 0, rank, perPeer ? it / N : it);
      }, a.epoch);
    }
  }

  tracePhase(tr, 1);
  // ---------------- phase 2: wait + decode ----------------
  constexpr bool reduce = FORM == kFormReduce || FORM == kFormTwoShot;
  // the slots are laid out on 16 bytes unless a caller's geometry says otherwise
  const bool aligned = ((reinterpret_cast<uintptr_t>(myWs) | (uintptr_t)a.slotBytes | (uintptr_t)a.regionBOffset) & 15u) == 0;
  {
    const int items = reduce ? slices : slices * N;
    const int nq = reduce ? N : 1, B = batchOf(items);
    for (int it0 = blockIdx.x; it0 < items; it0 += B * (int)gridDim.x) {
      int nb = 1;
      while (nb < B && it0 + nb * (int)gridDim.x < items) ++nb;
      // {source, slice} of flag i of the batch
      auto from = [&](int i) {
        const int it = it0 + i / nq * (int)gridDim.x;
        return make_int2(reduce ? i % nq : peer(it), reduce ? it : it / N);
      };
      if (!waitAll(nb * nq, [&](int i) { return flagPtr(myFlags, 0, from(i).x, from(i).y); }, from, a.epoch, a.timeoutNs, st, 2,
                   failed)) failed = true;
      for (int j = 0; j < nb; ++j) {
        const int2 qs = from(j * nq);
        const int q0 = qs.x;
        const long t0 = (long)qs.y * a.sliceTiles;
        const long t1 = min(tiles, t0 + (long)a.sliceTiles);
        if constexpr (!reduce) {
          decodeTiles<T, Codec, FORM == kFormGatherDelta>(myWs + (long)q0 * a.slotBytes, out + (long)q0 * a.count, L, c, t0, t1, aligned,
                                                          stage[0], sm);
          continue;
        }
        for (long t = t0; t < t1; ++t) {
          const long e0 = t * kTileElems, left = L.count - e0;
          const long e = e0 + (long)threadIdx.x * kElemsPerThread;
          float acc[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = 0.f;
          decodeSum<Codec>(myWs, a.slotBytes, N, L, c, e, FORM == kFormTwoShot ? 1.f : Codec::finishScale(c), acc, sm, aligned,
                           FORM != kFormTwoShot);
          if constexpr (FORM == kFormTwoShot) {
            // stay in the rotated domain: the sum of rotated values is the rotation of the sum
            const typename Codec::Enc enc = Codec::encode(acc, c, false, sm, ((uint64_t)(0x80 + rank) << 40) + (uint64_t)e);
            if (COCCL_CHUNK_RANGE_OK(Codec, L, c, e, 3))
              for (int d = 0; d < N; ++d) Codec::store(enc, a.ws[peerAt(d)] + a.regionBOffset + (long)rank * a.slotBytes, L, c, e);
          } else {
            Codec::finish(acc, c, TileIO<T, false>::window(stage[0]));
            TileIO<T, false>::storeTile(out + e0, left, TileIO<T, false>::fast(out + e0, left), stage[0], acc);
          }
        }
      }
      if (FORM == kFormTwoShot)
        publish(nb * N, [&](int i) { return flagPtr(a.flags[peerAt(i % N)], 1, rank, it0 + i / N * (int)gridDim.x); }, a.epoch);
    }
  }

  tracePhase(tr, 2);
  // ---------------- phase 3 (two-shot all-reduce): gather reduced chunks ----------------
  if constexpr (FORM == kFormTwoShot) {
    const int items = slices * N;
    const int B = batchOf(items);
    for (int it0 = blockIdx.x; it0 < items; it0 += B * (int)gridDim.x) {
      int nb = 1;
      while (nb < B && it0 + nb * (int)gridDim.x < items) ++nb;
      auto from = [&](int i) {
        const int it = it0 + i * (int)gridDim.x;
        return make_int2(peer(it), it / N);
      };
      if (!waitAll(nb, [&](int i) { return flagPtr(myFlags, 1, from(i).x, from(i).y); }, from, a.epoch, a.timeoutNs, st, 3,
                   failed)) failed = true;
      for (int j = 0; j < nb; ++j) {
        const int2 qs = from(j);
        const long t0 = (long)qs.y * a.sliceTiles;
        const long t1 = min(tiles, t0 + (long)a.sliceTiles);
        decodeTiles<T, Codec, false>(myWs + a.regionBOffset + (long)qs.x * a.slotBytes, out + (long)qs.x * a.count, L, c, t0, t1, aligned,
                                     stage[0], sm);
      }
    }
  }
  tracePhase(tr, 3);
}

// ---------------------------------------------------------------------------
// Standalone codec kernels (plugin path, tests, autotune profiling).
// ---------------------------------------------------------------------------
struct CodecArgs {
  const void* in;      // raw input (encode) or encoded input (decode)
  void* out;           // encoded output (encode / drc) or raw output (decode)
  long count;          // elements per chunk
  long chunks;         // encode: input chunks; decode: OUTPUT chunks
  long reduce;         // decode / drc: encoded copies summed per output chunk (>=1)
  long rawPitch;       // elements between consecutive raw chunks
  long encStrideIn;    // bytes between encoded input chunks
  long encStrideOut;   // bytes between encoded output chunks
  int dtype;
  CodecCfg codec;
  CodecCfg codecOut;   // drc: codec of the re-encoded output (same family)
};

// These kernels are bound by instruction issue, then by the loads in flight. With packed fp32 arithmetic, digits dequantised
// where they stand, no divisions and four copies in flight (8 chunks, 4-bit groups of 128, rotated): encode of 256 MiB fp32
// with stochastic rounding 68.6 -> 54.6 us, now 52.3 (290 MB: 44 us to copy), decode + sum 30.6 -> 26.4 us, now 16.7 (codecs.cuh, sums);
// chunks of 5,000,003 bf16 elements (misaligned: see tile_io.cuh) 74.4 -> 30.0 us, now 29.0.
//
// whether every encoded input chunk starts on 16 bytes
__device__ __forceinline__ bool encodedAligned(const CodecArgs& a) {
  return ((reinterpret_cast<uintptr_t>(a.in) | (uintptr_t)a.encStrideIn) & 15u) == 0;
}

// The tiles of all chunks in order, `gridDim.x` apart: (chunk, tile) and every address that belongs to it advance by fixed
// steps with one carry, because a 64-bit division per tile and thread was a fifth of the instructions of these kernels.
struct TileWalk {
  unsigned tiles, t, stepT;   // 2^32 tiles would be 2^45 elements
  long chunks, ch, stepCh;
  bool carried;               // whether the last step began another chunk
  __device__ __forceinline__ TileWalk(long count, long chunks_) : chunks(chunks_), carried(false) {
    tiles = (unsigned)((count + kTileElems - 1) / kTileElems);
    ch = blockIdx.x / tiles; t = blockIdx.x % tiles; stepCh = gridDim.x / tiles; stepT = gridDim.x % tiles;
  }
  __device__ __forceinline__ bool more() const { return ch < chunks; }
  __device__ __forceinline__ void next() {
    const unsigned rest = tiles - t;   // the sum itself may pass 2^32
    carried = stepT >= rest;
    ch += stepCh + (carried ? 1 : 0);
    t = carried ? stepT - rest : t + stepT;
  }
};
// An address that grows by `pitch` with the chunk and by `tileElems` with the tile.
template <class P>
struct Along {
  P* p;
  long step, carry;
  __device__ __forceinline__ Along(P* base, long pitch, long tileElems, const TileWalk& w)
      : p(base + w.ch * pitch + w.t * tileElems), step(w.stepCh * pitch + w.stepT * tileElems), carry(pitch - (long)w.tiles * tileElems) {}
  __device__ __forceinline__ void next(const TileWalk& w) { p += w.carried ? step + carry : step; }
};

template <typename T, class Codec>
__global__ void __launch_bounds__(kTileThreads, Codec::kEncodeBlocks) encodeKernel(const CodecArgs a) {
  constexpr int S = kEncodeStages<T, Codec>;
  __shared__ TileStage<T> stage[S];
  __shared__ __align__(16) float sm[Codec::kSmemFloats];
  Codec::initShared(sm);
  __syncthreads();
  const ChunkLayout L = makeChunkLayout(a.codec, a.count, 4);
  TileWalk w(a.count, a.chunks);
  Along<const T> src(reinterpret_cast<const T*>(a.in), a.rawPitch, kTileElems, w);
  Along<uint8_t> dst(reinterpret_cast<uint8_t*>(a.out), a.encStrideOut, 0, w);
  auto start = [&](int s) {
    const long left = L.count - (long)w.t * kTileElems;
    if (w.more()) TileIO<T>::template bring<S == 2>(src.p, left, w.t == 0, TileIO<T>::fast(src.p, left), stage[s]);
    if (S == 2) commitCopies();
  };
  if (S == 2) start(0);
  for (int s = 0; w.more(); s ^= S - 1) {
    const T* tile = src.p;
    uint8_t* out = dst.p;
    const long e0 = (long)w.t * kTileElems, left = L.count - e0, ch = w.ch;
    __syncwarp();   // the stage that is filled next has been read
    if (S == 1) start(0);
    w.next();
    src.next(w);
    dst.next(w);
    if (S == 2) start(s ^ 1);
    if (S == 2) waitCopies<1>();
    float v[32];
    TileIO<T>::take(tile, left, e0 == 0, TileIO<T>::fast(tile, left), stage[s], v);
    const long e = e0 + (long)threadIdx.x * kElemsPerThread;
    const typename Codec::Enc enc = Codec::encode(v, a.codec, true, sm, ((uint64_t)ch << 40) + (uint64_t)e, TileIO<T>::window(stage[s]));
    if (COCCL_CHUNK_RANGE_OK(Codec, L, a.codec, e, 1)) Codec::store(enc, out, L, a.codec, e);
  }
}

// out chunk j = decode(in chunk j): one copy (all-gather, all-to-all), for codecs with direct sums. The next tile's words are loaded
// before this one is transformed and stored (4 bits, groups of 128, rotated: 8 x 8 Mi bf16 41.5 -> 33.6 us, 8 x 5,000,003 35.1 ->
// 24.9 us, of which tile_io.cuh has the greater part). A kernel of its own: in one with the sums' code both spilled (TACO fp32 88 bytes, asymmetric 4 bits 28).
template <typename T, class Codec>
__global__ void __launch_bounds__(kTileThreads, Codec::kDecodeBlocks) decodeKernel(const CodecArgs a) {
  __shared__ TileStage<T> stage;
  __shared__ __align__(16) float sm[Codec::kSmemFloats];
  Codec::initShared(sm);
  __syncthreads();
  const ChunkLayout L = makeChunkLayout(a.codec, a.count, 4);
  TileWalk w(a.count, a.chunks);
  Along<const uint8_t> src(reinterpret_cast<const uint8_t*>(a.in), a.encStrideIn, 0, w);
  Along<T> dst(reinterpret_cast<T*>(a.out), a.rawPitch, kTileElems, w);
  auto fetch = [&] { return Codec::ahead(src.p, L, a.codec, (long)w.t * kTileElems + (long)threadIdx.x * kElemsPerThread); };
  typename Codec::Ahead r;
  if (w.more()) r = fetch();
  while (w.more()) {
    T* tile = dst.p;
    const long left = L.count - (long)w.t * kTileElems;
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    Codec::addAhead(r, a.codec, Codec::finishScale(a.codec), acc);
    w.next();
    src.next(w);
    dst.next(w);
    if (w.more()) r = fetch();
    Codec::finish(acc, a.codec, TileIO<T>::window(stage));
    TileIO<T>::storeTile(tile, left, TileIO<T>::fast(tile, left), stage, acc);
  }
}

// out chunk j = sum_{i<reduce} decode(in chunk i*chunks + j)
template <typename T, class Codec, int BLOCKS>
__global__ void __launch_bounds__(kTileThreads, BLOCKS) decodeReduceKernel(const CodecArgs a) {
  __shared__ TileStage<T> stage;
  __shared__ __align__(16) float sm[Codec::kSmemFloats];
  Codec::initShared(sm);
  __syncthreads();
  const ChunkLayout L = makeChunkLayout(a.codec, a.count, 4);
  TileWalk w(a.count, a.chunks);
  Along<const uint8_t> src(reinterpret_cast<const uint8_t*>(a.in), a.encStrideIn, 0, w);
  Along<T> dst(reinterpret_cast<T*>(a.out), a.rawPitch, kTileElems, w);
  for (; w.more(); w.next(), src.next(w), dst.next(w)) {
    const long e0 = (long)w.t * kTileElems, left = L.count - e0;
    const long e = e0 + (long)threadIdx.x * kElemsPerThread;
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    decodeSum<Codec>(src.p, a.chunks * a.encStrideIn, (int)a.reduce, L, a.codec, e, Codec::finishScale(a.codec), acc, sm, encodedAligned(a), true);
    Codec::finish(acc, a.codec, TileIO<T>::window(stage));
    TileIO<T>::storeTile(dst.p, left, TileIO<T>::fast(dst.p, left), stage, acc);
  }
}

// decode + reduce + re-encode without leaving registers
// (reference kernel: sdp4bit/quantization/dequant_reduce_quant.cu:14-179).
template <class Codec>
__global__ void __launch_bounds__(kTileThreads, Codec::kMinBlocks) decodeReduceEncodeKernel(const CodecArgs a) {
  __shared__ __align__(16) float sm[Codec::kSmemFloats];
  Codec::initShared(sm);
  __syncthreads();
  const ChunkLayout L = makeChunkLayout(a.codec, a.count, 4);
  TileWalk w(a.count, a.chunks);
  Along<const uint8_t> src(reinterpret_cast<const uint8_t*>(a.in), a.encStrideIn, 0, w);
  Along<uint8_t> dst(reinterpret_cast<uint8_t*>(a.out), a.encStrideOut, 0, w);
  for (; w.more(); w.next(), src.next(w), dst.next(w)) {
    const long e = (long)w.t * kTileElems + (long)threadIdx.x * kElemsPerThread;
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    decodeSum<Codec>(src.p, a.chunks * a.encStrideIn, (int)a.reduce, L, a.codec, e, 1.f, acc, sm, encodedAligned(a), false);
    const typename Codec::Enc o = Codec::encode(acc, a.codec, false, sm, ((uint64_t)(0x40 + w.ch) << 40) + (uint64_t)e);
    Codec::store(o, dst.p, L, a.codec, e);
  }
}

}  // namespace coccl
