// Raw-value tile I/O for the codec and collective kernels.
//
// A CTA of 256 threads owns a tile of 8192 consecutive elements; thread t owns the aligned run of 32
// elements [32 t, 32 t + 32) and keeps it in registers as fp32. A run is one Hadamard block and a whole
// number of quantisation groups (or a fraction 1/lpg of one), so the transform and most of the group
// statistics need no cross-lane traffic.
//
// Global memory is still accessed with fully coalesced 16-byte vectors: a warp reads its 1024 elements as
// consecutive uint4, parks them in a per-warp shared-memory window with the 16-byte chunks XOR-swizzled by
// the run index, and every thread then picks up its own run with conflict-free 16-byte shared loads (and the
// reverse for stores). A chunk that does not start on a 16-byte boundary (an odd number of 16-bit elements per rank) and
// the ragged last tile move the same way: the vectors that lie wholly inside the chunk travel as vectors, the up to seven
// elements at either end one by one. The window is staged as it lies in memory, and the distance between a vector and the
// elements of a run is a template parameter, chosen per tile by a switch that is uniform over the CTA: a value is then
// unpacked from (packed into) the word it lies in, at no cost beyond the one more vector that a run touches. Shifting words
// by a run-time distance took up to 80 instructions a run: 4 bits, groups of 128, rotated, 8 x 5,000,003 bf16: encode 29.5 ->
// 27.2 us, decode 35.4 -> 29.4 us (24.9 with the next tile loaded ahead: decodeKernel).
#pragma once
#include "common.cuh"
#include <type_traits>

namespace coccl {

// 16 bytes from global to shared memory without a register in between; bytes = 0 writes zeros and reads nothing.
__device__ __forceinline__ void copyAsync16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void commitCopies() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>   // waits for the calling thread's copies but those of the last PENDING groups
__device__ __forceinline__ void waitCopies() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Shared staging of one CTA: 8192 elements of T, and per warp the vector behind a misaligned window.
template <typename T>
struct TileStage {
  uint4 buf[kTileElems * sizeof(T) / 16];
  uint4 extra[kTileThreads / 32];
};

// 8 packed 16-bit values <-> 8 floats
template <typename T> struct Pack16;
template <> struct Pack16<__nv_bfloat16> {
  static __device__ __forceinline__ float low(uint32_t w) { return __uint_as_float(w << 16); }
  static __device__ __forceinline__ float high(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
  static __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ void unpack(const uint4& a, float* v) {
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  static __device__ __forceinline__ uint4 pack(const float* v) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <> struct Pack16<__half> {
  static __device__ __forceinline__ float low(uint32_t w) { return __low2float(*reinterpret_cast<const __half2*>(&w)); }
  static __device__ __forceinline__ float high(uint32_t w) { return __high2float(*reinterpret_cast<const __half2*>(&w)); }
  static __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ void unpack(const uint4& a, float* v) {
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ uint4 pack(const float* v) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};

// SHIFTS: every distance between a vector and the elements of a run as code of its own (stand-alone kernels). Without it one
// piece of code moves the words by a run-time distance: the fused collectives have many more instances, in which the other takes
// twice as long to compile as all the rest.
template <typename T, bool SHIFTS = true>
struct TileIO {
  static constexpr bool k32 = sizeof(T) == 4;
  static constexpr int kChunksPerRun = 32 * sizeof(T) / 16;       // 16-byte chunks in one run: 8 | 4
  static constexpr int kWarpChunks = 32 * kChunksPerRun;          // chunks in a warp's window: 256 | 128
  static constexpr int kRunsPerInstr = 32 / kChunksPerRun;        // runs covered by one warp-wide vector: 4 | 8

  // swizzled position of chunk c of run r inside the warp window
  static __device__ __forceinline__ int slot(int r, int c) {
    return k32 ? r * 8 + (c ^ (r & 7)) : r * 4 + (c ^ ((r >> 1) & 3));
  }

  // the warp's window: at least 2 KiB
  static __device__ __forceinline__ uint4* window(TileStage<T>& st) { return st.buf + (threadIdx.x >> 5) * kWarpChunks; }
  // position of vector vi (0 .. kWarpChunks) of the warp's window
  static __device__ __forceinline__ uint4* place(TileStage<T>& st, int warp, int vi) {
    return vi == kWarpChunks ? st.extra + warp : st.buf + warp * kWarpChunks + slot(vi / kChunksPerRun, vi % kChunksPerRun);
  }
  // f(integral_constant<M>) for the distance m between a vector and the window (a multiple of sizeof(T), uniform over the CTA)
  template <class F>
  static __device__ __forceinline__ void byShift(int m, F&& f) {
    switch (m / (int)sizeof(T)) {
      case 1: f(std::integral_constant<int, 1 * (int)sizeof(T)>{}); break;
      case 2: f(std::integral_constant<int, 2 * (int)sizeof(T)>{}); break;
      case 3: f(std::integral_constant<int, 3 * (int)sizeof(T)>{}); break;
      case 4: if constexpr (!k32) f(std::integral_constant<int, 8>{}); break;
      case 5: if constexpr (!k32) f(std::integral_constant<int, 10>{}); break;
      case 6: if constexpr (!k32) f(std::integral_constant<int, 12>{}); break;
      case 7: if constexpr (!k32) f(std::integral_constant<int, 14>{}); break;
      default: f(std::integral_constant<int, 0>{}); break;
    }
  }
  // w[i] <- bytes [4 i + shift, +4) of the words w (shift < 16, a multiple of sizeof(T), uniform over the CTA)
  template <int N>
  static __device__ __forceinline__ void shiftWords(uint32_t (&w)[N], int shift) {
    if (shift & 8) {
#pragma unroll
      for (int i = 0; i + 2 < N; ++i) w[i] = w[i + 2];
    }
    if (shift & 4) {
#pragma unroll
      for (int i = 0; i + 1 < N; ++i) w[i] = w[i + 1];
    }
    if (!k32 && (shift & 2)) {
#pragma unroll
      for (int i = 0; i + 1 < N; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], 16);
    }
  }
  // The run of lane `lane` from the window's stage, which it starts M (M < 0: m) bytes into.
  template <int M>
  static __device__ __forceinline__ void stagedRun(TileStage<T>& st, int warp, int lane, int m, float (&v)[32]) {
    constexpr int D = M < 0 ? 0 : M;
    uint4 p = *place(st, warp, lane * kChunksPerRun);
#pragma unroll
    for (int c = 0; c < kChunksPerRun; ++c) {
      uint4 y = make_uint4(0, 0, 0, 0);
      if (M != 0 || c + 1 < kChunksPerRun) y = *place(st, warp, lane * kChunksPerRun + c + 1);
      uint32_t w[8] = {p.x, p.y, p.z, p.w, y.x, y.y, y.z, y.w};
      if constexpr (M < 0) shiftWords(w, m);
      if constexpr (k32) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * c + i] = __uint_as_float(w[D / 4 + i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int h = D / 2 + i;
          v[8 * c + i] = (h & 1) ? Pack16<T>::high(w[h >> 1]) : Pack16<T>::low(w[h >> 1]);
        }
      }
      p = y;
    }
  }
  // The run of lane `lane` into the window's stage, M bytes on: a lane writes the kChunksPerRun vectors that end inside its run,
  // whose first words come from the lane before it; the last one also what reaches past the window.
  template <int M>
  static __device__ __forceinline__ void stageRun(const float (&v)[32], TileStage<T>& st, int warp, int lane) {
    constexpr int n = 4 * kChunksPerRun, k = M / 4;
    constexpr bool odd = M % 4 != 0;   // 16-bit elements: a word holds the elements (2 i - 1, 2 i) of the run, i = 0 .. n
    const float prev = odd ? __shfl_up_sync(0xffffffffu, v[31], 1) : 0.f;
    auto word = [&](int i) -> uint32_t {
      if constexpr (k32) return i < n ? __float_as_uint(v[i < n ? i : 0]) : 0u;
      else if constexpr (!odd) return i < n ? Pack16<T>::pack2(v[i < n ? 2 * i : 0], v[i < n ? 2 * i + 1 : 0]) : 0u;
      else return Pack16<T>::pack2(i == 0 ? prev : v[i == 0 ? 0 : 2 * i - 1], i < n ? v[i < n ? 2 * i : 0] : 0.f);
    };
    uint32_t before[k + 1];
#pragma unroll
    for (int i = 0; i < k; ++i) before[i] = __shfl_up_sync(0xffffffffu, word(n - k + i), 1);
    before[k] = 0;
    auto at = [&](int i) { return i < k ? before[i < k ? i : 0] : word(i < k ? 0 : i - k); };
#pragma unroll
    for (int c = 0; c < kChunksPerRun; ++c)
      *place(st, warp, lane * kChunksPerRun + c) = make_uint4(at(4 * c), at(4 * c + 1), at(4 * c + 2), at(4 * c + 3));
    auto past = [&](int i) { return i <= k ? word(i <= k ? n - k + i : 0) : 0u; };
    if (M != 0 && lane == 31) st.extra[warp] = make_uint4(past(0), past(1), past(2), past(3));
  }

  // A tile is given by its first element, the number of elements from there to the end of its chunk and whether it is the
  // chunk's first; `fast` (uniform over the CTA): whole and aligned. `m` bytes separate the 16-byte boundary before a warp's
  // window from its first element.
  struct Window {
    const char* at;        // the window's first element
    int m, nv, full, first;
    __device__ __forceinline__ Window(const T* tile, long left, bool head, int warp) {
      at = reinterpret_cast<const char*>(tile + warp * 1024);
      m = (int)(reinterpret_cast<uintptr_t>(tile) & 15u);
      const int n = left > 2 * kTileElems ? 2 * kTileElems : (int)left;   // elements of the chunk from the tile on
      const int mine = n - warp * 1024;
      nv = mine < 0 ? 0 : (mine > 1088 ? 1088 : mine);               // more than the window: a whole vector past it
      full = (nv * (int)sizeof(T) + m) / 16;                         // vectors [first, full) lie inside the chunk
      first = (head && warp == 0 && m != 0) ? 1 : 0;
    }
  };
  // Brings the warp's window into its stage, which must not be in use: the vectors that lie wholly inside the chunk, zeros for the
  // others. ASYNC: the copies are the calling thread's cp.async, to be committed and waited for; otherwise through registers,
  // which is faster where nothing is done meanwhile (block-scaled FP8 of 8 x 8 Mi bf16: 32.9 us, 35.1 with cp.async).
  template <bool ASYNC>
  static __device__ __forceinline__ void bring(const T* tile, long left, bool head, bool fast, TileStage<T>& st) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint4 x[kChunksPerRun];
    if (fast) {
      const uint4* g = reinterpret_cast<const uint4*>(tile) + warp * kWarpChunks;
      uint4* w = st.buf + warp * kWarpChunks;
      auto to = [&](int j) { return w + slot(j * kRunsPerInstr + lane / kChunksPerRun, lane % kChunksPerRun); };
      if constexpr (ASYNC) {
#pragma unroll
        for (int j = 0; j < kChunksPerRun; ++j) copyAsync16(to(j), g + j * 32 + lane, 16);
      } else {
#pragma unroll
        for (int j = 0; j < kChunksPerRun; ++j) x[j] = __ldg(g + j * 32 + lane);
#pragma unroll
        for (int j = 0; j < kChunksPerRun; ++j) *to(j) = x[j];
      }
      return;
    }
    const Window w(tile, left, head, warp);
    const uint4* g = reinterpret_cast<const uint4*>(w.at - w.m);
    auto in = [&](int vi) { return vi >= w.first && vi < w.full; };
    if constexpr (ASYNC) {
      // a vector outside the chunk names an address that is not read
      const void* none = reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(tile) & ~(uintptr_t)15);
      auto one = [&](int vi) { copyAsync16(place(st, warp, vi), in(vi) ? g + vi : none, in(vi) ? 16 : 0); };
#pragma unroll
      for (int j = 0; j < kChunksPerRun; ++j) one(j * 32 + lane);
      if (lane == 0) one(kWarpChunks);
    } else {
      uint4 xe = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < kChunksPerRun; ++j) x[j] = in(j * 32 + lane) ? __ldg(g + j * 32 + lane) : make_uint4(0, 0, 0, 0);
      if (lane == 0 && in(kWarpChunks)) xe = __ldg(g + kWarpChunks);
#pragma unroll
      for (int j = 0; j < kChunksPerRun; ++j) *place(st, warp, j * 32 + lane) = x[j];
      if (lane == 0) st.extra[warp] = xe;
    }
  }
  // v <- elements [32 t, +32) of the tile (zero beyond the chunk) from the stage that bring filled for the same arguments;
  // every lane of the warp has waited for its copies.
  static __device__ __forceinline__ void take(const T* tile, long left, bool head, bool fast, TileStage<T>& st, float (&v)[32]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncwarp();
    if (fast) { stagedRun<0>(st, warp, lane, 0, v); return; }
    const Window w(tile, left, head, warp);
    auto one = [&](int e) {   // element e of the window, on its own
      const int b = e * (int)sizeof(T) + w.m;
      reinterpret_cast<T*>(place(st, warp, b / 16))[(b % 16) / sizeof(T)] = reinterpret_cast<const T*>(w.at)[e];
    };
    if (w.first == 1 && lane < (16 - w.m) / (int)sizeof(T) && lane < w.nv) one(lane);
    const int tail = (w.full * 16 - w.m) / (int)sizeof(T) + lane;        // from the first element of vector `full` on
    if (w.full >= w.first && w.full <= kWarpChunks && lane < 16 / (int)sizeof(T) && tail >= 0 && tail < w.nv) one(tail);
    __syncwarp();
    if constexpr (SHIFTS) byShift(w.m, [&](auto M) { stagedRun<decltype(M)::value>(st, warp, lane, 0, v); });
    else stagedRun<-1>(st, warp, lane, w.m, v);
  }

  static __device__ __forceinline__ void storeAny(T* tile, long left, TileStage<T>& st, const float (&v)[32]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    char* at = reinterpret_cast<char*>(tile + warp * 1024);
    const int m = (int)(reinterpret_cast<uintptr_t>(tile) & 15u);
    const int n = left > kTileElems ? kTileElems : (int)left, mine = n - warp * 1024;
    const int nv = mine < 0 ? 0 : (mine > 1024 ? 1024 : mine);
    __syncwarp();
    if constexpr (SHIFTS) byShift(m, [&](auto M) { stageRun<decltype(M)::value>(v, st, warp, lane); });
    else stageRun<0>(v, st, warp, lane);
    __syncwarp();
    // vector k of memory holds the window's bytes [16 k - m, 16 k - m + 16); those in [first, full) are whole
    const int first = m != 0 ? 1 : 0, full = (nv * (int)sizeof(T) + m) / 16, staged = SHIFTS ? m : 0;
#pragma unroll(SHIFTS ? kChunksPerRun : 2)
    for (int j = 0; j < kChunksPerRun; ++j) {
      const int k = j * 32 + lane;
      if (k < first || k >= full) continue;
      uint4 y = *place(st, warp, k);
      if (!SHIFTS && m != 0) {
        const uint4 p = *place(st, warp, k - 1);
        uint32_t w[8] = {p.x, p.y, p.z, p.w, y.x, y.y, y.z, y.w};
        shiftWords(w, 16 - m);
        y = make_uint4(w[0], w[1], w[2], w[3]);
      }
      reinterpret_cast<uint4*>(at - m)[k] = y;
    }
    auto one = [&](int e) {
      const int b = e * (int)sizeof(T) + staged;
      reinterpret_cast<T*>(at)[e] = reinterpret_cast<const T*>(place(st, warp, b / 16))[(b % 16) / sizeof(T)];
    };
    if (first == 1 && lane < (16 - m) / (int)sizeof(T) && lane < nv) one(lane);
    const int tail = (full * 16 - m) / (int)sizeof(T) + lane;
    if (full >= first && lane < 16 / (int)sizeof(T) && tail >= 0 && tail < nv) one(tail);
  }

  // v <- elements [e0 + 32 t, +32) of `chunk` (zero beyond `count`). `fast` must be uniform over the CTA.
  static __device__ __forceinline__ void load(const T* chunk, long count, long e0, bool fast, TileStage<T>& st,
                                              float (&v)[32]) {
    __syncwarp();  // the previous user of the window is done
    bring<false>(chunk + e0, count - e0, e0 == 0, fast, st);
    take(chunk + e0, count - e0, e0 == 0, fast, st, v);
  }

  // elements [e0 + 32 t, +32) of `chunk` <- v (nothing beyond `count`).
  static __device__ __forceinline__ void store(T* chunk, long count, long e0, bool fast, TileStage<T>& st,
                                               const float (&v)[32]) {
    storeTile(chunk + e0, count - e0, fast, st, v);
  }
  static __device__ __forceinline__ void storeTile(T* tile, long left, bool fast, TileStage<T>& st, const float (&v)[32]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (fast) {
      uint4* w = st.buf + warp * kWarpChunks;
      __syncwarp();
#pragma unroll
      for (int c = 0; c < kChunksPerRun; ++c) {
        uint4 y;
        if constexpr (k32) {
          y = make_uint4(__float_as_uint(v[4 * c]), __float_as_uint(v[4 * c + 1]), __float_as_uint(v[4 * c + 2]),
                         __float_as_uint(v[4 * c + 3]));
        } else {
          y = Pack16<T>::pack(&v[8 * c]);
        }
        w[slot(lane, c)] = y;
      }
      __syncwarp();
      uint4* g = reinterpret_cast<uint4*>(tile) + warp * kWarpChunks;
#pragma unroll
      for (int j = 0; j < kChunksPerRun; ++j)
        g[j * 32 + lane] = w[slot(j * kRunsPerInstr + lane / kChunksPerRun, lane % kChunksPerRun)];
    } else {
      storeAny(tile, left, st, v);
    }
  }

  static __device__ __forceinline__ bool fast(const T* tile, long left) { return aligned16(tile) && left >= kTileElems; }
  // whether the tile starting at element e0 can take the vector path
  static __device__ __forceinline__ bool fastTile(const T* chunk, long count, long e0) {
    return aligned16(chunk) && e0 + kTileElems <= count;
  }
};

}  // namespace coccl
