// In-place FFT of a tile of pencils in shared memory (device code), for the passes of
// the displacement-space CG (disp.cuh).
//
// A length m = r1 * r2 (both at most 17, on 2-D grids 32) takes two stages on one buffer:
//   forward  stage 1: for each y < r2, DFT_r1 over the slots y r1 + t (t < r1), which
//                     hold x[y + r2 t] (the "split" order); results stay in their slots;
//            stage 2: for each j < r1, slots j + r1 y times W_m^(j y), DFT_r2, giving
//                     X[j + r1 r] in slot j + r1 r (natural order);
//   inverse  the mirror: natural order in, IDFT_r2 and conjugate twiddles over the
//            slots j + r1 r, then IDFT_r1 over y r1 + t, split order out.
// Both stages read and write the same slots of the same thread, so there is one
// barrier per stage and no second buffer, and a forward transform takes the order an
// inverse one leaves.
//
// Lengths with a prime factor above 17 run Bluestein's algorithm over such an m >=
// 2 n - 1: chirp and zero padding ride on stage 1, the filter on the point between the
// two middle stages (the same butterflies of the same thread), and the output chirp on
// the last stage: four shared-memory passes, split order in and out.  Lengths that
// need three or more factors ping-pong between two buffers in
// natural order and read their twiddles from global memory (the table would not leave
// room for the pencils of the longest axes).
//
// Kernels come with a compile-time plan (two stages inline, indices folded) or a runtime
// one: its two stages are inline too, one body per radix; Bluestein and three or more
// factors are one out-of-line function (tile_stages.cuh, linked into every kernel that
// calls it), which addresses shared memory by its 32-bit window address.
#pragma once

#include "fft_device.cuh"

namespace musg {

// Slots of a pencil: groups of r1, S >= r1 places apart (S > r1 pads), so the inner stage
// works on the places y S + t, the outer one on j + S r.  Place of (slot, pencil): slot *
// se + pencil * sp.  Pencil-fast tiles (strided axes): se = P, sp = 1, S = r1; slot-fast
// tiles (the contiguous axis): se = 1, sp = the pencil's stride.
struct TileLay {
  int se, sp, S, pencil_fast;
  __device__ __forceinline__ int at(int slot, int p) const { return slot * se + p * sp; }
  // f(j, p) over the tasks (j < nj, p < P) of a stage, the faster one as the layout says
  template <typename F> __device__ __forceinline__ void each(int nj, int P, F f) const {
    const FDiv fd(pencil_fast ? P : nj);
    for (int t = threadIdx.x; t < nj * P; t += blockDim.x) {
      int lo;
      const int hi = fd.div(t, lo);
      pencil_fast ? f(hi, lo) : f(lo, hi);
    }
  }
};
// a pencil-fast tile over whole rows of P threads: a thread keeps its pencil p and walks
// over j, so nothing is divided inside the loops.  Threads past the last whole row (only
// in grouped launches, whose block fits the largest problem) take no part.
constexpr int kNoRow = 1 << 28;
struct PencilMap {
  int P, p, j0, dj;
  __device__ __forceinline__ explicit PencilMap(int P_) : P(P_) {
    const FDiv f(P_);
    dj = f.div((int)blockDim.x);
    j0 = f.div((int)threadIdx.x, p);
    if (j0 >= dj) j0 = kNoRow;
  }
  __device__ __forceinline__ int stride(int r1) const { return r1; }
  __device__ __forceinline__ int at(int slot, int q) const { return slot * P + q; }
  template <typename F> __device__ __forceinline__ void each(int nj, int, F f) const {
    for (int j = j0; j < nj; j += dj) f(j, p);
  }
  __device__ __forceinline__ TileLay lay(int r1) const { return TileLay{P, 1, r1, 1}; }
};
// Strides of a slot-fast tile of two-stage pencils: S and the pencil stride with the
// fewest bank conflicts over the four ways a half-warp walks it (16 lanes of 8 bytes:
// consecutive indices in natural and in split order, the butterflies of the inner and of
// the outer stage, going over to the next pencil), the smallest among equals.  At 16 x 8
// the pixel phase had 4-way conflicts with one pad entry per 16 slots.
struct RowStrides {
  int S, sp;
};
__host__ __device__ constexpr int bank_cost(int r1, int r2, int S, int sp) {
  int cost = 0;
  for (int pat = 0; pat < 4; ++pat) {
    int cnt[16] = {}, most = 0;
    for (int i = 0; i < 16; ++i) {
      const int a = pat == 0 ? (i / r1) * S + i % r1
                    : pat == 1 ? (i % r2) * S + i / r2
                    : pat == 2 ? (i % r2) * S + (i / r2) * sp
                               : i % r1 + (i / r1) * sp;
      const int k = ++cnt[a & 15];
      if (k > most) most = k;
    }
    cost += most;
  }
  return cost;
}
__host__ __device__ constexpr RowStrides row_strides(int r1, int r2) {
  RowStrides best{r1, r1 * r2};
  int cost = 1000;
  for (int S = r1; S < r1 + 16; ++S)
    for (int sp = (r2 - 1) * S + r1; sp < (r2 - 1) * S + r1 + 16; ++sp) {
      const int c = bank_cost(r1, r2, S, sp);
      if (c < cost || (c == cost && sp < best.sp)) {
        cost = c;
        best = RowStrides{S, sp};
      }
    }
  return best;
}

// a slot-fast tile; CR1 > 0: factors known at compile time
template <int CR1, int CR2> struct RowMap {
  int S, sp;
  __device__ __forceinline__ RowMap(int S_, int sp_) {
    constexpr RowStrides r = row_strides(CR1 > 0 ? CR1 : 1, CR2 > 0 ? CR2 : 1);
    S = CR1 > 0 ? r.S : S_;
    sp = CR1 > 0 ? r.sp : sp_;
  }
  __device__ __forceinline__ int stride(int) const { return S; }
  __device__ __forceinline__ int at(int slot, int p) const { return slot + p * sp; }
  template <typename F> __device__ __forceinline__ void each(int nj, int P, F f) const {
    if constexpr (CR1 > 0) {  // nj is a constant the compiler divides by with a multiplication
      for (int t = threadIdx.x; t < nj * P; t += blockDim.x) f(t % nj, t / nj);
    } else {
      const FDiv fd(nj);
      for (int t = threadIdx.x; t < nj * P; t += blockDim.x) {
        int j;
        const int p = fd.div(t, j);
        f(j, p);
      }
    }
  }
  __device__ __forceinline__ TileLay lay(int) const { return TileLay{1, sp, S, 0}; }
};

__device__ __forceinline__ uint32_t smem_window(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory access by window address (for the out-of-line stages, where the
// address space of a pointer argument is not visible)
__device__ __forceinline__ float2 sld(uint32_t a, float2) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double2 sld(uint32_t a, double2) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sst(uint32_t a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sst(uint32_t a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
// a tile buffer: an ordinary pointer into shared memory, or its window address
template <typename T> struct PtrBuf {
  T *p;
  __device__ __forceinline__ T ld(int i) const { return p[i]; }
  __device__ __forceinline__ void st(int i, T v) const { p[i] = v; }
};
template <typename T> struct WinBuf {
  uint32_t a;
  __device__ __forceinline__ T ld(int i) const { return sld(a + (uint32_t)i * (uint32_t)sizeof(T), T{}); }
  __device__ __forceinline__ void st(int i, T v) const { sst(a + (uint32_t)i * (uint32_t)sizeof(T), v); }
};

enum TileOp : int {
  OP_F1 = 0,  // forward stage 1
  OP_F2 = 1,  // forward stage 2 (twiddles first)
  OP_I1 = 2,  // inverse stage 1 (twiddles last)
  OP_I2 = 3,  // inverse stage 2
  OP_B1 = 4,  // Bluestein: chirp, zero padding, forward stage 1
  OP_BM = 5,  // Bluestein: forward stage 2, filter, inverse stage 1
  OP_B2 = 6   // Bluestein: inverse stage 2, chirp
};
template <typename T> struct TileStageArgs {
  int P, ra, S;           // pencils; the other factor; stride of the slot groups
  int n, conj;            // Bluestein: the transform's length; conj: the inverse transform
  const T *chirp, *bf;    // Bluestein tables (global memory)
};

template <typename T> __device__ __forceinline__ T conj_if(T v, bool c) {
  if (c) v.y = -v.y;
  return v;
}

// one stage over all butterflies of the tile.  ld(e, slot, p) gives input e of the
// transform's axis (slot: its place in the tile), st(e, slot, p, v) takes output e
template <int RAD, int OP, typename T, typename MAP, typename TWB, typename LD, typename ST>
__device__ __forceinline__ void tile_stage(const MAP &map, const TWB tw, const TileStageArgs<T> &a, LD ld, ST st) {
  const int nj = a.ra;
  constexpr bool kOuter = OP == OP_F2 || OP == OP_I1 || OP == OP_BM;  // slots j + S r, else y S + t
  map.each(nj, a.P, [&](int j, int p) {
    T v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) v[r] = ld(j + nj * r, kOuter ? j + a.S * r : j * a.S + r, p);
    if (OP == OP_B1) {
#pragma unroll
      for (int r = 0; r < RAD; ++r) {
        const int e = j + nj * r;
        v[r] = e < a.n ? cmul(conj_if(v[r], a.conj != 0), __ldg(&a.chirp[e])) : T{0, 0};
      }
    }
    if (OP == OP_F2 || OP == OP_BM) {
#pragma unroll
      for (int r = 1; r < RAD; ++r) v[r] = cmul(v[r], tw.ld(j * r));
    }
    if (OP == OP_F1 || OP == OP_F2 || OP == OP_B1 || OP == OP_BM) Dft<RAD, false, T>::run(v);
    if (OP == OP_BM) {
#pragma unroll
      for (int r = 0; r < RAD; ++r) v[r] = cmul(v[r], __ldg(&a.bf[j + nj * r]));
    }
    if (OP == OP_I1 || OP == OP_I2 || OP == OP_BM || OP == OP_B2) Dft<RAD, true, T>::run(v);
    if (OP == OP_I1 || OP == OP_BM) {
#pragma unroll
      for (int r = 1; r < RAD; ++r) v[r] = cmul(v[r], conj_if(tw.ld(j * r), true));
    }
    if (OP == OP_B2) {
#pragma unroll
      for (int r = 0; r < RAD; ++r) {
        const int e = j + nj * r;
        if (e < a.n) v[r] = conj_if(cmul(v[r], __ldg(&a.chirp[e])), a.conj != 0);
      }
    }
#pragma unroll
    for (int r = 0; r < RAD; ++r) st(j + nj * r, kOuter ? j + a.S * r : j * a.S + r, p, v[r]);
  });
}
// Where an index sits in a tile: split order (what a forward transform takes and an
// inverse one leaves) and natural order (the other side).  <CR1, CR2>: factors known at
// compile time; <0, 0> and <-1, -1>: a runtime plan, where three and more factors keep natural order
// throughout and Bluestein keeps split order throughout.
template <int CR1, int CR2> struct SlotMap {
  int S;
  template <typename R> __device__ __forceinline__ SlotMap(const TilePlanD<R> &, int S_) : S(S_) {}
  __device__ __forceinline__ int split(int e) const { return (e % CR2) * S + e / CR2; }
  __device__ __forceinline__ int nat(int e) const { return (e / CR1) * S + e % CR1; }
};
struct SlotMapRt {
  int r1, blu, S;
  FDiv f, f1;
  template <typename R>
  __device__ __forceinline__ SlotMapRt(const TilePlanD<R> &pl, int S_)
      : r1(pl.r1), blu(pl.blu), S(S_), f(pl.r1 ? pl.r2 : 1), f1(pl.r1 ? pl.r1 : 1) {}
  __device__ __forceinline__ int split(int e) const {
    if (!r1) return e;
    int lo;
    const int hi = f.div(e, lo);
    return lo * S + hi;
  }
  __device__ __forceinline__ int nat(int e) const {
    if (blu) return split(e);
    if (S == r1 || !r1) return e;
    int lo;
    const int hi = f1.div(e, lo);
    return hi * S + lo;
  }
};
template <> struct SlotMap<0, 0> : SlotMapRt { using SlotMapRt::SlotMapRt; };
template <> struct SlotMap<-1, -1> : SlotMapRt { using SlotMapRt::SlotMapRt; };
template <> struct SlotMap<-2, -2> : SlotMapRt { using SlotMapRt::SlotMapRt; };

// The transform of P pencils.  run: from shared memory to shared memory, in place in buf
// (buf2: the second buffer of a plan of three or more factors, unused otherwise); the
// caller synchronises before, a barrier ends the call, and the buffer that holds the
// result is returned.  io: inputs from ld(e, slot, p), outputs to st(e, slot, p, v),
// with the exchange between the stages in buf; the caller synchronises before if ld reads
// shared memory, and after before buf is used again.

// runtime plans, out of line (tile_stages.cuh): true when the result is in the second buffer.
// tile_fft_rt: radices up to 17, in the registers of the 3-D kernels; tile_fft_rt2: those of
// 2-D grids, up to 32, in theirs (401^2 mixed 19.4 -> 17.6 ms, 449^2 23.1 -> 20.2)
#define MUSG_TILE_FFT_RT(NAME, T)                                                                                    \
  __device__ bool NAME(bool inv, int n, int m, int r1, int r2, int nst, unsigned long long rcode, int blu, const T *tw, \
                       const T *chirp, const T *bf, const TileLay lay, uint32_t buf, uint32_t buf2, int P, uint32_t tws);
MUSG_TILE_FFT_RT(tile_fft_rt, float2)
MUSG_TILE_FFT_RT(tile_fft_rt, double2)
MUSG_TILE_FFT_RT(tile_fft_rt2, float2)
MUSG_TILE_FFT_RT(tile_fft_rt2, double2)

#define MUSG_TILE_RADICES(X) \
  X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17)
// two factors up to 32 cover the axes of 2-D grids up to 1024
#define MUSG_TILE_RADICES_2D(X) \
  X(18) X(20) X(21) X(22) X(24) X(25) X(26) X(27) X(28) X(30) X(32)

template <int CR1, int CR2> struct TileRun {
  template <bool INV, typename R, typename MAP, typename LD, typename ST>
  static __device__ __forceinline__ void io(const TilePlanD<R> &, const MAP &map, typename V2<R>::T *buf,
                                            typename V2<R>::T *, int P, const typename V2<R>::T *tws, LD ld, ST st) {
    using T = typename V2<R>::T;
    const PtrBuf<T> tw{const_cast<T *>(tws)};
    const int S = map.stride(CR1);
    const TileStageArgs<T> a{P, CR2, S, CR1 * CR2, 0, nullptr, nullptr}, c{P, CR1, S, CR1 * CR2, 0, nullptr, nullptr};
    auto rd = [&](int, int s, int p) { return buf[map.at(s, p)]; };
    auto wr = [&](int, int s, int p, T v) { buf[map.at(s, p)] = v; };
    if constexpr (INV) {
      tile_stage<CR2, OP_I1, T>(map, tw, c, ld, wr);
      __syncthreads();
      tile_stage<CR1, OP_I2, T>(map, tw, a, rd, st);
    } else {
      tile_stage<CR1, OP_F1, T>(map, tw, a, ld, wr);
      __syncthreads();
      tile_stage<CR2, OP_F2, T>(map, tw, c, rd, st);
    }
  }
  template <bool INV, typename R, typename MAP>
  static __device__ __forceinline__ typename V2<R>::T *run(const TilePlanD<R> &pl, const MAP &map,
                                                           typename V2<R>::T *buf, typename V2<R>::T *buf2, int P,
                                                           const typename V2<R>::T *tws) {
    using T = typename V2<R>::T;
    io<INV, R>(pl, map, buf, buf2, P, tws, [&](int, int s, int p) { return buf[map.at(s, p)]; },
               [&](int, int s, int p, T v) { buf[map.at(s, p)] = v; });
    __syncthreads();
    return buf;
  }
};
// runtime plans, every stage out of line
template <bool WIDE> struct TileRunOut {
  template <bool INV, typename R, typename MAP>
  static __device__ __forceinline__ typename V2<R>::T *run(const TilePlanD<R> &pl, const MAP &map,
                                                           typename V2<R>::T *buf, typename V2<R>::T *buf2, int P,
                                                           const typename V2<R>::T *tws) {
    bool second;
    if constexpr (WIDE)
      second = tile_fft_rt2(INV, pl.n, pl.m, pl.r1, pl.r2, pl.nst, pl.rcode, pl.blu, pl.tw, pl.chirp, pl.bf,
                            map.lay(pl.r1), smem_window(buf), smem_window(buf2), P, smem_window(tws));
    else
      second = tile_fft_rt(INV, pl.n, pl.m, pl.r1, pl.r2, pl.nst, pl.rcode, pl.blu, pl.tw, pl.chirp, pl.bf,
                           map.lay(pl.r1), smem_window(buf), smem_window(buf2), P, smem_window(tws));
    return second ? buf2 : buf;
  }
  template <bool INV, typename R, typename MAP, typename LD, typename ST>
  static __device__ __forceinline__ void io(const TilePlanD<R> &pl, const MAP &map, typename V2<R>::T *buf,
                                            typename V2<R>::T *buf2, int P, const typename V2<R>::T *tws, LD ld, ST st) {
    const SlotMap<-1, -1> slots(pl, map.stride(pl.r1));
    map.each(pl.n, P, [&](int e, int p) {
      const int s = INV ? slots.nat(e) : slots.split(e);
      buf[map.at(s, p)] = ld(e, s, p);
    });
    __syncthreads();
    const typename V2<R>::T *res = run<INV, R>(pl, map, buf, buf2, P, tws);
    map.each(pl.n, P, [&](int e, int p) {
      const int s = INV ? slots.split(e) : slots.nat(e);
      st(e, s, p, res[map.at(s, p)]);
    });
  }
};
// the FP64 grouped passes of 3-D grids
template <> struct TileRun<-1, -1> : TileRunOut<false> {};
// runtime plans of the iteration's passes: the two stages inline (one body per radix; WIDE:
// radices up to 32, 2-D), Bluestein and three or more factors out of line
template <bool WIDE> struct TileRunRt {
  template <bool INV, typename R, typename MAP, typename LD, typename ST>
  static __device__ __forceinline__ void two(const TilePlanD<R> &pl, const MAP &map, typename V2<R>::T *buf, int P,
                                             const typename V2<R>::T *tws, LD ld, ST st) {
    using T = typename V2<R>::T;
    const PtrBuf<T> tw{const_cast<T *>(tws)};
    const int S = map.stride(pl.r1);
    const TileStageArgs<T> a{P, pl.r2, S, pl.n, 0, nullptr, nullptr};  // radix r1
    const TileStageArgs<T> c{P, pl.r1, S, pl.n, 0, nullptr, nullptr};  // radix r2
    auto rd = [&](int, int s, int p) { return buf[map.at(s, p)]; };
    auto wr = [&](int, int s, int p, T v) { buf[map.at(s, p)] = v; };
    if constexpr (INV) {
      switch (pl.r2) {
#define MUSG_TS(RAD) \
  case RAD: tile_stage<RAD, OP_I1, T>(map, tw, c, ld, wr); break;
        MUSG_TS(1) MUSG_TILE_RADICES(MUSG_TS)
#undef MUSG_TS
#define MUSG_TS(RAD) \
  case RAD: if constexpr (WIDE) tile_stage<RAD, OP_I1, T>(map, tw, c, ld, wr); break;
        MUSG_TILE_RADICES_2D(MUSG_TS)
#undef MUSG_TS
      }
      __syncthreads();
      switch (pl.r1) {
#define MUSG_TS(RAD) \
  case RAD: tile_stage<RAD, OP_I2, T>(map, tw, a, rd, st); break;
        MUSG_TILE_RADICES(MUSG_TS)
#undef MUSG_TS
#define MUSG_TS(RAD) \
  case RAD: if constexpr (WIDE) tile_stage<RAD, OP_I2, T>(map, tw, a, rd, st); break;
        MUSG_TILE_RADICES_2D(MUSG_TS)
#undef MUSG_TS
        default: tile_stage<1, OP_I2, T>(map, tw, a, rd, st); break;
      }
    } else {
      switch (pl.r1) {
#define MUSG_TS(RAD) \
  case RAD: tile_stage<RAD, OP_F1, T>(map, tw, a, ld, wr); break;
        MUSG_TILE_RADICES(MUSG_TS)
#undef MUSG_TS
#define MUSG_TS(RAD) \
  case RAD: if constexpr (WIDE) tile_stage<RAD, OP_F1, T>(map, tw, a, ld, wr); break;
        MUSG_TILE_RADICES_2D(MUSG_TS)
#undef MUSG_TS
        default: tile_stage<1, OP_F1, T>(map, tw, a, ld, wr); break;
      }
      __syncthreads();
      switch (pl.r2) {
#define MUSG_TS(RAD) \
  case RAD: tile_stage<RAD, OP_F2, T>(map, tw, c, rd, st); break;
        MUSG_TS(1) MUSG_TILE_RADICES(MUSG_TS)
#undef MUSG_TS
#define MUSG_TS(RAD) \
  case RAD: if constexpr (WIDE) tile_stage<RAD, OP_F2, T>(map, tw, c, rd, st); break;
        MUSG_TILE_RADICES_2D(MUSG_TS)
#undef MUSG_TS
      }
    }
  }
  template <bool INV, typename R, typename MAP, typename LD, typename ST>
  static __device__ __forceinline__ void io(const TilePlanD<R> &pl, const MAP &map, typename V2<R>::T *buf,
                                            typename V2<R>::T *buf2, int P, const typename V2<R>::T *tws, LD ld, ST st) {
    if (!pl.r1 || pl.blu) TileRunOut<WIDE>::template io<INV, R>(pl, map, buf, buf2, P, tws, ld, st);
    else two<INV, R>(pl, map, buf, P, tws, ld, st);
  }
  template <bool INV, typename R, typename MAP>
  static __device__ __forceinline__ typename V2<R>::T *run(const TilePlanD<R> &pl, const MAP &map,
                                                           typename V2<R>::T *buf, typename V2<R>::T *buf2, int P,
                                                           const typename V2<R>::T *tws) {
    using T = typename V2<R>::T;
    if (!pl.r1 || pl.blu) return TileRunOut<WIDE>::template run<INV, R>(pl, map, buf, buf2, P, tws);
    two<INV, R>(pl, map, buf, P, tws, [&](int, int s, int p) { return buf[map.at(s, p)]; },
                [&](int, int s, int p, T v) { buf[map.at(s, p)] = v; });
    __syncthreads();
    return buf;
  }
};

template <> struct TileRun<0, 0> : TileRunRt<false> {};
template <> struct TileRun<-2, -2> : TileRunRt<true> {};

}  // namespace musg
