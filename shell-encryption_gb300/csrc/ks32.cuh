// 32-bit arithmetic of the key switch that runs in three auxiliary primes
// (ks32.cu): residues modulo primes p < 2^30, p = 1 mod 2^16, with Shoup
// products in 32 bits (one high and two low multiplies against nine
// multiplies of the 64-bit lazy product).
//
// A 128-element row or an Ntt4 column is transformed by NttCore's passes with
// 16 values per thread.  Ranges:
//   exact (p < 2^30): forward [0, 4p) (Harvey), inverse [0, 2p);
//   LZ (p < 2^28, at most 7 levels per phase): forward levels add 2p without
//     any correction (below 2p + 14p = 16p <= 2^32), inverse sums double for
//     three levels before one Barrett step brings them back below 2p.
#pragma once
#include "ntt4.cuh"

namespace shg {

__device__ __forceinline__ uint32_t min_sub32(uint32_t x, uint32_t m) { return min(x, x - m); }

// x w mod p in [0, 2p) for any x < 2^32, w < p, wp = floor(w 2^32 / p).
__device__ __forceinline__ uint32_t shoup32(uint32_t x, uint2 w, uint32_t p) {
  return x * w.x - __umulhi(x, w.y) * p;
}

// x mod p in [0, 2p) for any x < 2^32, bar = floor(2^32 / p).
__device__ __forceinline__ uint32_t barrett32(uint32_t x, uint32_t bar, uint32_t p) {
  return x - __umulhi(x, bar) * p;
}

template <bool LZ>
__device__ __forceinline__ void bf32_ct(uint32_t& X, uint32_t& Y, uint2 w, const Pr32& P) {
  const uint32_t x = LZ ? X : min_sub32(X, P.p2);
  const uint32_t t = shoup32(Y, w, P.p);
  X = x + t;
  Y = x - t + P.p2;
}

// Twiddles u, u + 1 of a level come in one 16-byte load (their index is even
// whenever the level has at least two per thread).  PAIR_STEP: distance of
// consecutive pairs, in twiddles.
template <int CNT, bool SHARED = false, int PAIR_STEP = 2>
__device__ __forceinline__ void load_tw32(uint2 (&w)[8], const uint2* tw) {
  if constexpr (CNT == 1) {
    w[0] = SHARED ? *tw : __ldg(tw);
  } else {
#pragma unroll
    for (int u = 0; u < CNT; u += 2) {
      const uint4* q = reinterpret_cast<const uint4*>(tw + u / 2 * PAIR_STEP);
      const uint4 v = SHARED ? *q : __ldg(q);
      w[u] = make_uint2(v.x, v.y);
      w[u + 1] = make_uint2(v.z, v.w);
    }
  }
}

// Forward pass PASS of a 2^LOG transform (NttCore's order and layouts).
// SHARED: tw is in shared memory.
template <int LOG, int PASS, bool LZ, bool SHARED = false>
__device__ __forceinline__ void fwd_pass32(uint32_t (&x)[16], int tid, const uint2* tw,
                                           int tw_mult, const Pr32& P) {
  using C = NttCore<LOG, 4>;
  constexpr int clo = C::fwd_clo(PASS), RR = C::R(PASS);
  const int tid_high = tid >> clo;
  static_for<0, RR>([&](auto ii) {
    constexpr int lb = RR - 1 - decltype(ii)::value;
    constexpr int s = LOG - 1 - (clo + lb), CNT = 16 >> (lb + 1);
    uint2 w[8];
    if constexpr (SHARED && PASS == 1)  // row_tw_pos's order
      load_tw32<CNT, true, 16>(w, tw + (1 << s) + 2 * tid);
    else
      load_tw32<CNT, SHARED>(w, tw + tw_mult * (1 << s) + (tid_high << (3 - lb)));
    static_for<0, CNT>([&](auto uu) {
      static_for<0, (1 << lb)>([&](auto ll) {
        constexpr int k0 = (decltype(uu)::value << (lb + 1)) | decltype(ll)::value;
        bf32_ct<LZ>(x[k0], x[k0 | (1 << lb)], w[decltype(uu)::value], P);
      });
    });
  });
}

// Inverse pass; bit_off and row as in NttCore::inv_pass.  LZ: before level b
// the values lie below 2^(1 + b mod 3) p.
template <int LOG, int PASS, bool LZ, bool SHARED = false>
__device__ __forceinline__ void inv_pass32(uint32_t (&x)[16], int tid, const uint2* tw,
                                           int nfull, int bit_off, int row, const Pr32& P) {
  using C = NttCore<LOG, 4>;
  constexpr int clo = C::inv_clo(PASS), plo = C::inv_plo(PASS), RR = C::R(PASS);
  const int tid_high = tid >> clo;
  static_for<0, RR>([&](auto ii) {
    constexpr int lb = plo + decltype(ii)::value;
    constexpr int b = clo + lb, CNT = 16 >> (lb + 1);
    const uint32_t bound = !LZ || b % 3 == 0 ? P.p2 : (b % 3 == 1 ? P.p4 : P.p8);
    uint2 w[8];
    if constexpr (SHARED && PASS == 0 && CNT > 1)
      load_tw32<CNT, true, 16>(w, tw + (128 - (128 >> b)) + 2 * tid);
    else
      load_tw32<CNT, SHARED>(w, tw + (nfull - (nfull >> (b + bit_off)) + (row << (LOG - b - 1)) +
                                      (tid_high << (3 - lb))));
    static_for<0, CNT>([&](auto uu) {
      static_for<0, (1 << lb)>([&](auto ll) {
        constexpr int k0 = (decltype(uu)::value << (lb + 1)) | decltype(ll)::value;
        constexpr int k1 = k0 | (1 << lb);
        const uint32_t s = x[k0] + x[k1], d = x[k0] - x[k1] + bound;
        if constexpr (!LZ)
          x[k0] = min_sub32(s, P.p2);
        else if constexpr (b % 3 == 2)
          x[k0] = barrett32(s, P.bar, P.p);
        else
          x[k0] = s;
        x[k1] = shoup32(d, w[decltype(uu)::value], P.p);
      });
    });
  });
}

// Exchange tile of COLS interleaved columns.  Sixteen columns put two
// elements on the 32 banks: flipping bit 0 by bit 4 of the element index keeps
// the two threads rows of a warp apart in both register layouts.
struct ColTile32 {
  uint32_t* sm;
  int cols, j;
  __device__ __forceinline__ uint32_t& operator()(int i) const {
    return sm[(i ^ ((i >> 4) & 1)) * cols + j];
  }
};

template <int LOG>
__device__ __forceinline__ void exchange32(uint32_t (&x)[16], int tid, const ColTile32& m,
                                           int clo_a, int clo_b) {
  using C = NttCore<LOG, 4>;
#pragma unroll
  for (int k = 0; k < 16; ++k) m(C::idx(tid, k, clo_a)) = x[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; ++k) x[k] = m(C::idx(tid, k, clo_b));
  __syncthreads();
}

template <int LOG, bool LZ>
__device__ __forceinline__ void fwd_cols32(uint32_t (&x)[16], int tid, const ColTile32& m,
                                           const uint2* tw, const Pr32& P) {
  using C = NttCore<LOG, 4>;
  static_for<0, C::P>([&](auto pp) {
    constexpr int ps = decltype(pp)::value;
    fwd_pass32<LOG, ps, LZ>(x, tid, tw, 1, P);
    if constexpr (ps + 1 < C::P) exchange32<LOG>(x, tid, m, C::fwd_clo(ps), C::fwd_clo(ps + 1));
  });
}

template <int LOG, bool LZ>
__device__ __forceinline__ void inv_cols32(uint32_t (&x)[16], int tid, const ColTile32& m,
                                           const uint2* tw, int nfull, const Pr32& P) {
  using C = NttCore<LOG, 4>;
  static_for<0, C::P>([&](auto pp) {
    constexpr int ps = decltype(pp)::value;
    inv_pass32<LOG, ps, LZ>(x, tid, tw, nfull, kNtt4RowBits, 0, P);
    if constexpr (ps + 1 < C::P) exchange32<LOG>(x, tid, m, C::inv_clo(ps), C::inv_clo(ps + 1));
  });
}

// Tile of 128-element rows, 136 words apart.  Element i sits at word i with
// bits 3 and 2 flipped by its bits 5 and 6, so that the accesses of a warp on
// four rows (eight threads t each) at 8 k + t and, 16 bytes wide, at 16 t + 4 m,
// and 8-byte accesses along one row, all run without bank conflicts, and the
// first are two bases plus constants (an XOR swizzle over all bits cost a
// fifth of the row kernel's instructions in address arithmetic).
constexpr int kRow32 = 136;
__device__ __forceinline__ int row_word32(int i) { return i ^ ((i >> 2) & 8) ^ ((i >> 4) & 4); }

// The places of one thread's 16 values of a row: elements 8 k + t and
// 16 t + 4 m ... + 3.
struct RowPos32 {
  uint32_t *b0, *b1, *w[4];
  __device__ __forceinline__ RowPos32(uint32_t* row, int t) {
    b0 = row + t;
    b1 = row + (t ^ 4);
#pragma unroll
    for (int m = 0; m < 4; ++m) w[m] = row + row_word32(16 * t + 4 * m);
  }
  template <int k>
  __device__ __forceinline__ uint32_t& at() const {
    return (k < 8 ? b0 : b1)[(8 * k) ^ ((k & 4) << 1)];
  }
  __device__ __forceinline__ void load_wide(uint32_t (&x)[16]) const {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint4 v = *reinterpret_cast<const uint4*>(w[m]);
      x[4 * m] = v.x;
      x[4 * m + 1] = v.y;
      x[4 * m + 2] = v.z;
      x[4 * m + 3] = v.w;
    }
  }
  __device__ __forceinline__ void store_wide(const uint32_t (&x)[16]) const {
#pragma unroll
    for (int m = 0; m < 4; ++m)
      *reinterpret_cast<uint4*>(w[m]) =
          make_uint4(x[4 * m], x[4 * m + 1], x[4 * m + 2], x[4 * m + 3]);
  }
};

// Twiddles of one row in shared memory: forward entry i of level s (of the
// row's seven, (R + row) 2^s + i in the prime's table) at 2^s + i, inverse
// entry i of level b at 128 - 2^(7 - b) + i, which is how the passes index a
// 128-element transform of its own (tw_mult 1; nfull 128, row 0).  Levels with
// 8 or 4 twiddles per thread t (32 and 64 entries; i = 8 t + u or 4 t + u) keep
// pair u / 2 of all eight threads together, so their 16-byte loads meet no
// bank conflicts.
constexpr int kRowTw32 = 128;
__device__ __forceinline__ int row_tw_pos(int i, int per_thread) {
  const int t = i / per_thread, u = i % per_thread;
  return ((u >> 1) * 8 + t) * 2 + (u & 1);
}
__device__ __forceinline__ int row_tw_fwd_pos(int e) {
  return e >= 64 ? 64 + row_tw_pos(e - 64, 8) : (e >= 32 ? 32 + row_tw_pos(e - 32, 4) : e);
}
__device__ __forceinline__ int row_tw_inv_pos(int e) {
  return e < 64 ? row_tw_pos(e, 8) : (e < 96 ? 64 + row_tw_pos(e - 64, 4) : e);
}
__device__ __forceinline__ uint2 row_tw_fwd(const uint2* tw, int R, int row, int e) {
  const int s = 31 - __clz(e | 1);
  return e ? __ldg(tw + (((R + row) << s) + e - (1 << s))) : make_uint2(0, 0);
}
__device__ __forceinline__ uint2 row_tw_inv(const uint2* tw, int nfull, int row, int e) {
  const int z = 128 - e;  // 2^(6 - b) < z <= 2^(7 - b)
  if (e == 127) return make_uint2(0, 0);
  const int b = 7 - (32 - __clz(z - 1));
  return __ldg(tw + (nfull - (nfull >> b) + (row << (6 - b)) + e - (128 - (128 >> b))));
}

// Forward transform of one row in place by eight threads (t) of one warp;
// every thread of the warp calls it.  fin takes the results (below 16p for
// LZ, else 4p).
template <bool LZ, class Fin>
__device__ __forceinline__ void fwd_row32(uint32_t* row, int t, const uint2* tw, const Pr32& P,
                                          Fin&& fin) {
  const RowPos32 r(row, t);
  uint32_t x[16];
  static_for<0, 16>([&](auto k) { x[decltype(k)::value] = r.at<decltype(k)::value>(); });
  fwd_pass32<7, 0, LZ, true>(x, t, tw, 1, P);
  static_for<0, 16>([&](auto k) { r.at<decltype(k)::value>() = x[decltype(k)::value]; });
  __syncwarp();
  r.load_wide(x);
  fwd_pass32<7, 1, LZ, true>(x, t, tw, 1, P);
#pragma unroll
  for (int k = 0; k < 16; ++k) x[k] = fin(x[k]);
  r.store_wide(x);
}

// Inverse transform of one row (values below 2p); x[k] becomes element
// 8 k + t of the row, below 2p.
template <bool LZ>
__device__ __forceinline__ void inv_row32(uint32_t (&x)[16], uint32_t* row_sm, int t,
                                          const uint2* tw, const Pr32& P) {
  const RowPos32 r(row_sm, t);
  r.load_wide(x);
  inv_pass32<7, 0, LZ, true>(x, t, tw, 128, 0, 0, P);
  r.store_wide(x);
  __syncwarp();
  static_for<0, 16>([&](auto k) { x[decltype(k)::value] = r.at<decltype(k)::value>(); });
  inv_pass32<7, 1, LZ, true>(x, t, tw, 128, 0, 0, P);
  if constexpr (LZ) {  // the last level left its sums below 4p
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = min_sub32(x[k], P.p2);
  }
}

}  // namespace shg
