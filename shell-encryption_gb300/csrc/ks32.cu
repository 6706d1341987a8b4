// Gadget key switch in three auxiliary 30-bit primes.
//
// For every output limb l and key component c the key switch needs
//   S = sum_j d_j * K_j  in Z[X]/(X^n + 1),  reduced mod q_l,
// with d_j the gadget digits (the same small integers for every limb) and
// K_j the key row modulo q_l, taken as integers in (-q_l/2, q_l/2).  Every
// coefficient satisfies |S| <= n * sum_j max(d_j) * q_l/2, so three primes
// p_0 p_1 p_2 = P > 2 |S| determine it exactly.  The digits are transformed
// modulo the three p_a instead of modulo all L primes q_l, in 32-bit
// arithmetic: per ciphertext 3 k forward and 6 L inverse 32-bit transforms and
// 2 L forward 64-bit ones take the place of k L forward 64-bit ones (n = 2^14,
// L = 6, k = 18: 54 + 36 + 12 against 108).  This is the evaluation of gadget
// products over a second RNS basis of Kim, Lee, Seo and Song ("Accelerating HE
// operations from key decomposition technique", CRYPTO 2023), used here with
// the key's own digits, so results equal the reference's bit for bit.
//
//   k32_digit_cols  digit extraction + column phase of its three transforms
//   k32_rows        row phase of all digits, inner product with the key,
//                   inverse row phase of the 2 L sums, per prime
//   k32_crt_cols    inverse column phase in the three primes, reconstruction
//                   modulo q_l, column phase of the forward 64-bit transform
//   launch4_rows_add (ntt4.cu)  its row phase + base
#include "ks32.cuh"

namespace shg {
namespace {

template <int LOG_N>
struct K32 {
  using S = Ntt4<LOG_N>;
  using C = typename S::CC;  // layouts of the 16-value column transform
  // Columns per CTA of the 32-bit column kernels: 128-byte rows of words
  // below n = 2^14, 64 bytes above (CTAs of at most 256 threads).
  static constexpr int COLS = LOG_N <= 13 ? 32 : 16;
  static constexpr int TILES = (1 << S::B) / COLS;
  static constexpr int THREADS = C::T * COLS;
};

// Column phase of one digit transform per (prime, digit): the CTA takes COLS
// columns of limb l of ciphertext p, reads the exported coefficients once and
// runs its share (part of nsplit) of the limb's digits x three primes.
// D [count][k][3][n].
template <int LOG_N, bool LZ>
__global__ void __launch_bounds__(K32<LOG_N>::THREADS, 768 / K32<LOG_N>::THREADS)
    k32_digit_cols(const uint64_t* X, const DigitDesc* digits, Ks32Digits first, int k, int L,
                   int nsplit, uint32_t* D, const __grid_constant__ W32 w) {
  after_previous();
  using S = Ntt4<LOG_N>;
  using G = K32<LOG_N>;
  using C = typename G::C;
  __shared__ uint32_t smem[G::COLS << S::A];
  int b = blockIdx.x;
  const int tile = b % G::TILES;
  b /= G::TILES;
  const int part = b % nsplit;
  b /= nsplit;
  const int l = b % L;
  const size_t p = (size_t)(b / L);
  const int jc = threadIdx.x % G::COLS, t = threadIdx.x / G::COLS;
  const int col = tile * G::COLS + jc;
  const uint64_t* src = X + ((p * L + l) << LOG_N);
  uint64_t v[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) v[e] = src[(C::fwd_in_idx(t, e) << S::B) | col];
  const int j0 = first.j[l], nd = first.j[l + 1] - j0;
  const ColTile32 tile32{smem, G::COLS, jc};
#pragma unroll 1
  for (int it = part; it < 3 * nd; it += nsplit) {
    const int j = j0 + it / 3, a = it % 3;
    const int dj = dbg_index(j, k, kDbgDigit);
    const int shift = digits[dj].shift;
    const uint32_t mask = (uint32_t)digits[dj].mask;
    uint32_t x[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = (uint32_t)(v[e] >> shift) & mask;
    const Pr32& P = w.pr[a];
    fwd_cols32<S::A, LZ>(x, t, tile32, w.fwd + ((size_t)a << LOG_N), P);
    uint32_t* dst = D + (((p * k + j) * 3 + a) << LOG_N);
#pragma unroll
    for (int e = 0; e < 16; ++e)
      dst[(C::fwd_out_idx(t, e) << S::B) | col] = LZ ? barrett32(x[e], P.bar, P.p) : x[e];
  }
}

__device__ __forceinline__ void cp_async16(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src));
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Key words: read once per CTA, so they leave L1 to the twiddles.
__device__ __forceinline__ uint2 ld_key(const uint32_t* p) {
  uint2 v;
  asm("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// hi * (2^32 mod p) + lo of a 64-bit sum: congruent and below 2^32 (p + 1).
__device__ __forceinline__ uint64_t fold32(uint64_t acc, uint32_t r) {
  return (uint64_t)(uint32_t)(acc >> 32) * r + (uint32_t)acc;
}
// acc 2^-32 mod p below 2p, for a folded acc.
__device__ __forceinline__ uint32_t redc32(uint64_t acc, uint32_t p, uint32_t pinv) {
  return (uint32_t)(acc >> 32) - __umulhi((uint32_t)acc * pinv, p) + p;
}

constexpr int kPf = 3;  // digits whose key words are prefetched

__host__ __device__ constexpr int rows32_digit_rows(int k, int T) { return (k * T + 3) & ~3; }
// Sums of one inner-product round: both components of NT / 64 limbs.
__host__ __device__ constexpr int rows32_sum_rows(int T, int NT) {
  return (NT / 32 * T + 3) & ~3;
}

// One row (128 positions) of one prime for T ciphertexts: forward row phase
// of their k digit transforms (rows j * T + t of the tile, four per warp at a
// time), then per round of NT / 64 limbs the inner product with the key (two
// positions of both components of one limb and all T ciphertexts per thread;
// 64-bit sums folded every w.chunk terms) and the inverse row phase of the
// round's sums.  key [3][n/128][k][L][2][128], premultiplied by
// 2^32 n^-1 (P/p_a)^-1 mod p_a; E [count][2][L][3][n].  Ciphertext groups are
// the fastest block index, so a key row stays in L2 for all of them.
//
// Bound by the multiply pipe and its latency: n = 2^14, L = 6, 16 ciphertexts
// take 72 us (105 us with XOR-swizzled addresses, unprefetched key words and
// twiddles from global memory), multiply pipe 59 % and issue slots 45 % busy,
// 103 MB of DRAM reads (the digit transforms and the key once).  80 registers
// and 55 KB keep four 192-thread CTAs on an SM; 64 registers for five spilled
// (80 us), and at k = 36 (n = 2^15, L = 12), where only two CTAs fit, 384
// threads take 299 us for 10 ciphertexts against 368.
template <int LOG_N, bool LZ, int T, int NT>
__global__ void __launch_bounds__(NT, 768 / NT)
    k32_rows(const uint32_t* D, const uint32_t* key, uint32_t* E, int k, int L, int count,
             const __grid_constant__ W32 w) {
  after_previous();
  extern __shared__ __align__(16) uint32_t sm32[];
  constexpr int R = 1 << (LOG_N - 7), kLimbs = NT / 64;
  const int groups = (count + T - 1) / T;
  const int p0 = (blockIdx.x % groups) * T;
  const int ar = blockIdx.x / groups, row = ar % R, a = ar / R;
  const Pr32& P = w.pr[a];
  uint2* twf = reinterpret_cast<uint2*>(sm32);
  uint2* twi = twf + kRowTw32;
  uint32_t* dig = sm32 + 4 * kRowTw32;
  uint32_t* sums = dig + rows32_digit_rows(k, T) * kRow32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int sub = warp; sub < k * T; sub += NT / 32) {
    const size_t p = (size_t)min(p0 + sub % T, count - 1);
    cp_async16(dig + sub * kRow32 + row_word32(4 * lane),
               D + (((p * k + sub / T) * 3 + a) << LOG_N) + row * 128 + 4 * lane);
  }
  if (tid < kRowTw32) {
    twf[row_tw_fwd_pos(tid)] = row_tw_fwd(w.fwd + ((size_t)a << LOG_N), R, row, tid);
    twi[row_tw_inv_pos(tid)] = row_tw_inv(w.inv + ((size_t)a << LOG_N), 1 << LOG_N, row, tid);
  }
  // kPf digits' key words at a time, fetched one step ahead: the first before
  // the digit transforms, a later round's before its predecessor's inverse
  // rows.  (Loaded where they are used, every step held for an L2 round trip:
  // 105 us a launch of 16 ciphertexts at n = 2^14, L = 6 against 92.)  The last
  // fetches run past the row's digits, into the next row or the key's padding
  // (kKs32PadDigits digits), and are not used.
  static_assert(kKs32PadDigits >= 3 * kPf, "fetches past the last digit");
  const int lg = tid >> 6, pp = tid & 63, kstep = L * 256;
  const uint32_t* key_row = key + (size_t)ar * k * L * 256 + 2 * pp;
  const uint32_t* kq = key_row + min(lg, L - 1) * 256;
  uint2 kb[2][kPf], ka[2][kPf];
  auto fetch = [&](auto slot) {
    constexpr int z = decltype(slot)::value;
#pragma unroll
    for (int f = 0; f < kPf; ++f) {
      kb[z][f] = ld_key(kq);
      ka[z][f] = ld_key(kq + 128);
      kq += kstep;
    }
  };
  using Z0 = std::integral_constant<int, 0>;
  using Z1 = std::integral_constant<int, 1>;
  fetch(Z0{});
  cp_async_wait_all();
  __syncthreads();
  for (int s0 = warp * 4; s0 < rows32_digit_rows(k, T); s0 += NT / 8)
    fwd_row32<LZ>(dig + (s0 + (lane >> 3)) * kRow32, lane & 7, twf, P, [&](uint32_t x) {
      // below 2p (LZ: from below 16p) or canonical (from below 4p)
      return LZ ? barrett32(x, P.bar, P.p) : min_sub32(min_sub32(x, P.p2), P.p);
    });
  __syncthreads();
  const uint32_t* dp = dig + row_word32(2 * pp);
  for (int l0 = 0; l0 < L; l0 += kLimbs) {
    const int l = l0 + lg;
    if (l < L) {
      uint64_t acc[2][T][2];
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int t = 0; t < T; ++t) acc[c][t][0] = acc[c][t][1] = 0;
      auto mac = [&](int j, auto slot) {
        constexpr int z = decltype(slot)::value;
#pragma unroll
        for (int f = 0; f < kPf; ++f) {
          if (j + f >= k) break;
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const uint2 d = *reinterpret_cast<const uint2*>(dp + ((j + f) * T + t) * kRow32);
            acc[0][t][0] += (uint64_t)d.x * kb[z][f].x;
            acc[0][t][1] += (uint64_t)d.y * kb[z][f].y;
            acc[1][t][0] += (uint64_t)d.x * ka[z][f].x;
            acc[1][t][1] += (uint64_t)d.y * ka[z][f].y;
          }
        }
      };
      int left = w.chunk;
      for (int j = 0; j < k; j += 2 * kPf) {
        fetch(Z1{});
        mac(j, Z0{});
        fetch(Z0{});
        mac(j + kPf, Z1{});
        left -= 2 * kPf;
        if (left < 2 * kPf || j + 2 * kPf >= k) {
          left = w.chunk;
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int t = 0; t < T; ++t) {
              acc[c][t][0] = fold32(acc[c][t][0], P.r);
              acc[c][t][1] = fold32(acc[c][t][1], P.r);
            }
        }
      }
      kq = key_row + min(l + kLimbs, L - 1) * 256;
      if (l0 + kLimbs < L) fetch(Z0{});
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int t = 0; t < T; ++t)
          *reinterpret_cast<uint2*>(sums + ((lg * 2 + c) * T + t) * kRow32 +
                                    row_word32(2 * pp)) =
              make_uint2(redc32(acc[c][t][0], P.p, P.pinv), redc32(acc[c][t][1], P.p, P.pinv));
    }
    __syncthreads();
    for (int s0 = warp * 4; s0 < rows32_sum_rows(T, NT); s0 += NT / 8) {
      const int es = s0 + (lane >> 3), t8 = lane & 7;
      uint32_t x[16];
      inv_row32<LZ>(x, sums + es * kRow32, t8, twi, P);
      const int lc = es / T, el = l0 + (lc >> 1), p = p0 + es % T;
      if (lc < 2 * kLimbs && el < L && p < count) {
        uint32_t* dst =
            E + (((((size_t)p * 2 + (lc & 1)) * L + el) * 3 + a) << LOG_N) + row * 128 + t8;
#pragma unroll
        for (int e = 0; e < 16; ++e) dst[8 * e] = x[e];
      }
    }
    __syncthreads();
  }
}

// Inverse column phase of one sum in the three primes (the key carries
// (P/p_a)^-1, so the results y_a are S's digits over the basis P/p_a:
// S = sum_a y_a P/p_a - u P with u = round(sum_a y_a / p_a); |S| < 0.499 P
// and single precision leave no doubt about u), S mod q_l, and the column
// phase of the forward transform modulo q_l.  The CTA takes 16 columns of one
// (ciphertext, component, limb).  out [count][2][L][n], lazily reduced.
template <int LOG_N, bool LZ>
__global__ void __launch_bounds__(Ntt4<LOG_N>::COL_THREADS, 640 / Ntt4<LOG_N>::COL_THREADS)
    k32_crt_cols(const uint32_t* E, const Crt32* crt, int L, uint64_t* out, const __grid_constant__ W32 w, CtxDev c) {
  after_previous();
  using S = Ntt4<LOG_N>;
  using C = typename S::CC;
  __shared__ __align__(16) uint64_t smem[S::COLS << S::A];
  const int g = blockIdx.x / S::COL_TILES, tile = blockIdx.x % S::COL_TILES;
  const int jc = threadIdx.x % S::COLS, t = threadIdx.x / S::COLS;
  const int col = tile * S::COLS + jc;
  const int l = dbg_index(g % L, c.L, kDbgLimb);
  const uint32_t* src = E + ((size_t)g * 3 << LOG_N);
  const ColTile32 tile32{reinterpret_cast<uint32_t*>(smem), S::COLS, jc};
  uint32_t y[3][16];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int e = 0; e < 16; ++e)
      y[a][e] = src[((size_t)a << LOG_N) + ((C::inv_in_idx(t, e) << S::B) | col)];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
    inv_cols32<S::A, LZ>(y[a], t, tile32, w.inv + ((size_t)a << LOG_N), S::N, w.pr[a]);
  const uint64_t q = c.primes[l].q, two_q = c.primes[l].two_q;
  const Crt32 m = crt[l];
  uint64_t x[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const float f = (float)y[0][e] * w.finv[0] + (float)y[1][e] * w.finv[1] +
                    (float)y[2][e] * w.finv[2];
    const uint32_t u = (uint32_t)__float2int_rn(f);
    x[e] = shoup_lazy_x32(y[0][e], m.w[0], m.wp[0], q) +
           shoup_lazy_x32(y[1][e], m.w[1], m.wp[1], q) +
           shoup_lazy_x32(y[2][e], m.w[2], m.wp[2], q) + u * m.neg_p;
  }
  C::template forward_m<true, true, typename C::ColMap>(
      x, t, typename C::ColMap{smem, S::COLS, jc}, c.tw_fwd + ((size_t)l << LOG_N), 1, q, two_q);
  uint64_t* dst = out + ((size_t)g << LOG_N);
#pragma unroll
  for (int e = 0; e < 16; ++e) dst[(C::fwd_out_idx(t, e) << S::B) | col] = x[e];
}

// Key import, column phase: coefficients of key rows [k][L][n] modulo q_l, as
// integers in (-q_l/2, q_l/2), to [k][L][3][n].  Runs once per key.
template <int LOG_N>
__global__ void __launch_bounds__(K32<LOG_N>::THREADS)
    k32_key_cols(const uint64_t* rows, int L, uint32_t* out, const __grid_constant__ W32 w, CtxDev c) {
  using S = Ntt4<LOG_N>;
  using G = K32<LOG_N>;
  using C = typename G::C;
  __shared__ uint32_t smem[G::COLS << S::A];
  const int tile = blockIdx.x % G::TILES;
  const size_t g = blockIdx.x / G::TILES;
  const uint64_t q = c.primes[g % L].q;
  const int jc = threadIdx.x % G::COLS, t = threadIdx.x / G::COLS;
  const int col = tile * G::COLS + jc;
  for (int a = 0; a < 3; ++a) {
    const uint32_t pr = w.pr[a].p;
    uint32_t x[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const uint64_t v = rows[(g << LOG_N) + ((C::fwd_in_idx(t, e) << S::B) | col)];
      x[e] = v > q / 2 ? pr - (uint32_t)((q - v) % pr) : (uint32_t)(v % pr);
    }
    fwd_cols32<S::A, false>(x, t, ColTile32{smem, G::COLS, jc}, w.fwd + ((size_t)a << LOG_N),
                            w.pr[a]);
    uint32_t* dst = out + ((g * 3 + a) << LOG_N);
#pragma unroll
    for (int e = 0; e < 16; ++e) dst[(C::fwd_out_idx(t, e) << S::B) | col] = x[e];
  }
}

// Key import, row phase: the CTA takes one row of digits j .. j + nj - 1 and every
// limb of one prime and writes them, times `scale`, to their places in the key of
// k32_rows (k digits, component comp).
template <int LOG_N>
__global__ void __launch_bounds__(128)
    k32_key_rows(const uint32_t* in, int j, int nj, int k, int L, int comp, uint32_t* key,
                 const __grid_constant__ W32 w) {
  __shared__ __align__(16) uint32_t sm[16 * kRow32];
  __shared__ __align__(16) uint2 tw[kRowTw32];
  constexpr int R = 1 << (LOG_N - 7);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int a = blockIdx.x / R, row = blockIdx.x % R;
  const Pr32& P = w.pr[a];
  tw[row_tw_fwd_pos(threadIdx.x)] =
      row_tw_fwd(w.fwd + ((size_t)a << LOG_N), R, row, threadIdx.x);
  __syncthreads();
  uint32_t* tile = sm + warp * 4 * kRow32;
  for (int q0 = warp * 4; q0 < nj * L; q0 += 16) {
    for (int i = lane; i < 512; i += 32) {
      const size_t jl = min(q0 + (i >> 7), nj * L - 1);
      tile[(i >> 7) * kRow32 + row_word32(i & 127)] =
          in[((jl * 3 + a) << LOG_N) + row * 128 + (i & 127)];
    }
    __syncwarp();
    fwd_row32<false>(tile + (lane >> 3) * kRow32, lane & 7, tw, P, [&](uint32_t x) {
      return (uint32_t)((uint64_t)x * P.scale % P.p);
    });
    __syncwarp();
    for (int i = lane; i < 512; i += 32) {
      const int jl = q0 + (i >> 7);
      if (jl < nj * L)
        key[(((size_t)blockIdx.x * k + j) * L + jl) * 256 + comp * 128 + (i & 127)] =
            tile[(i >> 7) * kRow32 + row_word32(i & 127)];
    }
    __syncwarp();
  }
}

#define SHG_DISPATCH32(log_n, F) \
  switch (log_n) {               \
    case 12: F(12); break;       \
    case 13: F(13); break;       \
    case 14: F(14); break;       \
    case 15: F(15); break;       \
    default: break;              \
  }

template <int LOG_N, bool LZ>
void run_rows(const Ks32& ks, const uint32_t* D, uint32_t* E, int k, int L, int count,
              cudaStream_t s) {
  // Ciphertexts per CTA: four share every key load, while two CTAs' digit rows
  // still fit an SM; fewer when the batch has no more.
  // 192 threads where four CTAs' rows fit an SM, else 384 (two CTAs).
  auto smem = [&](int T, int NT) {
    return (rows32_digit_rows(k, T) + rows32_sum_rows(T, NT)) * kRow32 * 4 + 16 * kRowTw32;
  };
  constexpr int kFourPerSm = 56 * 1024, kTwoPerSm = 113 * 1024;
  auto go = [&](auto tt, auto nt) {
    constexpr int T = decltype(tt)::value, NT = decltype(nt)::value;
    auto kern = k32_rows<LOG_N, LZ, T, NT>;
    const int bytes = smem(T, NT);
    if (bytes > 48 * 1024)
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    const int groups = (count + T - 1) / T;
    launch_next(true, kern, 3 * (1 << (LOG_N - 7)) * groups, NT, bytes, s, D, ks.key, E, k, L,
                count, ks.w);
  };
  using N192 = std::integral_constant<int, 192>;
  using N384 = std::integral_constant<int, 384>;
  using T1 = std::integral_constant<int, 1>;
  using T2 = std::integral_constant<int, 2>;
  using T4 = std::integral_constant<int, 4>;
  if (count >= 3 && smem(4, 192) <= kFourPerSm)
    go(T4{}, N192{});
  else if (count >= 3 && smem(4, 384) <= kTwoPerSm)
    go(T4{}, N384{});
  else if (count >= 2 && smem(2, 192) <= kFourPerSm)
    go(T2{}, N192{});
  else
    go(T1{}, N192{});
}

}  // namespace

void launch_ks32(const CtxDev& c, const Ks32& ks, uint64_t* scratch, const uint64_t* X,
                 const DigitDesc* digits, int k, uint64_t* out, const uint64_t* base,
                 size_t base_ct_elems, CtMap map, int base1_zero, int subst_power, int count,
                 int L, cudaStream_t s) {
  const size_t n = (size_t)1 << c.log_n;
  // D, and once it has been read the 64-bit sums, then E.
  uint32_t* D = reinterpret_cast<uint32_t*>(scratch);
  uint64_t* Y = scratch;
  uint32_t* E = reinterpret_cast<uint32_t*>(
      reinterpret_cast<uint8_t*>(scratch) + ks32_digit_bytes(k, L) * n * count);
  {
    LaunchScope scope_("ks32_digits", s);
#define F(LN)                                                                          \
  {                                                                                    \
    using G = K32<LN>;                                                                 \
    /* one CTA per limb tile while that fills the GPU, else one per prime, else one */ \
    /* per prime and digit */                                                          \
    const long long ctas = (long long)count * L * G::TILES;                            \
    const int split = ctas >= 4LL * c.sms ? 1 : (ctas * 3 >= 2LL * c.sms ? 3 : 9);     \
    auto kern = ks.lazy ? k32_digit_cols<LN, LN <= 14> : k32_digit_cols<LN, false>;    \
    launch_next(c.follows, kern, (int)(ctas * split), G::THREADS, 0, s, X, digits, \
                ks.first, k, L, split, D, ks.w);                                       \
  }
    SHG_DISPATCH32(c.log_n, F)
#undef F
  }
  {
    LaunchScope scope_("ks32_rows", s);
#define F(LN)                                           \
  if (ks.lazy)                                          \
    run_rows<LN, LN <= 14>(ks, D, E, k, L, count, s);   \
  else                                                  \
    run_rows<LN, false>(ks, D, E, k, L, count, s);
    SHG_DISPATCH32(c.log_n, F)
#undef F
  }
  {
    LaunchScope scope_("ks32_crt", s);
#define F(LN)                                                                         \
  {                                                                                   \
    using S = Ntt4<LN>;                                                               \
    auto kern = ks.lazy ? k32_crt_cols<LN, LN <= 14> : k32_crt_cols<LN, false>;       \
    launch_next(true, kern, count * 2 * L * S::COL_TILES, S::COL_THREADS, 0, s, E, ks.crt, L, Y, \
                ks.w, c);                                                             \
  }
    SHG_DISPATCH32(c.log_n, F)
#undef F
  }
  LaunchScope scope_("ks32_out", s);
  launch4_rows_add(c, Y, out, base, base_ct_elems, map, base1_zero, subst_power, count, L, s);
}

void launch_ks32_key(const CtxDev& c, const W32& w, const uint64_t* rows, uint32_t* tmp, int j,
                     int nj, int k, int L, int comp, uint32_t* key, cudaStream_t s) {
  LaunchScope scope_("ks32_key", s);
  g_launch_count++;  // second phase kernel
#define F(LN)                                                                          \
  {                                                                                    \
    k32_key_cols<LN><<<nj * L * K32<LN>::TILES, K32<LN>::THREADS, 0, s>>>(rows, L, tmp, w, c); \
    k32_key_rows<LN><<<3 * (1 << (LN - 7)), 128, 0, s>>>(tmp, j, nj, k, L, comp, key, w); \
  }
  SHG_DISPATCH32(c.log_n, F)
#undef F
}

unsigned take_debug_word_ks32() {
  unsigned v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, g_shg_dbg, sizeof(v)) != cudaSuccess) return 0;
  if (v) cudaMemcpyToSymbol(g_shg_dbg, &z, sizeof(z));
  return v;
}

}  // namespace shg
