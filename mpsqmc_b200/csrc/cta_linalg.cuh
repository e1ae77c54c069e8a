// CTA-cooperative FP64 dense linear algebra for the walker kernels (sm_100a).
//
// All matrices are column-major with an explicit leading dimension and may live in shared or
// global memory (generic pointers).  Every routine is called by all threads of the CTA and
// returns without a trailing barrier unless stated; callers place __syncthreads() between
// dependent calls.
//
// FP64 products use the tensor-core DMMA instructions (mma.sync .f64; tcgen05 has no f64 kind, so
// this is Blackwell's FP64 tensor path).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace mq {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxWarps = 16;  // of the QR-free FP64 sweep (any power of two of threads up to 512)

// Operand of a grouped product: element (x, k) of group g and K block kb at
// p[x*ix + k*ik + g*sg + kb*sk] (x: a row of the left, a column of the right factor).
template <typename T>
struct Mat {
  const T *p;
  int ix, ik;
  long sg, sk;
};
template <typename T, bool K>
struct MatK : Mat<T> {};  // K: k contiguous (ik == 1)
template <typename T>
__device__ __forceinline__ MatK<T, false> cols(const T *p, int ld, long sg = 0, long sk = 0) {  // [x + ld k]
  return {{p, 1, ld, sg, sk}};
}
template <typename T>
__device__ __forceinline__ MatK<T, true> rows(const T *p, int ld, long sg = 0, long sk = 0) {  // [k + ld x]
  return {{p, ld, 1, sg, sk}};
}

// A grouped product as the CTA's warps read it: each warp keeps its own copy in shared memory.  As
// function arguments the thirty words would live in registers beside the fragments and be spilled;
// from here a warp takes them when it sets up a tile.
template <typename T>
struct alignas(16) GemmOpT {
  const T *a, *b;
  T *c;
  int M, N, K, GM, GN, GK;
  int aix, aik, bix, bik;
  int ldc, ca, cb, beta;
  long asg, ask, bsg, bsk;
};
using GemmOp = GemmOpT<double>;
template <typename T = double>
__device__ __forceinline__ GemmOpT<T> *warp_op() {
  __shared__ GemmOpT<T> ops[kMaxWarps];
  return ops + (threadIdx.x >> 5);
}
constexpr int kOpBytes = kMaxWarps * sizeof(GemmOp);  // static shared memory of every kernel with products
template <typename T, bool KA, bool KB>
__device__ __forceinline__ void set_op(int M, int N, int K, const MatK<T, KA> &A, int GM, const MatK<T, KB> &B,
                                       int GN, int GK, bool beta, T *C, int ldc, int ca, int cb) {
  __syncwarp();
  *warp_op<T>() = GemmOpT<T>{A.p, B.p, C,  M,   N,  K,  GM,   GN,   GK,   A.ix, A.ik,
                       B.ix, B.ik, ldc, ca, cb, beta, A.sg, A.sk, B.sg, B.sk};
  __syncwarp();
}

// Quotient and remainder of a by b where the quotient is small, by subtraction (an integer division
// costs more than the few rounds).
__device__ __forceinline__ int take_out(int &a, int b) {
  int q = 0;
#pragma unroll 1
  while (a >= b) {
    a -= b;
    ++q;
  }
  return q;
}
// mma.sync m8n8k4 .f64.  Fragments (PTX ISA), g = lane >> 2, t = lane & 3: A[g][t], B[t][g],
// D[g][2t], D[g][2t + 1].
__device__ __forceinline__ void dmma884(double &d0, double &d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// Output tiles of a grouped FP64 product, for every (ga < GM, gb < GN):
//   sum_{kb < GK} sum_{k < K} A(ga, kb)[m, k] B(gb, kb)[k, n],   m < M, n < N,
// handed to epi.put(ga, gb, m, n, v, w, two): v of row m and (two) w of row m + 1.  KA, KB: k is
// contiguous in A, in B (ik == 1).  A warp owns a tile of 16 rows (of one left group) by NP
// 8-column pieces (16-column blocks of any right groups; one piece of 8 when NP == 1).
//
// What bounds it is the FP64 tensor pipe (64 FMA per clock and SM) once a warp gets by with few
// instructions besides its DMMAs: a warp's dependent instructions issue every four to five cycles,
// and four warps share a scheduler.  So the loads are 16 bytes wide wherever the operands are
// aligned (V): the MMA's row, column and k slots are dealt out so that a lane's two rows (2g,
// 2g+1), its columns in two neighbouring pieces (2g, 2g+1) or its two k (2t, 2t+1) are adjacent
// in memory.  With leading dimensions of 4 mod 8 the k-contiguous shared-memory reads are free of
// bank conflicts.  The left factor, which may come from L2, is loaded a chunk of eight k ahead.
// Rows and columns beyond M, N read a valid neighbour and are not handed out; a last partial chunk
// is read element by element, masked.
// The tile of an element depends on M, N, GM, GN only: two calls with the same ones may
// accumulate into the same output without a barrier.
template <int NP, bool KA, bool KB, bool V, class Epi>
__device__ __forceinline__ void dmma_tiles(const volatile GemmOp &op, Epi &epi) {
  constexpr bool kPair = KA || KB;            // a lane's two k: 2t, 2t+1 (else t, t+4)
  constexpr int kNext = kPair ? 1 : 4, kW = NP == 1 ? 8 : 16, kBlk = NP == 1 ? 1 : NP / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3, kl = kPair ? 2 * t : t;
  int mt, tiles, per, span;
  {
    const int n1 = (op.N + kW - 1) / kW, GN = op.GN;
    mt = op.GM * ((op.M + 15) >> 4);
    // blocks are dealt out from all right groups in a row, or (kOneGroup) group by group
    span = Epi::kOneGroup ? n1 : GN * n1;
    per = (span + kBlk - 1) / kBlk;
    tiles = mt * per * (Epi::kOneGroup ? GN : 1);
  }
  int mi = warp, ti = 0;
#pragma unroll 1
  for (int tile = warp; tile < tiles; tile += nw, mi += nw) {
    const int n1 = (op.N + kW - 1) / kW;
    ti += take_out(mi, mt);
    int m0 = mi, pi = ti;
    const int ga = take_out(m0, (op.M + 15) >> 4);
    m0 = (m0 << 4) + 2 * g;
    const int sp = Epi::kOneGroup ? take_out(pi, per) : 0;
    const int left = span - pi * kBlk;  // blocks from the tile's first on
    int p0 = pi * kBlk;
    const int gb0 = Epi::kOneGroup ? sp : take_out(p0, n1);
    double acc[NP][4];
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
#pragma unroll 1
    for (int kb = 0; kb < op.GK; ++kb) {
      const int K = op.K, full = K >> 3, aik = KA ? 1 : op.aik, bik = KB ? 1 : op.bik;
      // row 2g and, where rows are not contiguous, 2g + 1
      const double *pa0, *pa1;
      {
        const int M1 = op.M - 1, aix = op.aix;
        const int r0 = (KA || !V) ? min(m0, M1) : min(m0, M1 & ~1);
        pa0 = op.a + (ga * op.asg + kb * op.ask + (long)r0 * aix + kl * aik);
        pa1 = (KA || !V) ? pa0 + (long)(min(m0 + 1, M1) - r0) * aix : pa0 + kNext * aik;
      }
      const double *pb[NP];
      {
        const double *b0 = op.b + (kb * op.bsk + kl * bik);
        const int N1 = op.N - 1, bix = op.bix;
        const long bsg = op.bsg;
        int gb = gb0, pc = p0;
#pragma unroll
        for (int j = 0; j < kBlk; ++j) {
          const double *bg = b0 + gb * bsg;
          if (NP == 1) {
            pb[0] = bg + (long)min(pc * 8 + g, N1) * bix;
          } else if (KB || !V) {
            pb[2 * j] = bg + (long)min(pc * 16 + 2 * g, N1) * bix;
            pb[2 * j + 1] = bg + (long)min(pc * 16 + 2 * g + 1, N1) * bix;
          } else {  // the column pair at this lane's first and second k
            pb[2 * j] = bg + min(pc * 16 + 2 * g, N1 & ~1);
            pb[2 * j + 1] = pb[2 * j] + kNext * bik;
          }
          if (j + 1 < left && ++pc == n1) {
            pc = 0;
            ++gb;
          }
        }
      }
      double a[4], an[4], b[NP][2];  // a: [row 2g, 2g+1] at the first k, then at the second
      auto load_a = [&](double (&x)[4]) {
        if (V) {
          const double2 u = *reinterpret_cast<const double2 *>(pa0), v = *reinterpret_cast<const double2 *>(pa1);
          x[0] = u.x;
          x[3] = v.y;
          x[KA ? 2 : 1] = u.y;
          x[KA ? 1 : 2] = v.x;
        } else {
          x[0] = pa0[0];
          x[1] = pa1[0];
          x[2] = pa0[kNext * aik];
          x[3] = pa1[kNext * aik];
        }
        pa0 += 8 * aik;
        pa1 += 8 * aik;
      };
      auto load_b = [&]() {
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if (V && (KB || NP > 1)) {
            const double2 u = *reinterpret_cast<const double2 *>(pb[j]);
            b[KB ? j : (j & ~1)][KB ? 0 : (j & 1)] = u.x;
            b[KB ? j : (j | 1)][KB ? 1 : (j & 1)] = u.y;
          } else {
            b[j][0] = pb[j][0];
            b[j][1] = pb[j][kNext * bik];
          }
          pb[j] += 8 * bik;
        }
      };
      const bool i0 = (full << 3) + kl < K, i1 = (full << 3) + kl + kNext < K;  // this lane's k of the last chunk
      auto tail_a = [&](double (&x)[4]) {
        constexpr bool pairs = V && !KA;  // pa1 is the second k of row 2g, else the first k of row 2g + 1
        const bool odd = !pairs || m0 + 1 < op.M;
        x[0] = i0 ? pa0[0] : 0.0;
        x[1] = i0 && odd ? (pairs ? pa0[1] : pa1[0]) : 0.0;
        x[2] = i1 ? (pairs ? pa1[0] : pa0[kNext * aik]) : 0.0;
        x[3] = i1 && odd ? (pairs ? pa1[1] : pa1[kNext * aik]) : 0.0;
      };
      auto tail_b = [&]() {
        constexpr bool pairs = V && !KB && NP > 1;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          const double *q = pairs ? pb[j & ~1] + (j & 1) : pb[j];
          b[j][0] = i0 ? q[0] : 0.0;
          b[j][1] = i1 ? q[kNext * bik] : 0.0;
        }
      };
      auto mma = [&]() {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < NP; ++j) {
            dmma884(acc[j][0], acc[j][1], a[2 * h], b[j][h]);
            dmma884(acc[j][2], acc[j][3], a[2 * h + 1], b[j][h]);
          }
      };
      if (full > 0) load_a(a);
#pragma unroll 1
      for (int c = 1; c < full; ++c) {
        load_b();
        load_a(an);
        mma();
#pragma unroll
        for (int q = 0; q < 4; ++q) a[q] = an[q];
      }
      if (full > 0) {
        load_b();
        mma();
      }
      if (K & 7) {
        tail_a(a);
        tail_b();
        mma();
      }
    }
    const int M = op.M, N = op.N;
    if (m0 < M) {
      const bool two = m0 + 1 < M;
      int gb = gb0, pc = p0;
#pragma unroll
      for (int j = 0; j < kBlk; ++j)
        if (j < left) {
          if (NP == 1) {
            const int n = pc * 8 + 2 * t;
            if (n < N) epi.put(ga, gb, m0, n, acc[0][0], acc[0][2], two);
            if (n + 1 < N) epi.put(ga, gb, m0, n + 1, acc[0][1], acc[0][3], two);
          } else {
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
              for (int h = 0; h < 2; ++h) {  // slot 2t + e of piece h: column 2 (2t + e) + h
                const int n = pc * 16 + 4 * t + 2 * e + h;
                if (n < N) epi.put(ga, gb, m0, n, acc[2 * j + h][e], acc[2 * j + h][2 + e], two);
              }
          }
          epi.block();
          if (++pc == n1) {
            pc = 0;
            ++gb;
          }
        }
    }
    if (Epi::kOneGroup) epi.done(ga, sp);
  }
}

// Pieces per tile: the wider tiles where they still give every warp one.  A CTA of kMaxWarps warps has its
// SM to itself, and nothing fills the warps that wait for a last round of tiles: there the pieces
// take the fewest rounds, a tile's work being its pieces and one more (its set-up and left factor):
// four for more blocks than warps, but for 33 to 48 blocks two (three rounds of 3, not two of 5); two
// for more than half as many (one round of 3, not two of 2).  Measured (ms a step, few walkers): 6x6
// lattice, 64/48, 20 walkers 26.2, now 19.4; two rows of 8, 96/48, 148 walkers 9.4, now 8.6.
template <typename T>
__device__ __forceinline__ int tile_pieces(const volatile GemmOpT<T> &op) {
  const int N = op.N, blocks = op.GM * ((op.M + 15) >> 4) * op.GN * ((N + 15) >> 4), nw = blockDim.x >> 5;
  const bool alone = std::is_same<T, double>::value && nw == kMaxWarps;  // (the TF32 sweep has eight warps)
  if (alone ? blocks > kMaxWarps && (unsigned)(blocks - 2 * kMaxWarps - 1) >= (unsigned)kMaxWarps : blocks >= 2 * nw) return 4;
  return blocks >= (alone ? kMaxWarps / 2 + 1 : nw) && N > 8 ? 2 : 1;
}

// One function per tile shape: together in one body they share what can be computed in front of the
// choice, and the registers that takes push fragments to local memory.
template <int NP, bool KA, bool KB, bool V, class Epi>
static __device__ __noinline__ void run_tiles(double *red) {
  const volatile GemmOp &op = *warp_op();
  Epi epi(op, red);
  dmma_tiles<NP, KA, KB, V>(op, epi);
}
template <bool KA, bool KB, class Epi>
__device__ __forceinline__ void dmma_groups(double *red = nullptr) {
  const volatile GemmOp &op = *warp_op();
  const int np = tile_pieces(op);
  // pairs are 16-byte aligned: even strides and an even base
  const long odd = (KA ? op.aix : op.aik) | op.asg | op.ask | (KB ? op.bix : op.bik) | op.bsg | op.bsk;
  const uintptr_t at = reinterpret_cast<uintptr_t>(op.a) | reinterpret_cast<uintptr_t>(op.b);
  if (!(odd & 1) && !(at & 15)) {
    if (np == 4) run_tiles<4, KA, KB, true, Epi>(red);
    else if (np == 2) run_tiles<2, KA, KB, true, Epi>(red);
    else run_tiles<1, KA, KB, true, Epi>(red);
  } else {
    if (np == 4) run_tiles<4, KA, KB, false, Epi>(red);
    else if (np == 2) run_tiles<2, KA, KB, false, Epi>(red);
    else run_tiles<1, KA, KB, false, Epi>(red);
  }
}

template <typename T>
struct alignas(2 * sizeof(T)) Pair {
  T x, y;
};
template <typename T>
struct StoreEpi {
  static constexpr bool kOneGroup = false;
  const volatile GemmOpT<T> &op;
  __device__ __forceinline__ StoreEpi(const volatile GemmOpT<T> &o, double *) : op(o) {}
  __device__ __forceinline__ void put(int ga, int gb, int m, int n, T v, T w, bool two) {
    const int ldc = op.ldc, ca = op.ca, cb = op.cb;
    const bool beta = op.beta,
               wide = ((ldc | ca | cb) & 1) == 0 && (reinterpret_cast<uintptr_t>(op.c) & (2 * sizeof(T) - 1)) == 0;
    T *c = op.c + ((long)ga * ca + (long)gb * cb + m + (long)ldc * n);
    if (wide && two) {  // row pairs are aligned
      Pair<T> x{v, w};
      if (beta) {
        const Pair<T> y = *reinterpret_cast<const Pair<T> *>(c);
        x.x += y.x;
        x.y += y.y;
      }
      *reinterpret_cast<Pair<T> *>(c) = x;
    } else {
      c[0] = beta ? v + c[0] : v;
      if (two) c[1] = beta ? w + c[1] : w;
    }
  }
  __device__ __forceinline__ void block() {}
  __device__ __forceinline__ void done(int, int) {}
};

// C(ga, gb)[m + ldc n] = sum_kb A(ga, kb) B(gb, kb) + (beta ? C : 0), C(ga, gb) = C + ga*ca + gb*cb, of
// the warp's op.
template <bool KA, bool KB>
__device__ __forceinline__ void cta_gemm_groups() {
  dmma_groups<KA, KB, StoreEpi<double>>();
}

// The same product for small matrices, one output element per thread and round: a tile's set-up,
// some 300 dependent instructions, costs more than the products of up to 8 x 8 x 8 elements do this
// way (the bonds of the smallest walks, and the ends of every chain).
__host__ __device__ constexpr bool small_product(int M, int N, int K) { return M * N <= 512 && M * N * K <= 512; }
static_assert(!small_product(4096, 128, 4096), "the product of the sizes exceeds an int");
template <typename T>
static __device__ __noinline__ void cta_gemm_small() {
  const volatile GemmOpT<T> &op = *warp_op<T>();
  const int M = op.M, N = op.N, K = op.K, GM = op.GM, GK = op.GK, aik = op.aik, bik = op.bik;
  const int sm = 32 - __clz(M - 1), sn = 32 - __clz(N - 1);  // (N, M == 1: no bits)
  for (int e = threadIdx.x; e < (GM * op.GN) << (sm + sn); e += blockDim.x) {
    const int m = e & ((1 << sm) - 1), n = (e >> sm) & ((1 << sn) - 1);
    int ga = e >> (sm + sn);
    const int gb = take_out(ga, GM);
    if (m >= M || n >= N) continue;
    const T *a = op.a + (ga * op.asg + m * op.aix), *b = op.b + (gb * op.bsg + n * op.bix);
    T *c = op.c + (ga * op.ca + gb * op.cb + m + op.ldc * n);
    T sum = op.beta ? *c : T(0);
    for (int kb = 0; kb < GK; ++kb) {
#pragma unroll 4
      for (int k = 0; k < K; ++k) sum += a[k * aik] * b[k * bik];
      a += op.ask;
      b += op.bsk;
    }
    *c = sum;
  }
}

// ---------------------------------------------------------------------------------------------
// FP32 storage, TF32 tensor cores (the mixed-precision sweep)
//
// mma.sync.m16n8k8 .tf32 with FP32 accumulation.  Fragment layouts (PTX ISA, m16n8k8 .tf32),
// g = lane >> 2, t = lane & 3:
//   A (16x8, row):  a0 A[g][t], a1 A[g+8][t], a2 A[g][t+4], a3 A[g+8][t+4]
//   B (8x8, col):   b0 B[t][g], b1 B[t+4][g]
//   C/D (16x8):     c0 C[g][2t], c1 C[g][2t+1], c2 C[g+8][2t], c3 C[g+8][2t+1]
// NP = 1: operands rounded to TF32 (10-bit mantissa) once.  NP = 3: each operand split into a
// TF32 head and a TF32 tail, three products (tail*head + head*tail + head*head), which carries
// the FP32 operands' precision through the tensor cores.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tf32_bits(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// x = head + tail, both TF32 (NP == 1: head alone)
template <int NP>
__device__ __forceinline__ void tf32_split(float x, uint32_t &head, uint32_t &tail) {
  head = tf32_bits(x);
  if (NP == 3) tail = tf32_bits(x - __uint_as_float(head));
}

// The FP32 counterpart of dmma_tiles: the same tiles (16 rows by NP 8-column pieces) and epilogues, K in
// chunks of 16 (two MMAs deep).  A lane's four k of a chunk are 4t .. 4t + 3 and its two rows 2g, 2g + 1,
// so that k-contiguous operands are read 16 bytes and row- or column-contiguous ones 8 bytes at a
// time (VA, VB: where the operand's strides and base allow it; a trial of bonds that are no
// multiples of four does not).  What bounds it is instructions: an element that is loaded is split
// into head and tail (PASSES == 3) for every tile it is part of, so a tile is as wide as
// leaves every warp one; the left factor, which may come from L2, is loaded a chunk ahead.
// Each chunk is summed in accumulators of its own, the small products first, and these are then added
// up in FP32: the tensor cores' sums truncate, and a chain over all of K costs accuracy.  Measured on
// the L = 64 chain (D_T = 64, D_W = 32, 1,024 walkers): 25.2 ms a step with 16x16 blocks, one
// 4-byte load per element and one chain over K, 20.7 ms with these tiles (19.6 ms with the reads of
// the elementwise loops in flight together).  Error against 64 bits on one population: 8.2e-6 before,
// 1.1e-5 with the long chain, 5.5e-6 as it is; on another 8.2e-7 before and 7.5e-7 as it is.
template <int PASSES, int NP, bool KA, bool KB, bool VA, bool VB, class Epi>
__device__ __forceinline__ void tf32_tiles(const volatile GemmOpT<float> &op, Epi &epi) {
  constexpr int kW = NP == 1 ? 8 : 16, kBlk = NP == 1 ? 1 : NP / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3, kl = 4 * t;
  int mt, tiles, per, span;
  {
    const int n1 = (op.N + kW - 1) / kW, GN = op.GN;
    mt = op.GM * ((op.M + 15) >> 4);
    span = Epi::kOneGroup ? n1 : GN * n1;
    per = (span + kBlk - 1) / kBlk;
    tiles = mt * per * (Epi::kOneGroup ? GN : 1);
  }
  int mi = warp, ti = 0;
#pragma unroll 1
  for (int tile = warp; tile < tiles; tile += nw, mi += nw) {
    const int n1 = (op.N + kW - 1) / kW;
    ti += take_out(mi, mt);
    int m0 = mi, pi = ti;
    const int ga = take_out(m0, (op.M + 15) >> 4);
    m0 = (m0 << 4) + 2 * g;
    const int sp = Epi::kOneGroup ? take_out(pi, per) : 0;
    const int left = span - pi * kBlk;  // blocks from the tile's first on
    int p0 = pi * kBlk;
    const int gb0 = Epi::kOneGroup ? sp : take_out(p0, n1);
    float sum[NP][4];
#pragma unroll
    for (int j = 0; j < NP; ++j) sum[j][0] = sum[j][1] = sum[j][2] = sum[j][3] = 0.f;
#pragma unroll 1
    for (int kb = 0; kb < op.GK; ++kb) {
      const int K = op.K, full = K >> 4, aik = KA ? 1 : op.aik, bik = KB ? 1 : op.bik;
      const float *pa0, *pa1;  // row 2g and row 2g + 1 (pairs of rows: pa0 alone)
      {
        const int M1 = op.M - 1, aix = op.aix;
        const int r0 = (KA || !VA) ? min(m0, M1) : min(m0, M1 & ~1);
        pa0 = op.a + (ga * op.asg + kb * op.ask + (long)r0 * aix + kl * aik);
        pa1 = pa0 + (long)(min(m0 + 1, M1) - r0) * aix;
      }
      const float *pb[NP];
      {
        const float *b0 = op.b + (kb * op.bsk + kl * bik);
        const int N1 = op.N - 1, bix = op.bix;
        const long bsg = op.bsg;
        int gb = gb0, pc = p0;
#pragma unroll
        for (int j = 0; j < kBlk; ++j) {
          const float *bg = b0 + gb * bsg;
          if (NP == 1) {
            pb[0] = bg + (long)min(pc * 8 + g, N1) * bix;
          } else if (KB || !VB) {
            pb[2 * j] = bg + (long)min(pc * 16 + 2 * g, N1) * bix;
            pb[2 * j + 1] = bg + (long)min(pc * 16 + 2 * g + 1, N1) * bix;
          } else {  // the column pair
            pb[2 * j] = pb[2 * j + 1] = bg + min(pc * 16 + 2 * g, N1 & ~1);
          }
          if (j + 1 < left && ++pc == n1) {
            pc = 0;
            ++gb;
          }
        }
      }
      float a[4][2], an[4][2], b[NP][4];  // a[k][row], b[piece][k]
      auto load_a = [&](float (&x)[4][2]) {
        if constexpr (VA && KA) {
          const float4 u = *reinterpret_cast<const float4 *>(pa0), v = *reinterpret_cast<const float4 *>(pa1);
          x[0][0] = u.x;
          x[1][0] = u.y;
          x[2][0] = u.z;
          x[3][0] = u.w;
          x[0][1] = v.x;
          x[1][1] = v.y;
          x[2][1] = v.z;
          x[3][1] = v.w;
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if constexpr (VA) {
              const float2 u = *reinterpret_cast<const float2 *>(pa0 + k * aik);
              x[k][0] = u.x;
              x[k][1] = u.y;
            } else {
              x[k][0] = pa0[k * aik];
              x[k][1] = pa1[k * aik];
            }
          }
        }
        pa0 += 16 * aik;
        pa1 += 16 * aik;
      };
      auto load_b = [&]() {
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if constexpr (VB && KB) {
            const float4 u = *reinterpret_cast<const float4 *>(pb[j]);
            b[j][0] = u.x;
            b[j][1] = u.y;
            b[j][2] = u.z;
            b[j][3] = u.w;
          } else if constexpr (VB && NP > 1) {
            if (!(j & 1)) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 u = *reinterpret_cast<const float2 *>(pb[j] + k * bik);
                b[j][k] = u.x;
                b[j | 1][k] = u.y;
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) b[j][k] = pb[j][k * bik];
          }
          pb[j] += 16 * bik;
        }
      };
      const int kt = K - (full << 4) - kl;  // how many of this lane's four k the last chunk has
      auto tail_a = [&](float (&x)[4][2]) {
        constexpr bool pairs = VA && !KA;
        const bool odd = !pairs || m0 + 1 < op.M;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x[k][0] = k < kt ? pa0[k * aik] : 0.f;
          x[k][1] = k < kt && odd ? (pairs ? pa0[k * aik + 1] : pa1[k * aik]) : 0.f;
        }
      };
      auto tail_b = [&]() {
        constexpr bool pairs = VB && !KB && NP > 1;
#pragma unroll
        for (int j = 0; j < NP; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) b[j][k] = k < kt ? pb[j][k * bik + (pairs ? j & 1 : 0)] : 0.f;
      };
      auto mma = [&]() {
        float acc[NP][4];
#pragma unroll
        for (int j = 0; j < NP; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
        uint32_t ah[2][4], at[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 4; ++q) tf32_split<PASSES>(a[2 * h + (q >> 1)][q & 1], ah[h][q], at[h][q]);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          uint32_t bh[4], bt[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) tf32_split<PASSES>(b[j][q], bh[q], bt[q]);
          if (PASSES == 3) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              mma_tf32(acc[j], at[h][0], at[h][1], at[h][2], at[h][3], bh[2 * h], bh[2 * h + 1]);
              mma_tf32(acc[j], ah[h][0], ah[h][1], ah[h][2], ah[h][3], bt[2 * h], bt[2 * h + 1]);
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) mma_tf32(acc[j], ah[h][0], ah[h][1], ah[h][2], ah[h][3], bh[2 * h], bh[2 * h + 1]);
        }
#pragma unroll
        for (int j = 0; j < NP; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) sum[j][q] += acc[j][q];
      };
      if (full > 0) load_a(a);
#pragma unroll 1
      for (int c = 1; c < full; ++c) {
        load_b();
        load_a(an);
        mma();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a[k][0] = an[k][0];
          a[k][1] = an[k][1];
        }
      }
      if (full > 0) {
        load_b();
        mma();
      }
      if (K & 15) {
        tail_a(a);
        tail_b();
        mma();
      }
    }
    const int M = op.M, N = op.N;
    if (m0 < M) {
      const bool two = m0 + 1 < M;
      int gb = gb0, pc = p0;
#pragma unroll
      for (int j = 0; j < kBlk; ++j)
        if (j < left) {
          if (NP == 1) {
            const int n = pc * 8 + 2 * t;
            if (n < N) epi.put(ga, gb, m0, n, sum[0][0], sum[0][2], two);
            if (n + 1 < N) epi.put(ga, gb, m0, n + 1, sum[0][1], sum[0][3], two);
          } else {
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int n = pc * 16 + 4 * t + 2 * e + h;
                if (n < N) epi.put(ga, gb, m0, n, sum[2 * j + h][e], sum[2 * j + h][2 + e], two);
              }
          }
          epi.block();
          if (++pc == n1) {
            pc = 0;
            ++gb;
          }
        }
    }
    if (Epi::kOneGroup) epi.done(ga, sp);
  }
}

template <int PASSES, int NP, bool KA, bool KB, bool VA, bool VB, class Epi>
static __device__ __noinline__ void run_tf32(double *red) {
  const volatile GemmOpT<float> &op = *warp_op<float>();
  Epi epi(op, red);
  tf32_tiles<PASSES, NP, KA, KB, VA, VB>(op, epi);
}
template <int PASSES, bool KA, bool KB, class Epi>
__device__ __forceinline__ void tf32_groups(double *red = nullptr) {
  const volatile GemmOpT<float> &op = *warp_op<float>();
  const int np = tile_pieces(op);
  // an operand's quadruples of k are 16-byte aligned, its pairs of rows or columns 8-byte aligned
  const bool va = !(((KA ? op.aix : op.aik) | op.asg | op.ask) & 3) && !(reinterpret_cast<uintptr_t>(op.a) & 15);
  const bool vb = !(((KB ? op.bix : op.bik) | op.bsg | op.bsk) & 3) && !(reinterpret_cast<uintptr_t>(op.b) & 15);
  if (va && vb) {
    if (np == 4) run_tf32<PASSES, 4, KA, KB, true, true, Epi>(red);
    else if (np == 2) run_tf32<PASSES, 2, KA, KB, true, true, Epi>(red);
    else run_tf32<PASSES, 1, KA, KB, true, true, Epi>(red);
  } else if (vb) {
    if (np == 4) run_tf32<PASSES, 4, KA, KB, false, true, Epi>(red);
    else if (np == 2) run_tf32<PASSES, 2, KA, KB, false, true, Epi>(red);
    else run_tf32<PASSES, 1, KA, KB, false, true, Epi>(red);
  } else {
    if (np == 4) run_tf32<PASSES, 4, KA, KB, false, false, Epi>(red);
    else if (np == 2) run_tf32<PASSES, 2, KA, KB, false, false, Epi>(red);
    else run_tf32<PASSES, 1, KA, KB, false, false, Epi>(red);
  }
}

// Sixteen closures of two-site branch products, fused with the products that form them:
//   out[k + 4 (s + 2 t)] = sum_{m < M, n < N} (A_s B_t)[m, n] P_k[m, n],   s, t in {0, 1}, k < 4,
// A_s = A + s*sa (M x K, ld lda), B_t = B + t*sb (K x N, ld ldb), P_k = P + k*sp (ld ldp).  The
// products are never stored: a warp dots its tile with the four P tiles in the epilogue and adds
// to its own column of red (16 doubles per warp).  Ends with a barrier.
template <typename T>
struct ClosureEpi {
  static constexpr bool kOneGroup = true;
  const volatile GemmOpT<T> &op;  // c: P, ldc: its leading dimension, ca: its block stride
  double *red;                    // of this warp
  double w[4];
  float x[4];                     // FP32: the sums of one block, before they join w
  __device__ __forceinline__ ClosureEpi(const volatile GemmOpT<T> &o, double *r) : op(o), red(r), w{0.0, 0.0, 0.0, 0.0}, x{0.f, 0.f, 0.f, 0.f} {}
  __device__ __forceinline__ void put(int, int, int m, int n, T v, T v1, bool two) {
    const T *pp = op.c + m + (long)op.ldc * n;
    const int sp = op.ca;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      auto &at = [&]() -> auto & {
        if constexpr (std::is_same<T, double>::value) return w[k];
        else return x[k];
      }();
      at += v * pp[(long)k * sp];
      if (two) at += v1 * pp[(long)k * sp + 1];
    }
  }
  __device__ __forceinline__ void block() {
    if constexpr (!std::is_same<T, double>::value) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[k] += (double)x[k];
        x[k] = 0.f;
      }
    }
  }
  __device__ __forceinline__ void done(int s, int t) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      double v = w[k];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == k) red[(4 * (s + 2 * t) + k) * nw] += v;
      w[k] = 0.0;
    }
  }
};
// The warps' sums in red (16 per warp) added up.  Starts and ends with a barrier.
__device__ __forceinline__ void add_warps(const double *red, double *out) {
  const int nw = blockDim.x >> 5;
  __syncthreads();
  if (threadIdx.x < 16) {
    double sum = 0.0;
    for (int w = 0; w < nw; ++w) sum += red[threadIdx.x * nw + w];
    out[threadIdx.x] = sum;
  }
  __syncthreads();
}
template <typename T, int NP = 0>
static __device__ __forceinline__ void cta_closure_groups(double *red) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double *mine = red + (threadIdx.x >> 5);
  if (lane < 16) mine[lane * nw] = 0.0;
  __syncwarp();
  if constexpr (std::is_same<T, double>::value) dmma_groups<false, true, ClosureEpi<double>>(mine);
  else tf32_groups<NP, false, true, ClosureEpi<float>>(mine);
}
template <int NP = 0, typename T>
__device__ __forceinline__ void cta_closure16(int M, int N, int K, const T *A, int lda, int sa, const T *B, int ldb,
                                              int sb, T *P, int ldp, int sp, double *red, double *out) {
  set_op(M, N, K, cols(A, lda, sa), 2, rows(B, ldb, sb), 2, 1, false, P, ldp, sp, 0);
  cta_closure_groups<T, NP>(red);
  add_warps(red, out);
}

// Overloads that let the sweep be written once for FP64 (DMMA) and FP32 (TF32) work buffers.
template <int NP, bool KA, bool KB>
__device__ __forceinline__ void gemm_g(int M, int N, int K, const MatK<double, KA> &A, int GM, const MatK<double, KB> &B,
                                       int GN, int GK, bool beta, double *C, int ldc, long ca = 0, long cb = 0) {
  set_op(M, N, K, A, GM, B, GN, GK, beta, C, ldc, (int)ca, (int)cb);
  if (small_product(M, N, K)) cta_gemm_small<double>();
  else cta_gemm_groups<KA, KB>();
}
template <int NP, bool KA, bool KB>
__device__ __forceinline__ void gemm_g(int M, int N, int K, const MatK<float, KA> &A, int GM, const MatK<float, KB> &B,
                                       int GN, int GK, bool beta, float *C, int ldc, long ca = 0, long cb = 0) {
  set_op(M, N, K, A, GM, B, GN, GK, beta, C, ldc, (int)ca, (int)cb);
  if (small_product(M, N, K)) cta_gemm_small<float>();
  else tf32_groups<NP, KA, KB, StoreEpi<float>>();
}

// Sum of v over the CTA; result returned to every thread.  red: >= one double per warp of smem.
__device__ __forceinline__ double cta_sum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll 8
  for (int w = 0; w < nw; ++w) s += red[w];
  return s;
}

// Four sums at once (one pair of barriers).  red: >= four doubles per warp.
__device__ __forceinline__ void cta_sum4(double v[4], double *red) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < 4; ++q) red[q * nw + warp] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[q * nw + w];
    v[q] = s;
  }
}

// dlarfg's coefficients for a column with head alpha and squared tail norm xnorm2 > 0:
// beta = -sign(alpha) ||(alpha, x)||, tau = (beta - alpha) / beta, scale of the tail 1/(alpha - beta).
// FP64 square roots and divisions are long dependent sequences on this GPU, and this sits on the
// QR's critical path (once per column): one sqrt of alpha^2 + xnorm2 (no overflow at the
// magnitudes of normalised MPS tensors) and one division serve all three.
__device__ __forceinline__ void reflector_coeffs(double alpha, double xnorm2, double &beta, double &tau,
                                                 double &scale) {
  const double mag = sqrt(fma(alpha, alpha, xnorm2));
  beta = (alpha >= 0.0) ? -mag : mag;
  const double dd = alpha - beta;  // nonzero: |beta| > 0 and of opposite sign to alpha
  const double r = 1.0 / (beta * dd);
  tau = -dd * dd * r;               // (beta - alpha) / beta
  scale = beta * r;                 // 1 / (alpha - beta)
}

// Apply H = I - tau v v^T (v = (1, col[i+1..m)) stored below the diagonal of column i) to the
// columns j > i that this warp owns (j = warp mod kWarps), all of them at once: partial dot
// products for every owned column first, then one interleaved butterfly, then the updates.
// MAXC bounds the owned columns (n <= MAXC * kWarps).
template <int MAXC>
static __device__ __forceinline__ void warp_apply_reflector(int m, int n, int i, const double *col,
                                                            double tau, double *A, int lda) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = i + 1 + (((warp - (i + 1)) % kWarps) + kWarps) % kWarps;
  double part[MAXC], head[MAXC];
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int j = first + c * kWarps;
    part[c] = 0.0;
    head[c] = 0.0;
    if (j < n) {
      const double *cj = A + (long)lda * j;
      head[c] = cj[i];
      for (int r = i + 1 + lane; r < m; r += 32) part[c] += col[r] * cj[r];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < MAXC; ++c) part[c] += __shfl_xor_sync(0xffffffffu, part[c], o);
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int j = first + c * kWarps;
    if (j < n) {
      double *cj = A + (long)lda * j;
      const double f = tau * (part[c] + head[c]);
      for (int r = i + 1 + lane; r < m; r += 32) cj[r] -= f * col[r];
      if (lane == 0) cj[i] = head[c] - f;
    }
  }
  __syncwarp();
}

// Register-resident Householder QR (same conventions and results as cta_householder_qr below).
// Column j belongs to warp j % kWarps; the warp keeps rows lane + 32*q (q < RPL) of its columns
// (at most MAXC of them) in registers for the whole factorisation, so updates never go through
// shared memory.  Reflector vectors are published in A below the diagonal (and tau[]), one
// barrier per column in the factorisation; forming Q reads the published reflectors only and
// needs no barrier.  Requires m <= 32*RPL and n <= kWarps*MAXC.
template <int RPL, int MAXC>
static __device__ __noinline__ void cta_qr_reg(int m, int n, double *__restrict__ A, int lda,
                                               double *__restrict__ R, int ldr, double *__restrict__ tau) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned full = 0xffffffffu;
  double x[MAXC][RPL];
  __syncthreads();
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int j = warp + c * kWarps;
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const int r = lane + 32 * q;
      x[c][q] = (j < n && r < m) ? A[r + lda * j] : 0.0;
    }
  }
  // dgeqr2; ci: slot of column i in its owner's registers.  The slots are unrolled: picked at run time, a
  // column is copied through selects of all of them, and how many registers that moves differs from
  // one version of this file to the next (left-normalisation, L = 64, D_W = 32, 148 walkers: 2.85 ms,
  // 3.09 ms without a change here; unrolled 2.80 ms).
#pragma unroll
  for (int ci = 0; ci < MAXC; ++ci)
#pragma unroll 1
    for (int i = ci * kWarps; i < min(n, (ci + 1) * kWarps); ++i) {
      if (warp == i % kWarps) {
        double part = 0.0, alpha = 0.0;
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          const int r = lane + 32 * q;
          if (r > i && r < m) part += x[ci][q] * x[ci][q];
          if (r == i) alpha = x[ci][q];
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(full, part, o);
        alpha = __shfl_sync(full, alpha, i & 31);
        double ti = 0.0, beta = alpha, sc = 1.0;
        if (m - i > 1 && part > 0.0) reflector_coeffs(alpha, part, beta, ti, sc);
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          const int r = lane + 32 * q;
          if (r > i && r < m) {
            if (ti != 0.0) x[ci][q] *= sc;
            A[r + lda * i] = x[ci][q];  // published reflector below the diagonal
          }
          if (r == i) x[ci][q] = beta;
        }
        if (lane == 0) tau[i] = ti;
      }
      __syncthreads();
      const double ti = tau[i];
      if (ti != 0.0) {
        double v[RPL];
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          const int r = lane + 32 * q;
          v[q] = (r > i && r < m) ? A[r + lda * i] : (r == i ? 1.0 : 0.0);
        }
        double part[MAXC];
#pragma unroll
        for (int c = 0; c < MAXC; ++c) {
          part[c] = 0.0;
#pragma unroll
          for (int q = 0; q < RPL; ++q) part[c] += v[q] * x[c][q];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int c = 0; c < MAXC; ++c) part[c] += __shfl_xor_sync(full, part[c], o);
#pragma unroll
        for (int c = 0; c < MAXC; ++c) {
          const int j = warp + c * kWarps;
          if (j > i && j < n) {
            const double f = ti * part[c];
#pragma unroll
            for (int q = 0; q < RPL; ++q) x[c][q] -= f * v[q];
          }
        }
      }
    }
  // R: upper triangle of the reduced columns
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int j = warp + c * kWarps;
    if (j < n) {
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const int r = lane + 32 * q;
        if (r < n) R[r + ldr * j] = (r <= j) ? x[c][q] : 0.0;
      }
    }
  }
  // dorg2r: columns start as unit vectors, H_i applied for i = n-1 .. 0
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int j = warp + c * kWarps;
#pragma unroll
    for (int q = 0; q < RPL; ++q) x[c][q] = (lane + 32 * q == j) ? 1.0 : 0.0;
  }
  for (int i = n - 1; i >= 0; --i) {
    const double ti = tau[i];
    double v[RPL];
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const int r = lane + 32 * q;
      v[q] = (r > i && r < m) ? A[r + lda * i] : (r == i ? 1.0 : 0.0);
    }
    if (ti != 0.0) {
      double part[MAXC];
#pragma unroll
      for (int c = 0; c < MAXC; ++c) {
        part[c] = 0.0;
#pragma unroll
        for (int q = 0; q < RPL; ++q) part[c] += v[q] * x[c][q];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < MAXC; ++c) part[c] += __shfl_xor_sync(full, part[c], o);
#pragma unroll
      for (int c = 0; c < MAXC; ++c) {
        const int j = warp + c * kWarps;
        if (j > i && j < n) {
          const double f = ti * part[c];
#pragma unroll
          for (int q = 0; q < RPL; ++q) x[c][q] -= f * v[q];
        }
      }
    }
    // column i := H_i e_i
#pragma unroll
    for (int c = 0; c < MAXC; ++c) {
      const int j = warp + c * kWarps;
      if (j == i) {
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          const int r = lane + 32 * q;
          x[c][q] = (r > i) ? -ti * v[q] : (r == i ? 1.0 - ti : 0.0);
        }
      }
    }
  }
  __syncthreads();  // every warp has read the published reflectors
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int j = warp + c * kWarps;
    if (j < n) {
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const int r = lane + 32 * q;
        if (r < m) A[r + lda * j] = x[c][q];
      }
    }
  }
  __syncthreads();
}

// Householder QR of A (m x n, m >= n, ld lda, shared memory) in LAPACK's conventions
// (dgeqr2 + dorg2r, with dlarfg's beta = -sign(alpha)*||x||, tau = 0 when the column below the
// diagonal is zero or m - i == 1).  On exit A holds Q (m x n, orthonormal columns) and R
// (n x n, ld ldr, upper triangular) holds the triangular factor.  tau: >= n doubles of shared
// memory.  Starts and ends with a barrier.
//
// Column j belongs to warp j % kWarps for the whole factorisation: the owner builds reflector j
// and every warp applies published reflectors to its own columns, so one barrier per column
// and pass is enough (a warp updates its columns in program order).
static __device__ __noinline__ void cta_householder_qr(int m, int n, double *A, int lda, double *R, int ldr,
                                                double *tau) {
  if (m <= 64 && n <= 4 * kWarps) {
    cta_qr_reg<2, 4>(m, n, A, lda, R, ldr, tau);
    return;
  }
  if (m <= 128 && n <= 8 * kWarps) {
    cta_qr_reg<4, 8>(m, n, A, lda, R, ldr, tau);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned full = 0xffffffffu;
  __syncthreads();
  // dgeqr2
  for (int i = 0; i < n; ++i) {
    double *col = A + (long)lda * i;
    if (warp == i % kWarps) {
      double part = 0.0;
      for (int r = i + 1 + lane; r < m; r += 32) part += col[r] * col[r];
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(full, part, o);
      const double alpha = col[i];
      double ti = 0.0;
      if (m - i > 1 && part > 0.0) {
        double beta, sc;
        reflector_coeffs(alpha, part, beta, ti, sc);
        for (int r = i + 1 + lane; r < m; r += 32) col[r] *= sc;
        __syncwarp();
        if (lane == 0) col[i] = beta;
      }
      if (lane == 0) tau[i] = ti;
    }
    __syncthreads();
    const double ti = tau[i];
    if (ti != 0.0) {
      if (n <= 4 * kWarps) warp_apply_reflector<4>(m, n, i, col, ti, A, lda);
      else if (n <= 8 * kWarps) warp_apply_reflector<8>(m, n, i, col, ti, A, lda);
      else warp_apply_reflector<16>(m, n, i, col, ti, A, lda);
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < n * n; q += kThreads) {
    const int r = q % n, c = q / n;
    R[r + (long)ldr * c] = (r <= c) ? A[r + (long)lda * c] : 0.0;
  }
  __syncthreads();
  // dorg2r, k = n: Q = H_0 ... H_{n-1} applied to the first n unit columns
  for (int i = n - 1; i >= 0; --i) {
    const double *col = A + (long)lda * i;
    const double ti = tau[i];
    if (ti != 0.0 && i < n - 1) {
      if (n <= 4 * kWarps) warp_apply_reflector<4>(m, n, i, col, ti, A, lda);
      else if (n <= 8 * kWarps) warp_apply_reflector<8>(m, n, i, col, ti, A, lda);
      else warp_apply_reflector<16>(m, n, i, col, ti, A, lda);
    }
    __syncthreads();
    if (warp == i % kWarps) {
      double *ci = A + (long)lda * i;
      for (int r = lane; r < m; r += 32) {
        if (r > i) ci[r] *= -ti;
        else if (r == i) ci[r] = 1.0 - ti;
        else ci[r] = 0.0;
      }
    }
  }
  __syncthreads();
}

}  // namespace mq
