// gbdx_mlp_fm.cuh -- the MLP-field integrator on the fifth-generation tensor
// cores with the field's features on the accumulator's lanes.
//
// A group of 8 warps integrates a tile of R trajectories ("rows") in lockstep, as
// a CTA of mlp_fused_kernel does (gbdx_mlp.cuh: the same rows, controller and
// outputs); the G groups of a CTA share its weights and nothing else, and while
// one waits for its products the others compute.
// Each layer of the field is one product with the weights as the M operand,
//   acc[feature, (piece, row)] = W[feature, k] * x[k, (piece, row)],
// so that the 128 lanes of a tcgen05 accumulator are 128 features and a tile
// needs only as many columns as it has rows: 3 R, the three BF16 pieces of every
// activation side by side (gbdx_mlp.cuh: why three), each weight read once for
// all of them and the three column groups summed in FP32 when they are read
// back.  Tiles of 16 or 32 rows thus keep the tensor cores fed, where a tile with
// the trajectories on the lanes needs 128 rows and leaves most SMs without one.
// The weights stay on the SM for the launch.  A thread owns one feature and a
// run of rows, so it writes its part of the next operand as 16-byte runs (the
// MN-major layout) and its Runge--Kutta state stays in its registers.
//
// Lane maps.  Where a layer has fewer than 128 features its rows of W are stored
// 128 / features times, so every lane holds results and the copies split the
// tile's rows; the M = 128 product costs what an M = 64 one does.  At width 256
// the hidden layers are two 128-feature blocks, one after the other on the
// group's accumulator, and W0 and W1 are A operands in tensor memory (64 and 256
// of its columns): shared memory has no room for them beside two groups'
// operands.
//
// Tile size: a product takes ~46 cycles up to N = 48 (one thread's issue rate) and
// 49 (A in tensor memory) to 57 at N = 96, so 32 rows rather than 16; four groups
// of 16 rows and 4 warps measured 8700 cycles a stage of 64 rows at width 128
// against 6400 with two of 32 rows and 8 warps.
//
// Bound: the serial chain of a stage (three products, the waits for their completion and
// the reads of their sums, barriers of eight warps), which two groups overlap in part, and
// in it the epilogues' issue slots (~27 a warp and element: tanh, splitting and storing,
// sums; about 3500 of a stage's 6400 cycles with 64 rows at width 128).  Counters at 8192
// rows: issue slots 37 % (61 % on the fullest SM), tensor pipe 19 %, of 10.8 warp cycles an
// issue 2.4 on those reads and 2.3 on barriers; width 256, 16384 rows: 40 (59), 28 %, 2.7
// of 9.9 and 0.8.  Measured (Tsit5 PID(1e-5, 1e-7) on [0, 1], kernel
// time) against the mma.sync row tiles that it replaced: 64-128-128-64 at 8192 rows
// 421 -> 210 us, at 19456 902 -> 371 us (445 us with 128 trajectories on the lanes);
// 64-256-256-64 with 32 saves at 16384 rows 2240 -> 780 us.
//
// Reference semantics: diffrax/_integrate.py:302-885 and the files cited in
// gbdx_mlp.cuh.
#pragma once

#include "gbdx_f2.cuh"
#include "gbdx_f64i.cuh"
#include "gbdx_launch.h"
#include "gbdx_mlp.cuh"
#include "gbdx_tc.cuh"

namespace gbdx {

// Polls of a product's completion barrier before it counts as lost (a test's build sets
// another number), and of the one that says at the end that none is left in flight.
#ifndef GBDX_FM_POLLS
#define GBDX_FM_POLLS (1u << 22)
#endif
constexpr uint32_t kFmWait = GBDX_FM_POLLS, kFmDrain = 1u << 22;

template <int D_, int H_>
struct FmShape {
  static constexpr int D = D_, H = H_;
  static constexpr bool WIDE = H >= 256;            // W0, W1 in tensor memory, two blocks
  static constexpr int R = 32;                      // rows per tile
  static constexpr int GT = 256;                    // threads per group
  static constexpr int G = 2;                       // groups per CTA
  static constexpr int THREADS = G * GT;
  static constexpr int MB = H > 128 ? H / 128 : 1;  // 128-feature blocks of a hidden layer
  static constexpr int N = 3 * R;                   // accumulator columns of one product
  static constexpr int NE = R * D / GT;             // state elements per thread (one feature)
  static constexpr int HR = R * H / (GT * MB);      // rows per thread and hidden feature
  static constexpr int NPART = D / 32;              // error-norm partials per row
  static constexpr int TW0 = G * N, TW1 = TW0 + D;  // WIDE: the weights' TMEM columns
  static constexpr int TMEM_COLS = WIDE ? 512 : 256;
  static constexpr int MAX_SAVES = GT / R;          // ts saves of a row per pass
  // operand buffers: one, read whole before the next is written; WIDE: bufa (the
  // first hidden layer, then the second's upper half) and bufb (the stage input,
  // then the second's lower half)
  static constexpr int BUFA = N * H, BUFB = WIDE ? N * H / 2 : 0;
  static_assert(!WIDE || TW1 + H == TMEM_COLS, "tensor memory");
  static_assert(NE % 4 == 0 && HR % 8 == 0, "owned rows");
  // flat parameter offsets (FP32, row-major [out][in])
  static constexpr int OW0 = 0, OB0 = OW0 + H * D, OW1 = OB0 + H, OB1 = OW1 + H * H,
                       OW2 = OB1 + H, OB2 = OW2 + D * H;
};

template <int M, bool XO>
struct FmEvents {};
template <int M>
struct FmEvents<M, true> : RowEvents<M> {};

template <class SH, bool XO>
struct __align__(128) FmGroup {
  // the current operand, [k][(piece, row)]: a group of 8 (piece, row)s is K * 16
  // bytes.  Between products bufa holds the save weights (FmSaves) or the events'
  // scratch.
  __nv_bfloat16 bufa[SH::BUFA], bufb[SH::WIDE ? SH::BUFB : 8];
  alignas(16) RowState<SH::R> rows;
  float part[SH::R][2];  // the error norm's partial sums
  FmEvents<SH::R, XO> ev;
  uint64_t bar, drain;
  int err;  // a product of this group did not complete
};

template <class SH, bool XO>
struct __align__(128) FmSmem {
  __nv_bfloat16 w0[SH::WIDE ? 8 : 128 * SH::D], w1[SH::WIDE ? 8 : 128 * SH::H];
  __nv_bfloat16 w2[128 * SH::H];
  FmGroup<SH, XO> group[SH::G];
  uint32_t slot;
};

// Per row and save of one pass: the interpolant's weights at theta (Tsit5: of
// its seven stages; other solvers: theta itself in [7]).
template <class SH>
struct FmSaves {
  float w[SH::R][SH::MAX_SAVES][8];
  int n[SH::R];
};

// Barriers of one group.
__device__ __forceinline__ void fm_sync(int g) {
  asm volatile("bar.sync %0, 256;" :: "r"(g + 1) : "memory");
}
__device__ __forceinline__ int fm_sync_or(int g, int x) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, 256, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(x), "r"(g + 1) : "memory");
  return r;
}

// K-major copy of the BF16-rounded rows W[m % ROWS][0..K), m < STORED.  A group
// of 8 lanes writes one core matrix (128 contiguous bytes).
template <int ROWS, int STORED, int K>
__device__ __forceinline__ void fm_stage(__nv_bfloat16 *dst, const float *W, int tid, int nt,
                                         bool vec) {
#pragma unroll 4
  for (int i = tid; i < STORED * (K / 8); i += nt) {
    const int m = (i / (8 * (K / 8))) * 8 + (i & 7), k8 = (i >> 3) % (K / 8);
    const float *s = W + (m % ROWS) * K + 8 * k8;
    float v[8];
    if (vec) {
      *reinterpret_cast<float4 *>(v) = __ldg(reinterpret_cast<const float4 *>(s));
      *reinterpret_cast<float4 *>(v + 4) = __ldg(reinterpret_cast<const float4 *>(s) + 1);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = __ldg(s + j);
    }
    __nv_bfloat162 h[4];
#pragma unroll
    for (int j = 0; j < 4; j++) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(dst) +
                               tc::kmajor_offset(m, 8 * k8, K)) =
        *reinterpret_cast<const uint4 *>(h);
  }
}

// Rows W[row0 + lane of the accumulator][0..K) as an A operand in the TMEM columns
// from tcol on; called by the eight warps of a group, each set of four for half of K.
template <int K>
__device__ __forceinline__ void fm_stage_tmem(uint32_t tcol, const float *W, int t, bool vec) {
  const float *s = W + (t & 127) * K;
  const int c0 = (t >> 7) * (K / 2);
#pragma unroll 4
  for (int c = c0; c < c0 + K / 2; c += 8) {
    float v[8];
    if (vec) {
      *reinterpret_cast<float4 *>(v) = __ldg(reinterpret_cast<const float4 *>(s + c));
      *reinterpret_cast<float4 *>(v + 4) = __ldg(reinterpret_cast<const float4 *>(s + c) + 1);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = __ldg(s + c + j);
    }
    uint32_t h[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      h[j] = *reinterpret_cast<const uint32_t *>(&b);
    }
    tc::tmem_st4(tcol + c / 2, h);
  }
}

// v as three BF16 pieces, written as feature f's rows row0 .. row0 + 2 NP of a
// K-feature operand with R rows.
template <int R, int K, int NP>
__device__ __forceinline__ void fm_put(unsigned char *act, int f, int row0, const F2 (&v)[NP]) {
  uint32_t p[3][NP];
  auto pair = [](float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
  };
  // x minus the BF16 pair h
  auto rest = [](F2 x, uint32_t h) {
    return f2_fma(f2_pack(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)),
                  f2_set(-1.f), x);
  };
#pragma unroll
  for (int j = 0; j < NP; j++) {
    F2 x = v[j];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      float a, b;
      f2_unpack(x, a, b);
      p[q][j] = pair(a, b);
      if (q < 2) x = rest(x, p[q][j]);
    }
  }
  unsigned char *a = act + (f >> 3) * 128 + (f & 7) * 16 + (row0 >> 3) * (K * 16);
#pragma unroll
  for (int q = 0; q < 3; q++) {
    unsigned char *o = a + q * (R / 8) * (K * 16);
    if constexpr (NP == 4) {
      *reinterpret_cast<uint4 *>(o) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    } else {
      *reinterpret_cast<uint2 *>(o + (row0 & 4) * 2) = make_uint2(p[q][0], p[q][1]);
    }
  }
}

// acc[lane, column] (+)= A[128 x 16 KS] x[16 KS x N].  A in shared memory, or (TA)
// in tensor memory.
template <int N, int KS>
__device__ __forceinline__ void fm_issue(uint32_t acc, uint64_t da, uint64_t db) {
  constexpr uint32_t id = tc::idesc_bf16_f32(128, N, false, true);
#pragma unroll
  for (int k = 0; k < KS; k++) tc::mma_bf16(acc, da + 16u * k, db + 16u * k, id, k > 0 ? 1u : 0u);
}
template <int N, int KS>
__device__ __forceinline__ void fm_issue_ta(uint32_t acc, uint32_t ta, uint64_t db) {
  constexpr uint32_t id = tc::idesc_bf16_f32(128, N, false, true);
#pragma unroll
  for (int k = 0; k < KS; k++)
    tc::mma_bf16_ta(acc, ta + 8u * k, db + 16u * k, id, k > 0 ? 1u : 0u);
}

// What thread t of a group owns.  Its warps 0..3 and 4..7 each cover the 128 lanes
// of the accumulators (tl) and split the rows.
template <class SH>
struct FmMap {
  int t, tl;
  int f, row0;      // state: feature and first of NE rows
  int hf, hrow0;    // hidden layers: (first) feature and first of HR rows
  uint32_t acc;     // TMEM address of the group's accumulator, column 0 of lane 0
  uint32_t lanes;   // the same of the warp's lane group
  __device__ FmMap(int t_, uint32_t acc_) : t(t_), tl(t_ & 127), acc(acc_) {
    lanes = acc + (uint32_t(tl & 96) << 16);
    f = tl & (SH::D - 1);
    row0 = (t / SH::D) * SH::NE;
    hf = SH::H < 128 ? tl & (SH::H - 1) : tl;
    hrow0 = (t / (SH::H < 128 ? SH::H : 128)) * SH::HR;
  }
};

// F = W2 tanh(W1 tanh(W0 x + b0) + b1) + b2 of the owned elements, for the stage
// input already written by put() (not yet synchronised).  On return every product
// has completed; ok is false after a timeout.
template <class SH, bool XO>
struct FmEval {
  FmSmem<SH, XO> &sm;
  FmGroup<SH, XO> &gs;
  const FmMap<SH> &m;
  const int g;
  const uint32_t tmem;
  float b0[SH::MB], b1[SH::MB], b2;  // the biases of the thread's features
  uint32_t phase = 0;
  bool ok = true;
  __device__ FmEval(FmSmem<SH, XO> &s, int gi, const FmMap<SH> &mm, uint32_t t, const float *W)
      : sm(s), gs(s.group[gi]), m(mm), g(gi), tmem(t) {
#pragma unroll
    for (int b = 0; b < SH::MB; b++) {
      b0[b] = W[SH::OB0 + m.hf + 128 * b];
      b1[b] = W[SH::OB1 + m.hf + 128 * b];
    }
    b2 = W[SH::OB2 + m.f];
  }
  __device__ __forceinline__ unsigned char *bufa() {
    return reinterpret_cast<unsigned char *>(gs.bufa);
  }
  __device__ __forceinline__ unsigned char *bufx() {
    return reinterpret_cast<unsigned char *>(SH::WIDE ? gs.bufb : gs.bufa);
  }
  __device__ __forceinline__ void put(const float (&Y)[SH::NE]) {
#pragma unroll
    for (int e = 0; e < SH::NE; e += SH::NE < 8 ? 4 : 8) {
      F2 v[SH::NE < 8 ? 2 : 4];
#pragma unroll
      for (int j = 0; j < (SH::NE < 8 ? 2 : 4); j++) v[j] = f2_pack(Y[e + 2 * j], Y[e + 2 * j + 1]);
      fm_put<SH::R, SH::D>(bufx(), m.f, m.row0 + e, v);
    }
  }
  // this group's operand writes and accumulator reads are done
  __device__ __forceinline__ void publish() {
    tc::fence_async_smem();
    tc::fence_before_sync();
    fm_sync(g);
  }
  __device__ __forceinline__ void wait() {
    ok = ok && tc::mbar_wait(&gs.bar, phase, kFmWait);
    phase ^= 1u;
    tc::fence_after_sync();
  }
  // tanh(acc + bias) of the owned hidden rows as feature f of a K-feature operand
  template <int K>
  __device__ __forceinline__ void hidden(float bias, unsigned char *dst, int f) {
#pragma unroll
    for (int c = 0; c < SH::HR; c += 8) {
      F2 v[4];
      tc::tmem_sum3(m.lanes + m.hrow0 + c, SH::R, v);
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = tanh2(f2_add(v[j], f2_set(bias)));
      fm_put<SH::R, K>(dst, f, m.hrow0 + c, v);
    }
  }
  template <int K>
  __device__ __forceinline__ uint64_t a_desc(const __nv_bfloat16 *w) const {
    return tc::smem_desc(tc::smem_u32(w), 128u, K * 16u);
  }
  template <int K>
  __device__ __forceinline__ uint64_t x_desc(const unsigned char *b) const {
    return tc::smem_desc(tc::smem_u32(b), 128u, K * 16u);
  }
  __device__ __forceinline__ void operator()(float (&F)[SH::NE]) {
    constexpr int D = SH::D, H = SH::H, N = SH::N;
    const bool issuer = m.t == 0;
    if constexpr (SH::WIDE) {
#pragma unroll
      for (int b = 0; b < 2; b++) {
        publish();
        if (issuer) {
          tc::fence_after_sync();
          fm_issue_ta<N, D / 16>(m.acc, tmem + SH::TW0 + b * (D / 2), x_desc<D>(bufx()));
          tc::mma_commit(&gs.bar);
        }
        wait();
        hidden<H>(b0[b], bufa(), m.hf + 128 * b);
      }
#pragma unroll
      for (int b = 0; b < 2; b++) {
        publish();
        if (issuer) {
          tc::fence_after_sync();
          fm_issue_ta<N, H / 16>(m.acc, tmem + SH::TW1 + b * (H / 2), x_desc<H>(bufa()));
          tc::mma_commit(&gs.bar);
        }
        wait();
        hidden<128>(b1[b], b == 0 ? bufx() : bufa(), m.hf);
      }
      publish();
      if (issuer) {
        tc::fence_after_sync();
        constexpr uint32_t id = tc::idesc_bf16_f32(128, N, false, true);
        const uint64_t da = a_desc<H>(sm.w2);
#pragma unroll
        for (int k = 0; k < 16; k++)
          tc::mma_bf16(m.acc, da + 16u * k, x_desc<128>(k < 8 ? bufx() : bufa()) + 16u * (k & 7),
                       id, k > 0 ? 1u : 0u);
        tc::mma_commit(&gs.bar);
      }
      wait();
    } else {
      publish();
      if (issuer) {
        tc::fence_after_sync();
        fm_issue<N, D / 16>(m.acc, a_desc<D>(sm.w0), x_desc<D>(bufx()));
        tc::mma_commit(&gs.bar);
      }
      wait();
      hidden<H>(b0[0], bufa(), m.hf);
      publish();
      if (issuer) {
        tc::fence_after_sync();
        fm_issue<N, H / 16>(m.acc, a_desc<H>(sm.w1), x_desc<H>(bufa()));
        tc::mma_commit(&gs.bar);
      }
      wait();
      hidden<H>(b1[0], bufa(), m.hf);
      publish();
      if (issuer) {
        tc::fence_after_sync();
        fm_issue<N, H / 16>(m.acc, a_desc<H>(sm.w2), x_desc<H>(bufa()));
        tc::mma_commit(&gs.bar);
      }
      wait();
    }
    // (rows in eights or fours: the group's lanes hold R columns a piece)
#pragma unroll
    for (int e = 0; e < SH::NE; e += SH::NE < 8 ? 4 : 8) {
      F2 v[SH::NE < 8 ? 2 : 4];
      tc::tmem_sum3(m.lanes + m.row0 + e, SH::R, v);
#pragma unroll
      for (int j = 0; j < (SH::NE < 8 ? 2 : 4); j++)
        f2_unpack(f2_add(v[j], f2_set(b2)), F[e + 2 * j], F[e + 2 * j + 1]);
    }
  }
};

// Sums of s[e] over the features of each owned row, in NPART parts: halving
// exchanges give each lane one row, then plain butterflies.  (The sum of a row
// does not depend on where in the tile it sits.)
template <class SH>
__device__ __forceinline__ void fm_row_sums(float (&part)[SH::R][2], const FmMap<SH> &m,
                                            float (&s)[SH::NE]) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = m.tl & 31;
  int row = m.row0, bit = 16;
#pragma unroll
  for (int n = SH::NE / 2; n >= 1; n /= 2, bit /= 2) {
    const bool up = lane & bit;
#pragma unroll
    for (int j = 0; j < n; j++) {
      const float keep = up ? s[n + j] : s[j], give = up ? s[j] : s[n + j];
      s[j] = keep + __shfl_xor_sync(full, give, bit);
    }
    row += up ? n : 0;
  }
  float t = s[0];
#pragma unroll
  for (int b = 16 / SH::NE; b >= 1; b /= 2) t += __shfl_xor_sync(full, t, b);
  if ((lane & (32 / SH::NE - 1)) == 0) part[row][SH::D == 64 ? (m.tl >> 5) & 1 : 0] = t;
}

// Four or eight row values from shared memory.
template <int NE, class T>
__device__ __forceinline__ void fm_rows(const T *a, int row0, T (&v)[NE]) {
  static_assert(sizeof(T) == 4, "32-bit row values");
#pragma unroll
  for (int e = 0; e < NE; e += 4)
    *reinterpret_cast<int4 *>(v + e) = *reinterpret_cast<const int4 *>(a + row0 + e);
}

// XO (extended outputs: SaveAt(steps=n), SaveAt(dense=True), the clip controller,
// events, resume records) is a template flag, as in the trajectory kernels.
template <int SOLVER, int D, int H, bool XO>
__global__ void __launch_bounds__((FmShape<D, H>::THREADS), 1) mlp_fm_kernel(SolveParams P) {
  using SH = FmShape<D, H>;
  using TB = Tab<SOLVER>;
  constexpr int S = TB::S, NE = SH::NE, M = SH::R, NT = SH::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FmSmem<SH, XO> &sm = *reinterpret_cast<FmSmem<SH, XO> *>(smem_raw);
  const int tid = threadIdx.x, g = tid / SH::GT, t = tid % SH::GT;
  FmGroup<SH, XO> &gs = sm.group[g];
  RowState<M> &R = gs.rows;
  RowEvents<M> *EV = nullptr;
  if constexpr (XO) EV = &gs.ev;
  using Step = RowEventStep<M, 2>;
  [[maybe_unused]] Step &ES = *reinterpret_cast<Step *>(gs.bufa);
  static_assert(sizeof(Step) <= sizeof(gs.bufa), "the events' scratch fits the operand");

  if (tid < 32) tc::tmem_alloc(&sm.slot, SH::TMEM_COLS);
  const float *W = P.mlp;
  const bool vec = (reinterpret_cast<uintptr_t>(W) & 15) == 0;
  if constexpr (!SH::WIDE) {
    fm_stage<H, 128, D>(sm.w0, W + SH::OW0, tid, NT, vec);
    fm_stage<H, 128, H>(sm.w1, W + SH::OW1, tid, NT, vec);
  }
  fm_stage<D, 128, H>(sm.w2, W + SH::OW2, tid, NT, vec);
  // Take trajectory q of the work order for row t.  A group's first tile is
  // fixed (tiles go round the CTAs, then round their groups, so a small batch
  // spreads over the SMs); the queue hands out the rest.
  auto take = [&](unsigned long long q) {
    const bool got = q < (unsigned long long)P.batch;
    if (got)
      row_init<M, XO>(R, EV, t, P.order ? (int64_t)P.order[q] : (int64_t)q, P, D,
                         TB::FSAL);
    else
      R.active[t] = 0;
    R.loaded[t] = got;
  };
  const unsigned long long queued = (unsigned long long)gridDim.x * SH::G * M;
  if (t < M) {
    R.idx[t] = 0;
    R.keep[t] = 0;
    take(((unsigned long long)g * gridDim.x + blockIdx.x) * M + t);
  }
  if (t == 0) {
    tc::mbar_init(&gs.bar, 1);
    tc::mbar_init(&gs.drain, 1);
    gs.err = 0;
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = sm.slot;
  if constexpr (SH::WIDE) {
    // group b stages block b of both hidden layers
    const uint32_t lanes = tmem + (uint32_t(t & 96) << 16);
    fm_stage_tmem<D>(lanes + SH::TW0 + g * (D / 2), W + SH::OW0 + g * 128 * D, t, vec);
    fm_stage_tmem<H>(lanes + SH::TW1 + g * (H / 2), W + SH::OW1 + g * 128 * H, t, vec);
    tc::tmem_st_wait();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  }
  const FmMap<SH> m(t, tmem + g * SH::N);
  FmEval<SH, XO> eval(sm, g, m, tmem, W);
  bool ev_steady = false;
  if constexpr (XO) {
#pragma unroll
    for (int e = 0; e < GBDX_MAX_EVENTS; e++)
      ev_steady |= e < P.n_event && P.ev_kind[e] == GBDX_EV_STEADY;
  }
  // the steady-state condition's norms of the owned elements
  [[maybe_unused]] auto steady = [&](const float (&F)[NE], const float (&Y)[NE]) {
    float s[NE];
#pragma unroll
    for (int e = 0; e < NE; e++) s[e] = F[e] * F[e];
    fm_row_sums<SH>(ES.pf, m, s);
#pragma unroll
    for (int e = 0; e < NE; e++) s[e] = Y[e] * Y[e];
    fm_row_sums<SH>(ES.py, m, s);
  };

  float Y0[NE], F0[NE];
#pragma unroll
  for (int e = 0; e < NE; e++) Y0[e] = F0[e] = 0.f;
  // Initial state of freshly loaded rows: y0, a zero FSAL vector, the t0 save and
  // the first state checkpoint.
  auto load = [&]() {
#pragma unroll
    for (int e = 0; e < NE; e++) {
      const int row = m.row0 + e;
      if (R.loaded[row]) {
        const int64_t i = R.idx[row];
        Y0[e] = reinterpret_cast<const float *>(P.y0)[i * D + m.f];
        F0[e] = 0.f;
        if (P.save_t0)
          *GBDX_AT(P, reinterpret_cast<float *>(P.ys_out), i * P.n_save * D + m.f, 1,
                   P.batch * P.n_save * D, GBDX_SITE_YS) = Y0[e];
        // a resumed row's FSAL value (row_init cleared its `first`)
        if constexpr (XO && TB::FSAL) {
          if (P.state_in && !R.first[row])
            F0[e] = float(*GBDX_AT(
                P, P.state_in, i * int64_t(GBDX_STATE_HEAD + D) + GBDX_STATE_HEAD + m.f, 1,
                P.batch * (GBDX_STATE_HEAD + D), GBDX_SITE_STATE));
        }
      }
    }
  };
  load();
  fm_sync(g);
  if (t < M) R.loaded[t] = 0;

  float K[S][NE], F[NE];
  while (fm_sync_or(g, t < M && R.active[t])) {
    // ---- one lockstep step -------------------------------------------------
    int live = 0, first_live = 0;
    if (t < M) {
      live = row_running(R, t, P.max_steps);
      first_live = live && R.first[t];
      R.live[t] = live;
      R.anynan[t] = 0;
      // control h = dir * dt as FP32 (WrapTerm, _term.py:742-745)
      R.h[t] = live ? float(R.dir[t] > 0 ? R.dtc[t] : -R.dtc[t]) : 0.f;
    }
    const int any_first = fm_sync_or(g, first_live);
    float h[NE];
    fm_rows<NE>(R.h, m.row0, h);
    // The stages share one copy of the field's code (seven unrolled copies,
    // ~200 KB, missed the instruction caches: twice the epilogues' time); the
    // stage vectors stay in registers, each case naming its own.  Stage 0 reuses
    // the FSAL value unless some row is on its first step.
    float Yi[NE];
#pragma unroll
    for (int e = 0; e < NE; e++) F[e] = F0[e];
#pragma unroll 1
    for (int i = 0; i < S; i++) {
      stage_input<SOLVER, 1>(i, Y0, K, Yi);
      if (i > 0 || !TB::FSAL || any_first) {
        eval.put(Yi);
        eval(F);
      }
      // a steady-state condition already true at (t0, y0) ends the solve before
      // its first step (_integrate.py:1333-1426); F holds f(y0) for a fresh row
      if constexpr (XO) {
        if (i == 0 && ev_steady) {
          const int fresh = t < M && live && R.nsteps[t] == 0;
          if (fm_sync_or(g, fresh)) {
            steady(F, Y0);
            fm_sync(g);
            if (fresh) {
#pragma unroll
              for (int e = 0; e < GBDX_MAX_EVENTS; e++) {
                if (e < P.n_event && P.ev_kind[e] == GBDX_EV_STEADY) {
                  const double v = steady_value<D, SH::NPART>(P, ES, t, e);
                  EV->evv[t][e] = v;
                  if (EV->evi[t] < 0 && v != 0.0) EV->evi[t] = e;
                }
              }
              if (EV->evi[t] >= 0) {
                R.result[t] = GBDX_EVENT_OCCURRED;
                live = 0;
                R.live[t] = 0;
              }
            }
            fm_sync(g);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < S; j++)
        if (i == j) {
#pragma unroll
          for (int e = 0; e < NE; e++) K[j][e] = F[e] * h[e];
        }
    }
    if (!eval.ok) gs.err = 1;
    // y1, error estimate, per-row scaled error norm
    float Y1[NE];
#pragma unroll
    for (int e = 0; e < NE; e++) {
      if constexpr (TB::SSAL) {
        Y1[e] = Yi[e];
      } else {
        float a = Y0[e];
#pragma unroll
        for (int j = 0; j < S; j++) a = fmaf(float(TB::b(j)), K[j][e], a);
        Y1[e] = a;
      }
    }
    if (P.controller == GBDX_PID) {
      // a row with a NaN in y1 is scaled by y0 alone (pid.py:466-492)
      bool nan1 = false;
#pragma unroll
      for (int e = 0; e < NE; e++) nan1 |= isnan(Y1[e]);
      const bool somenan = fm_sync_or(g, nan1);
      if (somenan) {
#pragma unroll
        for (int e = 0; e < NE; e++)
          if (isnan(Y1[e])) R.anynan[m.row0 + e] = 1;
        fm_sync(g);
      }
      float s[NE];
#pragma unroll
      for (int e = 0; e < NE; e++) {
        float er = 0.f;
#pragma unroll
        for (int j = 0; j < S; j++)
          if (TB::e(j) != 0.0) er = fmaf(float(TB::e(j)), K[j][e], er);
        er = isnan(er) ? INFINITY : er;
        const bool nanrow = somenan && R.anynan[m.row0 + e];
        const float ym = fmaxf(fabsf(Y0[e]), fabsf(nanrow ? Y0[e] : Y1[e]));
        const float q = __fdividef(er, fmaf(ym, P.rtol_f, P.atol_f));
        s[e] = q * q;
      }
      fm_row_sums<SH>(gs.part, m, s);
      fm_sync(g);
    }
    if (t < M && live) {
      float a = 0.f;
#pragma unroll
      for (int n = 0; n < SH::NPART; n++) a += gs.part[t][n];
      R.acc[t] = a;
      row_control<M, XO>(R, t, D, P);
    }
    fm_sync(g);
    // ---- events at the new state (_integrate.py:542-633) --------------------
    // The first condition (in order) that fires ends the solve; with a root
    // finder the final time is the root inside this step and no save after
    // it is made.
    if constexpr (XO) {
      if (P.n_event > 0) {
        if constexpr (!TB::FSAL) {
          // f(y1) for a steady-state condition (FSAL solvers have it in F)
          if (ev_steady && fm_sync_or(g, t < M && live && R.keep[t])) {
            eval.put(Y1);
            eval(F);
            if (!eval.ok) gs.err = 1;
          }
        }
        if (m.f < 4) {
#pragma unroll
          for (int e = 0; e < NE; e++) {
            const int row = m.row0 + e;
            if (R.live[row] && R.keep[row]) {
              ES.ey0[row][m.f] = Y0[e];
              ES.ey1[row][m.f] = Y1[e];
#pragma unroll
              for (int j = 0; j < S; j++) ES.ek[row][j][m.f] = K[j][e];
            }
          }
        }
        if (ev_steady) steady(F, Y1);
        fm_sync(g);
        if (t < M) {
          EV->tsave[t] = R.tn_old[t];
          if (live && R.keep[t]) row_events<SOLVER, S, D, SH::NPART>(R, *EV, ES, t, P);
        }
        fm_sync(g);
      }
    }
    // ---- SaveAt(ts) inside accepted steps (_integrate.py:456-487) ----------
    // MAX_SAVES lanes look at a row's next save times at once and leave the
    // interpolant's weights for all; passes repeat while some row filled one.
    // The pass is latency: place without an FP64 division (~1200 cycles) and weights in
    // two 16-byte reads.  16384 trajectories 64-256-256-64 with 32 saves: 790 to 710 us.
    while (P.n_ts > 0) {
      constexpr int MS = SH::MAX_SAVES;
      FmSaves<SH> &sv = *reinterpret_cast<FmSaves<SH> *>(gs.bufa);
      static_assert(sizeof(FmSaves<SH>) <= sizeof(gs.bufa), "save weights fit the operand");
      const int row = t / MS, c = t % MS;
      const int first = R.ts_index[row], slot = R.save_index[row];
      double tsv = 0.0, tsd = 0.0;
      bool hit = false;
      if (R.live[row] && R.keep[row] && first + c < P.n_ts) {
        tsv = __ldg(P.save_ts + first + c);
        tsd = R.dir[row] * tsv;
        double last = R.tn_old[row];
        if constexpr (XO) {
          if (P.n_event > 0) last = EV->tsave[row];
        }
        hit = tsd <= last;
      }
      // hits before the row's first miss
      const unsigned seg = (__ballot_sync(0xffffffffu, hit) >> (t & 31 & ~(MS - 1))) &
                           ((1u << MS) - 1u);
      const int n = __ffs(~seg) - 1;
      if (c < n) {
        const double tp = R.tp_old[row], tn = R.tn_old[row];
        const float th = tp == tn ? 0.f : f64i_quotient_f32(tsd - tp, tn - tp);
        *GBDX_AT(P, P.ts_out, R.idx[row] * P.n_save + slot + c, 1, P.batch * P.n_save,
                 GBDX_SITE_TS) = tsv;
        if constexpr (SOLVER == GBDX_TSIT5) {
#pragma unroll
          for (int j = 0; j < 7; j++) sv.w[row][c][j] = tsit5_w<float>(j, th);
        } else {
          sv.w[row][c][7] = th;
        }
      }
      if (c == 0) {
        sv.n[row] = n;
        R.sslot[row] = slot;
        R.ts_index[row] = first + n;
        R.save_index[row] = slot + n;
      }
      if (!fm_sync_or(g, n)) break;
#pragma unroll
      for (int e = 0; e < NE; e++) {
        const int r = m.row0 + e, ns = sv.n[r];
        for (int k = 0; k < ns; k++) {
          float w[8];
          *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(sv.w[r][k]);
          *reinterpret_cast<float4 *>(w + 4) = *reinterpret_cast<const float4 *>(sv.w[r][k] + 4);
          float v;
          if constexpr (SOLVER == GBDX_TSIT5) {
            v = 0.f;
#pragma unroll
            for (int j = 0; j < 7; j++) v = fmaf(w[j], K[j < S ? j : 0][e], v);
            v += Y0[e];
          } else {
            v = mlp_interp<SOLVER, S, false>(w[7], Y0[e], Y1[e], [&](int j) { return K[j][e]; });
          }
          *GBDX_AT(P, reinterpret_cast<float *>(P.ys_out),
                   (R.idx[r] * P.n_save + R.sslot[r] + k) * D + m.f, 1, P.batch * P.n_save * D,
                   GBDX_SITE_YS) = v;
        }
      }
      if (!fm_sync_or(g, n == MS)) break;
    }
    // ---- SaveAt(steps=n), after the step's ts saves (_integrate.py:492-527),
    // and SaveAt(dense=True) step times (:529-540) ----------------------------
    if (XO && (P.save_steps > 0 || P.dense_ts != nullptr)) {
      if (t < M) {
        R.stslot[t] = -1;
        if (live && R.keep[t]) {
          const int64_t i = R.idx[t];
          if (P.save_steps > 0 && --R.sdown[t] == 0) {
            R.sdown[t] = P.save_steps;
            // not past an event's root
            if (!(P.n_event > 0 && order_key(R.tn_old[t]) > order_key(EV->tsave[t]))) {
              R.stslot[t] = R.save_index[t]++;
              *GBDX_AT(P, P.ts_out, i * P.n_save + R.stslot[t], 1, P.batch * P.n_save,
                       GBDX_SITE_TS) = R.dir[t] * R.tn_old[t];
            }
          }
          // nacc already counts this step
          if (P.dense_ts)
            *GBDX_AT(P, P.dense_ts, i * (P.max_steps + 1) + R.nacc[t], 1,
                     P.batch * (P.max_steps + 1), GBDX_SITE_DENSE_TS) = R.tn_old[t];
        }
      }
      fm_sync(g);
    }
    // ---- accept: advance the state, FSAL vector ----------------------------
    int kept[NE];
    {
      int lv[NE];
      fm_rows<NE>(R.live, m.row0, lv);
      fm_rows<NE>(R.keep, m.row0, kept);
#pragma unroll
      for (int e = 0; e < NE; e++) kept[e] = kept[e] && lv[e];
    }
#pragma unroll
    for (int e = 0; e < NE; e++) {
      if (kept[e]) {
        if constexpr (XO) {
          const int row = m.row0 + e;
          if (R.stslot[row] >= 0)
            *GBDX_AT(P, reinterpret_cast<float *>(P.ys_out),
                     (R.idx[row] * P.n_save + R.stslot[row]) * D + m.f, 1,
                     P.batch * P.n_save * D, GBDX_SITE_YS) = Y1[e];
          if (P.dense_info) {
            // the step's (y0, y1, k_0..k_{S-1}), component f of each
            constexpr int REC = (2 + S) * D;
            float *rec = GBDX_AT(P, static_cast<float *>(P.dense_info),
                                 (R.idx[row] * P.max_steps + R.nacc[row] - 1) * REC, REC,
                                 P.batch * P.max_steps * REC, GBDX_SITE_DENSE_INFO);
            rec[m.f] = Y0[e];
            rec[D + m.f] = Y1[e];
#pragma unroll
            for (int j = 0; j < S; j++) rec[(2 + j) * D + m.f] = K[j][e];
          }
          if (P.n_event > 0 && EV->evi[row] >= 0 && EV->thfin[row] >= 0.f) {
            // the state at the event's root (or the step's end for a boolean)
            Y1[e] = mlp_interp<SOLVER, S, false>(EV->thfin[row], Y0[e], Y1[e],
                                                 [&](int j) { return K[j][e]; });
          }
        }
        Y0[e] = Y1[e];
        if (TB::FSAL) F0[e] = F[e];  // field value of the last stage (FSAL)
      }
    }
    // ---- finished rows: t1 save, outputs, refill ----------------------------
    // (a product that did not complete makes this the group's last step, and every
    // row that it had a part in an internal error)
    const bool lost = *reinterpret_cast<volatile int *>(&gs.err);
    int fin = 0;
    if (t < M) {
      R.fin[t] = 0;
      if (R.active[t] && !row_running(R, t, P.max_steps)) {
        const int64_t i = R.idx[t];
        const int dir = R.dir[t];
        const double t0 = P.t0[i * P.time_stride] * dir;
        int si = R.save_index[t];
        R.nfill[t] = (t0 == R.t1[t]) ? P.n_ts : 0;
        R.sslot[t] = si;  // first slot written by the element pass
        [[maybe_unused]] const int64_t tse = P.batch * P.n_save;
        for (int n = 0; n < R.nfill[t]; n++)
          *GBDX_AT(P, P.ts_out, i * P.n_save + si + n, 1, tse, GBDX_SITE_TS) = t0 * dir;
        si += R.nfill[t];
        // the t1 value is already saved when SaveAt(steps=n) saved the last
        // step (_integrate.py:847-877); with an event root finder the final
        // value is saved whenever the steps saved the t1 value, as that save
        // fell after the event (:860-872), and the final time is the event's
        R.sflag[t] = P.save_t1;
        double tf = R.tprev[t];
        if constexpr (XO) {
          const bool via_steps = P.save_steps > 0 && R.sdown[t] == P.save_steps;
          const bool root = P.n_event > 0 && P.event_root;
          R.sflag[t] = root ? (P.save_t1 || via_steps) : (P.save_t1 && !via_steps);
          if (root && EV->evi[t] >= 0) tf = EV->tfin[t];
          if (P.event_index) P.event_index[i] = EV->evi[t];
          if (P.dense_n) P.dense_n[i] = R.nacc[t] + 1;
          if (P.state_out) {
            // SaveAt(controller_state=, solver_state=, made_jump=)
            // (_integrate.py:1489-1500): the head of the record; the
            // element pass writes the FSAL value
            double *so = GBDX_AT(P, P.state_out, i * int64_t(GBDX_STATE_HEAD + D),
                                 GBDX_STATE_HEAD, P.batch * (GBDX_STATE_HEAD + D),
                                 GBDX_SITE_STATE);
            if (P.controller == GBDX_PID) {
              so[0] = exp2(double(R.hist1[t]));
              so[1] = exp2(double(R.hist2[t]));
              so[2] = R.at_dtmin[t] ? 1.0 : 0.0;
              so[3] = 0.0;
            } else {
              so[0] = R.sc[t];
              so[1] = R.nc[t];
              so[2] = R.t0s[t];
              so[3] = R.t1s[t];
            }
            so[4] = 1.0;
            so[5] = (TB::FSAL && !R.first[t]) ? 0.0 : 1.0;
            so[6] = 0.0;  // made_jump: set by a ClipStepSizeController only
          }
        }
        if (R.sflag[t])
          *GBDX_AT(P, P.ts_out, i * P.n_save + si++, 1, tse, GBDX_SITE_TS) = tf * dir;
        if (!XO || !P.saves_prefilled)
          for (int n = si; n < P.n_save; n++)  // direction * inf
            *GBDX_AT(P, P.ts_out, i * P.n_save + n, 1, tse, GBDX_SITE_TS) =
                dir > 0 ? INFINITY : -INFINITY;
        int res = R.result[t];
        if (res == GBDX_SUCCESSFUL && order_key(R.tprev[t]) < order_key(R.t1[t]))
          res = GBDX_MAX_STEPS_REACHED;
        if (lost) res = GBDX_INTERNAL_ERROR;
        P.result_out[i] = res;
        P.stats_out[i * 3 + 0] = R.nsteps[t];
        P.stats_out[i * 3 + 1] = R.nacc[t];
        P.stats_out[i * 3 + 2] = R.nrej[t];
        R.fin[t] = 1;
        fin = 1;
      }
    }
    if (fm_sync_or(g, fin)) {
#pragma unroll
      for (int e = 0; e < NE; e++) {
        const int row = m.row0 + e;
        if (R.fin[row]) {
          float *o = reinterpret_cast<float *>(P.ys_out);
          const int64_t b0 = R.idx[row] * P.n_save * D + m.f;
          [[maybe_unused]] const int64_t ext = P.batch * P.n_save * D;
          int si = R.sslot[row];
          for (int n = 0; n < R.nfill[row]; n++)
            *GBDX_AT(P, o, b0 + (si + n) * D, 1, ext, GBDX_SITE_YS) = Y0[e];
          si += R.nfill[row];
          if (R.sflag[row]) *GBDX_AT(P, o, b0 + (si++) * D, 1, ext, GBDX_SITE_YS) = Y0[e];
          if (!XO || !P.saves_prefilled)
            for (int n = si; n < P.n_save; n++)
              *GBDX_AT(P, o, b0 + n * D, 1, ext, GBDX_SITE_YS) = INFINITY;
          if constexpr (XO) {
            if (P.state_out)  // the record's FSAL value (0 where there is none)
              *GBDX_AT(P, P.state_out,
                       R.idx[row] * int64_t(GBDX_STATE_HEAD + D) + GBDX_STATE_HEAD + m.f, 1,
                       P.batch * (GBDX_STATE_HEAD + D), GBDX_SITE_STATE) =
                  (TB::FSAL && !R.first[row]) ? double(F0[e]) : 0.0;
          }
        }
      }
      fm_sync(g);
      if (t < M && R.fin[t]) {
        if (lost)
          R.active[t] = 0;
        else
          take(queued + atomicAdd(P.queue, 1ull));
      }
      fm_sync(g);
      load();
      fm_sync(g);
      if (t < M) R.loaded[t] = 0;
    }
    if (lost) {
      // the rows still under way, and those that no group may be left to take
      if (t < M) {
        if (R.active[t]) P.result_out[R.idx[t]] = GBDX_INTERNAL_ERROR;
        for (unsigned long long q = queued + atomicAdd(P.queue, 1ull);
             q < (unsigned long long)P.batch; q = queued + atomicAdd(P.queue, 1ull))
          P.result_out[P.order ? (int64_t)P.order[q] : (int64_t)q] = GBDX_INTERNAL_ERROR;
      }
      // the operands and accumulators stay until no product uses them
      if (t == 0) {
        tc::mma_commit(&gs.drain);
        tc::mbar_wait(&gs.drain, 0, kFmDrain);
      }
      break;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 32) tc::tmem_dealloc(tmem, SH::TMEM_COLS);
}

template <int SOLVER, int D, int H, bool XO>
cudaError_t launch_fm(const SolveParams &P, const LaunchCfg &cfg, cudaStream_t s) {
  using SH = FmShape<D, H>;
  // one CTA per SM: two could not both have their tensor memory
  constexpr size_t need = sizeof(FmSmem<SH, XO>), half = 114 * 1024;
  constexpr size_t bytes = need < half ? half : need;
  static_assert(bytes <= 227 * 1024, "shared memory of one CTA");
  auto k = mlp_fm_kernel<SOLVER, D, H, XO>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  if (P.batch <= 0) return cudaSuccess;
  k<<<cfg.grid, SH::THREADS, bytes, s>>>(P);
  return cudaGetLastError();
}

inline cudaError_t occupancy_fm(int, int *ctas) {
  *ctas = 1;
  return cudaSuccess;
}

template <int D, int H, bool XO>
OdeEntry fm_entry(int solver) {
  switch (solver) {
    case GBDX_EULER: return OdeEntry{&launch_fm<GBDX_EULER, D, H, XO>, &occupancy_fm};
    case GBDX_HEUN: return OdeEntry{&launch_fm<GBDX_HEUN, D, H, XO>, &occupancy_fm};
    case GBDX_DOPRI5: return OdeEntry{&launch_fm<GBDX_DOPRI5, D, H, XO>, &occupancy_fm};
    case GBDX_TSIT5: return OdeEntry{&launch_fm<GBDX_TSIT5, D, H, XO>, &occupancy_fm};
    default: return OdeEntry{nullptr, nullptr};
  }
}

}  // namespace gbdx
