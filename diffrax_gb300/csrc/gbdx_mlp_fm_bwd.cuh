// gbdx_mlp_fm_bwd.cuh -- RecursiveCheckpointAdjoint backward of the MLP fields on
// the fifth-generation tensor cores (BF16 products).
//
// The walk of mlp_bwd_kernel (gbdx_mlp_bwd.cuh: the tape, the recompute and
// backpropagation iterations of a row, what is differentiated), with the field
// and its VJP in the feature-major layout of gbdx_mlp_fm.cuh: 8 warps own a tile
// of R = 32 rows, a thread one feature and a run of rows, and a ninth warp issues
// the products.  Per stage
//   forward   x -> a1 = tanh(W0 x + b0) -> a2 = tanh(W1 a1 + b1) -> F
//   reverse   g2 = (W2^T g3)(1 - a2^2), g1 = (W1^T g2)(1 - a1^2), gY = W0^T g1
// are products of the weights (as stored, or MN-major for the transposes: one
// copy serves both) with the three pieces of an operand side by side, and the
// weight gradients
//   dW1 += g2 a1^T, dW2^T += a2 g3^T, dW0 += g1 x^T
// contract over the rows of the same operand buffers (there K-major), six products
// of pieces each, the smallest first, into an accumulator of their own; they run
// behind the chain's products while the epilogues compute.  The tensor core cuts
// each sum short of rounding, so the running sum is not its accumulator: every
// stage's gradient is added, rounded, to sums in other columns of tensor memory
// (one accumulator for all stages of an iteration lost a factor of 2 in dW1), and
// those of a few iterations, compensated, to the CTA's partials.
//
// Work left out because it adds exact zeros: a stage whose increment has no
// cotangent (the last one of an SSAL tableau without a save inside the step), and
// forward stages that only it would read.
//
// Every weight is stored 128 x 128, its rows and columns repeated up to that, so
// the accumulators' lanes are full in both directions (gbdx_mlp_fm.cuh: lane maps).
//
// Bound: the serial chain of a stage (six products, their completion latency and
// epilogues), one tile a CTA: at 64-128 and 8192 rows issue slots 27 %, tensor pipe 18 %; the
// neural SDE 24 and 11 %.
#pragma once

#include "gbdx_mlp_bwd.cuh"
#include "gbdx_mlp_fm.cuh"

namespace gbdx {

template <int D_, int H_, bool SDE_>
struct FbShape {
  static constexpr int D = D_, H = H_;
  static constexpr bool SDE = SDE_;
  static constexpr int R = 32, M = R;     // rows per tile
  static constexpr int GT = 256;          // threads that own elements
  static constexpr int THREADS = GT + 32; // and the issuing warp
  static constexpr int N = 3 * R;
  static constexpr int NE = R * D / GT, HR = R * H / GT;
  static_assert(H <= 128 && 128 % H == 0 && 128 % D == 0, "repeated weights");
  // weight gradients: accumulator rows (M = 64 leaves them in 16 lanes of each
  // 32); TMEM columns behind the chain's accumulator(s): the sums, then a stage's
  // accumulator
  static constexpr int MW = H < 128 ? 64 : 128;
  static constexpr int T1 = N * (SDE ? 2 : 1), T2 = T1 + H, T0 = T2 + D, TS = T0 + D;
  static constexpr int TA = TS + (SDE ? D : 0);
  static_assert(TA + 128 <= 512 && 2 * D <= 128, "tensor memory");
  static constexpr int OW0 = 0, OB0 = OW0 + H * D, OW1 = OB0 + H, OB1 = OW1 + H * H,
                       OW2 = OB1 + H, OB2 = OW2 + D * H, OWS = OB2 + D, OBS = OWS + D * D;
};

template <class SH>
struct __align__(128) FbSmem {
  __nv_bfloat16 w0[128 * 128], w1[128 * 128], w2[128 * 128], ws[SH::SDE ? 128 * 128 : 8];
  // operands, [k][(piece, row)] as gbdx_mlp_fm.cuh
  __nv_bfloat16 x[SH::N * SH::D], a1[SH::N * SH::H], a2[SH::N * SH::H];
  __nv_bfloat16 g3[SH::N * SH::D], g2[SH::N * SH::H], g1[SH::N * SH::H];
  __nv_bfloat16 gs[SH::SDE ? SH::N * SH::D : 8];
  BwdRows<SH::R> rows;
  float bias[4][SH::GT];
  uint64_t bar, barw;  // a chain product is done; a weight-gradient product is
  uint64_t drain;
  int job;
  int issued, issuedw;  // products of either kind issued so far
  uint32_t slot;
  int err;
};

// Iterations between additions to the partials: their traffic (16 bytes a
// parameter) took 15000 cycles of an iteration's 185000 at width 128.
constexpr int kFbFlush = 8;

// Products the issuing warp runs.
enum { kFbF0 = 0, kFbF1, kFbF2, kFbB2, kFbB1, kFbB0, kFbExit };

// K-major 128 x 128 copy of the BF16-rounded W[m % ROWS][k % COLS].
template <int ROWS, int COLS>
__device__ __forceinline__ void fb_stage(__nv_bfloat16 *dst, const float *W, int tid, int nt,
                                         bool vec) {
#pragma unroll 2
  for (int i = tid; i < 128 * 16; i += nt) {
    const int m = (i >> 7) * 8 + (i & 7), k8 = (i >> 3) & 15;
    const float *s = W + (m % ROWS) * COLS + (8 * k8) % COLS;
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
                               tc::kmajor_offset(m, 8 * k8, 128)) =
        *reinterpret_cast<const uint4 *>(h);
  }
}

// acc (+)= n products along K: descriptors da, db stepping by sa, sb.  (The issuing
// warp's loops stay rolled: unrolled, its code was fetched anew for every product.)
__device__ __forceinline__ void fb_seq(uint32_t acc, uint64_t da, uint64_t db, uint32_t sa,
                                       uint32_t sb, uint32_t id, int n, bool add) {
  uint32_t on = add ? 1u : 0u;
#pragma unroll 1
  for (int k = 0; k < n; k++) {
    tc::mma_bf16(acc, da, db, id, on);
    on = 1u;
    da += sa;
    db += sb;
  }
}

// acc (+)= W x (T: W^T x) for a K-feature operand x.
template <int N, int K, bool T>
__device__ __forceinline__ void fb_chain(uint32_t acc, const __nv_bfloat16 *w,
                                         const __nv_bfloat16 *x, bool add) {
  // W's 16-column slices lie 256 bytes apart, its 16-row slices 2 x 2048
  fb_seq(acc,
         T ? tc::smem_desc(tc::smem_u32(w), 2048u, 128u)
           : tc::smem_desc(tc::smem_u32(w), 128u, 2048u),
         tc::smem_desc(tc::smem_u32(x), 128u, K * 16u), T ? 256u : 16u, 16u,
         tc::idesc_bf16_f32(128, N, T, true), K / 16, add);
}

// acc[o, n] = sum over the rows of u[o, row] v[n, row], u and v operands of KU and
// KV features in three pieces: the six products of pieces whose size is at least
// 2^-18 of the leading one, the smallest first.
template <int MW, int NW, int KU, int KV, int R>
__device__ __forceinline__ void fb_outer(uint32_t acc, const __nv_bfloat16 *u,
                                         const __nv_bfloat16 *v) {
  const uint64_t du = tc::smem_desc(tc::smem_u32(u), KU * 16u, 128u);
  const uint64_t dv = tc::smem_desc(tc::smem_u32(v), KV * 16u, 128u);
  constexpr uint32_t id = tc::idesc_bf16_f32(MW, NW, false, false);
#pragma unroll 1
  for (int j = 0; j < 6; j++) {
    // pieces (2, 0), (0, 2), (1, 1), (1, 0), (0, 1), (0, 0)
    const uint32_t pu = (0x001102u >> (4 * j)) & 3u, pv = (0x010120u >> (4 * j)) & 3u;
    // 16 rows a product: two groups of 8
    fb_seq(acc, du + pu * uint32_t(R / 8 * KU), dv + pv * uint32_t(R / 8 * KV), 2 * KU, 2 * KV,
           id, R / 16, j > 0);
  }
}

// Barriers between the threads that own elements and the issuing warp: a product is
// wanted; the weight-gradient accumulator is free.
constexpr int kFbWant = 2, kFbFree = 3;
__device__ __forceinline__ void fb_arrive(int id) {
  asm volatile("bar.arrive %0, 288;" :: "r"(id) : "memory");
}
__device__ __forceinline__ void fb_await(int id) {
  asm volatile("bar.sync %0, 288;" :: "r"(id) : "memory");
}

// The issuing warp: runs the wanted products until told to leave (the others always
// tell it, after a timeout of theirs too: FbField::wait).
template <class SH>
__device__ void fb_issuer(FbSmem<SH> &sm, uint32_t tmem) {
  constexpr int D = SH::D, H = SH::H, N = SH::N, R = SH::R, MW = SH::MW;
  const bool lead = (threadIdx.x & 31) == 0;
  int issued = 0, issuedw = 0;
  while (true) {
    fb_await(kFbWant);
    // the leading lane's: its product lets the others post the next job, which a lane
    // behind it would read
    const int job =
        __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int *>(&sm.job), 0);
    if (job == kFbExit) {
      // the operands and accumulators stay until no product uses them
      if (lead && *reinterpret_cast<volatile int *>(&sm.err)) {
        tc::mma_commit(&sm.drain);
        tc::mbar_wait(&sm.drain, 0, kFmDrain);
      }
      __syncwarp();
      return;
    }
    if (lead) {
      tc::fence_after_sync();
      switch (job) {
        case kFbF0:
          fb_chain<N, D, false>(tmem, sm.w0, sm.x, false);
          if constexpr (SH::SDE) fb_chain<N, D, false>(tmem + N, sm.ws, sm.x, false);
          break;
        case kFbF1: fb_chain<N, H, false>(tmem, sm.w1, sm.a1, false); break;
        case kFbF2: fb_chain<N, H, false>(tmem, sm.w2, sm.a2, false); break;
        case kFbB2: fb_chain<N, D, true>(tmem, sm.w2, sm.g3, false); break;
        case kFbB1: fb_chain<N, H, true>(tmem, sm.w1, sm.g2, false); break;
        default:
          fb_chain<N, H, true>(tmem, sm.w0, sm.g1, false);
          if constexpr (SH::SDE) fb_chain<N, D, true>(tmem, sm.ws, sm.gs, true);
          break;
      }
      tc::mma_commit(&sm.bar);
      *reinterpret_cast<volatile int *>(&sm.issued) = ++issued;
    }
    __syncwarp();
    if (job < kFbB2) continue;
    fb_await(kFbFree);
    if (lead) {
      tc::fence_after_sync();
      switch (job) {
        case kFbB2: fb_outer<MW, D, H, D, R>(tmem + SH::TA, sm.a2, sm.g3); break;
        case kFbB1: fb_outer<MW, H, H, H, R>(tmem + SH::TA, sm.g2, sm.a1); break;
        default:
          fb_outer<MW, D, H, D, R>(tmem + SH::TA, sm.g1, sm.x);
          if constexpr (SH::SDE) fb_outer<64, D, D, D, R>(tmem + SH::TA + D, sm.gs, sm.x);
          break;
      }
      tc::mma_commit(&sm.barw);
      *reinterpret_cast<volatile int *>(&sm.issuedw) = ++issuedw;
    }
    __syncwarp();
  }
}

// Feature f's 8 rows from row0 of a K-feature operand, the three pieces summed.
template <int R, int K>
__device__ __forceinline__ void fb_get(const __nv_bfloat16 *buf, int f, int row0, F2 (&v)[4]) {
  const unsigned char *a = reinterpret_cast<const unsigned char *>(buf) + (f >> 3) * 128 +
                           (f & 7) * 16 + (row0 >> 3) * (K * 16);
#pragma unroll
  for (int q = 2; q >= 0; q--) {
    const uint4 w = *reinterpret_cast<const uint4 *>(a + q * (R / 8) * (K * 16));
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const F2 p = f2_pack(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u));
      v[j] = q == 2 ? p : f2_add(v[j], p);
    }
  }
}

// The thread's part of a stage's weight gradient (NC TMEM columns at src), added to
// (first: made) the iteration's sum at dst.
template <int NC>
__device__ __forceinline__ void fb_accumulate(uint32_t lanes, int src, int dst, int t,
                                              bool first) {
  const int c0 = (t >> 7) * (NC / 2);
#pragma unroll 1
  for (int c = c0; c < c0 + NC / 2; c += 16) {
    float v[16], s[16];
    tc::tmem_ld16(lanes + uint32_t(src + c), v);
    if (!first) {
      tc::tmem_ld16(lanes + uint32_t(dst + c), s);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] += s[j];
    }
    tc::tmem_st16(lanes + uint32_t(dst + c), v);
  }
  tc::tmem_st_wait();
}

// A compensated sum in registers.
struct FbSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = x - c, t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

// KB_j += a_ij g for j < i.
template <int SOLVER, int I, int S, int NE>
__device__ __forceinline__ void fb_spread(int i, const float (&g)[NE], float (&KB)[S][NE]) {
  using TB = Tab<SOLVER>;
  if constexpr (I < S) {
    if (i == I) {
#pragma unroll
      for (int j = 0; j < I; j++)
        if (TB::a(I, j) != 0.0) {
#pragma unroll
          for (int e = 0; e < NE; e++) KB[j][e] = fmaf(float(TB::a(I, j)), g[e], KB[j][e]);
        }
    } else {
      fb_spread<SOLVER, I + 1>(i, g, KB);
    }
  }
}

// Brownian values at times tsel[row] of the owned elements of the rows with flag
// set.  The four lanes of a quad of dimensions each descend the tree for one of
// the four owned rows, for all four dimensions, and exchange.
template <class SH, bool DEEP>
__device__ __forceinline__ void fb_brownian(const SolveParams &P, const BwdRows<SH::R> &R,
                                            const int *flag, const double *tsel,
                                            VbtQuadCache &vc, float (&W)[SH::NE],
                                            const FmMap<SH> &m) {
  static_assert(SH::NE == 4, "a quad's lanes take one row each");
  const int me = m.tl & 3, row = m.row0 + me;
  float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
  if (flag[row]) w = vbt_w_quad<DEEP>(P, R.idx[row], tsel[row] * R.dir[row], m.f >> 2, vc);
  // round x: dimension me ^ x of my row goes to lane me ^ x, whose row's value
  // of my dimension comes back
#pragma unroll
  for (int x = 0; x < 4; x++) {
    const int d = me ^ x;
    const float give = d == 0 ? w.x : d == 1 ? w.y : d == 2 ? w.z : w.w;
    const float got = __shfl_xor_sync(0xffffffffu, give, x);
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (e == d) W[e] = got;
  }
}

// A product did not complete: err is set, and the thread goes on (false) once product n
// has been issued.  So it stays behind the issuing warp, as the barriers between them
// need, and the walk ends with the iteration.  Out of line: in each of the nine waits it
// cost the 32-64 neural SDE 4 % (9001 rows: 5.93 -> 6.15 ms).
static __device__ __noinline__ bool fb_lost(int *err, const int *issued, int n) {
  *reinterpret_cast<volatile int *>(err) = 1;
  for (uint32_t i = 0; i < kFmDrain && *reinterpret_cast<const volatile int *>(issued) <= n; i++)
    __nanosleep(100);
  return false;
}

// The products of the field and its VJP, from the threads that own elements.
template <class SH>
struct FbField {
  static constexpr int D = SH::D, H = SH::H, R = SH::R, NE = SH::NE;
  static constexpr int NP = NE < 8 ? 2 : 4;  // pairs of a run of rows
  FbSmem<SH> &sm;
  const FmMap<SH> &m;
  const uint32_t tmem;
  const float b0, b1, b2, bs;
  uint32_t done = 0, donew = 0;  // products of either kind waited for
  bool ok = true, pending = false;
  bool first = true;  // no weight gradient of this iteration yet
  FbSum d0, d1, d2, ds;  // bias gradients of the thread's features and rows
  __device__ FbField(FbSmem<SH> &s, const FmMap<SH> &mm, uint32_t tm, const float *W)
      : sm(s), m(mm), tmem(tm), b0(W[SH::OB0 + mm.hf]), b1(W[SH::OB1 + mm.hf]), b2(W[SH::OB2 + mm.f]),
        bs(SH::SDE ? W[SH::OBS + mm.f] : 0.f) {}

  // this thread's operand writes and accumulator reads so far are done; the
  // product runs once every thread's are
  __device__ __forceinline__ void post(int job) {
    tc::fence_async_smem();
    tc::fence_before_sync();
    if (m.t == 0) *reinterpret_cast<volatile int *>(&sm.job) = job;
    fb_arrive(kFbWant);
  }
  // the weight-gradient accumulator may be overwritten
  __device__ __forceinline__ void release() {
    tc::fence_before_sync();
    fb_arrive(kFbFree);
  }
  // The next product on bar is complete.  Once one was not within the limit (err), the
  // thread goes on when it has been issued: it stays behind the issuing warp, as the
  // barriers between them need, and the walk ends with the iteration.
  __device__ __forceinline__ void wait(uint64_t *bar, uint32_t &n, const int *issued) {
    if (!ok || !tc::mbar_wait(bar, n & 1u, kFmWait)) ok = fb_lost(&sm.err, issued, int(n));
    n++;
    tc::fence_after_sync();
  }
  __device__ __forceinline__ void wait_chain() { wait(&sm.bar, done, &sm.issued); }
  __device__ __forceinline__ void wait_weights() { wait(&sm.barw, donew, &sm.issuedw); }
  // the weight-gradient product in flight is done: NC columns to the sum at dst
  template <int NC>
  __device__ __forceinline__ void collect(int src, int dst) {
    fb_accumulate<NC>(tmem + (uint32_t(m.tl & 96) << 16), src, dst, m.t, first);
  }
  // the stage's last ones
  __device__ __forceinline__ void collect_last() {
    pending = false;
    collect<D>(SH::TA, SH::T0);
    if constexpr (SH::SDE) collect<D>(SH::TA + D, SH::TS);
    first = false;
  }
  __device__ __forceinline__ void drain() {
    if (!pending) return;
    wait_weights();
    collect_last();
  }
  __device__ __forceinline__ void put(__nv_bfloat16 *buf, const float (&Y)[NE]) {
#pragma unroll
    for (int e = 0; e < NE; e += 2 * NP) {
      F2 v[NP];
#pragma unroll
      for (int j = 0; j < NP; j++) v[j] = f2_pack(Y[e + 2 * j], Y[e + 2 * j + 1]);
      fm_put<R, D>(reinterpret_cast<unsigned char *>(buf), m.f, m.row0 + e, v);
    }
  }
  __device__ __forceinline__ void owned(uint32_t acc, float bias, float (&F)[NE]) {
#pragma unroll
    for (int e = 0; e < NE; e += 2 * NP) {
      F2 v[NP];
      tc::tmem_sum3(acc + m.row0 + e, R, v);
#pragma unroll
      for (int j = 0; j < NP; j++)
        f2_unpack(f2_add(v[j], f2_set(bias)), F[e + 2 * j], F[e + 2 * j + 1]);
    }
  }
  __device__ __forceinline__ void hidden(float bias, __nv_bfloat16 *dst) {
#pragma unroll
    for (int c = 0; c < SH::HR; c += 8) {
      F2 v[4];
      tc::tmem_sum3(m.lanes + m.hrow0 + c, R, v);
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = tanh2(f2_add(v[j], f2_set(bias)));
      fm_put<R, H>(reinterpret_cast<unsigned char *>(dst), m.hf, m.hrow0 + c, v);
    }
  }
  // x, a1, a2 of the stage input Y; F (unless last_only) and sigma
  __device__ __forceinline__ void forward(const float (&Y)[NE], float (&F)[NE],
                                          float (&sig)[NE], bool want_f) {
    if (pending) wait_weights();  // (the last stage's products read x)
    put(sm.x, Y);
    post(kFbF0);
    if (pending) collect_last();
    wait_chain();
    if constexpr (SH::SDE) {
      owned(m.lanes + SH::N, bs, sig);
#pragma unroll
      for (int e = 0; e < NE; e += 2)
        f2_unpack(f2_mul(tanh2(sig[e], sig[e + 1]), f2_set(0.1f)), sig[e], sig[e + 1]);
    }
    hidden(b0, sm.a1);
    post(kFbF1);
    wait_chain();
    hidden(b1, sm.a2);
    if (want_f) {
      post(kFbF2);
      wait_chain();
      owned(m.lanes, b2, F);
    }
  }
  // g = acc (1 - a^2) of the owned hidden rows as the next cotangent operand
  __device__ __forceinline__ void back(const __nv_bfloat16 *a, __nv_bfloat16 *dst, FbSum &db) {
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < SH::HR; c += 8) {
      F2 v[4], h[4];
      fb_get<R, H>(a, m.hf, m.hrow0 + c, h);
      tc::tmem_sum3(m.lanes + m.hrow0 + c, R, v);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        // 1 - a^2
        v[j] = f2_mul(v[j], f2_fma(f2_mul(h[j], f2_set(-1.f)), h[j], f2_set(1.f)));
        float p, q;
        f2_unpack(v[j], p, q);
        sum += p + q;
      }
      fm_put<R, H>(reinterpret_cast<unsigned char *>(dst), m.hf, m.hrow0 + c, v);
    }
    db.add(sum);
  }
  // gY = d<G, F> / dY + d<Gs, sigma> / dY for the stage that forward() left, and
  // its parameter gradients
  __device__ __forceinline__ void backward(const float (&G)[NE], const float (&Gs)[NE],
                                           const float (&sig)[NE], float (&gY)[NE]) {
    put(sm.g3, G);
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < NE; e++) sum += G[e];
    d2.add(sum);
    if constexpr (SH::SDE) {
      // sigma = 0.1 tanh(z): d sigma / dz = 0.1 (1 - (sigma / 0.1)^2)
      float gz[NE], t = 0.f;
#pragma unroll
      for (int e = 0; e < NE; e++) {
        gz[e] = Gs[e] * 0.1f * (1.f - 100.f * sig[e] * sig[e]);
        t += gz[e];
      }
      ds.add(t);
      put(sm.gs, gz);
    }
    post(kFbB2);
    release();
    wait_chain();
    back(sm.a2, sm.g2, d1);
    // a gradient is collected while the next product of the chain runs
    post(kFbB1);
    wait_weights();
    collect<D>(SH::TA, SH::T2);
    release();
    wait_chain();
    back(sm.a1, sm.g1, d0);
    post(kFbB0);
    wait_weights();
    collect<H>(SH::TA, SH::T1);
    release();
    wait_chain();
    pending = true;
    owned(m.lanes, 0.f, gY);
  }
};

// Adds an accumulated weight gradient (ROWS x NC, TMEM columns tcol on) to the CTA's
// compensated partials at psum, pcomp, laid out [NC / 4][ROWS][4] so that a warp's
// 16-byte accesses are contiguous.
template <int MW, int ROWS, int NC>
__device__ __forceinline__ void fb_flush(uint32_t lanes, int tcol, float *psum, float *pcomp,
                                         int t) {
  const int lane = t & 31, q = (t >> 5) & 3;
  const int row = MW == 64 ? 16 * q + (lane & 15) : 32 * q + lane;
  const bool mine = row < ROWS && (MW != 64 || lane < 16);
  const int c0 = (t >> 7) * (NC / 2);
#pragma unroll 1
  for (int c = c0; c < c0 + NC / 2; c += 16) {
    float v[16];
    tc::tmem_ld16(lanes + uint32_t(tcol + c), v);
    if (mine) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float4 *ps = reinterpret_cast<float4 *>(psum + ((c >> 2) + j) * (ROWS * 4) + row * 4);
        float4 *pc = reinterpret_cast<float4 *>(pcomp + ((c >> 2) + j) * (ROWS * 4) + row * 4);
        float4 s = *ps, k = *pc;
        auto add = [](float &sv, float &cv, float x) {
          const float y = x - cv, u = sv + y;
          cv = (u - sv) - y;
          sv = u;
        };
        add(s.x, k.x, v[4 * j]);
        add(s.y, k.y, v[4 * j + 1]);
        add(s.z, k.z, v[4 * j + 2]);
        add(s.w, k.w, v[4 * j + 3]);
        *ps = s;
        *pc = k;
      }
    }
  }
}

template <int SOLVER, int D, int H, bool SDE, bool DEEP = false>
__global__ void __launch_bounds__((FbShape<D, H, SDE>::THREADS), 1)
    mlp_fm_bwd_kernel(SolveParams P, BwdParams Q) {
  using SH = FbShape<D, H, SDE>;
  using TB = Tab<SOLVER>;
  constexpr int S = TB::S, NE = SH::NE, M = SH::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FbSmem<SH> &sm = *reinterpret_cast<FbSmem<SH> *>(smem_raw);
  BwdRows<M> &R = sm.rows;
  const int t = threadIdx.x;
  const int n_save = P.n_save;

  if (t < 32) tc::tmem_alloc(&sm.slot, 512);
  {
    const float *W = P.mlp;
    const bool vec = (reinterpret_cast<uintptr_t>(W) & 15) == 0;
    fb_stage<H, D>(sm.w0, W + SH::OW0, t, SH::THREADS, vec);
    fb_stage<H, H>(sm.w1, W + SH::OW1, t, SH::THREADS, vec);
    fb_stage<D, H>(sm.w2, W + SH::OW2, t, SH::THREADS, vec);
    if constexpr (SDE) fb_stage<D, D>(sm.ws, W + SH::OWS, t, SH::THREADS, vec);
  }
  // Take trajectory q of the work order for row t: the first tile is fixed, the
  // queue hands out the rest.
  auto take = [&](unsigned long long q) {
    const bool got = q < (unsigned long long)P.batch;
    if (got) {
      bwd_row_init<SH>(R, t, P.order ? (int64_t)P.order[q] : (int64_t)q, P);
    } else {
      R.active[t] = 0;
      R.ld_kind[t] = kLoadNone;
    }
    R.loaded[t] = got;
  };
  if (t < M) {
    R.idx[t] = 0;
    R.mode[t] = kModeBwd;
    take((unsigned long long)blockIdx.x * M + t);
  }
  if (t == 0) {
    tc::mbar_init(&sm.bar, 1);
    tc::mbar_init(&sm.barw, 1);
    tc::mbar_init(&sm.drain, 1);
    sm.err = sm.issued = sm.issuedw = 0;
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = sm.slot;
  if (t >= SH::GT) {
    fb_issuer<SH>(sm, tmem);
  } else {
    const FmMap<SH> m(t, tmem);
    FbField<SH> field(sm, m, tmem, P.mlp);
    float *psum = Q.part_sum + size_t(blockIdx.x) * Q.n_params;
    float *pcomp = Q.part_comp + size_t(blockIdx.x) * Q.n_params;
    const unsigned long long queued = (unsigned long long)gridDim.x * M;

    float Y[NE], GY[NE];
    // Newly loaded rows: the cotangent of the final state (the t1 save and,
    // when t0 == t1, every ts save), and y at the step the row starts from.
    auto load_rows = [&]() {
#pragma unroll
      for (int e = 0; e < NE; e++) {
        const int row = m.row0 + e;
        if (R.loaded[row]) {
          const int64_t i = R.idx[row];
          const float *gys = Q.grad_ys + i * n_save * D + m.f;
          float g = 0.f;
          int slot = (P.save_t0 ? 1 : 0) + R.k_hi[row];
          if (R.N[row] == 0) {
            for (int m2 = 0; m2 < P.n_ts; m2++)
              g += *GBDX_AT(P, gys, (slot + m2) * D, 1, (n_save - 1) * D + 1,
                            GBDX_SITE_GRAD_YS);
            slot += P.n_ts;
          }
          if (P.save_t1)
            g += *GBDX_AT(P, gys, slot * D, 1, (n_save - 1) * D + 1, GBDX_SITE_GRAD_YS);
          GY[e] = g;
          Y[e] = 0.f;
        }
        if (R.ld_kind[row] == kLoadCheckpoint)
          Y[e] = *GBDX_AT(P, P.tape_y, (R.idx[row] * P.checkpoints + R.ld_slot[row]) * D + m.f,
                          1, P.batch * P.checkpoints * D, GBDX_SITE_TAPE_Y);
        else if (R.ld_kind[row] == kLoadScratch)
          Y[e] = *GBDX_AT(P, Q.scratch, (R.idx[row] * Q.seg_max + R.ld_slot[row]) * D + m.f, 1,
                          P.batch * Q.seg_max * D, GBDX_SITE_SCRATCH);
      }
    };
#pragma unroll
    for (int e = 0; e < NE; e++) Y[e] = GY[e] = 0.f;
    load_rows();
    fm_sync(0);
    if (t < M) {
      R.loaded[t] = 0;
      R.ld_kind[t] = kLoadNone;
    }

    float K[S][NE], F[NE], sig[NE], dW[NE];
    float Wc[NE];  // the carried Brownian values of the owned elements
#pragma unroll
    for (int e = 0; e < NE; e++) Wc[e] = dW[e] = sig[e] = 0.f;
    VbtQuadCache vc;  // this lane's tree path (SDE)
    vc.traj = -1;
    vc.node = 0;
    // the sums of up to kFbFlush iterations into the CTA's partials
    int since = 0;
    auto flush = [&]() {
      since = 0;
      field.drain();
      if (field.first) return;
      field.first = true;
      const uint32_t lanes = tmem + (uint32_t(t & 96) << 16);
      fb_flush<SH::MW, H, H>(lanes, SH::T1, psum + SH::OW1, pcomp + SH::OW1, t);
      fb_flush<SH::MW, H, D>(lanes, SH::T2, psum + SH::OW2, pcomp + SH::OW2, t);
      fb_flush<SH::MW, H, D>(lanes, SH::T0, psum + SH::OW0, pcomp + SH::OW0, t);
      if constexpr (SDE) fb_flush<64, D, D>(lanes, SH::TS, psum + SH::OWS, pcomp + SH::OWS, t);
    };
    while (fm_sync_or(0, t < M && R.active[t])) {
      // ---- A. row set-up: the step this row works on -----------------------
      int fwd = 0;
      if (t < M) {
        R.h[t] = 0.f;
        R.fin[t] = 0;
        R.live[t] = 0;
        if (R.active[t] && (R.mode[t] == kModeFwd || R.n[t] >= 0)) {
          R.live[t] = 1;
          fwd = R.mode[t] == kModeFwd;
          const int j = R.mode[t] == kModeBwd ? R.n[t] : R.m[t];
          const double *tt = GBDX_AT(P, P.tape_t, R.idx[t] * (P.max_steps + 1) + j, 2,
                                     P.batch * (P.max_steps + 1), GBDX_SITE_TAPE_T) - j;
          R.t_lo[t] = tt[j];
          R.t_hi[t] = tt[j + 1];
          const double dt = tt[j + 1] - tt[j];
          R.h[t] = float(R.dir[t] > 0 ? dt : -dt);
          if (R.mode[t] == kModeBwd) {
            int k = R.k_hi[t];
            while (k > 0 && (j == 0 || R.dir[t] * P.save_ts[k - 1] > tt[j])) k--;
            R.k_lo[t] = k;
          } else {
            R.k_lo[t] = R.k_hi[t];
          }
        }
        if constexpr (SDE) {
          R.w_lo[t] = R.live[t] && !(R.wt[t] == R.t_lo[t]);
          R.w_hi[t] = R.live[t] && !(R.wt[t] == R.t_hi[t]);
        }
      }
      const bool anyfwd = fm_sync_or(0, fwd);
      const bool anybwd = fm_sync_or(0, t < M && R.live[t] && !fwd);
      float h[NE];
      int live[NE], mode[NE];
      fm_rows<NE>(R.h, m.row0, h);
      fm_rows<NE>(R.live, m.row0, live);
      fm_rows<NE>(R.mode, m.row0, mode);
      if constexpr (SDE) {
        // W at both ends of the step; a row's consecutive iterations share an end,
        // whose value its threads carry (gbdx_mlp_bwd.cuh)
        float wa[NE], wb[NE];
        fb_brownian<SH, DEEP>(P, R, R.w_lo, R.t_lo, vc, wa, m);
        fb_brownian<SH, DEEP>(P, R, R.w_hi, R.t_hi, vc, wb, m);
#pragma unroll
        for (int e = 0; e < NE; e++) {
          const int row = m.row0 + e;
          if (live[e]) {
            if (!R.w_lo[row]) wa[e] = Wc[e];
            if (!R.w_hi[row]) wb[e] = Wc[e];
            Wc[e] = mode[e] == kModeFwd ? wb[e] : wa[e];
          }
          dW[e] = wb[e] - wa[e];
        }
        if (t < M && R.live[t]) R.wt[t] = R.mode[t] == kModeFwd ? R.t_hi[t] : R.t_lo[t];
      }
      // ---- B. BWD rows: cotangents of the step's end and of the saves inside
      // it, y1 = last stage input (SSAL) or y0 + sum b_j k_j ------------------
      float KB[S][NE], GY0[NE], GY1[NE];
#pragma unroll
      for (int e = 0; e < NE; e++) {
#pragma unroll
        for (int j = 0; j < S; j++) KB[j][e] = 0.f;
        GY0[e] = 0.f;
        GY1[e] = live[e] && mode[e] == kModeBwd ? GY[e] : 0.f;
      }
      while (P.n_ts > 0) {
        int fl = 0;
        if (t < M) {
          R.sflag[t] = 0;
          if (R.live[t] && R.mode[t] == kModeBwd && R.k_lo[t] < R.k_hi[t]) {
            const int k = R.k_hi[t] - 1;
            const double tsd = R.dir[t] * P.save_ts[k];
            const double tp = R.t_lo[t], tn = R.t_hi[t];
            R.theta[t] = float(tp == tn ? 0.0 : (tsd - tp) / (tn - tp));
            R.sslot[t] = (P.save_t0 ? 1 : 0) + k;
            R.k_hi[t] = k;
            R.sflag[t] = 1;
            fl = 1;
          }
        }
        if (!fm_sync_or(0, fl)) break;
#pragma unroll
        for (int e = 0; e < NE; e++) {
          const int row = m.row0 + e;
          if (R.sflag[row]) {
            const float gb =
                *GBDX_AT(P, Q.grad_ys, (R.idx[row] * n_save + R.sslot[row]) * D + m.f, 1,
                         P.batch * n_save * D, GBDX_SITE_GRAD_YS);
            float ay0, ay1, gg[7];
            interp_coeffs<SOLVER>(R.theta[row], ay0, ay1, gg);
            GY0[e] = fmaf(ay0, gb, GY0[e]);
            GY1[e] = fmaf(ay1, gb, GY1[e]);
#pragma unroll
            for (int j = 0; j < S; j++) KB[j][e] = fmaf(gg[j], gb, KB[j][e]);
          }
        }
        fm_sync(0);
      }
      float YB[NE];  // cotangent of the current stage input
      int top = 0;
#pragma unroll
      for (int e = 0; e < NE; e++) {
        if constexpr (TB::SSAL) {
          YB[e] = GY1[e];
        } else {
          GY0[e] += GY1[e];
#pragma unroll
          for (int j = 0; j < S; j++) KB[j][e] = fmaf(float(TB::b(j)), GY1[e], KB[j][e]);
          YB[e] = 0.f;
        }
        top |= !(KB[S - 1][e] == 0.f);
      }
      const bool anytop = fm_sync_or(0, top);
      // ---- C. forward stages: those whose increments a later one reads ------
      const int nf = anyfwd   ? (TB::SSAL ? S - 1 : S)
                     : !anybwd ? 0
                               : (anytop || !TB::SSAL ? S - 1 : S - 2);
      float Yi[NE];
#pragma unroll 1
      for (int i = 0; i < nf; i++) {
        stage_input<SOLVER, 1>(i, Y, K, Yi);
        field.forward(Yi, F, sig, true);
#pragma unroll
        for (int j = 0; j < S; j++)
          if (i == j) {
#pragma unroll
            for (int e = 0; e < NE; e++)
              K[j][e] = SDE ? F[e] * h[e] + sig[e] * dW[e] : F[e] * h[e];
          }
      }
      float Y1[NE];
      if (anyfwd) {
        // ---- D. FWD rows: store the recomputed state -----------------------
        if constexpr (TB::SSAL) {
          stage_input<SOLVER, 1>(S - 1, Y, K, Y1);
        } else {
#pragma unroll
          for (int e = 0; e < NE; e++) {
            float a = Y[e];
#pragma unroll
            for (int j = 0; j < S; j++) a = fmaf(float(TB::b(j)), K[j][e], a);
            Y1[e] = a;
          }
        }
#pragma unroll
        for (int e = 0; e < NE; e++) {
          const int row = m.row0 + e;
          if (live[e] && mode[e] == kModeFwd)
            *GBDX_AT(P, Q.scratch,
                     (R.idx[row] * Q.seg_max + (R.m[row] - R.cs[row])) * D + m.f, 1,
                     P.batch * Q.seg_max * D, GBDX_SITE_SCRATCH) = Y1[e];
        }
      }
      // ---- E. reverse stage loop -------------------------------------------
#pragma unroll 1
      for (int i = anybwd ? S - 1 : -1; i >= 0; i--) {
        float G[NE], Gs[NE], gY[NE];
        if (i < S - 1 || anytop) {
#pragma unroll
          for (int j = 0; j < S; j++)
            if (i == j) {
#pragma unroll
              for (int e = 0; e < NE; e++) {
                G[e] = KB[j][e] * h[e];
                Gs[e] = SDE ? KB[j][e] * dW[e] : 0.f;
              }
            }
          stage_input<SOLVER, 1>(i, Y, K, Yi);
          field.forward(Yi, F, sig, false);  // x, a1, a2 (and sigma)
          field.backward(G, Gs, sig, gY);
        } else {
#pragma unroll
          for (int e = 0; e < NE; e++) gY[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < NE; e++) {
          if (i == S - 1) gY[e] += YB[e];
          GY0[e] += gY[e];
        }
        fb_spread<SOLVER, 1>(i, gY, KB);
      }
      if (anybwd && ++since == kFbFlush) flush();
      // ---- F. advance the rows ---------------------------------------------
#pragma unroll
      for (int e = 0; e < NE; e++) {
        if (live[e]) {
          if (mode[e] == kModeFwd)
            Y[e] = Y1[e];
          else
            GY[e] = GY0[e];
        }
      }
      fm_sync(0);
      int fin = 0;
      if (t < M) {
        R.ld_kind[t] = kLoadNone;
        if (R.active[t]) {
          if (R.mode[t] == kModeFwd) {
            R.m[t]++;
            if (R.m[t] == R.n[t]) R.mode[t] = kModeBwd;
          } else {
            const int n = R.n[t] - 1;
            R.n[t] = n;
            const int s = R.s[t];
            if (n < 0) {
              R.fin[t] = 1;
              fin = 1;
            } else if (n % s == 0) {
              R.ld_kind[t] = kLoadCheckpoint;
              R.ld_slot[t] = n / s;
              R.cs[t] = n;
            } else if (n > R.cs[t]) {
              R.ld_kind[t] = kLoadScratch;
              R.ld_slot[t] = n - R.cs[t] - 1;
            } else {
              const int cs = (n / s) * s;
              R.cs[t] = cs;
              R.m[t] = cs;
              R.mode[t] = kModeFwd;
              R.ld_kind[t] = kLoadCheckpoint;
              R.ld_slot[t] = cs / s;
            }
          }
        }
      }
      // a product that did not complete makes this the last iteration, and leaves no
      // gradients of the rows that it had a part in
      const bool lost = *reinterpret_cast<volatile int *>(&sm.err);
      if (fm_sync_or(0, fin)) {
        // finished rows: dL/dy0 (plus the t0 save's cotangent)
#pragma unroll
        for (int e = 0; e < NE; e++) {
          const int row = m.row0 + e;
          if (R.fin[row]) {
            const int64_t i = R.idx[row];
            float g = GY[e];
            if (P.save_t0) g += Q.grad_ys[(i * n_save) * D + m.f];
            Q.grad_y0[i * D + m.f] = lost ? NAN : g;
          }
        }
        fm_sync(0);
        if (t < M && R.fin[t]) {
          if (lost)
            R.active[t] = 0;
          else
            take(queued + atomicAdd(P.queue, 1ull));
        }
      }
      fm_sync(0);
      if (lost) {
        // the rows still under way, and those that no CTA may be left to take
#pragma unroll
        for (int e = 0; e < NE; e++)
          if (R.active[m.row0 + e]) Q.grad_y0[R.idx[m.row0 + e] * D + m.f] = NAN;
        if (t < M)
          for (unsigned long long q = queued + atomicAdd(P.queue, 1ull);
               q < (unsigned long long)P.batch; q = queued + atomicAdd(P.queue, 1ull)) {
            const int64_t i = P.order ? (int64_t)P.order[q] : (int64_t)q;
            for (int d = 0; d < D; d++) Q.grad_y0[i * D + d] = NAN;
          }
        break;
      }
      load_rows();
      fm_sync(0);
      if (t < M) R.loaded[t] = 0;
    }
    flush();
    // bias gradients: the threads that share a feature, in a fixed order
    sm.bias[0][t] = field.d0.s;
    sm.bias[1][t] = field.d1.s;
    sm.bias[2][t] = field.d2.s;
    sm.bias[3][t] = field.ds.s;
    fm_sync(0);
    if (sm.err)
      for (int p = t; p < Q.n_params; p += SH::GT) psum[p] = NAN;
    auto total = [&](int which, int width) {
      FbSum s;
      for (int k = t; k < SH::GT; k += width) s.add(sm.bias[which][k]);
      return sm.err ? NAN : s.s;
    };
    if (t < H) {
      psum[SH::OB0 + t] = total(0, H);
      psum[SH::OB1 + t] = total(1, H);
    }
    if (t < D) {
      psum[SH::OB2 + t] = total(2, D);
      if (SDE) psum[SH::OBS + t] = total(3, D);
    }
    field.post(kFbExit);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (t < 32) tc::tmem_dealloc(tmem, 512);
}

template <int SOLVER, int D, int H, bool SDE>
cudaError_t launch_fm_bwd(const SolveParams &P, const BwdParams &Q, int grid, cudaStream_t s) {
  using SH = FbShape<D, H, SDE>;
  constexpr size_t bytes = sizeof(FbSmem<SH>);
  static_assert(bytes <= 227 * 1024 && bytes > 114 * 1024, "one CTA per SM");
  auto k = mlp_fm_bwd_kernel<SOLVER, D, H, SDE>;
  if constexpr (SDE)
    if (P.vbt_deep) k = mlp_fm_bwd_kernel<SOLVER, D, H, SDE, true>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  if (P.batch <= 0) return cudaSuccess;
  k<<<grid, SH::THREADS, bytes, s>>>(P, Q);
  return cudaGetLastError();
}

inline cudaError_t occupancy_fm_bwd(int *ctas) {
  *ctas = 1;
  return cudaSuccess;
}

template <int D, int H, bool SDE>
BwdEntry fm_bwd_entry(int solver) {
  switch (solver) {
    case GBDX_EULER: return BwdEntry{&launch_fm_bwd<GBDX_EULER, D, H, SDE>, &occupancy_fm_bwd};
    case GBDX_HEUN: return BwdEntry{&launch_fm_bwd<GBDX_HEUN, D, H, SDE>, &occupancy_fm_bwd};
    case GBDX_DOPRI5:
      if constexpr (!SDE)
        return BwdEntry{&launch_fm_bwd<GBDX_DOPRI5, D, H, SDE>, &occupancy_fm_bwd};
      break;
    case GBDX_TSIT5:
      if constexpr (!SDE)
        return BwdEntry{&launch_fm_bwd<GBDX_TSIT5, D, H, SDE>, &occupancy_fm_bwd};
      break;
    default: break;
  }
  return BwdEntry{nullptr, nullptr};
}

}  // namespace gbdx
