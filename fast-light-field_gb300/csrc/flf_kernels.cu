// CUDA kernels of libflf.so (sm_103a): lenslet-grid FFTs, the fused spectral
// multiply-accumulate over planes and lenslet offsets, inverse transform with
// crop / plane reduction / Richardson-Lucy epilogues, and the PSF transfer
// matrix precompute.  Host code that sequences them is flf_api.cu.
#include "flf_internal.cuh"
#include "flf_fft.cuh"

#include <algorithm>
#include <cstdio>

namespace flf {

// ----------------------------------------------------------------------------
// Complex helpers, templated on the real type (float runtime, double precompute)
// ----------------------------------------------------------------------------
template <typename R> struct CT;
template <> struct CT<float> { typedef float2 T; };
template <> struct CT<double> { typedef double2 T; };

template <typename C> __device__ __forceinline__ C cmk(decltype(C::x) a, decltype(C::x) b) {
  C r; r.x = a; r.y = b; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return cmk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return cmk<C>(a.x - b.x, a.y - b.y); }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  return cmk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C> __device__ __forceinline__ C cconj(C a) { return cmk<C>(a.x, -a.y); }

// ----------------------------------------------------------------------------
// Shared-memory Stockham FFT (mixed radix 2/3/4/5/7), batched over the images
// a CTA holds.  Stage with radix p and span m: butterfly i of a transform
// reads x[i + j*n/p], applies w^(j*(i mod m)) with w = exp(-2 pi i/(p m)),
// does a p-point DFT and writes y[(i - i mod m)*p + i mod m + j*m].
// The output is in natural order after the last stage.
// ----------------------------------------------------------------------------
template <typename C>
__device__ __forceinline__ C twid(const C *W, int idx, bool inv) {
  C w = W[idx];
  return inv ? cconj(w) : w;
}

template <typename C, int P>
__device__ __forceinline__ void dft_small(C (&u)[P], const C *W, int n, bool inv) {
  if (P == 2) {
    C a = u[0], b = u[1];
    u[0] = cadd(a, b);
    u[1] = csub(a, b);
  } else if (P == 4) {
    C a = cadd(u[0], u[2]), b = csub(u[0], u[2]);
    C c = cadd(u[1], u[3]), d = csub(u[1], u[3]);
    // -i*d (forward) or +i*d (inverse)
    C id = inv ? cmk<C>(-d.y, d.x) : cmk<C>(d.y, -d.x);
    u[0] = cadd(a, c);
    u[2] = csub(a, c);
    u[1] = cadd(b, id);
    u[3] = csub(b, id);
  } else {
    C v[P];
    const int st = n / P;
#pragma unroll
    for (int l = 0; l < P; l++) {
      C s = u[0];
#pragma unroll
      for (int j = 1; j < P; j++) s = cadd(s, cmul(u[j], twid(W, ((j * l) % P) * st, inv)));
      v[l] = s;
    }
#pragma unroll
    for (int l = 0; l < P; l++) u[l] = v[l];
  }
}

template <typename C, int P>
__device__ void fft_stage(const C *__restrict__ src, C *__restrict__ dst, int imgStride, int nimg,
                          int ntrans, int es, int ts, int n, int m, const C *W, bool inv) {
  const int nb = n / P;
  const int step = n / (P * m);
  const int total = nimg * ntrans * nb;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int i = idx % nb;
    const int tr = idx / nb;
    const int img = tr / ntrans;
    const int tl = tr - img * ntrans;
    const int base = img * imgStride + tl * ts;
    const int k = i % m;
    C u[P];
#pragma unroll
    for (int j = 0; j < P; j++) u[j] = src[base + (i + j * nb) * es];
#pragma unroll
    for (int j = 1; j < P; j++) u[j] = cmul(u[j], twid(W, j * k * step, inv));
    dft_small<C, P>(u, W, n, inv);
    const int ob = (i - k) * P + k;
#pragma unroll
    for (int j = 0; j < P; j++) dst[base + (ob + j * m) * es] = u[j];
  }
}

// Runs all stages of plan `pl` on a batch of transforms; returns the buffer
// holding the result (A or B).
template <typename C>
__device__ C *fft_pass(C *A, C *B, int imgStride, int nimg, int ntrans, int es, int ts,
                       const FftPlan &pl, const C *W, bool inv) {
  C *src = A, *dst = B;
  int m = 1;
  for (int s = 0; s < pl.nst; s++) {
    const int p = pl.rad[s];
    switch (p) {
      case 2: fft_stage<C, 2>(src, dst, imgStride, nimg, ntrans, es, ts, pl.n, m, W, inv); break;
      case 3: fft_stage<C, 3>(src, dst, imgStride, nimg, ntrans, es, ts, pl.n, m, W, inv); break;
      case 4: fft_stage<C, 4>(src, dst, imgStride, nimg, ntrans, es, ts, pl.n, m, W, inv); break;
      case 5: fft_stage<C, 5>(src, dst, imgStride, nimg, ntrans, es, ts, pl.n, m, W, inv); break;
      default: fft_stage<C, 7>(src, dst, imgStride, nimg, ntrans, es, ts, pl.n, m, W, inv); break;
    }
    __syncthreads();
    C *t = src; src = dst; dst = t;
    m *= p;
  }
  return src;
}

// ----------------------------------------------------------------------------
// Forward real 2-D transform f x f -> f x (f/2+1) of contiguous images, in
// float or double (the transfer-matrix precompute; the hot-path transforms are
// the size-specialised kernels of flf_fft.cuh).  Two real rows are packed into
// one complex row for the row pass and split afterwards.
// ----------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(256) k_rfft2(Rfft2Params p) {
  typedef typename CT<R>::T C;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int f = p.plan.n, fh = f / 2 + 1, isz = f * fh;
  C *W = reinterpret_cast<C *>(smraw);
  C *A = W + f;
  C *Bf = A + p.imgs_per_cta * isz;
  const C *tw = reinterpret_cast<const C *>(p.twiddle);
  for (int i = threadIdx.x; i < f; i += blockDim.x) W[i] = tw[i];

  const int g0 = blockIdx.x * p.imgs_per_cta;
  const int nb = min(p.imgs_per_cta, p.nimg - g0);
  const int nq = p.nq_rows;

  for (int idx = threadIdx.x; idx < nb * nq * f; idx += blockDim.x) {
    const int c = idx % f;
    const int q = (idx / f) % nq;
    const int img = idx / (f * nq);
    const R *im = reinterpret_cast<const R *>(p.src_img) + (long long)(g0 + img) * f * f;
    A[img * isz + q * f + c] = cmk<C>(im[(2 * q) * f + c], im[(2 * q + 1) * f + c]);
  }
  __syncthreads();

  C *Rr = fft_pass<C>(A, Bf, isz, nb, nq, 1, f, p.plan, W, false);
  C *Yb = (Rr == A) ? Bf : A;

  const int half = f / 2;
  for (int idx = threadIdx.x; idx < nb * half * fh; idx += blockDim.x) {
    const int k = idx % fh;
    const int q = (idx / fh) % half;
    const int img = idx / (half * fh);
    C y0 = cmk<C>(0, 0), y1 = cmk<C>(0, 0);
    if (q < nq) {
      const C Z = Rr[img * isz + q * f + k];
      const C Zc = cconj(Rr[img * isz + q * f + ((f - k) % f)]);
      y0 = cmk<C>((Z.x + Zc.x) * (R)0.5, (Z.y + Zc.y) * (R)0.5);
      const C d = csub(Z, Zc);
      y1 = cmk<C>(d.y * (R)0.5, -d.x * (R)0.5);
    }
    Yb[img * isz + (2 * q) * fh + k] = y0;
    Yb[img * isz + (2 * q + 1) * fh + k] = y1;
  }
  __syncthreads();

  C *Out = fft_pass<C>(Yb, Rr, isz, nb, fh, fh, 1, p.plan, W, false);
  C *dst = reinterpret_cast<C *>(p.dst) + (long long)g0 * isz;
  for (int idx = threadIdx.x; idx < nb * isz; idx += blockDim.x) dst[idx] = Out[idx];
}

// ----------------------------------------------------------------------------
// Fused spectral multiply-accumulate (the hot kernel).
//
// Forward projection accumulates a group of planes in registers (the
// reference's plane sum moved into Fourier space), back projection writes one
// plane after the other.  Every stored matrix element is read once from HBM.
// This replaces the reference's expandX + calculateRows{,Mirrored} launches
// (projector.py:395-459) and CalculateRow/CalculateRowBoth
// (py_light_field.cpp:303-341), which read and wrote the accumulator once per
// lenslet offset.
// ----------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// Bulk-copy pipeline primitives (sm_90+ PTX: mbarrier, cp.async.bulk).
// Every wait is bounded by a wall-clock limit read from %globaltimer.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *ptr) {
  return (unsigned)__cvta_generic_to_shared(ptr);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}
// Wait for phase `parity` of `bar`; false after `limit_ns` nanoseconds.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity,
                                          unsigned long long limit_ns) {
  for (int i = 0; i < 32; i++)   // (the timer is slow to read)
    if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity))
    if (global_ns() - t0 > limit_ns) return false;
  return true;
}
// Global -> shared bulk copy completing `bytes` of transaction count on `bar`.
__device__ __forceinline__ void bulk_g2s(void *sdst, const void *gsrc, unsigned bytes,
                                         unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_u32(sdst)),
      "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Orders this thread's earlier generic-proxy shared-memory accesses (as seen
// through a CTA fence) before its later async-proxy (bulk copy) accesses.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}

constexpr unsigned long long kWaitLimitNs = 1000000000ull;   // 1 s per wait

// Barrier of the first n threads of the block (the helper warp stays out).
__device__ __forceinline__ void bar_sync(int n) { asm volatile("bar.sync 1, %0;\n" ::"r"(n) : "memory"); }

// Operand table of one plane, straight from the input spectra:
//   sv[half block][row][side][t][u / u*] = (p0, m0, p1, m1),
// the real factors with which the row (C, D of every channel pair) enters the
// accumulators of the receiving side,  P += C p0 + D p1,  M += C m0 + D m1.
// With sa the spectrum that multiplies the row's channel directly and sb the
// one that meets it through the Mxy mirror, w = sa + conj sb, v = sa - conj sb:
// (p0, m0, p1, m1) = (Re w, Im v, Im w, -Re v).  rowS names sa and sb per use
// (0: the half block's own side, 1: the other side, through the transpose);
// a second row (kRowSecond) counts nothing where the receiving frequency pair
// is self-paired (u = u*), since its first row says the same.  A channel's four
// values of quad kq (u, u* of side 0, then of side 1) lie side by side in its
// spectrum.  Each enters one or two entries, so staging the spectra first would
// cost more than it saves.
template <int TF>
__device__ void build_sv(float4 *sv, const MacParams &p, const MacGroup &G, int zs, const short4 *rowS, int nhalf, bool selfp0,
                         bool selfp1, int kq, int first, int step) {
  constexpr int U = 4;                                 // entries per round, loads first
  const int R = p.L.nrow, NN = p.L.NN, nT = p.L.nrowT;
  const int ss = 4 * G.nquads;                         // values of a spectrum
  const int n = min(TF, p.T) * nhalf * R * 4;
  for (int i0 = first; i0 < n; i0 += U * step) {
    float2 sa[U], sb[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const int idx = i0 + k * step;
      sa[k] = sb[k] = make_float2(0.f, 0.f);
      if (idx >= n) continue;
      const int e = idx & 3, side = e >> 1, rest = idx >> 2;
      const int tb = rest / R, row = rest - tb * R;    // t * nhalf + half block
      const int t = tb / nhalf, use = side != tb - t * nhalf;
      if (use && row >= nT) continue;                  // never read
      if ((rowS[2 * R + row].x & kRowSecond) && (side ? selfp1 : selfp0)) continue;
      const short4 si = rowS[use * R + row];
      const int ia = (e & 1) ? si.z : si.x, ib = (e & 1) ? si.w : si.y;
      const float2 *src = G.S + (long long)(t * G.nzS + zs) * NN * ss + 4 * kq + e;
      if (ia >= 0) sa[k] = __ldg(src + ia * ss);
      if (ib >= 0) sb[k] = __ldg(src + ib * ss);
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const int idx = i0 + k * step;
      if (idx >= n) continue;
      const int rest = idx >> 2, tb = rest / R, row = rest - tb * R;
      const int t = tb / nhalf, bs = tb - t * nhalf;
      sv[((bs * R + row) * 2 + ((idx >> 1) & 1)) * 2 * TF + t * 2 + (idx & 1)] =
          make_float4(sa[k].x + sb[k].x, sa[k].y + sb[k].y, sa[k].y - sb[k].y, sb[k].x - sa[k].x);
    }
  }
}

// Shared memory of k_mac: ring | operand tables (forward two, back projection
// one) | back projection: output exchange | rowS | mbarriers.  (Forward, the
// exchange uses the first operand table, which is the larger.)
size_t mac_smem_bytes(const Layout &L, int TF, int stages, int chunk_rows, bool fwd) {
  return sizeof(float4) * ((size_t)stages * chunk_rows * L.NP + (size_t)(fwd && TF == 1 ? 2 : 1) * TF * 2 * L.nrow * 4) +
         (fwd ? 0 : sizeof(float2) * (size_t)TF * 4 * L.NN) + sizeof(short4) * 3 * L.nrow +
         2 * sizeof(unsigned long long) * (stages + 2) + 16;
}

// Accumulators of one thread: per side, frame, channel pair and u / u* the lane
// pairs X = (P.x, M.x) and Y = (P.y, M.y) for the packed two-lane FMA
// (__ffma2_rn, two IEEE FMAs in one issue slot).  The operands come as lane pairs
// from shared memory, only the streamed elements are doubled into both lanes
// (four per channel pair and row, used on both sides and all frames); pairs of
// (re, im) with doubled operands took 2 % longer at one frame and 5 % at four,
// plain FMAs 3 % and 10 %.
template <int TF, int PPT, int SD> struct MacAcc {
  float2 X[SD][TF][PPT][2], Y[SD][TF][PPT][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int s = 0; s < SD; s++)
#pragma unroll
      for (int t = 0; t < TF; t++)
#pragma unroll
        for (int k = 0; k < PPT; k++)
#pragma unroll
          for (int uv = 0; uv < 2; uv++) X[s][t][k][uv] = Y[s][t][k][uv] = make_float2(0.f, 0.f);
  }
};

// One stored row into the accumulators S0 .. S1 - 1 of a thread's sides (svr:
// the row's operands of the thread's first side).
template <int TF, int PPT, int SD, int S0, int S1>
__device__ __forceinline__ void mac_row(const float4 *row, const int (&off)[PPT], const float4 *svr,
                                        MacAcc<TF, PPT, SD> &a) {
  float4 e[PPT];
#pragma unroll
  for (int k = 0; k < PPT; k++) e[k] = row[off[k]];
#pragma unroll
  for (int s = S0; s < S1; s++)
#pragma unroll
    for (int t = 0; t < TF; t++)
#pragma unroll
      for (int uv = 0; uv < 2; uv++) {
        const float4 q = svr[(s * TF + t) * 2 + uv];   // p0, m0, p1, m1
        const float2 q0 = make_float2(q.x, q.y), q1 = make_float2(q.z, q.w);
#pragma unroll
        for (int k = 0; k < PPT; k++) {
          a.X[s][t][k][uv] = __ffma2_rn(make_float2(e[k].x, e[k].x), q0, a.X[s][t][k][uv]);
          a.Y[s][t][k][uv] = __ffma2_rn(make_float2(e[k].y, e[k].y), q0, a.Y[s][t][k][uv]);
        }
#pragma unroll
        for (int k = 0; k < PPT; k++) {
          a.X[s][t][k][uv] = __ffma2_rn(make_float2(e[k].z, e[k].z), q1, a.X[s][t][k][uv]);
          a.Y[s][t][k][uv] = __ffma2_rn(make_float2(e[k].w, e[k].w), q1, a.Y[s][t][k][uv]);
        }
      }
}

// Threads: `cw` warps side by side cover the channel pairs (PPT per lane), `H`
// row shares of such warps take alternate rows of a chunk, with SD = 1 a warp
// for each side of the quad.  CTAs per SM the registers are asked to allow.
// (At one frame shared memory allows three CTAs: asking for four took registers
// from the row loop, 2 to 10 % of the forward time.  Side warps: three at two
// frames forward, Nnum 19, 760 x 760 px, 31 planes 1885 -> 1745 us a projection,
// Nnum 23 with two 719 -> 642; back projection, whose outputs need registers,
// loses 3 to 5 % by the same.)
template <int TF, int TH, int SD, bool FWD> struct MacOcc {
  static constexpr int v = SD == 1     ? (TH == 256 ? (TF == 2 && FWD ? 3 : 2) : TF == 2 && FWD ? 2 : 1)
                           : TH == 128 ? (TF <= 2 ? 3 : 2)
                                       : (TF == 1 ? 2 : 1);
};

// One CTA = one frequency quad {(uy, ux), (ux, uy)} and a group of planes.
// Every stored row of the quad's half blocks streams through shared memory
// once and feeds both sides (frequency pairs) of the quad: its own side, and,
// for the transposable rows (stored first), the other side through the
// transpose T_{Tr i, Tr j}[(uy, ux)] = T_ij[(ux, uy)].  A lane owns PPT pairs
// of output channels (j, Mxy j) on both sides: the pair (j, Mxy j) at u and the
// pair (My j, Mx j) at u*, with Tr j for j on side 1.  The row shares' sums,
// the two sides of a diagonal quad (one frequency pair) and the two sums of a
// self-paired frequency are added through shared memory when a plane's output
// is due, in a fixed order, so there is no atomic and every output has one
// writer.
//
// What bounds it.  Real operands against C and D halve the multiplications of
// the complex form (a stored complex number feeds 8 two-lane FMAs per frame, 16
// before), which leaves the stream of the matrices as the bound at one frame:
// per 1808-byte row (Nnum 15) an SM takes 77 cycles at the measured copy rate,
// against 32 of FMA issue and 46 of shared memory (PPT = 2: two column warps
// read the row once and 64 B of operands each; one pair per lane would read the
// operands four times, four pairs would keep 64 accumulators a lane).  From two
// frames on it is FMA issue (two-lane FMAs take two cycles of a scheduler), and
// about 440 SM cycles a chunk beside its rows.
// Measured (GB300, Nnum 15, sum of the launches of a projection; complex form
// first): 1005 x 1005 px, 41 planes, one frame: back 2776 -> 1509 us (3.7 -> 6.8
// TB/s, the copy rate), forward 3006 -> 1536 us; 437 x 608 px, 31 planes, three
// frames: back 3202 -> 953 us; 450 x 450 px, 31 planes, four frames a launch:
// forward 477 -> 185 us, back 462 -> 172 us a launch.
// The stored rows stream through a ring of shared-memory stages filled by
// bulk copies (crossing plane boundaries).  Forward projection accumulates the
// planes of the group (the group sums are added by the inverse transform), and
// a helper warp (the last but one) builds the next plane's operand table while the
// current plane streams; back projection writes each plane's spectra when the
// plane is done.
template <int TF, bool FWD, int PPT, int TH, int SD>
__global__ void __launch_bounds__(TH + (FWD && TF == 1 ? 64 : 0), MacOcc<TF, TH, SD, FWD>::v) k_mac(MacParams p) {
  constexpr bool HELP = FWD && TF == 1;         // a helper warp builds the operand tables, two in turn, and a copy
                                                // warp refills the ring
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int s_abort;
  __shared__ int s_issued;                      // chunks handed to the bulk-copy engine
  __shared__ int s_plane[kMacMaxZgroup];        // plane slots of this CTA's z range
  volatile int *abortf = &s_abort;
  const Layout &L = p.L;
  const int NN = L.NN, N = L.N, NP = L.NP, R = L.nrow, nT = L.nrowT, NN2 = 2 * L.NN;
  const int CH = p.chunk_rows, NST = p.stages, H = p.shares;
  const int svn = TF * 2 * R * 4;                                            // float4 of an operand table
  float4 *ring = reinterpret_cast<float4 *>(smraw);                          // [NST][CH][NP]
  float4 *sv0 = ring + (size_t)NST * CH * NP;                                // [1|2][2][R][2][TF][2]
  float2 *outs = reinterpret_cast<float2 *>(FWD ? sv0 : sv0 + svn);     // [TF][side][u | u*][NN]
  short4 *rowS = reinterpret_cast<short4 *>(FWD ? reinterpret_cast<float2 *>(sv0 + (HELP ? 2 : 1) * svn) : outs + TF * 4 * NN);
  unsigned long long *full = reinterpret_cast<unsigned long long *>(rowS + 3 * R);
  unsigned long long *svfull = full + NST;               // [2] operand table built (helper's lanes arrive)
  unsigned long long *svfree = svfull + 2;               // [2] operand table read (a lane of each warp arrives)
  unsigned long long *empty = svfree + 2;                // copy warp: [NST] chunk read (a lane of each warp arrives)
  int *released = reinterpret_cast<int *>(empty);        // else: [NST] warps done with each slot

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = (blockDim.x >> 5) - (HELP ? 2 : 0);  // streaming warps
  const int nthreads = 32 * nwarps;

  // quad k = ux (ux + 1) / 2 + uy, uy <= ux
  int gi = 0;
  while (gi + 1 < p.ngroups && (int)blockIdx.x >= p.g[gi + 1].cta0) gi++;
  const MacGroup &G = p.g[gi];
  const int zgi = ((int)blockIdx.x - G.cta0) / G.nquads;      // z group
  const int kq = (int)blockIdx.x - G.cta0 - zgi * G.nquads;
  int ux = (int)((sqrtf(8.f * (float)kq + 1.f) - 1.f) * 0.5f);
  while ((ux + 1) * (ux + 2) / 2 <= kq) ux++;
  while (ux * (ux + 1) / 2 > kq) ux--;
  const int uy = kq - ux * (ux + 1) / 2;
  const bool diag = (uy == ux);
  const int hb0 = 2 * kq - ux;                   // first half block of the quad
  const int nhalf = diag ? 1 : 2;
  const bool selfp0 = (uy == 0) || (2 * uy == G.f), selfp1 = (ux == 0) || (2 * ux == G.f);
  const int z0 = zgi * G.zgroup;
  const int z1 = min(z0 + G.zgroup, G.nz);
  const int cph = (R + CH - 1) / CH;             // chunks per half block, none across two
  const int cpb = nhalf * cph;                   // chunks per (quad, plane)
  const int total = (z1 - z0) * cpb;
  const size_t halfElems = (size_t)R * NP;       // float4

  // Chunk g goes to ring slot g % NST.  Thread 0 fills the whole ring before
  // anything else.  After that, the warp that releases a slot last (each warp
  // counts itself out once it has finished its rows of the chunk) refills it at
  // once with chunk g + NST, so no thread ever waits for a slot to drain; forward at
  // one frame, where the registers allow one warp more, a copy warp does so as soon
  // as every streaming warp has arrived on the slot's `empty` barrier (Nnum 23, 460
  // px, 15 planes 425 -> 383 us a projection, Nnum 19, 760 px, 31 planes 1143 -> 1104,
  // Nnum 15, 450 px 317 -> 312; with more frames it spills or evens out).
  // p.drop_chunk >= 0 (a test of the bounded waits only): the first CTA never
  // issues that chunk, so the waits on its slot run out after p.wait_ns
  const int drop = blockIdx.x == 0 ? p.drop_chunk : -1;
  auto issue = [&](int gn, const int *planes) {
    if (gn == drop) return;
    const int zl_n = gn / cpb, ch_n = gn - zl_n * cpb, sl = gn % NST;
    const int bs_n = ch_n >= cph ? 1 : 0;
    const int r0 = (ch_n - bs_n * cph) * CH;
    const int nr = min(CH, R - r0);
    const float4 *src = G.P + ((long long)planes[zl_n] * G.nkp + hb0 + bs_n) * (long long)halfElems + (long long)r0 * NP;
    const unsigned bytes = (unsigned)(nr * NP * sizeof(float4));
    mbar_arrive_expect_tx(full + sl, bytes);
    bulk_g2s(ring + (size_t)sl * CH * NP, src, bytes, full + sl);
  };
  if (tid == 0) {
    for (int i = 0; i < NST; i++) {
      mbar_init(full + i, 1);
      if (HELP) mbar_init(empty + i, nwarps);
      else released[i] = 0;
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(svfull + i, 32);
      mbar_init(svfree + i, nwarps);
    }
    *abortf = 0;
    fence_mbar_init();
    const int pre = min(NST, total);
    for (int g = 0; g < pre; g++) issue(g, G.planes + z0);
    s_issued = pre;
  }
  for (int i = tid; i < 3 * R; i += blockDim.x) rowS[i] = p.rowS[i];
  for (int i = tid; i < z1 - z0; i += blockDim.x) s_plane[i] = G.planes[z0 + i];
  __syncthreads();   // barriers initialised, row tables staged
  build_sv<TF>(sv0, p, G, FWD ? z0 : 0, rowS, nhalf, selfp0, selfp1, kq, tid, blockDim.x);
  __syncthreads();

  if (HELP && warp == nwarps + 1) {
    // copy warp
    if (lane == 0) {
      int sl = 0, par = 0;
      for (int g = min(NST, total); g < total; g++) {
        if (!mbar_wait(empty + sl, par, p.wait_ns)) {
          *abortf = 1;
          atomicExch(p.err, 2);
          break;
        }
        fence_proxy_async_smem();   // the warps' reads come before the copy that overwrites them
        issue(g, s_plane);
        s_issued = g + 1;
        if (++sl == NST) { sl = 0; par ^= 1; }
      }
    }
    __syncthreads();   // the streaming warps' last barrier
    return;
  }
  if (HELP && warp == nwarps) {
    // helper warp: operand tables of the planes after the first, two in turn
    for (int zl = 1; zl < z1 - z0; zl++) {
      const int b = zl & 1;
      if (zl > 1 && !mbar_wait(svfree + b, ((zl >> 1) - 1) & 1, p.wait_ns)) break;   // the waiting warps report it
      build_sv<TF>(sv0 + b * svn, p, G, z0 + zl, rowS, nhalf, selfp0, selfp1, kq, lane, 32);
      mbar_arrive(svfull + b);
    }
    __syncthreads();   // the streaming warps' last barrier
    return;
  }

  const int cw = SD == 1 ? nwarps / (2 * H) : nwarps / H;   // column warps
  const int hs = warp / cw;
  const int h = SD == 1 ? hs >> 1 : hs;          // row share
  const int side0 = SD == 1 ? hs & 1 : 0;        // first side of this thread
  const int p0 = (warp - hs * cw) * 32 * PPT + lane;
  int off[PPT];                                  // this lane's channel pairs (repeating the last one past the end)
#pragma unroll
  for (int k = 0; k < PPT; k++) off[k] = min(p0 + 32 * k, NP - 1);

  MacAcc<TF, PPT, SD> acc;
  acc.zero();

  bool dead = false;
  // The chunk's place, stepped along: half block, its first row, ring slot and phase.
  int zl = 0, bs = 0, lo = 0, slot = 0;
  unsigned phase = 0;
  const float4 *stage = ring;
  const float4 *svz = sv0 + side0 * 2 * TF;      // operands of the plane, the thread's first side
  for (int g = 0; g < total; g++) {
    const int zi = z0 + zl;
    const bool first = bs == 0 && lo == 0 && zl > 0;                // first chunk of a later plane
    const bool last = bs == nhalf - 1 && lo + CH >= R;              // last chunk of a plane
    if (FWD && !HELP && first) {
      bar_sync(nthreads);   // every warp is done with plane zi - 1
      build_sv<TF>(sv0, p, G, zi, rowS, nhalf, selfp0, selfp1, kq, tid, nthreads);
      bar_sync(nthreads);
    }
    // table zl: the helper's fill number zl >> 1 of buffer zl & 1 (buffer 0's first one is not counted)
    if (!dead && ((HELP && first && !mbar_wait(svfull + (zl & 1), ((zl - 1) >> 1) & 1, p.wait_ns)) ||
                  !mbar_wait(full + slot, phase, p.wait_ns))) {
      dead = true;
      *abortf = 1;
      atomicExch(p.err, 2);
    }
    if (!dead) {
      // the chunk's rows: the transposable ones feed both sides, the others the
      // half block's own.  (One row per loop turn: loops of two rows were slower
      // throughout, the more code a row is - Nnum 15, 450 px, 31 planes: one frame
      // 328 and 319 us a projection forward, four with side warps 951 and 916 - and
      // rows read ahead by hand slower too, 996.)
      const int nr = min(CH, R - lo), nb = min(nr, nT - lo);   // rows; transposable ones (may be negative)
      const float4 *e = stage + h * NP, *q = svz + ((size_t)bs * R + lo + h) * 4 * TF;
      const int estep = H * NP, qstep = H * 4 * TF;
      int n = h;
      if constexpr (SD == 1) {
        const int ne = bs == side0 ? nr : nb;
#pragma unroll 1
        for (; n < ne; n += H, e += estep, q += qstep) mac_row<TF, PPT, 1, 0, 1>(e, off, q, acc);
      } else {
#pragma unroll 1
        for (; n < nb; n += H, e += estep, q += qstep) mac_row<TF, PPT, 2, 0, 2>(e, off, q, acc);
        if (bs == 0) {
#pragma unroll 1
          for (; n < nr; n += H, e += estep, q += qstep) mac_row<TF, PPT, 2, 0, 1>(e, off, q, acc);
        } else {
#pragma unroll 1
          for (; n < nr; n += H, e += estep, q += qstep) mac_row<TF, PPT, 2, 1, 2>(e, off, q, acc);
        }
      }
    }
    __syncwarp();
    if (lane == 0 && !dead) {
      if (HELP) {
        mbar_arrive(empty + slot);
        if (last) mbar_arrive(svfree + (zl & 1));
      } else {
        __threadfence_block();                       // this warp's reads of the slot come first
        if (atomicAdd(released + slot, 1) == nwarps - 1 && g + NST < total && !*abortf) {
          released[slot] = 0;
          __threadfence_block();
          fence_proxy_async_smem();                  // ... before the bulk copy that overwrites it
          issue(g + NST, s_plane);
          atomicAdd(&s_issued, 1);
        }
      }
    }

    const bool out_due = last && (!FWD || zi + 1 == z1);
    if (out_due) {
      // the row shares add their channel values into outs in share order
      if (FWD) bar_sync(nthreads);   // every warp is done with the operand tables
      for (int hh = 0; hh < H; hh++) {
        if (h == hh) {
#pragma unroll
          for (int k = 0; k < PPT; k++) {
            const int pr = p0 + 32 * k;
            if (pr < NP) {
              const int b = pr / N, a = pr - b * N;             // channel j = pr of side 0
              const int my = (N - 1 - b) * N + a, tr = a * N + b, mytr = (N - 1 - a) * N + b;
#pragma unroll
              for (int sd = 0; sd < SD; sd++) {
                const int s = SD == 1 ? side0 : sd;
                const int j = s ? tr : pr, m = s ? mytr : my;    // first channels of the pair at u and at u*
#pragma unroll
                for (int t = 0; t < TF; t++) {
                  float2 *ou = outs + (size_t)(t * 2 + s) * NN2, *ov = ou + NN;
                  // first + conj(second) = 2 P, first - conj(second) = 2 i M (the halves are in C and D)
                  auto put = [&](float2 *o, int c1, float2 X, float2 Y) {   // X = (P.x, M.x), Y = (P.y, M.y)
                    float2 x = make_float2(X.x - Y.y, Y.x + X.y), y = make_float2(X.x + Y.y, X.y - Y.x);
                    const int c2 = NN - 1 - c1;                  // equal for the centre, then x = y
                    if (hh > 0) {
                      const float2 ox = o[c1], oy = o[c2];
                      x.x += ox.x; x.y += ox.y; y.x += oy.x; y.y += oy.y;
                    }
                    o[c1] = x;
                    o[c2] = y;
                  };
                  put(ou, j, acc.X[sd][t][k][0], acc.Y[sd][t][k][0]);
                  put(ov, m, acc.X[sd][t][k][1], acc.Y[sd][t][k][1]);
                }
              }
            }
          }
        }
        bar_sync(nthreads);
      }
      if (!dead) {
        // (back projection: two lanes write a channel's 32 bytes of the quad)
        const int nt = min(TF, p.T);
        for (int idx = tid; idx < nt * 2 * NN; idx += nthreads) {
          const int s = idx & 1, tq = idx >> 1;
          const int t = tq / NN, q = tq - t * NN;
          if (diag && s) continue;                   // the other side is the same frequency pair
          const float2 *o = outs + (size_t)(t * 2 + s) * NN2 + q;
          float2 u = o[0], v = o[NN];
          if (diag) {
            const float2 u1 = o[NN2], v1 = o[NN2 + NN];
            u.x += u1.x; u.y += u1.y; v.x += v1.x; v.y += v1.y;
          }
          if (s ? selfp1 : selfp0) {
            u.x += v.x; u.y += v.y;
          }
          if (FWD) {                                 // row order
            const int oy = s ? ux : uy;
            float2 *op = reinterpret_cast<float2 *>(G.O) +
                         ((long long)(zgi * p.T + t) * NN + q) * (G.f * G.fh) + (s ? uy : ux);
            op[oy * G.fh] = u;
            if (!(s ? selfp1 : selfp0)) op[(G.f - oy) * G.fh] = v;
          } else {                                   // quad order
            G.O[(((long long)(t * G.nzo + zi) * NN + q) * G.nquads + kq) * 2 + s] = make_float4(u.x, u.y, v.x, v.y);
          }
        }
      }
      acc.zero();
      if (g + 1 < total) bar_sync(nthreads);   // the exchange buffer is free again
    }
    lo += CH;
    if (lo >= R) {
      lo = 0;
      if (++bs == nhalf) {
        bs = 0;
        zl++;
        if (HELP) svz += (zl & 1) ? svn : -svn;
      }
    }
    stage += CH * NP;
    if (++slot == NST) {
      slot = 0;
      stage = ring;
      phase ^= 1;
    }
  }
  // Never leave a bulk copy in flight into this CTA's shared memory.
  __syncthreads();
  if (tid == 0 && *abortf) {
    const int issued = s_issued;
    for (int g = max(0, issued - NST); g < issued; g++)
      if (g != drop) mbar_wait(full + (g % NST), (g / NST) & 1, kWaitLimitNs / 10);
  }
}

// ----------------------------------------------------------------------------
// Precompute: lenslet-grid kernels K_iq (real f x f images, circular) built
// from the stored PSF quadrant through the reference's symmetry map
// (projector.py:159-189): offset (b, a) uses H[bb][aa] (aa >= bb) or the
// transpose of H[aa][bb], flipped along rows when b > c and columns when a > c.
// ----------------------------------------------------------------------------
template <typename R>
__global__ void k_build_k(BuildKParams p) {
  const int N = p.N, NN = N * N, c = N / 2, nh = c + 1, h = p.h, f = p.f, Rr = p.R;
  const int img = blockIdx.x;             // rl * NN + q
  const int rl = img / NN, q = img % NN;
  const int i = p.rep_ch[p.rep0 + rl];
  const int b = i / N, a = i % N, be = q / N, al = q % N;
  const int bb = min(b, N - 1 - b), aa = min(a, N - 1 - a);
  R *dst = reinterpret_cast<R *>(p.dst) + (long long)img * f * f;
  for (int e = threadIdx.x; e < f * f; e += blockDim.x) {
    const int mm = e / f, nn = e % f;
    const int m = (mm <= Rr) ? mm : ((mm >= f - Rr) ? mm - f : 1 << 20);
    const int n = (nn <= Rr) ? nn : ((nn >= f - Rr) ? nn - f : 1 << 20);
    R v = 0;
    if (m < (1 << 19) && n < (1 << 19)) {
      const int y = m * N + be - b + p.ch;
      const int x = n * N + al - a + p.ch;
      if (y >= 0 && y < h && x >= 0 && x < h) {
        const int yy = (b > c) ? h - 1 - y : y;
        const int xx = (a > c) ? h - 1 - x : x;
        float hv;
        if (aa >= bb) hv = p.H[((long long)(bb * nh + aa) * h + yy) * h + xx];
        else hv = p.H[((long long)(aa * nh + bb) * h + xx) * h + yy];
        v = (R)hv;
      }
    }
    dst[e] = v;
  }
}

// Packed matrices of a chunk of representatives: the value of frequency pair
// (fy, fx) goes to its half block (quad (fy, fx) side 0 when fy <= fx, quad
// (fx, fy) side 1 otherwise) as C and D of every channel pair (see Layout); a
// row pair also stores the row at (f - fy, fx), with its columns mirrored.
template <typename R>
__global__ void k_pack(PackParams p) {
  typedef typename CT<R>::T C;
  const Layout &L = p.L;
  const int N = L.N, NN = L.NN, NP = L.NP, ffh = p.f * p.fh;
  const long long total = (long long)p.nrep_chunk * NP * p.nkp;
  const R sc = (R)(0.5 * p.scale);
  // C = (A + B) / 2, D = i (A - B) / 2 with A = first, B = conj second
  auto cd = [&](C a, C s) {
    return make_float4((float)((a.x + s.x) * sc), (float)((a.y - s.y) * sc), (float)(-(a.y + s.y) * sc),
                       (float)((a.x - s.x) * sc));
  };
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int pr = (int)(idx % NP);
    const long long r2 = idx / NP;
    const int rl = (int)(r2 % p.nrep_chunk);
    const int kp = (int)(r2 / p.nrep_chunk);
    const int fy = kp / p.fq, fx = kp % p.fq;       // frequency pair (fy, fx)
    const int lo = min(fy, fx), hi = max(fy, fx);
    const int hb = 2 * (hi * (hi + 1) / 2 + lo) - hi + (fy > fx ? 1 : 0);
    const int fs = fy ? p.f - fy : 0;
    const int rep = p.rep0 + rl;
    const int row = p.rep_row[rep];
    const C *sp = reinterpret_cast<const C *>(p.spec) + (long long)rl * NN * ffh;
    // the second half block of a quad holds channel Tr j at the place of j
    const int b = pr / N, a = pr - b * N;
    const int jb = fy > fx ? a : b, ja = fy > fx ? b : a;
    const int j = jb * N + ja;
    float4 *dst = p.P + ((long long)hb * L.nrow + row) * NP + pr;
    const long long o = fy * p.fh + fx;
    dst[0] = cd(sp[(long long)j * ffh + o], sp[(long long)(NN - 1 - j) * ffh + o]);
    if (p.rep_kind[rep] != 0) {
      const int my = (N - 1 - jb) * N + ja;
      const long long os = fs * p.fh + fx;
      dst[NP] = cd(sp[(long long)my * ffh + os], sp[(long long)(NN - 1 - my) * ffh + os]);
    }
  }
}

// ----------------------------------------------------------------------------
// Launchers
// ----------------------------------------------------------------------------
size_t rfft2_smem_bytes(int f, int imgs, int fp64) {
  const size_t cs = fp64 ? sizeof(double2) : sizeof(float2);
  const size_t isz = (size_t)f * (f / 2 + 1);
  return cs * ((size_t)f + 2 * (size_t)imgs * isz);
}
// (a refusal is reported here and must not come up again as the next launch's last error)
static cudaError_t set_smem(const void *fn, size_t bytes) {
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// ----------------------------------------------------------------------------
// Lenslet interleave.  A pixel row y = r*N + b holds row r of the N channel
// images (b, a), a = 0..N-1, interleaved with stride N.  Both kernels work
// on one pixel row per CTA so that every global access is coalesced: the
// pixel row is read or written contiguously and each channel row is a
// contiguous run of Lxp floats.  This is the reference's strided sub-image
// access (special_fftconvolve.py:85-105, py_light_field.cpp:1001-1027 on
// input; projector.py:792-796 and the RL update of lfdeconv.py:112-183 on
// output) moved out of the transforms.
// ----------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_split(SplitParams p) {
  extern __shared__ float row[];                 // X floats
  const int y = blockIdx.x, s = blockIdx.y;
  const int N = p.N, NN = N * N, X = p.X, Lx = p.Lx, Lxp = p.Lxp, Ly = p.Ly;
  const int t = s / p.nz, zi = s - t * p.nz;
  const int r = y / N, b = y - r * N;
  const bool inside = y < p.Y;                   // rows of the last lenslet row beyond Y are zeros
  if (inside) {
    const int plane = p.planes ? p.planes[zi] : zi;
    const float *src = p.src + plane * p.src_sz + t * p.src_st + (long long)y * X;
    constexpr int U = 4;                         // loads in flight per thread
    for (int x0 = threadIdx.x; x0 < X; x0 += U * blockDim.x) {
      float v[U];
#pragma unroll
      for (int k = 0; k < U; k++) v[k] = x0 + k * blockDim.x < X ? __ldg(src + x0 + k * blockDim.x) : 0.f;
#pragma unroll
      for (int k = 0; k < U; k++)
        if (x0 + k * blockDim.x < X) row[x0 + k * blockDim.x] = v[k];
    }
  }
  __syncthreads();
  float *dst = p.dst + ((long long)s * NN + b * N) * Ly * Lxp + (long long)r * Lxp;
  const long long cstride = (long long)Ly * Lxp;
  for (int i = threadIdx.x; i < N * Lxp; i += blockDim.x) {
    const int a = (int)p.dlxp.div(i);
    const int c = i - a * Lxp;
    const int x = c * N + a;
    dst[a * cstride + c] = (inside && c < Lx && x < X) ? row[x] : 0.f;
  }
}

__global__ void __launch_bounds__(256) k_merge(MergeParams p) {
  extern __shared__ __align__(16) float sm[];    // N rows of `pitch` floats
  const int y = blockIdx.x, s = blockIdx.y;
  const int N = p.N, NN = N * N, X = p.X, Lxp = p.Lxp, Ly = p.Ly;
  const int n4 = Lxp / 4, pitch = 4 * (n4 | 1);  // 16-byte groups of a channel row; odd, so that channels spread over the banks
  const int t = s / p.nzo, zo = s - t * p.nzo;
  const int r = y / N, beta = y - r * N;
  const float *src = p.src + ((long long)s * NN + beta * N) * Ly * Lxp + (long long)r * Lxp;
  const long long cstride = (long long)Ly * Lxp;
  for (int i = threadIdx.x; i < N * n4; i += blockDim.x) {
    const int a = (int)p.dlx4.div(i);
    const int q = i - a * n4;
    const float *g = src + a * cstride + 4 * q;
    float4 v = __ldg(reinterpret_cast<const float4 *>(g));
    for (int k = 1; k < p.nsum; k++) {
      const float4 w = __ldg(reinterpret_cast<const float4 *>(g + k * p.sum_stride));
      v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    *reinterpret_cast<float4 *>(sm + a * pitch + 4 * q) = v;
  }
  __syncthreads();
  const int plane = p.planes ? p.planes[zo] : zo;
  const long long row = (long long)y * X;
  float *out = p.out.p + plane * p.out.sz + t * p.out.st + row;
  const float *aux = p.aux.p ? p.aux.p + plane * p.aux.sz + t * p.aux.st + row : nullptr;
  const float *nrm = p.norm.p ? p.norm.p + plane * p.norm.sz + t * p.norm.st + row : nullptr;
  const int epi = p.epi;
  const bool need_o = epi == EPI_ADD || epi == EPI_RL_PREVEDEL || epi == EPI_RL_STANDARD;
  const bool need_a = epi == EPI_DIVIDE || epi == EPI_RL_PREVEDEL;
  const bool need_n = epi == EPI_RL_STANDARD && nrm != nullptr;
  constexpr int U = 4;                           // pixels per thread per round, loads first
  for (int x0 = threadIdx.x; x0 < X; x0 += U * blockDim.x) {
    float v[U], ov[U], av[U], nv[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const int x = x0 + k * blockDim.x;
      const bool ok = x < X;
      const int c = ok ? (int)p.dn.div(x) : 0;
      v[k] = ok ? sm[(x - c * N) * pitch + c] : 0.f;
      ov[k] = (ok && need_o) ? out[x] : 0.f;
      av[k] = (ok && need_a) ? __ldg(aux + x) : 0.f;
      nv[k] = (ok && need_n) ? __ldg(nrm + x) : 1.f;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const int x = x0 + k * blockDim.x;
      if (x >= X) break;
      float res;
      switch (epi) {
        case EPI_STORE: res = v[k]; break;
        case EPI_ADD: res = ov[k] + v[k]; break;
        case EPI_DIVIDE: res = __fdiv_rn(av[k], v[k]); break;
        case EPI_RL_PREVEDEL:          // x * (Htf / Ht(H x)), lfdeconv.py:112-145
          res = __fmul_rn(ov[k], __fdiv_rn(av[k], v[k]));
          if (res != res) res = 0.f;
          break;
        default:                       // x * Ht(y / H x) [/ norm], lfdeconv.py:147-183
          res = __fmul_rn(ov[k], v[k]);
          if (need_n) res = __fdiv_rn(res, nv[k]);
          if (res != res) res = 0.f;
          break;
      }
      out[x] = res;
    }
  }
}

// Threads of a CTA of k_split and k_merge, which takes one pixel row: eight pixels
// each.  The kernels are bound by the loads they keep in flight and, with short rows,
// by the CTAs' set-up: with 256 threads and one load at a time back projections spent
// 195 us on 41 planes of 1005 x 1005 px in k_merge and 41 on four frames of nine 450 x
// 450 px planes, 107 and 22 so; k_split 135 and 26, 88 and 17 (128 threads at four
// pixels each 24 and 19).
static unsigned row_threads(int X) { return (unsigned)std::min(128, std::max(32, ((X + 7) / 8 + 31) / 32 * 32)); }

cudaError_t launch_split(const SplitParams &p0, cudaStream_t s) {
  if (p0.nsets == 0) return cudaSuccess;
  SplitParams p = p0;
  p.dlxp = Div16::make((unsigned)p.Lxp);
  const dim3 grid(p.Ly * p.N, p.nsets);
  k_split<<<grid, row_threads(p.X), p.X * sizeof(float), s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_merge(const MergeParams &p0, cudaStream_t s) {
  if (p0.nsets == 0) return cudaSuccess;
  MergeParams p = p0;
  p.dlx4 = Div16::make((unsigned)(p.Lxp / 4));
  p.dn = Div16::make((unsigned)p.N);
  const dim3 grid(p.Y, p.nsets);
  k_merge<<<grid, row_threads(p.X), p.N * (p.Lxp / 4 | 1) * sizeof(float4), s>>>(p);
  return cudaGetLastError();
}

// ----------------------------------------------------------------------------
// Rectification resample: bilinear interpolation of a float image at a
// separable grid of query coordinates, in double precision.  This is the
// reference's RectBivariateSpline(kx = ky = 1) evaluation (rectify.py:8-81):
// a degree-1 B-spline through the pixel values is the bilinear interpolant.
// Queries outside [0, H-1] x [0, W-1] are clamped to the edge.
// ----------------------------------------------------------------------------
__device__ __forceinline__ void bilinear_cell(double q, int n, int &i0, double &t) {
  if (n < 2) { i0 = 0; t = 0.0; return; }
  const double qc = fmin(fmax(q, 0.0), (double)(n - 1));
  i0 = min((int)floor(qc), n - 2);
  t = qc - (double)i0;
}

__global__ void __launch_bounds__(256) k_resample_bilinear(ResampleParams p) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)p.ny * p.nx) return;
  const int r = (int)(idx / p.nx), c = (int)(idx - (long long)r * p.nx);
  int y0, x0;
  double fy, fx;
  bilinear_cell(p.yq[r], p.H, y0, fy);
  bilinear_cell(p.xq[c], p.W, x0, fx);
  const int y1 = min(y0 + 1, p.H - 1), x1 = min(x0 + 1, p.W - 1);
  const float *row0 = p.img + (long long)y0 * p.W, *row1 = p.img + (long long)y1 * p.W;
  const double top = (1.0 - fx) * (double)row0[x0] + fx * (double)row0[x1];
  const double bot = (1.0 - fx) * (double)row1[x0] + fx * (double)row1[x1];
  p.out[idx] = (1.0 - fy) * top + fy * bot;
}

cudaError_t launch_resample_bilinear(const ResampleParams &p, cudaStream_t s) {
  const long long n = (long long)p.ny * p.nx;
  if (n == 0) return cudaSuccess;
  k_resample_bilinear<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(p);
  return cudaGetLastError();
}

// Transforms: the hot path runs the size-specialised kernels (flf_fft.cuh),
// one per even 7-smooth size up to kMaxF; the precompute (contiguous float or
// double images) runs the runtime-plan kernel above.
cudaError_t launch_rfft2(const Rfft2Params &p, int fp64, cudaStream_t s) {
  if (p.nimg == 0) return cudaSuccess;
  if (p.mode == 0) {
    if (fp64) return cudaErrorInvalidValue;
    switch (p.plan.n) {
#define FLF_CASE(F) \
      case F: return sfft::rfft2_sized<F>(p, s);
      FLF_SFFT_SIZES(FLF_CASE)
#undef FLF_CASE
      default: return cudaErrorInvalidValue;
    }
  }
  const size_t sm = rfft2_smem_bytes(p.plan.n, p.imgs_per_cta, fp64);
  const int grid = (p.nimg + p.imgs_per_cta - 1) / p.imgs_per_cta;
  cudaError_t e;
  if (fp64) {
    if ((e = set_smem((const void *)k_rfft2<double>, sm)) != cudaSuccess) return e;
    k_rfft2<double><<<grid, 256, sm, s>>>(p);
  } else {
    if ((e = set_smem((const void *)k_rfft2<float>, sm)) != cudaSuccess) return e;
    k_rfft2<float><<<grid, 256, sm, s>>>(p);
  }
  return cudaGetLastError();
}

cudaError_t launch_irfft2(const Irfft2Params &p, cudaStream_t s) {
  if (p.nimg == 0) return cudaSuccess;
  switch (p.plan.n) {
#define FLF_CASE(F) \
    case F: return sfft::irfft2_sized<F>(p, s);
    FLF_SFFT_SIZES(FLF_CASE)
#undef FLF_CASE
    default: return cudaErrorInvalidValue;
  }
}

int mac_max_frames() { return 4; }

// Warps side by side over the channel pairs, and row shares: about 128 threads
// per unit of p.split, at most 256; a small Nnum's single column warp keeps a unit's
// rows to itself, since a CTA then has few rows and its sums cost more to join than
// to make (Nnum 5, 31 planes of 250 x 300 px, four frames: back 129 us a launch with
// four shares, 76 with two, 58 with one; Nnum 7, 25 planes, one frame 44, 31, 31).
// Two pairs per lane from 33 pairs on.
// A warp for each side halves a thread's accumulators and its loop's code and
// doubles the warps, for twice the reads of the streamed rows from shared memory;
// us a projection with sides together and apart, back | forward:
//   Nnum  5, 250 px, 31 planes: 1 frame  39, 48 |  58, 60;  4 frames 175, 143 | 204, 161
//   Nnum 11, 330 px, 31 planes: 1 frame 138, 122 | 147, 129; 4 frames 721, 502 | 626, 457
//   Nnum 15, 450 px, 31 planes: 1 frame 303, 311 | 319, 357; 2 frames 561, 613 | 557, 613;
//                               3 frames 765, 704 | 798, 742; 4 frames 956, 900 | 969, 916
//   Nnum 19, 380 px, 21 planes: 1 frame 257, 246 | 282, 349; 2 frames 475, 408 | 499, 459;
//                               4 frames 1025, 842 | 811, 711
//   Nnum 23, 460 px, 15 planes: 1 frame 388, 377 | 425, 545; 2 frames 796, 634 | 706, 642;
//                               4 frames 1397, 1122 | 1389, 1097
// From seven column warps on a CTA has no room for more.
MacThreads mac_threads(const Layout &L, int split, int frames, bool fwd) {
  MacThreads t;
  t.ppt = L.NP > 32 ? 2 : 1;
  t.cw = (L.NP + 32 * t.ppt - 1) / (32 * t.ppt);
  t.sides = t.cw == 1   ? (frames >= 2 || t.ppt == 2 ? 1 : 2)
            : t.cw == 2 ? (frames >= 3 ? 1 : 2)
            : t.cw <= 6 ? (frames >= 2 || !fwd ? 1 : 2)
                        : 2;
  t.shares = t.sides == 1 && t.cw > 1 ? std::max(1, 4 / t.cw) : t.cw == 1 ? split : std::max(1, std::min(4 * split / t.cw, 8 / t.cw));
  return t;
}

template <int TF, bool FWD>
static cudaError_t launch_mac_tf(const MacParams &p0, cudaStream_t s) {
  MacParams p = p0;
  const MacThreads th = mac_threads(p.L, p.split, TF, FWD);
  p.shares = th.shares;
  const size_t sm = mac_smem_bytes(p.L, TF, p.stages, p.chunk_rows, FWD);
  int ctas = 0;
  for (int i = 0; i < p.ngroups; i++) {
    MacGroup &G = p.g[i];
    G.cta0 = ctas;
    ctas += G.nquads * ((G.nz + G.zgroup - 1) / G.zgroup);
  }
  const dim3 grid(ctas);
  const int threads = 32 * th.cw * th.shares * (th.sides == 1 ? 2 : 1);
  const int block = threads + (FWD && TF == 1 ? 64 : 0);   // and the helper and copy warps
  // (only the shapes that mac_threads gives for these frames and this direction are built)
  void (*fn)(MacParams) = nullptr;
  if (th.sides == 1) {
    if (th.ppt == 1) {
      if constexpr (TF >= 2) fn = k_mac<TF, FWD, 1, 256, 1>;
    } else if (threads <= 256) {
      fn = k_mac<TF, FWD, 2, 256, 1>;
    } else {
      if constexpr (TF >= 2 || !FWD) fn = k_mac<TF, FWD, 2, 384, 1>;
    }
  } else if (th.ppt == 1) {
    if constexpr (TF == 1) fn = k_mac<TF, FWD, 1, 128, 2>;
  } else if (threads <= 128) {
    if constexpr (TF <= 2) fn = k_mac<TF, FWD, 2, 128, 2>;
  } else {
    fn = k_mac<TF, FWD, 2, 256, 2>;
  }
  if (!fn) return cudaErrorInvalidValue;
  cudaError_t e = set_smem((const void *)fn, sm);
  if (e != cudaSuccess) return e;
  fn<<<grid, block, sm, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_mac(const MacParams &p, bool forward, cudaStream_t s) {
  if (p.T <= 1) return forward ? launch_mac_tf<1, true>(p, s) : launch_mac_tf<1, false>(p, s);
  if (p.T == 2) return forward ? launch_mac_tf<2, true>(p, s) : launch_mac_tf<2, false>(p, s);
  if (p.T == 3) return forward ? launch_mac_tf<3, true>(p, s) : launch_mac_tf<3, false>(p, s);
  return forward ? launch_mac_tf<4, true>(p, s) : launch_mac_tf<4, false>(p, s);
}

cudaError_t launch_build_k(const BuildKParams &p, int nimg, cudaStream_t s) {
  if (nimg == 0) return cudaSuccess;
  if (p.fp64) k_build_k<double><<<nimg, 256, 0, s>>>(p);
  else k_build_k<float><<<nimg, 256, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_pack(const PackParams &p, cudaStream_t s) {
  const long long total = (long long)p.nrep_chunk * p.L.NP * p.nkp;
  if (total == 0) return cudaSuccess;
  long long blocks = (total + 255) / 256;
  if (blocks > 65535LL * 16) blocks = 65535LL * 16;
  if (p.fp64) k_pack<double><<<(unsigned)blocks, 256, 0, s>>>(p);
  else k_pack<float><<<(unsigned)blocks, 256, 0, s>>>(p);
  return cudaGetLastError();
}

}  // namespace flf
