// The tiled PCG: the persistent solve of the forms with FP64 vectors (the
// algorithm of implizit.rs:370-426 with the release pass :908-943, as in
// k3d_solve.cuh), every CTA owning one compact tile of the mesh.
//
// What bounds it. The reference loop needs two global sums and one exchange
// of w per iteration; the rest is a 3x3-block row product (13 blocks a row on
// a regular mesh) whose blocks are the bulk of the bytes. So
//  * a CTA's rows are one tile (recursive bisection of the points at upload);
//    w (or c) of the tile and of its halo lie in shared memory, and the row
//    product gathers from there through 16-bit local columns;
//  * the vectors r, A c, c (or w) and, up to two rows a thread, dv stay in
//    registers for the whole solve;
//  * the blocks lie in slabs (32 rows of one warp x one rank, with their
//    columns). As many slabs as fit stay in shared memory for the whole
//    launch; the others (of regular sheets from 36 k points FP64 and 66 k FP32
//    blocks on: 45 % there, 86 % at 160 k FP32, all at 90 k FP64) pass through a
//    ring of bulk copies that each warp keeps full by itself, its first copies on
//    their way before the sum is in;
//  * halo values and the CTAs' partial sums travel as words that carry their
//    own sequence number beside 32 bits of payload: a reader polls the datum
//    itself, so an exchange costs one store and one load latency, without
//    fence, arrival counter or second round trip;
//  * with FP32 blocks the row product applies A to w and forms
//    A c = A w + beta A c_prev, so it runs while the sum that gives beta is
//    still travelling.
// Measured against the launch over ELL rows (k3d_solve.cuh) in one call on a
// B200, a solve through the host interface: 160 k points, FP32 blocks, 1813
// iterations 59.8 -> 33.8 ms; 36 k, FP64, 3320 iterations 36.7 -> 24.7 ms;
// 100 k, FP64, 5840 iterations 232 -> 129 ms; 66 k, FP32 blocks, 3386
// iterations 36.6 -> 26.2 ms; 6.6 k, FP64, 50 iterations 0.92 -> 0.61 ms. What
// is left of an iteration: the two sums and the halo (about 1500 cycles a hop,
// 2600 where 148 CTAs poll one another), the row product at 30 cycles a slab (23
// shared-memory wavefronts, 18 of the conversion unit), the streamed slabs, and
// the warps' unequal shares: a CTA's slices go to its 16 warps whole, so the
// longest warp has 1.4 times the mean at 160 k points, 1.5 at 104 k FP64 of a
// garment, 2.1 at 36 k FP64 (8 warps have none), and ncu puts the warps at
// barriers first. From L2 come 19.5 MB an iteration in 8.1 us at 66 k points, 98 MB
// in 19.8 us at 160 k (25 MB of it from memory), 19.8 MB in 8.6 us at 36 k FP64.
// Self-collision springs come as merged rows of blocks (federzeilen): with the
// launch over ELL rows, which forms each spring's products and sums them by
// point, 205 k points with 63 k springs, 3051 iterations, took 217 ms, here
// 117 ms; two layers of 3 k points, 907 iterations in ten solves, 30 ms and 16.
// Sums are deterministic: a fixed tree per CTA, then the CTAs' partials in
// CTA order in every CTA. Every wait is bounded (StepArgs::frist_ns). One that
// gives up records K3D_TIMEOUT, and the others, which look at that record now and
// then, give up too; waits for a warp's own copies do not, so no CTA leaves with
// copies under way into its shared memory. The CTA's threads leave together: a
// barrier lies between each look at sh.err and the next wait that may set it. A
// launch that finds the record set returns before its first copy.
#include "k3d_solve.cuh"

namespace k3d {
namespace {

constexpr int kNT = kSolveBlock;
constexpr int kNW = kNT / 32;

// A slab: 32 blocks as two 4-vectors and a scalar per lane, then the lanes'
// local columns.
template <typename R>
struct Satz {
  static constexpr unsigned v = 128 * sizeof(R), w = 256 * sizeof(R), spalte = 288 * sizeof(R);
  static constexpr unsigned bytes = kachel_satz(sizeof(R));
};

// The dynamic shared memory: KSh, the tile, the warps' slabs. Kept as offsets
// from this base, so that every access is known to be shared memory.
extern __shared__ __align__(128) char g_roh[];

struct KSh {
  unsigned long long bar[kNW][kKachelStufen + 1];  // per warp: its ring's stages, then its resident slabs
  double red[2][kNW];
  double arr[2][512 + 32];  // posted words (of warps: a gap after every 16)
  Grp g;
  KachelBlk b;
  unsigned bidx;
  unsigned federn;  // rows of springs of this CTA
  int err;
};

// ------------------------------------------------------------ words with a sequence number
__device__ __forceinline__ void st_wort(ulonglong2* p, double v, uint32_t ep) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)ep << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
               : "memory");
}
__device__ __forceinline__ bool ld_wort(const ulonglong2* p, uint32_t ep, double& v) {
  unsigned long long x, y;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
  v = __longlong_as_double((long long)((y << 32) | (x & 0xffffffffull)));
  return uint32_t(x >> 32) == ep && uint32_t(y >> 32) == ep;
}

// A bounded wait for another CTA: false when it is to give up (another wait did, or time is out).
struct Warten {
  unsigned n = 0;
  uint64_t t0 = 0;
};
__device__ __forceinline__ bool weiter(const StepArgs& a, KSh& sh, Warten& w) {
  if ((++w.n & 63u) != 0u) return true;
  if (*reinterpret_cast<volatile int*>(&sh.err) != 0) return false;
  const int e = ld_relaxed_i32(&a.sync->error);
  const uint64_t t = globaltimer();
  if (w.t0 == 0) w.t0 = t;
  if (e == 0 && t - w.t0 <= a.frist_ns) return true;
  if (e == 0) atomicCAS(&a.sync->error, 0, K3D_STATUS_TIMEOUT);
  *reinterpret_cast<volatile int*>(&sh.err) = K3D_STATUS_TIMEOUT;
  return false;
}
// Whether a wait of the CTA gave up. ohne_abbruch is the same in every thread
// where a barrier lies before it and another before the next wait; einig is both
// (its vote costs 400 cycles more than a barrier, so the loop has none).
__device__ __forceinline__ bool ohne_abbruch(KSh& sh) { return *reinterpret_cast<volatile int*>(&sh.err) == 0; }
__device__ __forceinline__ bool einig(KSh& sh) { return __syncthreads_or(ohne_abbruch(sh) ? 0 : 1) == 0; }
__device__ __forceinline__ double hol_wort(const StepArgs& a, KSh& sh, const ulonglong2* p, uint32_t ep) {
  double v;
  Warten w;
  while (!ld_wort(p, ep, v) && weiter(a, sh, w)) {
  }
  return v;
}

// The vector of three words a plane apart (its loads travel together).
__device__ __forceinline__ bool ld_wort3(const ulonglong2* p, int64_t ebene, uint32_t ep, D3& v) {
  const bool a = ld_wort(p, ep, v.x), b = ld_wort(p + ebene, ep, v.y), c = ld_wort(p + 2 * ebene, ep, v.z);
  return a && b && c;
}
__device__ __forceinline__ D3 hol_wort3(const StepArgs& a, KSh& sh, const ulonglong2* p, uint32_t ep) {
  D3 v;
  Warten w;
  while (!ld_wort3(p, a.n, ep, v) && weiter(a, sh, w)) {
  }
  return v;
}

// ------------------------------------------------------------ grid sums
// The posted parts of sum k under `seq`, copy c. Every CTA polls every other
// CTA's part, so each part is posted in several copies, and a CTA polls one
// of them: fewer readers wait on the same lines.
__device__ __forceinline__ ulonglong2* summe(const StepArgs& a, uint32_t seq, unsigned c, int k) {
  return a.ka_summe + (((size_t(seq & 1u) * 2 + k) * kKachelKopien) + c) * kKachelWorte;
}
// Posts this CTA's part of NV sums under the sequence number `seq`, its
// warps' sums or their sum in warp order. Every warp of the CTA has come this
// far when it returns.
template <int NV>
__device__ __forceinline__ void melden(const StepArgs& a, KSh& sh, double (&v)[NV], uint32_t seq) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool einzeln = sh.b.einzeln != 0;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (einzeln) {
      if (32 * unsigned(warp) < sh.b.rows && lane < kKachelKopien) st_wort(summe(a, seq, lane, k) + sh.b.wort0 + warp, x, seq);
    } else if (lane == 0) {
      sh.red[k][warp] = x;
    }
  }
  __syncthreads();
  if (!einzeln && warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double x = 0.0;
#pragma unroll
      for (int w = 0; w < kNW; ++w) x += sh.red[k][w];
      if (lane < kKachelKopien) st_wort(summe(a, seq, lane, k) + sh.b.wort0, x, seq);
    }
  }
}
// The sums posted under `seq` by every CTA of the group, the same bits in
// every thread (after a wait that gave up too, of no meaning then). Double-buffered
// by the number's parity: a CTA posts seq + 2 only after it has waited for seq + 1,
// which every CTA posts after its wait for seq.
// `vor`: this thread's part of the first sum as it was read ahead (vorab).
struct Vorab {
  double v = 0.0;
  bool da = false;
};
__device__ __forceinline__ void vorab(const StepArgs& a, const KSh& sh, Vorab& v, uint32_t seq) {
  if (threadIdx.x < sh.b.worte)
    v.da = ld_wort(summe(a, seq, sh.bidx % kKachelKopien, 0) + sh.b.gruppe0 + threadIdx.x, seq, v.v);
}
template <int NV>
__device__ __forceinline__ void sammeln(const StepArgs& a, KSh& sh, double (&v)[NV], uint32_t seq,
                                        Vorab vor = Vorab()) {
  const unsigned nb = sh.b.worte, lane = threadIdx.x & 31;
  const bool einzeln = sh.b.einzeln != 0;
  if (threadIdx.x < nb) {
    const unsigned i = einzeln ? threadIdx.x + threadIdx.x / 16 : threadIdx.x;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      sh.arr[k][i] = k == 0 && vor.da ? vor.v
                                      : hol_wort(a, sh, summe(a, seq, sh.bidx % kKachelKopien, k) + sh.b.gruppe0 + threadIdx.x, seq);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double x = 0.0;
    if (einzeln) {  // a lane adds 16 warps' words in order, as a CTA of 16 warps does
#pragma unroll
      for (unsigned w = 0; w < 16; ++w) x += 16 * lane + w < nb ? sh.arr[k][17 * lane + w] : 0.0;
    } else {
      double t[kKachelBloecke / 32];
#pragma unroll
      for (int j = 0; j < kKachelBloecke / 32; ++j) t[j] = lane + 32 * j < nb ? sh.arr[k][lane + 32 * j] : 0.0;
#pragma unroll
      for (int j = 0; j < kKachelBloecke / 32; ++j) x += t[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    v[k] = x;
  }
}

// ------------------------------------------------------------ the blocks of a warp
__device__ __forceinline__ uint32_t smem(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(unsigned long long* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem(b)) : "memory");
}
__device__ __forceinline__ void bar_erwarte(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_da(unsigned long long* b, unsigned par) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem(b)), "r"(par)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void kopiere(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem(dst)),
               "l"(src), "r"(bytes), "r"(smem(b))
               : "memory");
}

__device__ __forceinline__ void kopiere_weg(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
  unsigned long long regel;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(regel));
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
          smem(dst)),
      "l"(src), "r"(bytes), "r"(smem(b)), "l"(regel)
      : "memory");
}

// A warp's blocks: the streamed slabs (n of them, contiguous in memory, whole
// grips) pass through a ring of `stufen` stages in an endless cycle, the
// resident ones stay.
struct Band {
  const char* quelle;
  unsigned n, stufen;
  unsigned ring, fest;   // offsets in shared memory
  unsigned pj;           // the next slab to copy (n: all of this product's are on their way)
  unsigned stufe, par;   // the next stage to read and its parity
  unsigned offen;        // copies on their way or not yet read
  unsigned bleibt;       // slabs up to here are to stay in L2
};
template <typename R, int U>
__device__ __forceinline__ void band_hole(Band& g, unsigned long long* bar, unsigned stufe, int lane) {
  constexpr unsigned bytes = U * Satz<R>::bytes;
  if (lane == 0) {
    bar_erwarte(&bar[stufe], bytes);
    char* z = g_roh + g.ring + stufe * bytes;
    const char* q = g.quelle + size_t(g.pj) * Satz<R>::bytes;
    if (g.pj < g.bleibt)
      kopiere(z, q, bytes, &bar[stufe]);
    else
      kopiere_weg(z, q, bytes, &bar[stufe]);
  }
  g.pj += U;
  ++g.offen;
}
// The first stages' copies of the next product.
template <typename R, int U>
__device__ __forceinline__ void band_start(Band& g, unsigned long long* bar, int lane) {
  g.pj = 0;
  unsigned s = g.stufe;
  for (unsigned k = 0; k < g.stufen && g.pj < g.n; ++k) {
    band_hole<R, U>(g, bar, s, lane);
    if (++s == g.stufen) s = 0;
  }
}
// A wait for this warp's own copies. They end whatever else has failed, so it
// gives up only when its own time is out.
__device__ __forceinline__ void bar_warte(const StepArgs& a, KSh& sh, unsigned long long* b, unsigned par) {
  Warten w;
  while (!bar_da(b, par)) {
    if ((++w.n & 63u) != 0u) continue;
    const uint64_t t = globaltimer();
    if (w.t0 == 0) w.t0 = t;
    if (t - w.t0 <= a.frist_ns) continue;
    atomicCAS(&a.sync->error, 0, K3D_STATUS_TIMEOUT);
    *reinterpret_cast<volatile int*>(&sh.err) = K3D_STATUS_TIMEOUT;
    return;
  }
}

// One grip: U slabs at the offset `wo`. Their loads go out before the first
// product, and little else is done: a slab is 7 loads, 9 conversions (FP32
// blocks) and 18 FP64 operations, and what is issued beside them counts as much.
template <typename R, int U>
__device__ __forceinline__ void griff(unsigned wo, double& x, double& y, double& z) {
  const int lane = threadIdx.x & 31;
  const char* tile = g_roh + kachel_kopf(sizeof(KSh));
  const char* s = g_roh + wo;
  unsigned j[U];
  R4<R> u[U], v[U];
  R w[U];
  double px[U], py[U], pz[U];
#pragma unroll
  for (int t = 0; t < U; ++t) j[t] = reinterpret_cast<const uint16_t*>(s + t * Satz<R>::bytes + Satz<R>::spalte)[lane];
#pragma unroll
  for (int t = 0; t < U; ++t) {
    u[t] = reinterpret_cast<const R4<R>*>(s + t * Satz<R>::bytes)[lane];
    v[t] = reinterpret_cast<const R4<R>*>(s + t * Satz<R>::bytes + Satz<R>::v)[lane];
    w[t] = reinterpret_cast<const R*>(s + t * Satz<R>::bytes + Satz<R>::w)[lane];
  }
#pragma unroll
  for (int t = 0; t < U; ++t) {
    const double* p = reinterpret_cast<const double*>(tile + 24 * j[t]);
    px[t] = p[0];
    py[t] = p[1];
    pz[t] = p[2];
  }
#pragma unroll
  for (int t = 0; t < U; ++t) {
    x += double(u[t].x) * px[t] + double(u[t].y) * py[t] + double(u[t].z) * pz[t];
    y += double(u[t].w) * px[t] + double(v[t].x) * py[t] + double(v[t].y) * pz[t];
    z += double(v[t].z) * px[t] + double(v[t].w) * py[t] + double(w[t]) * pz[t];
  }
}
// o = (A t) of the warp's rows, t in the tile. strom, fest: the slices'
// streamed and resident slabs.
template <typename R, int Q>
__device__ __forceinline__ void produkt(const StepArgs& a, KSh& sh, Band& g, const unsigned (&strom)[Q],
                                        const unsigned (&fest)[Q], double (&o)[Q][3]) {
  constexpr int U = kachel_griff(sizeof(R), Q);
  constexpr int F = sizeof(R) == 4 && Q == 1 ? 4 : U;  // resident slabs at once, as the registers allow
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long* bar = sh.bar[warp];
  unsigned wo = g.fest;
  if (g.offen == 0) band_start<R, U>(g, bar, lane);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    double x = 0.0, y = 0.0, z = 0.0;
#pragma unroll 1
    for (unsigned k = 0; k < strom[q]; k += U) {
      if (!bar_da(&bar[g.stufe], g.par)) bar_warte(a, sh, &bar[g.stufe], g.par);
      griff<R, U>(g.ring + g.stufe * (U * Satz<R>::bytes), x, y, z);
      __syncwarp();  // the stage is free again
      --g.offen;
      if (g.pj < g.n) band_hole<R, U>(g, bar, g.stufe, lane);
      if (++g.stufe == g.stufen) {
        g.stufe = 0;
        g.par ^= 1u;
      }
    }
    unsigned k = fest[q];
#pragma unroll 1
    for (; k >= F; k -= F, wo += F * Satz<R>::bytes) griff<R, F>(wo, x, y, z);
#pragma unroll 1
    for (; k > 0; --k, wo += Satz<R>::bytes) griff<R, 1>(wo, x, y, z);
    o[q][0] = x;
    o[q][1] = y;
    o[q][2] = z;
  }
}

template <typename R>
__device__ __forceinline__ void vorkond(const R* P, int64_t i, R (&p)[6]) {
#pragma unroll
  for (int k = 0; k < 6; ++k) p[k] = P[6 * i + k];
}
template <typename R>
__device__ __forceinline__ D3 pmal(const R (&f)[6], D3 r) {
  double p[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) p[k] = double(f[k]);
  return d3(p[0] * r.x + p[3] * r.y + p[4] * r.z, p[3] * r.x + p[1] * r.y + p[5] * r.z,
            p[4] * r.x + p[5] * r.y + p[2] * r.z);
}
// S: the part along the contact normal removed
__device__ __forceinline__ D3 s_filter(D3 n, D3 x) {
  const double d = x.x * n.x + x.y * n.y + x.z * n.z;
  return d3(x.x - n.x * d, x.y - n.y * d, x.z - n.z * d);
}

// The self-collision springs' part of a product, t = F w, in their merged rows
// (SelbstArgs::sf_*). The points in contact lie in few tiles, so the rows are
// spread over every CTA: eight lanes a row take its blocks against the
// published words of its columns and publish t in turn, and the point's own
// thread adds it after the tile's product. What bounds it is latency, so the
// rows' heads lie in shared memory (kopf: starts, blocks, columns) and the
// blocks travel with the words.
__device__ __forceinline__ void federzeilen(const StepArgs& a, KSh& sh, const uint32_t* kopf, uint32_t ep) {
  const unsigned l = threadIdx.x & 7;
  const ulonglong2* wort = a.ka_wort + size_t(ep & 1u) * 3 * size_t(a.n);
  ulonglong2* aus = a.ka_wort + (2 + size_t(ep & 1u)) * 3 * size_t(a.n);
  const size_t cap = size_t(a.sf_cap);
#pragma unroll 1
  for (unsigned g = threadIdx.x >> 3; __any_sync(0xffffffffu, g < sh.federn); g += kNT / 8) {
    const bool nah = g < kFederZeilen;
    unsigned anf = 0, m = 0;
    if (g < sh.federn) {
      anf = nah ? kopf[g] : a.sf_anf[g * sh.g.nblk + sh.bidx];
      m = nah ? kopf[kFederZeilen + g] : a.sf_anz[g * sh.g.nblk + sh.bidx];
    }
    double x = 0.0, y = 0.0, z = 0.0;
    uint32_t i = 0;
#pragma unroll 1
    for (unsigned e = l; e < m; e += 8) {
      const uint32_t j =
          nah && e < kFederSpalten ? kopf[2 * kFederZeilen + kFederSpalten * g + e] : a.sf_spalte[anf + e];
      const double* b = a.sf_block + anf + e;
      const double bxx = b[0], byy = b[cap], bzz = b[2 * cap], bxy = b[3 * cap], bxz = b[4 * cap], byz = b[5 * cap];
      const D3 w = hol_wort3(a, sh, wort + j, ep);
      x += bxx * w.x + bxy * w.y + bxz * w.z;
      y += bxy * w.x + byy * w.y + byz * w.z;
      z += bxz * w.x + byz * w.y + bzz * w.z;
      if (e < 8) i = j;
    }
    __syncwarp();
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
      z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    i = __shfl_sync(0xffffffffu, i, 0, 8);  // the diagonal's column
    if (m > 0 && l < 3) st_wort(aus + l * size_t(a.n) + i, l == 0 ? x : l == 1 ? y : z, ep);
  }
}

enum : unsigned { kZeile = 1u, kFrei = 2u, kGehalten = 4u, kGrenze = 8u, kFedern = 16u };

// Q rows a thread (slices of 32 rows: warp, warp + 16, ...).
template <typename R, bool SC, int Q>
__global__ void __launch_bounds__(kNT, 1) kachel_kernel(const __grid_constant__ StepArgs a) {
  KSh& sh = *reinterpret_cast<KSh*>(g_roh);
  constexpr bool kRec = sizeof(R) == 4;  // A c from A w and the previous A c; the tile holds w (else c)
  constexpr bool kDv = Q <= 2;           // dv in registers (else read and written in place)
  constexpr bool kNah = Q == 1;          // preconditioner and normal in registers too
  constexpr bool kAp = kachel_ap(sizeof(R), Q);  // A c in shared memory
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    sh.err = ld_relaxed_i32(&a.sync->error);
    sh.g = a.grp[a.blk_grp[blockIdx.x]];
    sh.b = a.ka_blk[blockIdx.x];
    sh.bidx = blockIdx.x - sh.g.first_blk;
    if (SC) {
      const unsigned z = *a.sf_zahl;
      sh.federn = z > sh.bidx ? (z - sh.bidx + sh.g.nblk - 1) / sh.g.nblk : 0u;
    }
  }
  if (lane == 0) {
    for (int s = 0; s <= kKachelStufen; ++s) bar_init(&sh.bar[warp][s]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (!ohne_abbruch(sh)) return;  // a launch before this one gave up
  const unsigned ns = (sh.b.rows + 31) >> 5, halos = sh.b.halos, ts = 32 * ns + halos;
  const uint32_t slice0 = sh.b.row0 >> 5;
  double* tile = reinterpret_cast<double*>(g_roh + kachel_kopf(sizeof(KSh)));
  double* halo = tile + 3 * 32 * ns;
  const uint32_t* halo_pt = a.ka_halo + sh.b.halo0;
  // rows
  constexpr int U = kachel_griff(sizeof(R), Q);
  uint32_t pt[Q];
  unsigned fl[Q], strom[Q], fest[Q];
  Band g{};
  unsigned fest_n = 0, fest_1 = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const unsigned s = warp + kNW * q;
    pt[q] = 0;
    fl[q] = strom[q] = fest[q] = 0;
    if (s >= ns) continue;
    const uint4 sl = a.ka_slice[slice0 + s];
    if (q == 0) {
      g.quelle = static_cast<const char*>(a.bmat) + size_t(sl.x) * Satz<R>::bytes;
      fest_1 = sl.z;
    }
    strom[q] = sl.y;
    fest[q] = sl.w;
    g.n += sl.y;
    fest_n += sl.w;
    const unsigned r = 32 * s + lane;
    if (r < sh.b.rows) {
      const uint32_t z = a.ka_row[sh.b.row0 + r];
      pt[q] = z & 0x7fffffffu;
      fl[q] = kZeile | (a.frei[pt[q]] ? kFrei : 0u) | (z >> 31 ? kGrenze : 0u);
      if (SC && a.sc_off[pt[q]] != a.sc_off[pt[q] + 1]) fl[q] |= kGrenze | kFedern;
    }
  }
  // the warp's share of the shared memory behind the tile: its ring, then its
  // resident slabs
  {
    g.stufen = sh.b.stufen;
    g.bleibt = sh.b.bleibt;
    g.ring = unsigned(kachel_kopf(sizeof(KSh)) + kachel_tile(sizeof(R), ns, halos, kAp, SC)) +
             unsigned(warp) * sh.b.platz * Satz<R>::bytes;
    g.fest = g.ring + g.stufen * U * Satz<R>::bytes;
    unsigned long long* bar = sh.bar[warp];
    if (lane == 0 && fest_n > 0) {
      bar_erwarte(&bar[kKachelStufen], fest_n * Satz<R>::bytes);
      kopiere(g_roh + g.fest, static_cast<const char*>(a.bmat) + size_t(fest_1) * Satz<R>::bytes,
              fest_n * Satz<R>::bytes, &bar[kKachelStufen]);
    }
    if (g.n == 0) g.stufen = 0;
  }
  for (unsigned i = threadIdx.x; i < 3 * ts; i += kNT) tile[i] = 0.0;
  const uint32_t ep0 = *reinterpret_cast<volatile unsigned*>(sh.g.count);
  uint32_t ep = ep0, seq = ep0;
  const bool lead = sh.bidx == 0 && threadIdx.x == 0;  // one thread per group
  const bool any_held = a.stats[ST_HELD] > 0;
  const R* pinv = static_cast<const R*>(a.pinv);
  // beyond one row a thread the preconditioner, beyond two dv, as planes in
  // position order: a warp's loads are whole lines (point order is 24 or 48
  // bytes a lane, each line fetched three to six times), past the L1, which
  // keeps the held points' normals
  const size_t ebene = 32 * size_t(a.ka_slices);
  R* pv_g = static_cast<R*>(a.ka_pv);
  double* dv_g = a.ka_dv;
  auto platz = [&](int q) -> size_t { return sh.b.row0 + 32 * (warp + kNW * q) + lane; };
  auto vorkond_g = [&](int q, R (&p)[6]) {
#pragma unroll
    for (int k = 0; k < 6; ++k) p[k] = __ldcg(&pv_g[k * ebene + platz(q)]);
  };
  auto dv_lesen = [&](int q) -> D3 {
    return d3(__ldcg(&dv_g[platz(q)]), __ldcg(&dv_g[ebene + platz(q)]), __ldcg(&dv_g[2 * ebene + platz(q)]));
  };
  auto dv_schreiben = [&](int q, D3 d) {
    dv_g[platz(q)] = d.x;
    dv_g[ebene + platz(q)] = d.y;
    dv_g[2 * ebene + platz(q)] = d.z;
  };
  R* nrm_r = static_cast<R*>(a.nrm);
  double cw[Q][3], r[Q][3], ap[kAp ? 1 : Q][3] = {}, dv[kDv ? Q : 1][3], o[Q][3];
  R pv[1][6] = {};          // with kNah
  double nn[1][3] = {};
  __syncthreads();
  if (fest_n > 0) bar_warte(a, sh, &sh.bar[warp][kKachelStufen], 0u);

  auto normale = [&](int q) -> D3 {
    if (!(fl[q] & kGehalten)) return d3(0.0, 0.0, 0.0);
    if (kNah) return d3(nn[0][0], nn[0][1], nn[0][2]);
    return ld3(a.nrm_d, pt[q]);
  };
  auto wort = [&]() -> ulonglong2* { return a.ka_wort + size_t(ep & 1u) * 3 * size_t(a.n); };
  auto ausgeben = [&](int q, D3 v) {  // publishes a row's vector under `ep`
    if (fl[q] & kGrenze) {
      ulonglong2* p = wort() + pt[q];
      st_wort(p, v.x, ep);
      st_wort(p + a.n, v.y, ep);
      st_wort(p + 2 * a.n, v.z, ep);
    }
  };
  auto eigen = [&](int q, D3 v) {
    double* p = tile + 3 * (32 * (warp + kNW * q) + lane);
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
  };
  auto aus_kachel = [&](int q) -> D3 {
    const double* p = tile + 3 * (32 * (warp + kNW * q) + lane);
    return d3(p[0], p[1], p[2]);
  };
  double* ap_s = halo + 3 * halos;
  double* f_s = ap_s + (kAp ? 3 * 32 * ns : 0);  // with FP64 blocks the springs' part of A c
  uint32_t* fkopf = reinterpret_cast<uint32_t*>(g_roh + kachel_kopf(sizeof(KSh)) +
                                                kachel_vektoren(sizeof(R), ns, halos, kAp, SC));
  if (SC) {  // heads of the springs' rows
    const unsigned nf = sh.federn < kFederZeilen ? sh.federn : kFederZeilen;
    for (unsigned t = threadIdx.x; t < nf * kFederSpalten; t += kNT) {
      const unsigned z = t / kFederSpalten, e = t % kFederSpalten, k = z * sh.g.nblk + sh.bidx;
      const uint32_t anf = a.sf_anf[k], m = a.sf_anz[k];
      if (e == 0) {
        fkopf[z] = anf;
        fkopf[kFederZeilen + z] = m;
      }
      if (e < m) fkopf[2 * kFederZeilen + t] = a.sf_spalte[anf + e];
    }
    __syncthreads();
  }
  auto ap_lesen = [&](int q) -> D3 {
    if (!kAp) return d3(ap[kAp ? 0 : q][0], ap[kAp ? 0 : q][1], ap[kAp ? 0 : q][2]);
    const double* p = ap_s + 3 * (32 * (warp + kNW * q) + lane);
    return d3(p[0], p[1], p[2]);
  };
  auto ap_setzen = [&](int q, D3 v) {
    double* p = kAp ? ap_s + 3 * (32 * (warp + kNW * q) + lane) : ap[kAp ? 0 : q];
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
  };
  auto halo_holen = [&]() {
    for (unsigned t = threadIdx.x; t < halos; t += kNT) {
      const D3 v = hol_wort3(a, sh, wort() + halo_pt[t], ep);
      halo[3 * t] = v.x;
      halo[3 * t + 1] = v.y;
      halo[3 * t + 2] = v.z;
    }
  };
  // o += the springs' product, of the vector published under e: t of w, or
  // (FP64 blocks) of c = w + beta c_prev by t + beta times its last value
  auto federn = [&](uint32_t e, double bt, bool neu) {
    const ulonglong2* p = a.ka_wort + (2 + size_t(e & 1u)) * 3 * size_t(a.n);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!(fl[q] & kFedern)) continue;
      D3 t = hol_wort3(a, sh, p + pt[q], e);
      if (!kRec && !neu) {
        double* f = f_s + 3 * (32 * (warp + kNW * q) + lane);
        if (bt != 0.0) t = d3(fmar(bt, f[0], t.x), fmar(bt, f[1], t.y), fmar(bt, f[2], t.z));
        f[0] = t.x;
        f[1] = t.y;
        f[2] = t.z;
      }
      o[q][0] += t.x;
      o[q][1] += t.y;
      o[q][2] += t.z;
    }
  };
  // the tile takes dv, its halo too; so do the springs' rows
  auto dv_auslegen = [&]() -> bool {
    ++ep;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!(fl[q] & kZeile)) continue;
      const D3 d = kDv ? d3(dv[q % (kDv ? Q : 1)][0], dv[q % (kDv ? Q : 1)][1], dv[q % (kDv ? Q : 1)][2])
                       : dv_lesen(q);
      ausgeben(q, d);
      eigen(q, d);
    }
    halo_holen();
    if (SC) federzeilen(a, sh, fkopf, ep);
    return einig(sh);
  };

  bool gut = true;
#pragma unroll 1
  for (int pass = 0; pass < 2 && gut; ++pass) {
    // start: pinned points 0, held points get their normal target
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      cw[q][0] = cw[q][1] = cw[q][2] = 0.0;
      if (!kAp) ap_setzen(q, d3(0.0, 0.0, 0.0));
      r[q][0] = r[q][1] = r[q][2] = 0.0;
      if (!(fl[q] & kZeile)) continue;
      D3 d = ld3(a.dv, pt[q]);
      const D3 n = ld3(a.nrm_d, pt[q]);
      const bool gehalten = n.x != 0.0 || n.y != 0.0 || n.z != 0.0;
      fl[q] = (fl[q] & ~unsigned(kGehalten)) | (gehalten ? kGehalten : 0u);
      if (!(fl[q] & kFrei)) {
        d = d3(0, 0, 0);
      } else if (gehalten) {
        const double soll = a.adjoint ? 0.0 : a.vn_soll[pt[q]] - dot(ld3(a.v, pt[q]), n);
        d = (d - n * dot(d, n)) + n * soll;
      }
      if (kNah) {
        nn[0][0] = n.x;
        nn[0][1] = n.y;
        nn[0][2] = n.z;
        vorkond<R>(pinv, pt[q], pv[0]);
      } else if (pass == 0) {
        R p[6];
        vorkond<R>(pinv, pt[q], p);
#pragma unroll
        for (int k = 0; k < 6; ++k) pv_g[k * ebene + platz(q)] = p[k];
      }
      if (kDv) {
        dv[q % (kDv ? Q : 1)][0] = d.x;
        dv[q % (kDv ? Q : 1)][1] = d.y;
        dv[q % (kDv ? Q : 1)][2] = d.z;
      }
      if (!kDv) dv_schreiben(q, d);
    }
    if (!(gut = dv_auslegen())) break;
    produkt<R, Q>(a, sh, g, strom, fest, o);
    if (SC) federn(ep, 0.0, true);
    double red[2] = {0.0, 0.0};
    ++ep;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      D3 w = d3(0.0, 0.0, 0.0);
      if (fl[q] & kFrei) {
        const D3 b = ld3(a.b, pt[q]);
        D3 ad = d3(o[q][0], o[q][1], o[q][2]);
        const D3 n = normale(q);
        D3 rd = b - ad;
        rd = rd - n * dot(rd, n);
        const D3 f = s_filter(n, b);
        R p[6];
        if (kNah) {
#pragma unroll
          for (int k = 0; k < 6; ++k) p[k] = pv[0][k];
        } else {
          vorkond_g(q, p);
        }
        const D3 pf = pmal(p, f);
        red[1] += f.x * pf.x + f.y * pf.y + f.z * pf.z;
        w = s_filter(n, pmal(p, rd));
        red[0] += rd.x * w.x + rd.y * w.y + rd.z * w.z;
        r[q][0] = rd.x;
        r[q][1] = rd.y;
        r[q][2] = rd.z;
      }
      if (fl[q] & kZeile) ausgeben(q, w);
      o[q][0] = w.x;
      o[q][1] = w.y;
      o[q][2] = w.z;
    }
    ++seq;
    melden<2>(a, sh, red, seq);  // every warp has read the tile
    // w in the tile and c = 0 in registers, or c = 0 in the tile and w in registers
    if (kRec) {
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (fl[q] & kZeile) eigen(q, d3(o[q][0], o[q][1], o[q][2]));
    } else {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        cw[q][0] = o[q][0];
        cw[q][1] = o[q][1];
        cw[q][2] = o[q][2];
      }
      for (unsigned i = threadIdx.x; i < 3 * ts; i += kNT) tile[i] = 0.0;
    }
    double delta = 0.0, bb = 0.0, ziel = 0.0, beta = 0.0;
    int64_t it = 0;
    bool brk = false, erste = true;
    for (;;) {
      // w (published under ep) of the halo, then delta and beta from the sum under seq
      D3 hw = d3(0.0, 0.0, 0.0);
      bool da = false;
      Vorab vor;
      if (kRec) {
        halo_holen();
        if (SC) federzeilen(a, sh, fkopf, ep);
        __syncthreads();
        vorab(a, sh, vor, seq);  // its latency passes under the product
        produkt<R, Q>(a, sh, g, strom, fest, o);
        if (SC) federn(ep, 0.0, true);
      } else {  // the first chunk of the halo and the springs while the sum travels
        if (threadIdx.x < halos) da = ld_wort3(wort() + halo_pt[threadIdx.x], a.n, ep, hw);
        if (SC) federzeilen(a, sh, fkopf, ep);
      }
      if (erste) {
        double s[2];
        sammeln<2>(a, sh, s, seq, vor);
        delta = s[0];
        bb = s[1];
        ziel = fmax(a.tol * a.tol * fmax(bb, delta), sh.g.boden);
      } else {
        double s[1];
        sammeln<1>(a, sh, s, seq, vor);
        beta = s[0] / delta;
        delta = s[0];
        ++it;
      }
      if (!(delta > ziel && it < a.cg_max)) break;
      double ca[1] = {0.0};
      if (!kRec) {  // c = w + beta c over the tile and its halo, then A c
#pragma unroll
        for (int q = 0; q < Q; ++q)
          if (fl[q] & kZeile) {
            const D3 c = aus_kachel(q);
            eigen(q, d3(fmar(beta, c.x, cw[q][0]), fmar(beta, c.y, cw[q][1]), fmar(beta, c.z, cw[q][2])));
          }
        for (unsigned t = threadIdx.x; t < halos; t += kNT) {
          if (!(t == threadIdx.x && da)) hw = hol_wort3(a, sh, wort() + halo_pt[t], ep);
          halo[3 * t] = fmar(beta, halo[3 * t], hw.x);
          halo[3 * t + 1] = fmar(beta, halo[3 * t + 1], hw.y);
          halo[3 * t + 2] = fmar(beta, halo[3 * t + 2], hw.z);
        }
        __syncthreads();
        produkt<R, Q>(a, sh, g, strom, fest, o);
        if (SC) federn(ep, beta, false);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (!(fl[q] & kZeile)) continue;
        D3 c = aus_kachel(q);
        if (kRec) {
          c = d3(fmar(beta, cw[q][0], c.x), fmar(beta, cw[q][1], c.y), fmar(beta, cw[q][2], c.z));
          cw[q][0] = c.x;
          cw[q][1] = c.y;
          cw[q][2] = c.z;
        }
        D3 s = d3(0.0, 0.0, 0.0);
        if (fl[q] & kFrei) {
          s = d3(o[q][0], o[q][1], o[q][2]);
          if (fl[q] & kGehalten) s = s_filter(normale(q), s);
          if (kRec && beta != 0.0) {
            const D3 v = ap_lesen(q);
            s = d3(fmar(beta, v.x, s.x), fmar(beta, v.y, s.y), fmar(beta, v.z, s.z));
          }
        }
        ap_setzen(q, s);
        ca[0] += c.x * s.x + c.y * s.y + c.z * s.z;
      }
      erste = false;
      ++seq;
      melden<1>(a, sh, ca, seq);
      // the update's loads travel with the sum
      R p2[kNah ? 1 : Q][6];
      D3 dv2[kDv ? 1 : Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (!(fl[q] & kZeile)) continue;
        if (!kNah) vorkond_g(q, p2[kNah ? 0 : q]);
        if (!kDv) dv2[kDv ? 0 : q] = dv_lesen(q);
      }
      sammeln<1>(a, sh, ca, seq);
      if (!ohne_abbruch(sh)) break;  // the iteration's waits; melden's barrier lies before the next
      if (ca[0] <= DBL_MIN || !isfinite(ca[0])) {
        brk = true;
        break;
      }
      const double alpha = delta / ca[0];
      double rz[1] = {0.0};
      ++ep;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (!(fl[q] & kZeile)) continue;
        const D3 c = kRec ? d3(cw[q][0], cw[q][1], cw[q][2]) : aus_kachel(q);
        if (kDv) {
          double(&d)[3] = dv[q % (kDv ? Q : 1)];
          d[0] += c.x * alpha;
          d[1] += c.y * alpha;
          d[2] += c.z * alpha;
        } else {
          dv_schreiben(q, dv2[kDv ? 0 : q] + c * alpha);
        }
        D3 s = ap_lesen(q);
        const D3 n = normale(q);
        const D3 rn = d3(r[q][0] - alpha * s.x, r[q][1] - alpha * s.y, r[q][2] - alpha * s.z);
        r[q][0] = rn.x;
        r[q][1] = rn.y;
        r[q][2] = rn.z;
        D3 z = pmal(kNah ? pv[0] : p2[kNah ? 0 : q], rn);
        if (!(fl[q] & kFrei)) z = d3(0.0, 0.0, 0.0);
        const D3 w = (fl[q] & kGehalten) ? s_filter(n, z) : z;
        ausgeben(q, w);
        if (kRec) {
          eigen(q, w);
        } else {
          cw[q][0] = w.x;
          cw[q][1] = w.y;
          cw[q][2] = w.z;
        }
        rz[0] += rn.x * z.x + rn.y * z.y + rn.z * z.z;
      }
      if (it == a.stumm_nach && threadIdx.x == 0) ++sh.b.worte;
      ++seq;
      melden<1>(a, sh, rz, seq);
      // the next product's first copies travel with the halo and this sum; the
      // update above ran on a quiet memory system
      band_start<R, U>(g, sh.bar[warp], lane);
    }
    if (!(gut = einig(sh))) break;
    // |dv| maximum and the counters go to the statistics by atomics (the
    // groups of a batch finish at different times)
    double dvm = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!(fl[q] & kZeile)) continue;
      D3 d;
      if (kDv) {
        const double(&e)[3] = dv[q % (kDv ? Q : 1)];
        d = d3(e[0], e[1], e[2]);
      } else {
        d = dv_lesen(q);
      }
      st3(a.dv, pt[q], d);
      dvm = fmax(dvm, fmax(fabs(d.x), fmax(fabs(d.y), fabs(d.z))));
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) dvm = fmax(dvm, __shfl_xor_sync(0xffffffffu, dvm, s));
    if (lane == 0 && dvm > 0.0)
      atomicMax(reinterpret_cast<unsigned long long*>(&a.stat_rest_max[1]), (unsigned long long)__double_as_longlong(dvm));
    if (lead) {
      const double rest = sqrt(delta / fmax(bb, sh.g.boden));
      atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[ST_CG_ITERATIONS]), (unsigned long long)it);
      atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[ST_SOLVES]), 1ull);
      if (delta > ziel) atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[ST_UNCONVERGED]), 1ull);
      if (brk) atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[ST_BREAKDOWNS]), 1ull);
      if (rest > 0.0)
        atomicMax(reinterpret_cast<unsigned long long*>(&a.stat_rest_max[0]),
                  (unsigned long long)__double_as_longlong(rest));
      if (sh.g.first_blk == 0) a.stats[ST_LAST_ITERATIONS] = it;
    }
    if (a.mode == MODE_SOLVE || !any_held) break;
    // release pass (implizit.rs:924-942): the normal force from A dv - b; a
    // held point that pulls on the body is released
    if (!(gut = dv_auslegen())) break;
    produkt<R, Q>(a, sh, g, strom, fest, o);
    if (SC) federn(ep, 0.0, true);
    double los[1] = {0.0};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!(fl[q] & kZeile) || !(fl[q] & kGehalten)) continue;
      const D3 n = normale(q);
      D3 ad = d3(o[q][0], o[q][1], o[q][2]);
      const D3 rest = ad - ld3(a.b, pt[q]);
      const double fn = dot(rest, n) / a.h;
      if (fn < 0.0) {
        st3(a.nrm_d, pt[q], d3(0, 0, 0));
        nrm_r[3 * size_t(pt[q])] = nrm_r[3 * size_t(pt[q]) + 1] = nrm_r[3 * size_t(pt[q]) + 2] = R(0);
        los[0] += 1.0;
        // released after the last solve: held in dv's constraint, free in friction
        if (pass == 1 && a.rec_flags) a.rec_flags[pt[q]] |= 8u;
      } else {
        a.fnk[pt[q]] = fn;
      }
    }
    ++seq;
    melden<1>(a, sh, los, seq);
    sammeln<1>(a, sh, los, seq);
    if (!(gut = einig(sh))) break;
    if (lead && los[0] > 0.0)
      atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[ST_RELEASED]), (unsigned long long)los[0]);
    if (los[0] == 0.0) break;
  }
  // the sequence numbers go on from here in the next launch
  if (lead && gut) *sh.g.count = (ep - ep0 > seq - ep0 ? ep : seq) + 1u;
  // copies still in flight (of a product that the last sum ended or a wait that gave up kept from running)
  for (unsigned k = 0; k < g.offen; ++k) {
    bar_warte(a, sh, &sh.bar[warp][g.stufe], g.par);
    if (++g.stufe == g.stufen) {
      g.stufe = 0;
      g.par ^= 1u;
    }
  }
}

template <typename R, bool SC>
const void* fn_q(int q) {
  switch (q) {
    case 1: return (const void*)kachel_kernel<R, SC, 1>;
    case 2: return (const void*)kachel_kernel<R, SC, 2>;
    case 3: return (const void*)kachel_kernel<R, SC, 3>;
    default: return (const void*)kachel_kernel<R, SC, 4>;
  }
}
const void* fn_of(int rsize, bool sc, int q) {
  return rsize == 8 ? (sc ? fn_q<double, true>(q) : fn_q<double, false>(q))
                    : (sc ? fn_q<float, true>(q) : fn_q<float, false>(q));
}

}  // namespace

size_t kachel_kopf_bytes() { return kachel_kopf(sizeof(KSh)); }

size_t kachel_smem(int device) {
  int most = 0;
  if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return 0;
  return size_t(most);
}

bool kachel_bereit(int rsize, bool federn, int q, size_t smem) {
  const void* fn = fn_of(rsize, federn, q);
  cudaFuncAttributes at;
  return cudaFuncGetAttributes(&at, fn) == cudaSuccess && at.maxThreadsPerBlock >= kNT && at.sharedSizeBytes == 0 &&
         cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) == cudaSuccess;
}

cudaError_t launch_kachel(const StepArgs& a, cudaStream_t st) {
  const int rsize = a.ka_rsize;
  void* args[] = {(void*)&a};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(a.ka_blocks));
  cfg.blockDim = dim3(unsigned(kNT));
  cfg.dynamicSmemBytes = a.ka_smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn_of(rsize, a.sc_off != nullptr, a.ka_q), args);
}

}  // namespace k3d
