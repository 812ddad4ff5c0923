// Update by runs of flat indices (sm_103a): rooms whose rows are not 16-byte
// aligned, and large or awkwardly wide ones.
//
// The tensor maps of k_update_tma need 16-byte row strides and tiles that
// cover the rows well.  A run of a plane's flat indices needs neither: the
// 7-point neighbours of flat index i are i +- 1, i +- X and i +- X*Y (also across
// rows, as the reference indexes), so a CTA that owns the indices [s, s + L) of
// every plane it marches through needs [s - X, s + L + X) of P^n and [s, s + L) of
// P^{n-1} and of the class ids: three contiguous pieces a plane, each one untiled
// bulk copy from the 16-byte boundary before it, indexed from the remainder in
// shared memory.
//
//  * One producer thread issues the copies into a ring of stages; stage k holds
//    P^n of plane z0-1+k and P^{n-1} and class ids of plane z0+k-2.
//  * A consumer thread takes kPer nodes, a block's width apart, so that every
//    access to shared and global memory is 32 neighbouring values whatever the
//    alignment.  It keeps planes z-1 and z of its nodes in registers (three
//    planes a trip, the arrays' roles rotating), and updates its nodes in packed
//    pairs, operation for operation as k_update_tma.
//
// Measured (us an update, FP32 forward): against the z-march kernel 203 x 155 x
// 119 11.2 -> 9.7, 401 x 301 x 201 70.0 -> 48.3 (498 G node-updates/s, 6.5 TB/s at
// 13 bytes); against k_update_tma 384 x 320 x 256 73.5 -> 61.5, 320 x 240 x 200
// 38.1 -> 30.5, 512 x 384 x 256 99.9 -> 95.8 (6.77 TB/s, the copy rate).  HBM bounds
// the large rooms; those that fit the L2 are bound by latency at two CTAs a SM.
#include "common.cuh"
#include "mbar.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

namespace pfdtd {
namespace {

constexpr int kConsumers = 256, kThreads = kConsumers + 32, kPer = 8;
constexpr int kRange = kConsumers * kPer;   // flat indices of a CTA
constexpr int kMaxStages = 8;
constexpr size_t kSmemPerCta = 110 * 1024;  // two CTAs on an SM

struct alignas(16) Coef { float a, b, c; uint32_t pos; };

__host__ __device__ inline int round128(int b) { return (b + 127) / 128 * 128; }

// Bytes of a stage's three pieces: elements of es bytes, `halo` more of P^n on
// either side of the run.
struct Stage { int past, cls, bytes; };  // offsets of P^{n-1} and class ids, size
__host__ __device__ inline Stage stage_of(int halo, int es, int cs, int kshift) {
  Stage s;
  s.past = round128((kRange + 2 * halo) * es + 32);
  s.cls = s.past + round128(kRange * es + 32);
  s.bytes = s.cls + round128((kRange >> kshift) * cs + 32);
  return s;
}

// Copy the elements [first, first + n) of `base` (16-byte aligned) to dst from
// the 16-byte boundary before them; the bytes copied.
template <typename T>
__device__ __forceinline__ uint32_t piece_bytes(int64_t first, int n) {
  constexpr int64_t kA = 16 / (int64_t)sizeof(T);
  const int64_t a = first & ~(kA - 1);
  return (uint32_t)(((first + n - a + kA - 1) & ~(kA - 1)) * (int64_t)sizeof(T));
}
template <typename T>
__device__ __forceinline__ void copy_piece(unsigned char* dst, const T* base, int64_t first, int n,
                                           uint32_t bar) {
  constexpr int64_t kA = 16 / (int64_t)sizeof(T);
  const T* src = base + (first & ~(kA - 1));
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(piece_bytes<T>(first, n)), "r"(bar)
      : "memory");
}
// Where element `first` lies in the copied piece.
template <typename T> __device__ __forceinline__ int remainder_of(int64_t first) {
  return (int)(first & (16 / (int64_t)sizeof(T) - 1));
}

// The producer thread: stage k receives `halo` elements around the run of P^n
// plane z0-1+k and, from k = 2 on, the run of P^{n-1} and the class ids of plane
// z0+k-2.  Every wait is bounded; on expiry it raises the error and abort flags,
// and every copy in flight has landed before it returns.
template <typename S, typename C>
__device__ __forceinline__ void produce(unsigned char* smem, const Stage& lay, uint32_t full,
                                        uint32_t empty, int* abort_flag, const S* P, const S* past,
                                        const C* cls, int halo, int64_t XY, int64_t s0, int n, int z0,
                                        int loads, int stages, int ks, int kshift, int* err,
                                        uint64_t wait_ns) {
  int issued = 0;
  for (int k = 0; k < loads; ++k) {
    const int slot = k % stages;
    if (k >= stages && !mbar_wait(empty + 8 * slot, (uint32_t)((k / stages - 1) & 1), wait_ns)) {
      atomicExch(err, 1);
      *(volatile int*)abort_flag = 1;
      break;
    }
    if (*(volatile int*)abort_flag) break;
    unsigned char* st = smem + (size_t)slot * lay.bytes;
    const uint32_t bar = full + 8 * slot;
    const int64_t fp = (int64_t)(z0 - 1 + k) * XY + s0 - halo;
    const int64_t fq = (int64_t)(z0 + k - 2) * XY + s0;
    uint32_t bytes = piece_bytes<S>(fp, n + 2 * halo);
    const int nc = (n + ks - 1) >> kshift;
    if (k >= 2) bytes += piece_bytes<S>(fq, n) + piece_bytes<C>(fq >> kshift, nc);
    mbar_expect_tx(bar, bytes);
    copy_piece<S>(st, P, fp, n + 2 * halo, bar);
    if (k >= 2) {
      copy_piece<S>(st + lay.past, past, fq, n, bar);
      copy_piece<C>(st + lay.cls, cls, fq >> kshift, nc, bar);
    }
    issued = k + 1;
  }
  for (int k = max(0, issued - stages); k < issued; ++k)
    mbar_wait(full + 8 * (k % stages), (uint32_t)((k / stages) & 1));
}

template <typename S, typename C, int SCHEME>
__global__ void __launch_bounds__(kThreads, 2)
k_update_flat(const S* __restrict__ P, S* __restrict__ Pp, const S* __restrict__ past,
              const C* __restrict__ cls, ClassTab<float> tab, int XE, int64_t XY, int z_last, int zc,
              int stages, int ks, int kshift, float l2, float nzf, unsigned air, uint64_t wait_ns,
              int* __restrict__ err) {
  using namespace px;
  using St = Store<S>;
  constexpr bool kSmemTab = sizeof(C) == 1;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  __shared__ Coef stab[kSmemTab ? 256 : 1];
  __shared__ __align__(8) uint64_t bars[2 * kMaxStages];
  __shared__ int abort_flag;
  const Stage lay = stage_of(XE, sizeof(S), sizeof(C), kshift);
  const int t = threadIdx.x, lane = t & 31;
  const int64_t s0 = (int64_t)blockIdx.x * kRange;  // the CTA's first index of a plane
  const int n = (int)(XY - s0 < kRange ? XY - s0 : (int64_t)kRange);
  const int z0 = 1 + blockIdx.y * zc, z1 = min(z0 + zc, z_last), nplanes = z1 - z0;
  const uint32_t full = smem_u32(bars), empty = full + 8 * kMaxStages;
  if (t == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, kConsumers / 32);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (kSmemTab)
    for (int i = t; i < tab.n; i += kThreads)
      stab[i] = Coef{tab.a[i], tab.b[i], tab.c[i], tab.pos[i]};
  __syncthreads();
  step_wait();
  step_ready();
  if (*(volatile int*)err) return;
  if (nplanes <= 0) return;

  if (t >= kConsumers) {
    if (lane == 0)
      produce<S, C>(smem, lay, full, empty, &abort_flag, P, past, cls, XE, XY, s0, n, z0, nplanes + 2,
                    stages, ks, kshift, err, wait_ns);
    return;
  }

  // ---------------- consumers ----------------
  auto plane_ptr = [&](int k) {  // the thread's first node in stage k's P^n
    const int64_t fp = (int64_t)(z0 - 1 + k) * XY + s0 - XE;
    return (const S*)(smem + (size_t)(k % stages) * lay.bytes) + remainder_of<S>(fp) + XE + t;
  };
  const f2 l22 = pk2(l2, l2), nz = pk2(nzf, nzf);
  auto coef = [&](unsigned c) -> Coef {
    if (kSmemTab) return stab[c];
    return Coef{__ldg(tab.a + c), __ldg(tab.b + c), __ldg(tab.c + c), __ldg(tab.pos + c)};
  };
  Coef ka{0.f, 0.f, 0.f, 0u};  // open air, most of a room
  if (air != 0xFFFFFFFFu) ka = coef(air);
  bool ok = mbar_wait(full, 0, wait_ns) && mbar_wait(full + 8, 0, wait_ns);
  float F0[kPer], F1[kPer], F2[kPer];
  if (ok) {
    const S *p0 = plane_ptr(0), *p1 = plane_ptr(1);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      F0[j] = St::load(p0[j * kConsumers]);
      F1[j] = St::load(p1[j * kConsumers]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty);  // plane z0-1 is in registers
  }
  auto step = [&](int j, const float (&fm)[kPer], const float (&fc)[kPer], float (&fn)[kPer]) -> bool {
    const int sp = (j + 2) % stages;
    if (!mbar_wait(full + 8 * sp, (uint32_t)(((j + 2) / stages) & 1), wait_ns)) return false;
    const S* pn = plane_ptr(j + 2);
    const S* pc = plane_ptr(j + 1);
    const int64_t fq = (int64_t)(z0 + j) * XY + s0;
    const unsigned char* st = smem + (size_t)sp * lay.bytes;
    const S* pq = (const S*)(st + lay.past) + remainder_of<S>(fq) + t;
    const C* cl = (const C*)(st + lay.cls) + remainder_of<C>(fq >> kshift);
    S* out = Pp + fq + t;
#pragma unroll
    for (int e = 0; e < kPer; ++e) fn[e] = St::load(pn[e * kConsumers]);
#pragma unroll
    for (int e = 0; e < kPer; e += 2) {
      const S *a = pc + e * kConsumers, *b = a + kConsumers;
      const int i0 = t + e * kConsumers, i1 = i0 + kConsumers;
      // (past the range's end the piece holds anything: class 0)
      const unsigned c0 = i0 < n ? cl[i0 >> kshift] : 0u, c1 = i1 < n ? cl[i1 >> kshift] : 0u;
      const float xm0 = St::load(a[-ks]), xm1 = St::load(b[-ks]), xp0 = St::load(a[ks]), xp1 = St::load(b[ks]);
      const float ym0 = St::load(a[-XE]), ym1 = St::load(b[-XE]), yp0 = St::load(a[XE]), yp1 = St::load(b[XE]);
      const f2 xm = pk2(xm0, xm1), xp = pk2(xp0, xp1), ym = pk2(ym0, ym1), yp = pk2(yp0, yp1);
      const f2 po = pk2(St::load(pq[e * kConsumers]), St::load(pq[(e + 1) * kConsumers]));
      const f2 c2 = pk2(fc[e], fc[e + 1]), n2 = pk2(fn[e], fn[e + 1]), m2 = pk2(fm[e], fm[e + 1]);
      f2 o;
      if (SCHEME == 1 && __all_sync(0xffffffffu, c0 == air && c1 == air)) {
        // A warp in open air: no boundary neighbours to choose (times 0 they
        // stay), coefficients from registers, the exact products by +-1 left
        // out.  (401 x 301 x 201: 59.3 -> 51.8 us.  The forward update, whose
        // general form is short, took 3 % longer so.)
        const f2 sb6 = add2(add2(fma2(xm, 0ull, nz), fma2(ym, 0ull, nz)), fma2(n2, 0ull, nz));
        const f2 s7 = add2(add2(add2(add2(add2(add2(xm, xp), ym), yp), n2), m2), sb6);
        o = sub2(sub2(fma2(s7, l22, nz), fma2(pk2(ka.b, ka.b), c2, nz)), po);
      } else {
        Coef k0 = ka, k1 = ka;
        if (c0 != air) k0 = coef(c0);
        if (c1 != air) k1 = coef(c1);
        const f2 aa = pk2(k0.a, k1.a), bb = pk2(k0.b, k1.b), cc = pk2(k0.c, k1.c);
        if constexpr (SCHEME == 1) {
          const uint32_t q0 = k0.pos, q1 = k1.pos;
          const f2 bx = pk2((q0 & 0x10u) ? xp0 : xm0, (q1 & 0x10u) ? xp1 : xm1);
          const f2 by = pk2((q0 & 0x20u) ? yp0 : ym0, (q1 & 0x20u) ? yp1 : ym1);
          const f2 bz = pk2((q0 & 0x40u) ? fm[e] : fn[e], (q1 & 0x40u) ? fm[e + 1] : fn[e + 1]);
          const f2 dx = pk2((float)(q0 & 1u), (float)(q1 & 1u));
          const f2 dy = pk2((float)((q0 >> 1) & 1u), (float)((q1 >> 1) & 1u));
          const f2 dz = pk2((float)((q0 >> 2) & 1u), (float)((q1 >> 2) & 1u));
          const f2 sb6 = add2(add2(fma2(bx, dx, nz), fma2(by, dy, nz)), fma2(bz, dz, nz));
          const f2 s7 = add2(add2(add2(add2(add2(add2(xm, xp), ym), yp), n2), m2), sb6);
          o = mul2(aa, add2(sub2(fma2(s7, l22, nz), fma2(bb, c2, nz)), fma2(cc, po, nz)));
        } else {
          const f2 s6 = add2(add2(add2(add2(add2(n2, m2), yp), ym), xp), xm);
          if constexpr (SCHEME == 4) {
            const f2 ee = pk2(__uint_as_float(k0.pos), __uint_as_float(k1.pos));
            o = mul2(aa, add2(add2(fma2(ee, c2, nz), fma2(cc, sub2(c2, po), nz)),
                              fma2(l22, sub2(s6, fma2(bb, c2, nz)), nz)));
          } else {
            o = mul2(aa, sub2(add2(fma2(bb, c2, nz), fma2(l22, s6, nz)), fma2(cc, po, nz)));
          }
        }
      }
      float o0, o1;
      up2(o, o0, o1);
      if (i0 < n) out[e * kConsumers] = St::store(o0);
      if (i1 < n) out[(e + 1) * kConsumers] = St::store(o1);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + 8 * ((j + 1) % stages));  // plane z done
    return true;
  };
  for (int j = 0; j < nplanes && ok; j += 3) {
    ok = step(j, F0, F1, F2);
    if (!ok || j + 1 >= nplanes) break;
    ok = step(j + 1, F1, F2, F0);
    if (!ok || j + 2 >= nplanes) break;
    ok = step(j + 2, F2, F0, F1);
  }
  if (!ok) {
    atomicExch(err, 1);
    *(volatile int*)&abort_flag = 1;
  }
}

// IWB 27-point update by runs (no counterpart in the reference), one field per
// node: every node takes the open sums here, and a node with a closed neighbour
// (class flag bit 30) keeps P^{n-1} for the closure pass (k_iwb_closure,
// dif.cu), as in the tiled kernel without masks.
//
// The in-plane sums (iwb_sums) of plane z+1 are made once, from nine values of
// the stage; of planes z and z-1 the thread keeps what planes z+1 and z+2 still
// add to.  Open nodes all have a = c = 1 and one b, so that a class id is only
// looked up for its kind.  Order and rounding are those of k_update_iwb, in packed
// pairs with uncontractible products.
//
// Measured on 512 x 384 x 256 FP32: 105 us of a 137 us step against 114 of 145 for
// k_update_tma; HBM alone would take 96.  The shared-memory loads (12 wavefronts a
// node and warp) bound it.  Two splits with fewer loads were slower: rows of 4 to
// 8 nodes a thread from whole rows (117 against 90 us a step on 384 x 320 x 256, more
// address arithmetic than loads saved), and 256 x 8 strips by one copy a row (160
// us, the 26 copies of a plane).
enum Kind : uint8_t { kOpen = 0, kOutside = 1, kClosure = 2 };

__device__ __forceinline__ unsigned kind_of(uint32_t pos) {
  return ((pos >> 30) & 1u) ? kClosure : (pos & 0x7Fu) == 0 ? kOutside : kOpen;
}

template <typename S, typename C>
__global__ void __launch_bounds__(kThreads, 2)
k_iwb_flat(const S* __restrict__ P, S* __restrict__ Pp, const S* __restrict__ past,
           const C* __restrict__ cls, const uint32_t* __restrict__ pos, int n_classes, float b, int X,
           int64_t XY, int z_last, int zc, int stages, float l2, float nzf, uint64_t wait_ns,
           int* __restrict__ err) {
  using namespace px;
  using St = Store<S>;
  constexpr bool kSmemTab = sizeof(C) == 1;
  constexpr int kPairs = kPer / 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  __shared__ uint8_t kinds[kSmemTab ? 256 : 1];
  __shared__ __align__(8) uint64_t bars[2 * kMaxStages];
  __shared__ int abort_flag;
  const int halo = X + 1;
  const Stage lay = stage_of(halo, sizeof(S), sizeof(C), 0);
  const int t = threadIdx.x, lane = t & 31;
  const int64_t s0 = (int64_t)blockIdx.x * kRange;
  const int n = (int)(XY - s0 < kRange ? XY - s0 : (int64_t)kRange);
  const int z0 = 1 + blockIdx.y * zc, z1 = min(z0 + zc, z_last), nplanes = z1 - z0;
  const uint32_t full = smem_u32(bars), empty = full + 8 * kMaxStages;
  if (t == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, kConsumers / 32);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (kSmemTab)
    for (int i = t; i < n_classes; i += kThreads) kinds[i] = (uint8_t)kind_of(pos[i]);
  __syncthreads();
  step_wait();
  step_ready();
  if (*(volatile int*)err) return;
  if (nplanes <= 0) return;
  if (t >= kConsumers) {
    if (lane == 0)
      produce<S, C>(smem, lay, full, empty, &abort_flag, P, past, cls, halo, XY, s0, n, z0, nplanes + 2,
                    stages, 1, 0, err, wait_ns);
    return;
  }
  const f2 nz = pk2(nzf, nzf), l22 = pk2(l2, l2), w1 = pk2(0.25f, 0.25f), w2 = pk2(0.125f, 0.125f),
           w3 = pk2(0.0625f, 0.0625f), bb = pk2(b, b);
  // The in-plane sums of stage k, handed pair by pair to `use`.
  auto sums = [&](int k, auto&& use) {
    const int64_t fp = (int64_t)(z0 - 1 + k) * XY + s0 - halo;
    const S* p = (const S*)(smem + (size_t)(k % stages) * lay.bytes) + remainder_of<S>(fp) + halo + t;
    const S *u = p - X, *d = p + X;
#pragma unroll
    for (int h = 0; h < kPairs; ++h) {
      constexpr int o = kConsumers;
      auto at = [&](const S* q, int x) { return pk2(St::load(q[2 * h * o + x]), St::load(q[2 * h * o + o + x])); };
      use(h, at(p, 0), add2(add2(add2(at(u, 0), at(p, -1)), at(p, 1)), at(d, 0)),
          add2(add2(add2(at(u, -1), at(u, 1)), at(d, -1)), at(d, 1)));
    }
  };
  // of plane z: c0, c1, c2; of planes z and z-1 together: t1, t2, t3
  f2 c0[kPairs], c1[kPairs], c2[kPairs], t1[kPairs], t2[kPairs], t3[kPairs];
  bool ok = mbar_wait(full, 0, wait_ns) && mbar_wait(full + 8, 0, wait_ns);
  if (ok) {
    sums(0, [&](int h, f2 n0, f2 n1, f2 n2) { t1[h] = n0; t2[h] = n1; t3[h] = n2; });
    sums(1, [&](int h, f2 n0, f2 n1, f2 n2) {
      t1[h] = add2(n1, t1[h]);
      t2[h] = add2(n2, t2[h]);
      c0[h] = n0; c1[h] = n1; c2[h] = n2;
    });
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(empty);
      mbar_arrive(empty + 8);
    }
  }
  for (int j = 0; j < nplanes && ok; ++j) {
    const int sp = (j + 2) % stages;
    ok = mbar_wait(full + 8 * sp, (uint32_t)(((j + 2) / stages) & 1), wait_ns);
    if (!ok) break;
    const int64_t fq = (int64_t)(z0 + j) * XY + s0;
    const unsigned char* st = smem + (size_t)sp * lay.bytes;
    const S* pq = (const S*)(st + lay.past) + remainder_of<S>(fq) + t;
    const C* cl = (const C*)(st + lay.cls) + remainder_of<C>(fq) + t;
    S* out = Pp + fq + t;
    sums(j + 2, [&](int h, f2 n0, f2 n1, f2 n2) {
      const int e0 = 2 * h * kConsumers, e1 = e0 + kConsumers;
      const bool in0 = t + e0 < n, in1 = t + e1 < n;
      const S v0 = pq[e0], v1 = pq[e1];
      unsigned k0, k1;
      if (kSmemTab) {
        k0 = kinds[cl[e0]];
        k1 = kinds[cl[e1]];
      } else {
        k0 = in0 ? kind_of(__ldg(pos + cl[e0])) : (unsigned)kOutside;
        k1 = in1 ? kind_of(__ldg(pos + cl[e1])) : (unsigned)kOutside;
      }
      const f2 s1 = add2(t1[h], n0), s2 = add2(t2[h], n1), s3 = add2(t3[h], n2);
      const f2 sw = fma2(l22, add2(add2(fma2(s1, w1, nz), fma2(s2, w2, nz)), fma2(s3, w3, nz)), nz);
      const f2 o = sub2(add2(sw, fma2(bb, c0[h], nz)), pk2(St::load(v0), St::load(v1)));
      float o0, o1;
      up2(o, o0, o1);
      const S r0 = k0 == kClosure ? v0 : St::store(k0 == kOutside ? 0.f : o0);
      const S r1 = k1 == kClosure ? v1 : St::store(k1 == kOutside ? 0.f : o1);
      if (in0) out[e0] = r0;
      if (in1) out[e1] = r1;
      t1[h] = add2(n1, c0[h]);
      t2[h] = add2(n2, c1[h]);
      t3[h] = c2[h];
      c0[h] = n0; c1[h] = n1; c2[h] = n2;
    });
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + 8 * sp);
  }
  if (!ok) {
    atomicExch(err, 1);
    *(volatile int*)&abort_flag = 1;
  }
}

int flat_stages(const pfdtd_domain* d) {
  const int halo = (int)(d->X * d->K) + (d->class_scheme == PFDTD_IWB ? 1 : 0);
  const Stage lay = stage_of(halo, (int)d->esize, d->cls_bytes, d->kshift);
  return (int)std::min<int64_t>(kMaxStages, (int64_t)((kSmemPerCta - 8192) / lay.bytes));
}

// The shared-memory opt-in of a kernel, once per device.
template <typename K> int allow_smem(K kernel, std::atomic<bool>* done, std::mutex* mu, int device) {
  if (device >= 64) return fail(PFDTD_ERR_UNSUPPORTED, "device index above 63");
  if (!done[device].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lock(*mu);
    PFDTD_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kSmemPerCta - 6144)));
    done[device].store(true, std::memory_order_release);
  }
  return PFDTD_OK;
}

// Planes per CTA, as in launch_tma_t: two CTAs on an SM, and a chunk
// costs four planes more.
int64_t flat_chunk(const pfdtd_domain* d, int64_t gx) {
  const int64_t nz = d->Z - 2;
  int64_t best_c = 1;
  double best = 1e30;
  for (int64_t c = 1; c <= std::max<int64_t>(1, nz / 4); ++c) {
    const int64_t ctas = gx * c, resident = (int64_t)d->sm_count * 2;
    const int64_t waves = (ctas + resident - 1) / resident;
    const double cost = (double)(waves * resident) / (double)ctas * (1.0 + 4.0 * (double)c / (double)nz);
    if (cost < best - 1e-9) { best = cost; best_c = c; }
  }
  return (nz + best_c - 1) / best_c;
}

ClassTab<float> class_table(const pfdtd_domain* d) {
  const char* tb = (const char*)d->d_ctab;
  const size_t n = d->n_classes;
  return ClassTab<float>{(const float*)tb, (const float*)(tb + 4 * n), (const float*)(tb + 8 * n),
                         (const uint32_t*)(tb + 12 * n), d->n_classes};
}

template <typename S, typename C, int SCHEME>
int launch_flat_t(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  static std::atomic<bool> done[64];
  static std::mutex mu;
  const int64_t nz = d->Z - 2, XYE = d->XY * d->K;
  if (nz <= 0) return PFDTD_OK;
  if (int rc = allow_smem(k_update_flat<S, C, SCHEME>, done, &mu, d->device)) return rc;
  const int XE = (int)(d->X * d->K), stages = flat_stages(d);
  const int64_t gx = (XYE + kRange - 1) / kRange, zc = flat_chunk(d, gx);
  const Stage lay = stage_of(XE, sizeof(S), sizeof(C), d->kshift);
  PFDTD_CK(launch_step_kernel(k_update_flat<S, C, SCHEME>, dim3((unsigned)gx, (unsigned)((nz + zc - 1) / zc)),
                              dim3(kThreads), (size_t)stages * lay.bytes + 128, s, (const S*)cur, (S*)past,
                              (const S*)past, (const C*)d->d_cls, class_table(d), XE, XYE,
                              (int)(d->Z - 1), (int)zc, stages, d->K, d->kshift, (float)d->params[1],
                              -0.0f, (unsigned)d->air_class, d->wait_ns, d->d_err));
  count_launch();
  return PFDTD_OK;
}

template <typename S, typename C>
int launch_iwb_flat_t(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  static std::atomic<bool> done[64];
  static std::mutex mu;
  const int64_t nz = d->Z - 2;
  if (nz > 0) {
    if (int rc = allow_smem(k_iwb_flat<S, C>, done, &mu, d->device)) return rc;
    const int stages = flat_stages(d);
    const int64_t gx = (d->XY + kRange - 1) / kRange, zc = flat_chunk(d, gx);
    const Stage lay = stage_of((int)d->X + 1, sizeof(S), sizeof(C), 0);
    PFDTD_CK(launch_step_kernel(k_iwb_flat<S, C>, dim3((unsigned)gx, (unsigned)((nz + zc - 1) / zc)),
                                dim3(kThreads), (size_t)stages * lay.bytes + 128, s, (const S*)cur,
                                (S*)past, (const S*)past, (const C*)d->d_cls, class_table(d).pos,
                                d->n_classes, d->iwb_open_b, (int)d->X, d->XY, (int)(d->Z - 1), (int)zc,
                                stages, (float)d->params[1], -0.0f, d->wait_ns, d->d_err));
    count_launch();
  }
  return launch_iwb_closure(d, cur, past, s);
}

template <typename S, typename C>
int launch_flat_c(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  if (d->class_scheme == PFDTD_IWB) return launch_iwb_flat_t<S, C>(d, cur, past, s);
  if (d->class_scheme == PFDTD_SRL) return launch_flat_t<S, C, 1>(d, cur, past, s);
  if constexpr (std::is_same<S, float>::value) {
    if (d->class_form == PFDTD_FORM_DIFFERENCE) return launch_flat_t<S, C, 4>(d, cur, past, s);
  }
  return launch_flat_t<S, C, 0>(d, cur, past, s);
}

template <typename S>
int launch_flat_s(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  return d->cls_bytes == 1 ? launch_flat_c<S, uint8_t>(d, cur, past, s)
                           : launch_flat_c<S, uint16_t>(d, cur, past, s);
}

}  // namespace

// Whether the update by flat runs can take the room: 32-bit arithmetic, rows
// short enough for four stages; IWB with one field per node and its closure
// list.
bool flat_usable(const pfdtd_domain* d) {
  if (d->kernel_variant == PFDTD_KERNEL_ZMARCH || d->precision == PFDTD_F64) return false;
  if (d->class_scheme == PFDTD_IWB && !(d->K == 1 && d->iwb_closure_ready && d->iwb_open)) return false;
  return d->X * d->K <= 4096 && d->XY * d->K < ((int64_t)1 << 31) && flat_stages(d) >= 4;
}

// Whether a plane's last run is full enough: with 13 x 13 nodes of a run of 2048
// (1.5 M nodes in 9000 planes) an update took 32.7 us, 12.2 by the z-march kernel.
bool full_runs(const pfdtd_domain* d) {
  const int64_t n = d->XY * d->K;
  return 4 * n >= 3 * ((n + kRange - 1) / kRange) * kRange;
}

// Whether a 7-point room whose rows are not aligned takes the flat runs, or the
// z-march kernel: a CTA's stage ring only pays once there are enough runs to share.
// Us a step by single steps, FP32, z-march / runs: forward 50 x 41 x 36 4.9 / 6.3, 81 x
// 80 x 79 5.3 / 6.2, 90 x 91 x 89 (0.73 M) 5.7 / 6.3, two fields of 701 x 30 x 20 (0.84 M)
// 6.6 / 6.6, 97^3 (0.91 M) 8.0 / 6.2, 203 x 155 x 119 12.1 / 10.6; centred 5.2 / 8.1, 5.6 /
// 8.0, 5.8 / 8.1, 7.2 / 7.3, 9.1 / 8.0, 14.0 / 13.0; 16-bit fields alike.  Centred
// updates take longer a plane, and where some SMs have two CTAs and most one, or a
// chunk is all of a few planes, the runs lose: two fields of 96^3 (171 CTAs) 9.5 / 9.9,
// 131 x 127 x 125 (225) 9.8 / 10.5, two of 400 x 300 x 8 8.0 / 9.1; with 250 CTAs and more
// they win (161 x 120 x 110, 270: 9.8 / 8.8).
bool flat_pays(const pfdtd_domain* d) {
  if (!flat_usable(d)) return false;
  if (d->kernel_variant == PFDTD_KERNEL_TMA) return true;
  if (d->N * d->K < 850000 || !full_runs(d)) return false;
  if (d->class_scheme != PFDTD_SRL) return true;
  const int64_t nz = d->Z - 2, gx = (d->XY * d->K + kRange - 1) / kRange, zc = flat_chunk(d, gx);
  const int64_t ctas = gx * ((nz + zc - 1) / zc);
  return nz >= 8 && (ctas <= d->sm_count || 10 * ctas >= 16 * (int64_t)d->sm_count);
}

// Whether the next IWB update is by flat runs with the closure pass.
// Measured, us a step, FP32.  Rows that are not aligned, z-march / runs, with DIF
// walls: 97 x 81 x 65 11.9 / 13.9, 90 x 91 x 89 11.7 / 14.2, 101 x 103 x 99 (1.03 M) 15.3 /
// 14.6, 203 x 155 x 119 29.8 / 18.0; without, where the closure pass is all loss, 101 x
// 103 x 99 12.2 / 14.4, 401 x 300 x 12 (1.44 M) 10.9 / 13.5, 45 x 45 x 1000 (2.03 M) 22.3 /
// 15.5, 131 x 127 x 125 18.1 / 14.8.  Aligned rooms, tiles / runs, FP32 with DIF walls:
// 160^3 28.5 / 22.8, 384 x 320 x 256 103.9 / 91.6, 512 x 384 x 256 144.9 / 136.6,
// 256 x 192 x 128 29.7 / 29.3, 128^3 no difference (without walls 17.0 / 18.2); in
// FP16 512 x 384 x 256 without walls 150.6 / 157.2.
bool iwb_flat(const pfdtd_domain* d) {
  if (d->class_scheme != PFDTD_IWB || !flat_usable(d)) return false;
  if (!uses_tma(d))
    return d->kernel_variant == PFDTD_KERNEL_TMA ||
           (d->N >= (d->n_dif > 0 ? 1000000 : 1600000) && full_runs(d));
  return d->kernel_variant == PFDTD_KERNEL_AUTO && d->tma_tile < 0 && d->precision == PFDTD_F32 &&
         d->N >= 3000000 && full_runs(d);
}

int launch_update_flat(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  switch (d->precision) {
    case PFDTD_F32: return launch_flat_s<float>(d, cur, past, s);
    case PFDTD_F16: return launch_flat_s<__half>(d, cur, past, s);
    case PFDTD_BF16: return launch_flat_s<__nv_bfloat16>(d, cur, past, s);
  }
  return fail(PFDTD_ERR_UNSUPPORTED, "flat update needs FP32, FP16 or BF16 fields");
}

}  // namespace pfdtd
