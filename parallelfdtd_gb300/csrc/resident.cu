// Runs of small rooms with the whole grid resident on the SMs (sm_103a).
//
// A kernel per step costs a small room more than its work: on a 64^3 room the
// update and step-I/O launches took 11.1 us a step, of which the 262 k nodes'
// arithmetic is well under one.  Where the grid fits, one cooperative launch
// runs many steps instead: 1.9 us a step, of which about half is the exchange
// of faces (0.43 us one way through L2, and a failed poll costs a round trip).
// 128^3: 11.5 -> 6 us, bound by the instructions of the update and of the
// exchange at 16 warps a SM; FP64 64^3: 41 -> 8.5 us, bound by FP64 issue.  Each CTA owns a brick of nodes; the current field
// of the brick with a one-node halo lies in shared memory, the past field in
// registers, the class ids in shared memory, and a step's only global traffic
// is the brick's faces.
//
//  * A thread owns 4 neighbouring x nodes over up to NZ planes.  It marches z
//    with planes z-1, z, z+1 in registers, reads rows y -+ 1 from shared memory
//    and its x neighbours by warp shuffles, and leaves P^{n+1} in the registers
//    of P^{n-1}; after a barrier it swaps them with the brick's P^n.
//  * Faces go to the neighbouring bricks as {value, step tag} pairs, 64-bit
//    relaxed words, in an inbox per brick that alternates between two halves;
//    all threads share the sending and the receiving (a table in shared memory
//    gives each inbox value's node); the receiving thread polls the pair itself, so a value and its
//    arrival are one L2 round trip, with no fence, flag or grid barrier.  A
//    half is rewritten two steps later: by then the writer has received the
//    face that its neighbour computed from the earlier values, so they have
//    been read.
//  * Sources are injected by every CTA that holds the node in its brick or
//    halo, in source order; receivers are written by the owner each step.
//  * Planes 0 and Z-1 never change; the halo of the bricks next to them is
//    read from the fields each step.
//
// Arithmetic, order and rounding are those of k_update_tma (packed pairs with
// uncontractible products), so every result is the same.  As in the temporally
// blocked kernels the x and y faces must lie outside the room: then the
// flat-index wrap of the reference cannot matter while the fields are finite (a
// zero there may differ in sign).  A NaN or an infinity on a face goes on to the
// wrapped neighbour, so a room that can be foreseen to meet one (samples, materials,
// lambda) takes single steps; one that a caller has written into a field does not
// reach that neighbour here.  Every poll is bounded (the domain's wait limit): on expiry the kernel
// raises the error flag and returns, and the host reports it.
#include "common.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

namespace pfdtd {
namespace {

constexpr int kThreads = 512;        // one CTA per SM, 128 registers a thread
constexpr int kMaxSources = 32;      // of the domain; one lane of a warp each
constexpr int kMaxReceivers = 128;
constexpr size_t kSmemLimit = 227 * 1024;

struct Brick {
  int bx, by, bz;   // nodes of a brick (x a multiple of 4; z of planes 1..Z-2)
  int gx, gy, gz;   // bricks per axis
  int groups;       // thread groups along z
  int planes;       // planes per thread
  int pitch;        // values of a row in shared memory
};

template <typename A> struct alignas(4 * sizeof(A)) Coef { A a, b, c; uint32_t pos; };

template <typename S> struct Args {
  using A = typename Store<S>::A;
  S *cur, *past;               // fields at the first step
  const uint8_t* cls;
  ClassTab<A> tab;
  uint32_t air;                // class word of 4 air nodes (a = 1), 0xFFFFFFFF: none
  int X, Y, Z;
  Brick k;
  uint64_t* inbox;             // [2][bricks][words]
  int words;                   // 64-bit words of a brick's inbox half
  uint32_t tag;                // of the first step
  int64_t step0;
  int steps;
  int n_src, n_rec;
  const int64_t *src_idx, *rec_idx;
  const int32_t* src_mode;
  const A* samples;
  int64_t n_samples, inject_end;
  A* rec_out;
  int64_t rec_ld;
  A l2;
  float nzf;                   // -0, see common.cuh
  uint64_t wait_ns;
  int* err;
};

// ---- {value, tag} words -----------------------------------------------------

__device__ __forceinline__ uint64_t word(uint32_t v, uint32_t tag) {
  return (uint64_t)v | ((uint64_t)tag << 32);
}
__device__ __forceinline__ void st_word2(uint64_t* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_word2(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A value is one word (float) or two (the halves of a double).
template <typename A> constexpr int kWords = sizeof(A) / 4;

__device__ __forceinline__ bool tagged(uint64_t w, uint32_t tag) { return (uint32_t)(w >> 32) == tag; }

// ---- four nodes -------------------------------------------------------------

template <typename A> __device__ __forceinline__ void lds4(const A* p, A (&v)[4]) {
  if constexpr (sizeof(A) == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
    const double2 s = reinterpret_cast<const double2*>(p)[0], t = reinterpret_cast<const double2*>(p)[1];
    v[0] = s.x; v[1] = s.y; v[2] = t.x; v[3] = t.y;
  }
}
template <typename A> __device__ __forceinline__ void sts4(A* p, const A (&v)[4]) {
  if constexpr (sizeof(A) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
  }
}

// The 7-point update of 4 x neighbours, P^{n-1} in and P^{n+1} out through pp.
template <int SCHEME>
__device__ __forceinline__ void update4(const float (&fm)[4], const float (&fc)[4],
                                        const float (&fn)[4], const float (&ym)[4],
                                        const float (&yp)[4], float left, float right,
                                        const Coef<float> (&k)[4], bool, float l2, float nzf,
                                        float (&pp)[4]) {
  using namespace px;
  const f2 l22 = pk2(l2, l2), nz = pk2(nzf, nzf);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const Coef<float>& k0 = k[2 * h];
    const Coef<float>& k1 = k[2 * h + 1];
    const f2 pc = pk2(fc[2 * h], fc[2 * h + 1]), pm = pk2(fm[2 * h], fm[2 * h + 1]);
    const f2 pn = pk2(fn[2 * h], fn[2 * h + 1]), po = pk2(pp[2 * h], pp[2 * h + 1]);
    const f2 m2 = pk2(ym[2 * h], ym[2 * h + 1]), p2 = pk2(yp[2 * h], yp[2 * h + 1]);
    const float xm0 = h == 0 ? left : fc[1], xp1 = h == 0 ? fc[2] : right;
    const f2 xm = pk2(xm0, fc[2 * h]), xp = pk2(fc[2 * h + 1], xp1);
    const f2 aa = pk2(k0.a, k1.a), bb = pk2(k0.b, k1.b), cc = pk2(k0.c, k1.c);
    f2 o;
    if constexpr (SCHEME == 1) {
      float bx[2], by[2], bz[2], dx[2], dy[2], dz[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int e = 2 * h + q;
        const uint32_t cp = q == 0 ? k0.pos : k1.pos;
        const float vm = q == 0 ? xm0 : fc[2 * h], vp = q == 0 ? fc[2 * h + 1] : xp1;
        bx[q] = (cp & 0x10u) ? vp : vm;
        by[q] = (cp & 0x20u) ? yp[e] : ym[e];
        bz[q] = (cp & 0x40u) ? fm[e] : fn[e];
        dx[q] = (float)(cp & 1u);
        dy[q] = (float)((cp >> 1) & 1u);
        dz[q] = (float)((cp >> 2) & 1u);
      }
      const f2 sb6 = add2(add2(fma2(pk2(bx[0], bx[1]), pk2(dx[0], dx[1]), nz),
                               fma2(pk2(by[0], by[1]), pk2(dy[0], dy[1]), nz)),
                          fma2(pk2(bz[0], bz[1]), pk2(dz[0], dz[1]), nz));
      const f2 s7 = add2(add2(add2(add2(add2(add2(xm, xp), m2), p2), pn), pm), sb6);
      o = mul2(aa, add2(sub2(fma2(s7, l22, nz), fma2(bb, pc, nz)), fma2(cc, po, nz)));
    } else {
      const f2 s6 = add2(add2(add2(add2(add2(pn, pm), p2), m2), xp), xm);
      if constexpr (SCHEME == 4) {  // difference form, the pos word holds 1 + beta
        const f2 ee = pk2(__uint_as_float(k0.pos), __uint_as_float(k1.pos));
        o = mul2(aa, add2(add2(fma2(ee, pc, nz), fma2(cc, sub2(pc, po), nz)),
                          fma2(l22, sub2(s6, fma2(bb, pc, nz)), nz)));
      } else {
        o = mul2(aa, sub2(add2(fma2(bb, pc, nz), fma2(l22, s6, nz)), fma2(cc, po, nz)));
      }
    }
    up2(o, pp[2 * h], pp[2 * h + 1]);
  }
}

// In double an SM issues about two operations a cycle: four air nodes (lossy
// false: a = 1, c = +-1) leave their exact products by 1 out.
template <int SCHEME>
__device__ __forceinline__ void update4(const double (&fm)[4], const double (&fc)[4],
                                        const double (&fn)[4], const double (&ym)[4],
                                        const double (&yp)[4], double left, double right,
                                        const Coef<double> (&k)[4], bool lossy, double l2, float,
                                        double (&pp)[4]) {
  using R = Rn<double>;
  double v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const Coef<double>& c = k[e];
    const double xm = e == 0 ? left : fc[e > 0 ? e - 1 : 0], xp = e == 3 ? right : fc[e < 3 ? e + 1 : 3];
    if constexpr (SCHEME == 1) {
      const double dx = (double)(c.pos & 1u), dy = (double)((c.pos >> 1) & 1u),
                   dz = (double)((c.pos >> 2) & 1u);
      const double bx = (c.pos & 0x10u) ? xp : xm;
      const double by = (c.pos & 0x20u) ? yp[e] : ym[e];
      const double bz = (c.pos & 0x40u) ? fm[e] : fn[e];
      const double sb6 = R::add(R::add(R::mul(bx, dx), R::mul(by, dy)), R::mul(bz, dz));
      const double s7 =
          R::add(R::add(R::add(R::add(R::add(R::add(xm, xp), ym[e]), yp[e]), fn[e]), fm[e]), sb6);
      v[e] = R::sub(R::mul(s7, l2), R::mul(c.b, fc[e]));
    } else {
      const double s6 = R::add(R::add(R::add(R::add(R::add(fn[e], fm[e]), yp[e]), ym[e]), xp), xm);
      v[e] = R::add(R::mul(c.b, fc[e]), R::mul(l2, s6));
    }
  }
  if (lossy) {
#pragma unroll
    for (int e = 0; e < 4; ++e) pp[e] = R::mul(SCHEME == 1 ? -k[e].c : k[e].c, pp[e]);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) pp[e] = R::sub(v[e], pp[e]);
  if (lossy) {
#pragma unroll
    for (int e = 0; e < 4; ++e) pp[e] = R::mul(k[e].a, pp[e]);
  }
}

// Values of an inbox half's segments x-, x+, y-, y+, z-, z+ (two of each size).
struct Segments { int x, y, z; };
__host__ __device__ inline Segments segments(const Brick& k) {
  return Segments{(k.by * k.bz + 3) / 4 * 4, k.bx * k.bz, k.bx * k.by};
}
__host__ __device__ inline int inbox_values(const Brick& k) {
  const Segments s = segments(k);
  return 2 * (s.x + s.y + s.z);
}
// Shared-memory bytes of a brick: field with halo, coefficients, class ids and
// the place of every inbox value.
template <typename A> size_t brick_smem(const Brick& k) {
  return ((size_t)(k.bz + 2) * (k.by + 2) * k.pitch + 4) * sizeof(A) + 256 * sizeof(Coef<A>) +
         (size_t)k.bx * k.by * k.bz + 2 * (size_t)inbox_values(k) + 16;
}
constexpr int kNoPlace = 0xFFFF;     // an inbox value that nobody sends
constexpr int kBatch = 4;            // 16-byte inbox loads a thread has in flight

template <typename S, int SCHEME, int NZ>
__global__ void __launch_bounds__(kThreads, 1) k_resident(const __grid_constant__ Args<S> g) {
  using A = typename Store<S>::A;
  using St = Store<S>;
  constexpr int W = kWords<A>;
  constexpr bool CARRY = NZ * sizeof(A) <= 16;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int l_src[kMaxSources], l_rec[kMaxReceivers];   // shared-memory offsets
  __shared__ int l_src_id[kMaxSources], l_rec_id[kMaxReceivers];
  __shared__ int n_lsrc, n_lrec, gave_up;
  // One thread reads the flag, and the block leaves or stays as a whole: a block
  // of this launch whose wait expires may raise it while this one starts, and a
  // block that some threads have left would run on tables they never filled.
  if (threadIdx.x == 0) n_lsrc = n_lrec = gave_up = 0;
  if (__syncthreads_or(threadIdx.x == 0 && *(volatile int*)g.err != 0)) return;
  const Brick& k = g.k;
  // Rows of the brick start 4 values into a row of the array.  The left halo
  // node lies in the value before; the right one after the row, which may be
  // the first value of the next row's 4 (pitch >= bx + 4).
  const int pitch = k.pitch, rows = k.by + 2, plane = pitch * rows;
  A* P = (A*)smem;
  Coef<A>* tab = (Coef<A>*)(P + (size_t)plane * (k.bz + 2) + 4);
  uint8_t* cls = (uint8_t*)(tab + 256);
  uint16_t* place = (uint16_t*)(cls + k.bx * k.by * k.bz);  // k.bx is a multiple of 4
  const int t = threadIdx.x, lane = t & 31, b = blockIdx.x;
  const int ix = b % k.gx, iy = b / k.gx % k.gy, iz = b / (k.gx * k.gy);
  const int x0 = ix * k.bx, y0 = iy * k.by, z0 = 1 + iz * k.bz;
  const int xe = min(k.bx, g.X - x0), ye = min(k.by, g.Y - y0), ze = min(k.bz, g.Z - 1 - z0);
  const int64_t XY = (int64_t)g.X * g.Y;
  const int64_t origin = z0 * XY + (int64_t)y0 * g.X + x0;  // the brick's first node

  // field with halo, class ids (nodes past the grid: the all-zero class),
  // coefficients
  for (int i = t; i < plane * (k.bz + 2) + 4; i += kThreads) P[i] = (A)0;
  __syncthreads();
  for (int i = t; i < (k.bx + 2) * rows * (k.bz + 2); i += kThreads) {
    const int c = i % (k.bx + 2) - 1, r = i / (k.bx + 2) % rows - 1, z = i / ((k.bx + 2) * rows) - 1;
    const int x = x0 + c, y = y0 + r;
    if (x >= 0 && x < g.X && y >= 0 && y < g.Y && z0 + z < g.Z)
      P[(z + 1) * plane + (r + 1) * pitch + 4 + c] =
          St::load(g.cur[origin + z * XY + (int64_t)r * g.X + c]);
  }
  for (int i = t; i < k.bx * k.by * k.bz; i += kThreads) {
    const int c = i % k.bx, r = i / k.bx % k.by, z = i / (k.bx * k.by);
    cls[i] = (c < xe && r < ye && z < ze) ? g.cls[origin + z * XY + (int64_t)r * g.X + c]
                                          : (uint8_t)g.tab.n;
  }
  // the halo node of every inbox value
  const Segments sg = segments(k);
  const int xw = (xe + 3) / 4 * 4;
  for (int i = t; i < 2 * (sg.x + sg.y + sg.z); i += kThreads) {
    int o = kNoPlace, r = i;
    if (r < 2 * sg.x) {
      const int f = r >= sg.x, z = (r - f * sg.x) / k.by, y = (r - f * sg.x) % k.by;
      if (z < ze && y < ye && (f ? ix + 1 < k.gx : ix > 0))
        o = (z + 1) * plane + (y + 1) * pitch + (f ? 4 + k.bx : 3);
    } else if ((r -= 2 * sg.x) < 2 * sg.y) {
      const int f = r >= sg.y, z = (r - f * sg.y) / k.bx, x = (r - f * sg.y) % k.bx;
      if (z < ze && x < xw && (f ? iy + 1 < k.gy : iy > 0))
        o = (z + 1) * plane + (f ? k.by + 1 : 0) * pitch + 4 + x;
    } else {
      r -= 2 * sg.y;
      const int f = r >= sg.z, y = (r - f * sg.z) / k.bx, x = (r - f * sg.z) % k.bx;
      if (y < ye && x < xw && (f ? iz + 1 < k.gz : iz > 0))
        o = (f ? k.bz + 1 : 0) * plane + (y + 1) * pitch + 4 + x;
    }
    place[i] = (uint16_t)o;
  }
  for (int i = t; i < 256; i += kThreads)
    tab[i] = i < g.tab.n ? Coef<A>{g.tab.a[i], g.tab.b[i], g.tab.c[i], g.tab.pos[i]}
                         : Coef<A>{(A)0, (A)0, (A)0, 0u};
  // sources in the brick or its halo, receivers in the brick, in order
  if (t < 32) {
    auto collect = [&](const int64_t* idx, int n, int margin, int most, int* off, int* id) {
      int count = 0;
      for (int base = 0; base < n; base += 32) {
        const int s = base + lane;
        int o = -1;
        if (s < n && idx[s] >= 0) {
          const int64_t i = idx[s];
          const int z = (int)(i / XY) - z0, r = (int)(i % XY / g.X) - y0, c = (int)(i % g.X) - x0;
          // outside the brick on at most one axis, and there by one node
          const int out = (c < 0 || c >= xe) + (r < 0 || r >= ye) + (z < 0 || z >= ze);
          if (c >= -margin && c < xe + margin && r >= -margin && r < ye + margin && z >= -margin &&
              z < ze + margin && out <= margin)
            o = (z + 1) * plane + (r + 1) * pitch + 4 + c;
        }
        const unsigned m = __ballot_sync(0xffffffffu, o >= 0);
        const int at = count + __popc(m & ((1u << lane) - 1u));
        if (o >= 0 && at < most) {
          off[at] = o;
          id[at] = s;
        }
        count += __popc(m);
      }
      return count;
    };
    const int ns = collect(g.src_idx, g.n_src, 1, kMaxSources, l_src, l_src_id);
    const int nr = collect(g.rec_idx, g.n_rec, 0, kMaxReceivers, l_rec, l_rec_id);
    if (lane == 0) {
      n_lsrc = ns;
      n_lrec = nr;
    }
  }

  // the thread's nodes
  const int nvx = k.bx / 4, ncol = nvx * k.by;
  const int zq = t / ncol, col = t - zq * ncol;
  const int lx = col % nvx * 4, ly = col / nvx, kz = zq * k.planes;
  const bool active = zq < k.groups && ly < ye && lx < xe && kz < ze;
  // (a thread without nodes runs along on its group's first place)
  const int nz = active ? min(k.planes, ze - kz) : 0;
  const int si = active ? (kz + 1) * plane + (ly + 1) * pitch + 4 + lx : plane + pitch + 4;
  const int ci = active ? (kz * k.by + ly) * k.bx + lx : 0;
  const int64_t gi = origin + kz * XY + (int64_t)ly * g.X + lx;
  const bool shfl_l = lane > 0 && lx > 0, shfl_r = lane < 31 && lx + 4 < min(k.bx, (xe + 3) / 4 * 4);
  const bool warp_on = (t & ~31) < ncol * k.groups;
  // Past values, and (CARRY: few planes a thread) the current ones too, which
  // then need not be read back from shared memory: three 128-bit accesses a
  // plane instead of five.
  A pp[NZ][4], cu[CARRY ? NZ : 1][4];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NZ; ++j) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      pp[j][e] = (j < nz && lx + e < xe) ? St::load(g.past[gi + j * XY + e]) : (A)0;
    if constexpr (CARRY) lds4(P + si + min(j, max(nz - 1, 0)) * plane, cu[j]);
  }

  const int64_t half = (int64_t)gridDim.x * g.words;
  const bool z_first = active && kz == 0 && iz == 0, z_last = active && kz + nz == ze && iz + 1 == k.gz;
  const int units = (sg.x + sg.y + sg.z) * W;  // 16-byte units of an inbox half
  const A l2 = g.l2;
  A sample = (A)0;  // lane s of warp 0: the next sample of local source s
  __syncthreads();
  auto fetch = [&](int64_t n) {
    if (t < n_lsrc && n < g.inject_end && n < g.n_samples)
      sample = g.samples[(int64_t)l_src_id[t] * g.n_samples + n];
  };
  fetch(g.step0);
  const Coef<A> air = tab[g.air & 0xFFu];

  for (int n = 0; n < g.steps; ++n) {
    const uint32_t tag = g.tag + (uint32_t)n;
    uint64_t* own = g.inbox + (tag & 1) * half + (int64_t)b * g.words;
    // this step's source samples, in order
    if (n_lsrc > 0) {
      const int64_t step = g.step0 + n;
      if (t < 32) {
        if (step < g.inject_end && step < g.n_samples) {
          for (int s = 0; s < n_lsrc; ++s) {
            if (lane == s) {
              A& p = P[l_src[s]];
              p = St::load(St::store(g.src_mode[l_src_id[s]] == 0 ? sample : Rn<A>::add(p, sample)));
            }
            __syncwarp();
          }
        }
        fetch(step + 1);
      }
      __syncthreads();
    }
    // P^{n+1}: into the registers of P^{n-1} (CARRY: of P^n, which moves on)
    if (warp_on) {
      if constexpr (CARRY) {
        if (n_lsrc > 0) {
#pragma unroll
          for (int j = 0; j < NZ; ++j) lds4(P + si + min(j, max(nz - 1, 0)) * plane, cu[j]);
        }
      }
      A f[3][4];
      lds4(P + si - plane, f[0]);
      if constexpr (!CARRY) lds4(P + si, f[1]);
#pragma unroll
      for (int j = 0; j < NZ; ++j) {
        if (j < k.planes) {
          // past its last plane a thread computes that one again, into
          // registers that nobody reads
          const int jj = min(j, max(nz - 1, 0));
          const A* p = P + si + jj * plane;
          A fc[4], fm[4], fn[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            fm[e] = CARRY && j > 0 ? pp[j > 0 ? j - 1 : 0][e] : f[j % 3][e];
            fc[e] = CARRY ? cu[CARRY ? j : 0][e] : f[(j + 1) % 3][e];
          }
          if constexpr (CARRY) {
#pragma unroll
            for (int e = 0; e < 4; ++e) fn[e] = j + 1 < NZ ? cu[CARRY && j + 1 < NZ ? j + 1 : 0][e] : (A)0;
            if (j + 1 >= nz) lds4(p + plane, fn);
          } else {
            lds4(p + plane, fn);
#pragma unroll
            for (int e = 0; e < 4; ++e) f[(j + 2) % 3][e] = fn[e];
          }
          A ym[4], yp[4];
          lds4(p - pitch, ym);
          lds4(p + pitch, yp);
          const uint32_t w = *reinterpret_cast<const uint32_t*>(cls + ci + jj * k.bx * k.by);
          A left = __shfl_up_sync(0xffffffffu, fc[3], 1);
          A right = __shfl_down_sync(0xffffffffu, fc[0], 1);
          if (!shfl_l) left = p[-1];
          if (!shfl_r) right = p[4];
          // open air, most of a room: the coefficients kept in registers
          Coef<A> c[4] = {air, air, air, air};
          if (w != g.air) {
            c[0] = tab[w & 0xFFu];
            c[1] = tab[(w >> 8) & 0xFFu];
            c[2] = tab[(w >> 16) & 0xFFu];
            c[3] = tab[w >> 24];
          }
          update4<SCHEME>(fm, fc, fn, ym, yp, left, right, c, w != g.air, l2, g.nzf, pp[j]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if constexpr (sizeof(S) == 2) pp[j][e] = St::load(St::store(pp[j][e]));
            if constexpr (CARRY) {
              cu[j][e] = pp[j][e];
              pp[j][e] = fc[e];
            }
          }
        }
      }
    }
    __syncthreads();
    // P^{n+1} into the brick (without CARRY P^n into the registers)
#pragma unroll
    for (int j = 0; j < NZ; ++j) {
      if (j < nz) {
        A* p = P + si + j * plane;
        if constexpr (CARRY) {
          sts4(p, cu[j]);
        } else {
          A c[4];
          lds4(p, c);
          sts4(p, pp[j]);
#pragma unroll
          for (int e = 0; e < 4; ++e) pp[j][e] = c[e];
        }
      }
    }
    if (n + 1 < g.steps) {
      __syncthreads();
      // faces to the neighbours: an inbox value's place in the halo, moved one
      // node inwards, is the node that the neighbour across that face wants,
      // at the same index of its opposite segment
#pragma unroll 4
      for (int u = t; u < units; u += kThreads) {
        const int v = u * 2 / W;
        const bool fx = v < 2 * sg.x, fy = !fx && v < 2 * (sg.x + sg.y);
        const int first = fx ? 0 : (fy ? 2 * sg.x : 2 * (sg.x + sg.y));
        const int size = fx ? sg.x : (fy ? sg.y : sg.z);
        const int inward = fx ? 1 : (fy ? pitch : plane);
        const int far = fx ? 1 : (fy ? k.gx : k.gx * k.gy);  // bricks to the neighbour
        const int dir = v >= first + size ? 1 : -1;           // the + face
        uint64_t* to = own + (int64_t)(dir * far) * g.words + (int64_t)(v - dir * size) * W;
        if constexpr (W == 1) {
          const uint32_t pl = reinterpret_cast<const uint32_t*>(place)[u];
          const uint32_t p0 = pl & 0xFFFFu, p1 = pl >> 16;
          const float a = p0 == kNoPlace ? 0.f : P[(int)p0 - dir * inward];
          const float c = p1 == kNoPlace ? 0.f : P[(int)p1 - dir * inward];
          if (pl != 0xFFFFFFFFu) st_word2(to, word(__float_as_uint(a), tag), word(__float_as_uint(c), tag));
        } else {
          const int pl = place[v];
          const A a = pl == kNoPlace ? (A)0 : P[pl - dir * inward];
          if (pl != kNoPlace)
            st_word2(to, word((uint32_t)__double2loint(a), tag), word((uint32_t)__double2hiint(a), tag));
        }
      }
      // planes 0 and Z-1: the field that the update has made current
      const S* fixed = (n & 1) ? g.cur : g.past;
      if (z_first) {
        A v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = lx + e < xe ? St::load(fixed[gi - XY + e]) : (A)0;
        sts4(P + si - plane, v);
      }
      if (z_last) {
        A v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = lx + e < xe ? St::load(fixed[gi + nz * XY + e]) : (A)0;
        sts4(P + si + nz * plane, v);
      }
      // the neighbours' faces into the halo: every thread polls its share of
      // the inbox, kBatch 16-byte units (two floats or one double) in flight
      uint64_t t0 = 0;
      for (int base = t; base < units; base += kThreads * kBatch) {
        uint32_t to[kBatch], wanted = 0;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int u = base + i * kThreads;
          to[i] = 0xFFFFFFFFu;
          if (u < units) {
            if constexpr (W == 1) to[i] = reinterpret_cast<const uint32_t*>(place)[u];
            else to[i] = place[u] == kNoPlace ? 0xFFFFFFFFu : place[u];
          }
          if (to[i] != 0xFFFFFFFFu) wanted |= 1u << i;
        }
        for (uint32_t tries = 1; wanted != 0; ++tries) {
          uint64_t a[kBatch], c[kBatch];
#pragma unroll
          for (int i = 0; i < kBatch; ++i)
            if (wanted >> i & 1) ld_word2(own + 2 * (base + i * kThreads), a[i], c[i]);
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            if (!(wanted >> i & 1)) continue;
            if constexpr (W == 1) {
              const uint32_t p0 = to[i] & 0xFFFFu, p1 = to[i] >> 16;
              if ((p0 == kNoPlace || tagged(a[i], tag)) && (p1 == kNoPlace || tagged(c[i], tag))) {
                if (p0 != kNoPlace) P[p0] = __uint_as_float((uint32_t)a[i]);
                if (p1 != kNoPlace) P[p1] = __uint_as_float((uint32_t)c[i]);
                wanted &= ~(1u << i);
              }
            } else {
              if (tagged(a[i], tag) && tagged(c[i], tag)) {
                P[to[i]] = __hiloint2double((int)(uint32_t)c[i], (int)(uint32_t)a[i]);
                wanted &= ~(1u << i);
              }
            }
          }
          if (wanted != 0 && ((tries & 63) == 0 || g.wait_ns < 1000000ull)) {
            const uint64_t now = now_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > g.wait_ns || *(volatile int*)g.err) {
              gave_up = 1;
              break;
            }
          }
        }
        if (wanted != 0) break;
      }
    }
    __syncthreads();
    if (gave_up) {
      if (t == 0) atomicExch(g.err, 1);
      return;
    }
    // receivers of the finished step
    if (t < 32 && g.rec_out != nullptr && g.step0 + n < g.rec_ld) {
      for (int r = lane; r < n_lrec; r += 32)
        g.rec_out[(int64_t)l_rec_id[r] * g.rec_ld + g.step0 + n] = P[l_rec[r]];
      __syncwarp();
    }
  }

  // back to the fields: after an odd number of steps their roles have changed
  S* cur = (g.steps & 1) ? g.past : g.cur;
  S* past = (g.steps & 1) ? g.cur : g.past;
#pragma unroll
  for (int j = 0; j < NZ; ++j) {
    if (j < nz) {
      A c[4];
      lds4(P + si + j * plane, c);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (lx + e < xe) {
          cur[gi + j * XY + e] = St::store(c[e]);
          past[gi + j * XY + e] = St::store(pp[j][e]);
        }
    }
  }
}

// The split of the grid into at most `sms` bricks with the least estimated
// time a step: the busiest CTA's warp-planes (about 30 cycles each: shared
// memory bandwidth; in double about 900, its operations), its face nodes (a third
// of a cycle each) and a fixed exchange latency.  (With 60 cycles for doubles a
// 16^3 room was one brick: 15.2 us a step, 3.1 in many.)  false: the grid does not
// fit.
template <typename A>
bool plan_bricks(const pfdtd_domain* d, int max_planes, Brick* out, double* cycles) {
  double best = 1e30;
  const int64_t nz = d->Z - 2;
  for (int gx = 1; gx <= d->sm_count && gx <= d->X; ++gx) {
    Brick k;
    const int64_t bx = ((d->X + gx - 1) / gx + 3) / 4 * 4;
    if (bx / 4 > kThreads) continue;
    k.bx = (int)bx;
    k.gx = (int)((d->X + bx - 1) / bx);
    if (k.gx != gx) continue;
    for (int gy = 1; gx * gy <= d->sm_count && gy <= d->Y; ++gy) {
      const int64_t by = (d->Y + gy - 1) / gy;
      if (bx / 4 * by > kThreads) continue;
      k.by = (int)by;
      k.gy = (int)((d->Y + by - 1) / by);
      if (k.gy != gy) continue;
      const int64_t gz_max = std::min<int64_t>(nz, d->sm_count / (gx * gy));
      for (int64_t gz = 1; gz <= gz_max; ++gz) {
        const int64_t bz = (nz + gz - 1) / gz;
        k.bz = (int)std::min<int64_t>(bz, 1 << 20);
        k.gz = (int)((nz + bz - 1) / bz);
        if (k.gz != gz || bz > 1 << 20) continue;
        const int ncol = k.bx / 4 * k.by;
        k.groups = std::min(kThreads / ncol, k.bz);
        k.planes = (k.bz + k.groups - 1) / k.groups;
        // rows of a whole number of 32 values follow one another without bank
        // conflicts; others want their place in the banks kept from row to row
        k.pitch = k.bx + (k.bx % 32 != 0 ? 32 : 4);
        if (brick_smem<A>(k) > kSmemLimit - 4096) k.pitch = k.bx + 4;
        if (k.planes > max_planes || brick_smem<A>(k) > kSmemLimit - 4096) continue;
        if ((k.bz + 2) * (k.by + 2) * k.pitch + 4 > kNoPlace) continue;  // 16-bit places
        const int warps = (ncol * k.groups + 31) / 32;
        const double faces = (k.gx > 1 ? 2.0 * k.by * k.bz : 0) + (k.gy > 1 ? 2.0 * k.bx * k.bz : 0) +
                             (k.gz > 1 ? 2.0 * k.bx * k.by : 0);
        const double cost = (sizeof(A) == 8 ? 900.0 : 30.0) * k.planes * warps +
                            0.35 * (sizeof(A) / 4) * faces + (faces > 0 ? 2500.0 : 500.0);
        if (cost < best) {
          best = cost;
          *out = k;
        }
      }
    }
  }
  *cycles = best;
  return best < 1e30;
}

template <typename S, int SCHEME, int NZ>
int launch_nz(pfdtd_domain* d, const Args<S>& a, cudaStream_t s) {
  using A = typename Store<S>::A;
  static std::atomic<bool> attr_done[64];
  static std::mutex attr_mu;
  if (d->device >= 64) return fail(PFDTD_ERR_UNSUPPORTED, "device index above 63");
  if (!attr_done[d->device].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lock(attr_mu);
    PFDTD_CK(cudaFuncSetAttribute(k_resident<S, SCHEME, NZ>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemLimit - 4096)));
    attr_done[d->device].store(true, std::memory_order_release);
  }
  void* args[] = {(void*)&a};
  const cudaError_t e =
      cudaLaunchCooperativeKernel((const void*)k_resident<S, SCHEME, NZ>,
                                  dim3(a.k.gx * a.k.gy * a.k.gz), dim3(kThreads), args,
                                  brick_smem<A>(a.k), s);
  // Refused as a whole, where the process may not use as many SMs at once as
  // there are bricks: nothing has run, and the domain keeps to single steps.
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources ||
      e == cudaErrorNotSupported) {
    cudaGetLastError();
    d->resident.ok = false;
    return PFDTD_ERR_UNSUPPORTED;
  }
  PFDTD_CK(e);
  count_launch();
  return PFDTD_OK;
}

// Register arrays are sized at compile time: the smallest that holds the
// plan's planes per thread.  Eight planes of 4 nodes for 512 threads are 2.4 M
// nodes on the whole chip.  With 12 and 17 planes the FP32 kernel spilled: it
// took 13.2 us a step on 160^3 and 15.1 on 203 x 155 x 119, where single steps
// take 10.8, so larger rooms keep to single steps.  At the line, us a step,
// resident / single: FP32 forward 128^3 5.2 / 6.6, 128 x 150 x 124 6.5 / 7.2, 131 x 127
// x 125 6.8 / 8.6, centred 6.3 / 7.1, 7.8 / 7.7 and 7.7 / 10.7; FP16 forward 5.3 / 6.3, 6.6 /
// 6.4 and 7.0 / 9.0.
constexpr int kMaxPlanes = 8;
// Nodes per SM of an FP64 room.  The z-march kernel keeps the FP64 units busier
// once it fills the SMs.  Forward and centred, us a step, resident / single: 24^3
// 3.0 / 3.4 and 4.3 / 4.1, 64^3 8.2 / 9.3 and 12.8 / 14.3, 100 x 90 x 80 22.4 / 26.2 and
// 37.3 / 44.5, 92 x 90 x 92 20.8 / 22.9 and 33.7 / 38.9; beyond the line 128 x 96 x 64
// 23.0 / 20.3 and 36.9 / 34.1, 96^3 26.1 / 23.0 and 40.6 / 38.9, 128 x 96 x 100 33.2 / 29.4
// and 54.2 / 44.6, though 112 x 104 x 100 32.4 / 32.0 and 53.5 / 55.0.
constexpr int kMostDoubles = 5100;

template <typename S, int SCHEME>
int launch_scheme(pfdtd_domain* d, const Args<S>& a, cudaStream_t s) {
  const int p = a.k.planes;
  if (p <= 1) return launch_nz<S, SCHEME, 1>(d, a, s);
  if (p <= 2) return launch_nz<S, SCHEME, 2>(d, a, s);
  if (p <= 4) return launch_nz<S, SCHEME, 4>(d, a, s);
  if (p <= 8) return launch_nz<S, SCHEME, 8>(d, a, s);
  return fail(PFDTD_ERR_UNSUPPORTED, "brick too deep");
}

template <typename S>
int launch_t(pfdtd_domain* d, int64_t step0, int64_t steps, void* rec_out, int64_t rec_ld,
             int64_t inject_end, cudaStream_t s) {
  using A = typename Store<S>::A;
  const ResidentState& rs = d->resident;
  Args<S> a;
  a.cur = (S*)d->cur_field();
  a.past = (S*)d->past_field();
  a.cls = (const uint8_t*)d->d_cls;
  const size_t as = sizeof(A);
  const char* tb = (const char*)d->d_ctab;
  a.tab = ClassTab<A>{(const A*)tb, (const A*)(tb + as * d->n_classes),
                      (const A*)(tb + 2 * as * d->n_classes),
                      (const uint32_t*)(tb + 3 * as * d->n_classes), d->n_classes};
  a.air = d->air_class >= 0 ? 0x01010101u * (uint32_t)d->air_class : 0xFFFFFFFFu;
  a.X = (int)d->X;
  a.Y = (int)d->Y;
  a.Z = (int)d->Z;
  a.k = Brick{rs.brick[0], rs.brick[1], rs.brick[2], rs.brick[3],
              rs.brick[4], rs.brick[5], rs.brick[6], rs.brick[7], rs.brick[8]};
  a.inbox = (uint64_t*)rs.inbox;
  a.words = rs.words;
  a.tag = rs.tag;
  a.step0 = step0;
  a.steps = (int)steps;
  a.n_src = d->n_src;
  a.n_rec = d->n_rec;
  a.src_idx = d->d_src_idx;
  a.rec_idx = d->d_rec_idx;
  a.src_mode = d->d_src_mode;
  a.samples = (const A*)d->d_src_samples;
  a.n_samples = d->n_samples;
  a.inject_end = inject_end;
  a.rec_out = (A*)rec_out;
  a.rec_ld = rec_ld;
  a.l2 = (A)d->params[1];
  a.nzf = -0.0f;
  a.wait_ns = d->wait_ns;
  a.err = d->d_err;
  if (d->class_scheme == PFDTD_SRL) return launch_scheme<S, 1>(d, a, s);
  if constexpr (std::is_same<S, float>::value) {
    if (d->class_form == PFDTD_FORM_DIFFERENCE) return launch_scheme<S, 4>(d, a, s);
  }
  return launch_scheme<S, 0>(d, a, s);
}

// A resident launch holds every SM until it ends, and work of other streams
// waits behind it.  About a millisecond of it at a time is no more than they wait
// behind one update of a large batch (0.9 ms).  With 8192 steps a launch a single
// step beside a 64^3 run in another thread waited 21 ms, now 0.7 (at most 2);
// long runs take 1 % longer so at 64^3, 3 % at 128^3 (2 ms: 0.6, at most 4; 0.5 ms:
// 0.3, at most 1, but 2 % and 6 %).
constexpr double kLaunchNs = 1e6;

}  // namespace

// Whether the domain's steps can run resident; plans the bricks and allocates
// the inboxes on the domain's first call (a failed allocation or a refused
// launch leaves the per-step path in use).
bool resident_usable(pfdtd_domain* d) {
  if (d->kernel_variant != PFDTD_KERNEL_AUTO || d->tma_tile >= 0 || d->tb_depth >= 2) return false;
  if (d->K != 1 || d->Z < 3 || !d->tb_faces_ok || d->n_dif > 0) return false;
  if (d->class_scheme != PFDTD_SRL_FORWARD && d->class_scheme != PFDTD_SRL) return false;
  if (d->cls_bytes != 1 || d->n_classes > 255) return false;  // one id for nodes past the grid
  if (!d->passive || !d->src_finite) return false;  // values that are not finite: see above
  if (d->n_src > kMaxSources || d->n_rec > kMaxReceivers) return false;
  if (d->N > (int64_t)d->sm_count * (d->precision == PFDTD_F64 ? kMostDoubles : 40000)) return false;
  for (int64_t e : d->src_idx_h)
    if (e >= 0 && (e < d->XY || e >= d->N - d->XY)) return false;
  for (int64_t e : d->rec_idx_h)
    if (e >= 0 && (e < d->XY || e >= d->N - d->XY)) return false;
  ResidentState& rs = d->resident;
  if (!rs.planned) {
    rs.planned = true;
    rs.ok = false;
    Brick k{};
    double cycles = 0.0;
    const bool fits = d->precision == PFDTD_F64 ? plan_bricks<double>(d, kMaxPlanes, &k, &cycles)
                                                : plan_bricks<float>(d, kMaxPlanes, &k, &cycles);
    if (!fits) return false;
    // (0.58 ns a cycle of the estimate at 24^3 and 64^3, 0.72 at 128^3, 0.5 in FP64)
    rs.chunk = std::max<int64_t>(2, (int64_t)(kLaunchNs / (0.6 * cycles)));
    const int words = inbox_values(k) * (int)(d->arith_size() / 4);
    const size_t bytes = 2 * sizeof(uint64_t) * (size_t)words * k.gx * k.gy * k.gz;
    if (d->alloc(&rs.inbox, bytes) != cudaSuccess) {
      cudaGetLastError();
      rs.inbox = nullptr;
      return false;
    }
    if (cudaMemsetAsync(rs.inbox, 0, bytes, d->stream) != cudaSuccess) return false;
    const int v[9] = {k.bx, k.by, k.bz, k.gx, k.gy, k.gz, k.groups, k.planes, k.pitch};
    for (int i = 0; i < 9; ++i) rs.brick[i] = v[i];
    rs.words = words;
    rs.bytes = bytes;
    rs.tag = 1;
    rs.ok = true;
  }
  return rs.ok;
}

// Whether `steps` steps at a time run faster resident than one by one.  A launch
// fills the SMs and empties them again, which costs two or three single steps and
// more the more nodes there are.  Measured, us a call, resident / single steps:
// 24^3 of 1 step 51 / 45, of 3 50 / 60; 64^3 of 1 51 / 46, of 4 55 / 66; 128^3 of 1 75 /
// 55, of 8 113 / 105, of 12 131 / 134.
bool resident_pays(pfdtd_domain* d, int64_t steps) {
  return steps >= 3 + d->N / 230000 && resident_usable(d);
}

// Queue steps [step0, step0 + steps) as one launch: sources injected,
// receivers recorded, fields and their roles as after that many single steps.
// PFDTD_ERR_UNSUPPORTED with resident.ok cleared: refused, nothing queued.
int launch_resident(pfdtd_domain* d, int64_t step0, int64_t steps, void* rec_out, int64_t rec_ld,
                    int64_t inject_end, cudaStream_t s) {
  ResidentState& rs = d->resident;
  if (steps <= 0) return PFDTD_OK;
  if ((uint64_t)rs.tag + (uint64_t)steps >= 0xFFFFFFFFull) {  // tags start over
    PFDTD_CK(cudaMemsetAsync(rs.inbox, 0, rs.bytes, s));
    rs.tag = 1;
  }
  int rc = PFDTD_ERR_UNSUPPORTED;
  switch (d->precision) {
    case PFDTD_F32: rc = launch_t<float>(d, step0, steps, rec_out, rec_ld, inject_end, s); break;
    case PFDTD_F64: rc = launch_t<double>(d, step0, steps, rec_out, rec_ld, inject_end, s); break;
    case PFDTD_F16: rc = launch_t<__half>(d, step0, steps, rec_out, rec_ld, inject_end, s); break;
    case PFDTD_BF16:
      rc = launch_t<__nv_bfloat16>(d, step0, steps, rec_out, rec_ld, inject_end, s);
      break;
  }
  if (rc != PFDTD_OK) return rc;
  rs.tag += (uint32_t)steps;
  if (steps & 1) d->swap_fields();
  return PFDTD_OK;
}

}  // namespace pfdtd
