// Leapfrog pressure update kernels (SRL forward and centred, frequency-
// independent boundaries) and the per-step source/receiver kernel.
//
// Update rules follow ParallelFDTD src/kernels/kernels3d.cu:485-529
// (forward / Bilbao) and :608-665 (centred / Kowalczyk) operation for
// operation; the coefficients that depend only on the node's (position,
// material) pair are evaluated once per class on the host with the same
// expressions (classes_host.cpp), and every remaining product and sum is
// issued with an explicitly rounded intrinsic so nothing is contracted.
#include "common.cuh"

#include <algorithm>
#include <type_traits>
#include <cstring>

namespace pfdtd {

namespace {

constexpr int kBX = 32;   // threads along x (one warp = one row segment)
constexpr int kBY = 8;    // rows per block

// z-marching update.  One thread owns the column (x, y) for z in [z0, z1):
// P at z-1, z, z+1 stays in registers while the x/y neighbours at plane z are
// read through the read-only cache (they are other threads' centre values).
// Neighbour addressing is by flat offsets (+-1, +-X, +-X*Y) exactly as the
// reference indexes, so a node on an outer x or y face sees the same wrapped
// neighbour the reference kernel reads.
template <typename S, typename C, int SCHEME>
__global__ void __launch_bounds__(kBX * kBY)
k_update_zmarch(const C* __restrict__ cls, const S* __restrict__ P, S* __restrict__ Pp,
                ClassTab<typename Store<S>::A> tab, int X, int Y, int64_t XY, int z_last,
                int zc, typename Store<S>::A l2, int ks, int kshift, unsigned air) {
  using A = typename Store<S>::A;
  using R = Rn<A>;
  using St = Store<S>;
  constexpr bool kSmemTab = (sizeof(C) == 1);
  __shared__ A sa[kSmemTab ? 256 : 1], sb[kSmemTab ? 256 : 1], sc[kSmemTab ? 256 : 1];
  __shared__ uint32_t sp[kSmemTab ? 256 : 1];
  if (kSmemTab) {
    const int t = threadIdx.y * kBX + threadIdx.x;
    for (int i = t; i < tab.n; i += kBX * kBY) {
      sa[i] = tab.a[i];
      sb[i] = tab.b[i];
      sc[i] = tab.c[i];
      sp[i] = tab.pos[i];
    }
    __syncthreads();
  }
  step_wait();
  step_ready();
  // X and XY count field elements (nodes times ks fields); ks is the element
  // distance of the x neighbour.
  const int x = blockIdx.x * kBX + threadIdx.x;
  const int y = blockIdx.y * kBY + threadIdx.y;
  const int z0 = 1 + blockIdx.z * zc;
  const int z1 = min(z0 + zc, z_last);
  if (x >= X || y >= Y || z0 >= z1) return;
  int64_t idx = (int64_t)z0 * XY + (int64_t)y * X + x;
  A pm = St::load(P[idx - XY]);
  A pc = St::load(P[idx]);
  for (int z = z0; z < z1; ++z, idx += XY) {
    const A pn = St::load(P[idx + XY]);
    const A xm = St::load(P[idx - ks]);
    const A xp = St::load(P[idx + ks]);
    const A ym = St::load(P[idx - X]);
    const A yp = St::load(P[idx + X]);
    const unsigned c = cls[idx >> kshift];
    const A pp = St::load(Pp[idx]);
    A ca, cb, cc;
    uint32_t cp;
    if (kSmemTab) {
      ca = sa[c]; cb = sb[c]; cc = sc[c]; cp = sp[c];
    } else {
      ca = __ldg(tab.a + c); cb = __ldg(tab.b + c); cc = __ldg(tab.c + c); cp = __ldg(tab.pos + c);
    }
    A out;
    if constexpr (sizeof(A) == 8) {
      // FP64 operations bound this kernel: a warp in open air leaves out its
      // exact products by 1 and, centred, the zero of its boundary neighbours
      // (see k_update_tma)
      const bool plain = c == air && !(SCHEME == 1 && (not_finite(xm) || not_finite(ym) || not_finite(pn)));
      if (__all_sync(__activemask(), plain))
        out = srl_air_f64<SCHEME>(pc, pm, pn, xm, xp, ym, yp, pp, cb, l2);
      else
        out = srl_node_f64<SCHEME>(pc, pm, pn, xm, xp, ym, yp, pp, ca, cb, cc, cp, l2);
    } else if (SCHEME == 0 || SCHEME == 4) {
      // S = P[z+1] + P[z-1] + P[y+1] + P[y-1] + P[x+1] + P[x-1]  (kernels3d.cu:525)
      const A s6 = R::add(R::add(R::add(R::add(R::add(pn, pm), yp), ym), xp), xm);
      if (SCHEME == 4) {
        // difference form: a (((1+beta) p + (1-beta)(p - pp)) + l2 (S - K p)),
        // cb = K and the pos word holds the float 1 + beta
        const A e = (A)__uint_as_float(cp);
        out = R::mul(ca, R::add(R::add(R::mul(e, pc), R::mul(cc, R::sub(pc, pp))),
                                R::mul(l2, R::sub(s6, R::mul(cb, pc)))));
      } else {
        // sw/(1+beta) * ((2 - K l2) p + l2 S - (1 - beta) pp)   (kernels3d.cu:526)
        out = R::mul(ca, R::sub(R::add(R::mul(cb, pc), R::mul(l2, s6)), R::mul(cc, pp)));
      }
    } else {
      // Mirrored boundary neighbour per axis (kernels3d.cu:642-659).
      const A dx = (A)(cp & 1u), dy = (A)((cp >> 1) & 1u), dz = (A)((cp >> 2) & 1u);
      const A bx = (cp & 0x10u) ? xp : xm;
      const A by = (cp & 0x20u) ? yp : ym;
      const A bz = (cp & 0x40u) ? pm : pn;
      const A sb6 = R::add(R::add(R::mul(bx, dx), R::mul(by, dy)), R::mul(bz, dz));
      const A s7 = R::add(R::add(R::add(R::add(R::add(R::add(xm, xp), ym), yp), pn), pm), sb6);
      const A s = R::mul(s7, l2);
      // (S - (2 - 6 l2) p + (beta - 1) pp) * sw / (1 + beta)  (kernels3d.cu:663)
      out = R::mul(ca, R::add(R::sub(s, R::mul(cb, pc)), R::mul(cc, pp)));
    }
    Pp[idx] = St::store(out);
    pm = pc;
    pc = pn;
  }
}

// IWB 27-point update (no counterpart in the reference).  One thread per
// (x, y) column marching z; the 3 x 3 neighbourhood of planes z-1, z and z+1
// stays in registers and each step reads the 3 x 3 block of plane z+1 through
// the read-only cache.  Boundary closure (finite volume on the voxel grid): a
// neighbour whose bit is set in the node's closed mask (k_iwb_geometry)
// contributes the node's own value.  Sums follow the canonical order of the
// oracle (iwb_sums: in-plane sums of each plane, then combined).
template <typename S, typename C>
__global__ void __launch_bounds__(kBX * kBY)
k_update_iwb(const C* __restrict__ cls, const uint32_t* __restrict__ mask,
             const S* __restrict__ P, S* __restrict__ Pp, ClassTab<typename Store<S>::A> tab,
             int X, int Y, int64_t XY, int z_last, int zc, int ks, int kshift,
             typename Store<S>::A l2) {
  using A = typename Store<S>::A;
  using R = Rn<A>;
  using St = Store<S>;
  step_wait();
  step_ready();
  const int x = blockIdx.x * kBX + threadIdx.x;
  const int y = blockIdx.y * kBY + threadIdx.y;
  const int z0 = 1 + blockIdx.z * zc;
  const int z1 = min(z0 + zc, z_last);
  if (x >= X || y >= Y || z0 >= z1) return;
  // v[plane][dy+1][dx+1]: plane 0 = z-1, 1 = z, 2 = z+1
  A v[3][3][3];
  auto load_plane = [&](int slot, int64_t base) {
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx)
        v[slot][dy + 1][dx + 1] = St::load(__ldg(P + base + (int64_t)dy * X + dx * ks));
  };
  int64_t idx = (int64_t)z0 * XY + (int64_t)y * X + x;
  load_plane(0, idx - XY);
  load_plane(1, idx);
  for (int z = z0; z < z1; ++z, idx += XY) {
    load_plane(2, idx + XY);
    const unsigned c = cls[idx >> kshift];
    const uint32_t mk = __ldg(mask + (idx >> kshift));
    const A pp = St::load(Pp[idx]);
    const A ca = __ldg(tab.a + c), cb = __ldg(tab.b + c), cc = __ldg(tab.c + c);
    A m[3][3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int e = 0; e < 3; ++e) m[a][b][e] = v[a][b][e];
    if (mk) {
      int k = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            if (a == 1 && b == 1 && e == 1) continue;
            if ((mk >> k) & 1u) m[a][b][e] = v[1][1][1];
            ++k;
          }
    }
    A s1, s2, s3;
    iwb_sums(m, s1, s2, s3);
    const A sw = R::mul(l2, R::add(R::add(R::mul(s1, (A)0.25), R::mul(s2, (A)0.125)),
                                   R::mul(s3, (A)0.0625)));
    const A out = R::mul(ca, R::sub(R::add(sw, R::mul(cb, v[1][1][1])), R::mul(cc, pp)));
    Pp[idx] = St::store(ca == (A)0 ? (A)0 : out);  // a node outside the room holds +0
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        v[0][b][e] = v[1][b][e];
        v[1][b][e] = v[2][b][e];
      }
  }
}

// IWB geometry per node: bit k of the mask is set when the k-th of the 26
// neighbours (flat offsets dz*XY + dy*X + dx for dz, dy, dx in -1, 0, 1,
// skipping the centre) is closed: outside the grid or without the inside
// bit.  The code is 0 for a node without the inside bit, else
// 1 + W16 + 64 * face, W16 = 4 (closed faces) + 2 (closed edges) + (closed
// corners), face = 1 when a face neighbour is closed; it replaces the
// position byte in the IWB class key.
__global__ void k_iwb_geometry(const uint8_t* __restrict__ pos, int64_t N, int64_t X,
                               int64_t XY, uint32_t* __restrict__ mask,
                               uint8_t* __restrict__ code) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N;
       c += (int64_t)gridDim.x * blockDim.x) {
    uint32_t m = 0;
    int w16 = 0, face = 0, k = 0;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
      for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
          const int n = (dx != 0) + (dy != 0) + (dz != 0);
          if (n == 0) continue;
          const int64_t i = c + dz * XY + dy * X + dx;
          const bool open = i >= 0 && i < N && (pos[i] >> 7);
          if (!open) {
            m |= 1u << k;
            w16 += n == 1 ? 4 : (n == 2 ? 2 : 1);
            face |= n == 1;
          }
          ++k;
        }
    mask[c] = m;
    code[c] = (pos[c] >> 7) ? (uint8_t)(1 + w16 + 64 * face) : 0;
  }
}

// Between two updates: record receivers from the current field for the step
// just finished (kernels3d.cu:164-173), then inject this step's source
// samples into the current field in source order (kernels3d.cu:93-104).
//
// The kernel is one chain of dependent loads between two updates: 3.4 us of
// a step (step counter, index, field value, sample one after the other, each
// source by itself).  Now everything but the field is read before the update
// it follows has ended (the update starts it after the last k_step_io's end, so
// the counter stands), and after the wait one round trip to L2 is left.
template <typename S>
__global__ void k_step_io(S* cur, volatile int64_t* d_step, int n_rec,
                          const int64_t* __restrict__ rec_idx,
                          typename Store<S>::A* __restrict__ rec_out,
                          int64_t rec_ld, int n_src, const int64_t* __restrict__ src_idx,
                          const int32_t* __restrict__ src_mode,
                          const typename Store<S>::A* __restrict__ samples, int64_t n_samples,
                          int64_t inject_end, int advance, int64_t step) {
  using A = typename Store<S>::A;
  using St = Store<S>;
  const int t = threadIdx.x;
  const int64_t n = step >= 0 ? step : *d_step;  // the step index may come from the host
  const bool inject = n < inject_end && n < n_samples;
  // one warp injects, 32 sources at a time
  int64_t node = -1;
  int mode = 0;
  A sample = (A)0;
  auto fetch = [&](int k) {
    node = k < n_src ? src_idx[k] : -1;
    mode = k < n_src ? src_mode[k] : 0;
    sample = k < n_src ? samples[(int64_t)k * n_samples + n] : (A)0;
  };
  if (t < 32 && inject) fetch(t);
  const bool record = n > 0 && rec_out != nullptr && n - 1 < rec_ld;
  const int64_t mine = record && t < n_rec ? rec_idx[t] : -1;
  step_ready();
  step_wait();
  if (record) {
    if (mine >= 0) rec_out[(int64_t)t * rec_ld + (n - 1)] = St::load(cur[mine]);
    for (int r = t + blockDim.x; r < n_rec; r += blockDim.x) {
      const int64_t i = rec_idx[r];
      if (i >= 0) rec_out[(int64_t)r * rec_ld + (n - 1)] = St::load(cur[i]);
    }
  }
  __syncthreads();
  if (t < 32 && inject) {
    for (int base = 0; base < n_src; base += 32) {
      if (base > 0) fetch(base + t);
      // sources on one node: its first lane applies them all, in order
      const unsigned same = __match_any_sync(0xffffffffu, (unsigned long long)node);
      const bool first = node >= 0 && __ffs(same) - 1 == t;
      A v = first ? St::load(cur[node]) : (A)0;
      unsigned left = same;
      while (__any_sync(0xffffffffu, first && left != 0)) {
        const int j = left != 0 ? __ffs(left) - 1 : t;
        const A s = __shfl_sync(0xffffffffu, sample, j);
        const int m = __shfl_sync(0xffffffffu, mode, j);
        if (first && left != 0) v = St::load(St::store(m == 0 ? s : Rn<A>::add(v, s)));
        left &= left - 1;
      }
      if (first) cur[node] = St::store(v);
      __syncwarp();
    }
  }
  // A temporally blocked update that follows advances by its depth.
  if (t == 0) *d_step = n + advance;
}

// Receivers of the current field and the pipeline error flag into host memory
// (the flag in the first 16 bytes), for pfdtd_step.
template <typename S>
__global__ void k_step_out(const S* cur, int n_rec, const int64_t* __restrict__ rec_idx,
                           const int* err, void* host) {
  using A = typename Store<S>::A;
  step_wait();
  if (threadIdx.x == 0) *(volatile int*)host = *err;
  A* out = (A*)((char*)host + 16);
  for (int r = threadIdx.x; r < n_rec; r += blockDim.x) {
    const int64_t i = rec_idx[r];
    if (i >= 0) out[r] = Store<S>::load(cur[i]);
  }
}

// Presence of (pos, mat) keys over the updated planes z = 1..Z-2.
__global__ void k_key_presence(const uint8_t* __restrict__ pos, const uint8_t* __restrict__ mat,
                               int64_t begin, int64_t end, uint8_t* __restrict__ present) {
  for (int64_t i = begin + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < end;
       i += (int64_t)gridDim.x * blockDim.x)
    present[((unsigned)pos[i] << 8) | mat[i]] = 1;
}

template <typename C>
__global__ void k_map_classes(const uint8_t* __restrict__ pos, const uint8_t* __restrict__ mat,
                              int64_t n, const uint16_t* __restrict__ lut, C* __restrict__ cls) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    cls[i] = (C)lut[((unsigned)pos[i] << 8) | mat[i]];
}

constexpr int kResidentBlocks = 8;  // z-march blocks an SM holds (2048 threads)

// FP64 z-march updates are bound by the SMs' FP64 units, so what counts is that
// every SM gets the same work.  While all blocks are resident at once, they are
// dealt out whole: the planes of a chunk, at most `most`, are chosen for the least
// work on the busiest SM (a chunk's two more planes cost loads only, half a
// plane).  Us an update of rooms left to single steps, chunks of 8 planes / so:
// 24^3 9.8 / 3.2, 100 x 90 x 80 29.2 / 26.3, 101 x 103 x 99 36.1 / 32.1, centred 128 x 96 x
// 100 62.3 / 44.6.
//
// For the same reason such a room is launched plainly.  As a programmatic
// dependent its blocks are placed while those of the kernel before it are still
// there, two on one SM and none on another: us a step, dependent / plain, 100 x 90 x
// 80 40.3 / 29.2, centred 96^3 60.6 / 38.8, with DIF walls (whose pass the update
// follows) 64^3 17.9 / 13.9, 80^3 30.6 / 20.5.  Up to two blocks an SM (without DIF
// walls, half a block with) there is room beside them, and rooms of more blocks
// than are resident are dealt out as they go: both gain the gap, 0.7 us.
int64_t balanced_chunk(int64_t columns, int64_t nz, int64_t most, int sms) {
  int64_t best_c = most;
  double best = 1e30;
  for (int64_t c = most; c >= 1; --c) {
    const int64_t blocks = columns * ((nz + c - 1) / c), per = (blocks + sms - 1) / sms;
    if (per > kResidentBlocks) break;
    const double cost = (double)per * ((double)c + 0.5);
    if (cost < best - 1e-9) {
      best = cost;
      best_c = c;
    }
  }
  return best_c;
}

template <typename S, typename C, int SCHEME>
int launch_update_t(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  using A = typename Store<S>::A;
  const int64_t nz = d->Z - 2;
  if (nz <= 0) return PFDTD_OK;
  const int64_t XE = d->X * d->K;
  const int gx = (int)((XE + kBX - 1) / kBX);
  const int gy = (int)((d->Y + kBY - 1) / kBY);
  // Enough z-chunks for several waves of 8 resident blocks on each SM.
  const int64_t target = (int64_t)d->sm_count * 8 * 4;
  int64_t zc = std::max<int64_t>(8, (nz * (int64_t)gx * gy + target - 1) / target);
  zc = std::min<int64_t>(zc, nz);
  bool dependent = true;
  if (sizeof(A) == 8) {
    zc = balanced_chunk((int64_t)gx * gy, nz, zc, d->sm_count);
    const int64_t blocks = (int64_t)gx * gy * ((nz + zc - 1) / zc);
    const int64_t even = d->n_dif > 0 ? d->sm_count / 2 : 2 * (int64_t)d->sm_count;
    dependent = blocks <= even || blocks > kResidentBlocks * (int64_t)d->sm_count;
  }
  const int gz = (int)((nz + zc - 1) / zc);
  const size_t as = sizeof(A);
  const char* tb = (const char*)d->d_ctab;
  ClassTab<A> tab{(const A*)tb, (const A*)(tb + as * d->n_classes),
                  (const A*)(tb + 2 * as * d->n_classes),
                  (const uint32_t*)(tb + 3 * as * d->n_classes), d->n_classes};
  PFDTD_CK(launch_kernel(dependent, k_update_zmarch<S, C, SCHEME>, dim3(gx, gy, gz), dim3(kBX, kBY),
                         0, s, (const C*)d->d_cls, (const S*)cur, (S*)past, tab, (int)XE, (int)d->Y,
                         d->XY * d->K, (int)(d->Z - 1), (int)zc, (A)d->params[1], d->K, d->kshift,
                         (unsigned)d->air_class));
  count_launch();
  return PFDTD_OK;
}

template <typename S, typename C>
int launch_iwb_t(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  using A = typename Store<S>::A;
  const int64_t nz = d->Z - 2;
  if (nz <= 0) return PFDTD_OK;
  const int64_t XE = d->X * d->K;
  const int gx = (int)((XE + kBX - 1) / kBX);
  const int gy = (int)((d->Y + kBY - 1) / kBY);
  const int64_t target = (int64_t)d->sm_count * 8 * 4;
  int64_t zc = std::max<int64_t>(8, (nz * (int64_t)gx * gy + target - 1) / target);
  zc = std::min<int64_t>(zc, nz);
  const int gz = (int)((nz + zc - 1) / zc);
  const size_t as = sizeof(A);
  const char* tb = (const char*)d->d_ctab;
  ClassTab<A> tab{(const A*)tb, (const A*)(tb + as * d->n_classes),
                  (const A*)(tb + 2 * as * d->n_classes),
                  (const uint32_t*)(tb + 3 * as * d->n_classes), d->n_classes};
  // (of up to two blocks an SM, all resident at once, some would lie on one SM as
  // programmatic dependents: 81 x 80 x 79 8.8 us a step, plainly 7.5.  A DIF pass in
  // between leaves more time: 10.3 and 10.6.)
  const int64_t blocks = (int64_t)gx * gy * gz;
  const bool dependent =
      d->n_dif > 0 || 2 * blocks <= 3 * (int64_t)d->sm_count || blocks > 2 * (int64_t)d->sm_count;
  PFDTD_CK(launch_kernel(dependent, k_update_iwb<S, C>, dim3(gx, gy, gz), dim3(kBX, kBY), 0, s,
                         (const C*)d->d_cls, d->d_iwb_mask, (const S*)cur, (S*)past, tab, (int)XE,
                         (int)d->Y, d->XY * d->K, (int)(d->Z - 1), (int)zc, d->K, d->kshift,
                         (A)d->params[1]));
  count_launch();
  return PFDTD_OK;
}

template <typename S>
int launch_update_s(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  if (d->class_scheme == PFDTD_IWB)
    return d->cls_bytes == 1 ? launch_iwb_t<S, uint8_t>(d, cur, past, s)
                             : launch_iwb_t<S, uint16_t>(d, cur, past, s);
  const bool centred = (d->class_scheme == PFDTD_SRL);
  if constexpr (std::is_same<S, float>::value) {  // the difference form (FP32 fields)
    if (d->class_form == PFDTD_FORM_DIFFERENCE)
      return d->cls_bytes == 1 ? launch_update_t<S, uint8_t, 4>(d, cur, past, s)
                               : launch_update_t<S, uint16_t, 4>(d, cur, past, s);
  }
  if (d->cls_bytes == 1)
    return centred ? launch_update_t<S, uint8_t, 1>(d, cur, past, s)
                   : launch_update_t<S, uint8_t, 0>(d, cur, past, s);
  return centred ? launch_update_t<S, uint16_t, 1>(d, cur, past, s)
                 : launch_update_t<S, uint16_t, 0>(d, cur, past, s);
}

template <typename S>
int launch_io_t(pfdtd_domain* d, void* cur, void* rec_out, int64_t rec_ld, int64_t inject_end,
                cudaStream_t s, int advance, int64_t step) {
  using A = typename Store<S>::A;
  const int threads = std::max(32, std::min(1024, ((d->n_rec + 31) / 32) * 32));
  PFDTD_CK(launch_step_kernel(k_step_io<S>, dim3(1), dim3(threads), 0, s, (S*)cur, (volatile int64_t*)d->d_step,
                              d->n_rec, d->d_rec_idx, (A*)rec_out, rec_ld, d->n_src, d->d_src_idx,
                              d->d_src_mode, (const A*)d->d_src_samples, d->n_samples, inject_end,
                              advance, step));
  count_launch();
  return PFDTD_OK;
}

}  // namespace

// Host-side class coefficient evaluation (classes_host.cpp).
int eval_class_coefs(int precision, int scheme, int form, int quirks, const double* params,
                     const std::vector<double>& materials, int n_mat, int n_coef,
                     const std::vector<uint16_t>& keys, std::vector<uint8_t>& out_tab);

int launch_update(pfdtd_domain* d, const void* cur, void* past, cudaStream_t s) {
  if (iwb_flat(d)) return launch_update_flat(d, cur, past, s);
  if (uses_tma(d)) {
    if (d->class_scheme == PFDTD_IWB) return launch_iwb_tma(d, cur, past, s);
    return prefers_flat(d) ? launch_update_flat(d, cur, past, s) : launch_update_tma(d, cur, past, s);
  }
  if (d->class_scheme != PFDTD_IWB && flat_pays(d)) return launch_update_flat(d, cur, past, s);
  switch (d->precision) {
    case PFDTD_F32: return launch_update_s<float>(d, cur, past, s);
    case PFDTD_F64: return launch_update_s<double>(d, cur, past, s);
    case PFDTD_F16: return launch_update_s<__half>(d, cur, past, s);
    case PFDTD_BF16: return launch_update_s<__nv_bfloat16>(d, cur, past, s);
  }
  return fail(PFDTD_ERR_UNSUPPORTED, "unknown precision");
}

int launch_io(pfdtd_domain* d, void* cur, void* rec_out, int64_t rec_ld, int64_t inject_end,
              cudaStream_t s, int advance, int64_t step) {
  switch (d->precision) {
    case PFDTD_F32: return launch_io_t<float>(d, cur, rec_out, rec_ld, inject_end, s, advance, step);
    case PFDTD_F64: return launch_io_t<double>(d, cur, rec_out, rec_ld, inject_end, s, advance, step);
    case PFDTD_F16: return launch_io_t<__half>(d, cur, rec_out, rec_ld, inject_end, s, advance, step);
    case PFDTD_BF16:
      return launch_io_t<__nv_bfloat16>(d, cur, rec_out, rec_ld, inject_end, s, advance, step);
  }
  return fail(PFDTD_ERR_UNSUPPORTED, "unknown precision");
}

template <typename S>
static int launch_step_out_t(pfdtd_domain* d, const void* cur, cudaStream_t s) {
  PFDTD_CK(launch_step_kernel(k_step_out<S>, dim3(1), dim3(std::max(32, std::min(1024, (d->n_rec + 31) / 32 * 32))),
                              0, s, (const S*)cur, d->n_rec, d->d_rec_idx, (const int*)d->d_err, d->step_out_h));
  count_launch();
  return PFDTD_OK;
}

int launch_step_out(pfdtd_domain* d, const void* cur, cudaStream_t s) {
  switch (d->precision) {
    case PFDTD_F32: return launch_step_out_t<float>(d, cur, s);
    case PFDTD_F64: return launch_step_out_t<double>(d, cur, s);
    case PFDTD_F16: return launch_step_out_t<__half>(d, cur, s);
    case PFDTD_BF16: return launch_step_out_t<__nv_bfloat16>(d, cur, s);
  }
  return fail(PFDTD_ERR_UNSUPPORTED, "unknown precision");
}

// The class of open air: all neighbours present (forward K = 6, centred no
// boundary axis), inside, its loss factors exactly 1 (air nodes of material 0
// first); -1 if there is none.
template <typename A>
static int find_air(int scheme, const std::vector<uint16_t>& keys, const std::vector<uint8_t>& tab) {
  const unsigned pos = scheme == PFDTD_SRL ? 0x80u : 0x86u;
  const size_t n = keys.size();
  const A* a = (const A*)tab.data();
  const A c = scheme == PFDTD_SRL ? (A)-1 : (A)1;
  for (size_t i = 0; i < n; ++i)
    if ((keys[i] >> 8) == pos && a[i] == (A)1 && a[2 * n + i] == c) return (int)i;
  return -1;
}

// Whether no class of the 7-point schemes gains energy or is not finite: a =
// s/(1 + beta) and c = 1 - beta (centred beta - 1) of a beta from 0 on.
template <typename A>
static bool passive_classes(int scheme, size_t n, const std::vector<uint8_t>& tab) {
  const A* a = (const A*)tab.data();
  const A* c = a + 2 * n;
  const A sign = scheme == PFDTD_SRL ? (A)-1 : (A)1;
  for (size_t i = 0; i < n; ++i)
    if (!(a[i] >= (A)0 && a[i] <= (A)1 && sign * c[i] <= (A)1)) return false;
  return true;
}

// Whether the IWB classes outside the room and without closed neighbours (codes
// 0 and 1) have the coefficients these codes stand for; a material that is not
// finite makes others.
static bool iwb_open_classes(const std::vector<uint16_t>& keys, const std::vector<uint8_t>& tab, float* b) {
  const size_t n = keys.size();
  const float* a = (const float*)tab.data();
  *b = 0.f;
  for (size_t i = 0; i < n; ++i) {
    const unsigned code = keys[i] >> 8;
    if (code == 0 && a[i] != 0.f) return false;
    if (code != 1) continue;
    if (a[i] != 1.f || a[2 * n + i] != 1.f) return false;
    *b = a[n + i];
  }
  return true;
}

// Build the class ids and the coefficient table for the domain's current
// scheme, quirks, parameters and materials.
int build_classes(pfdtd_domain* d) {
  const int scheme = (d->scheme == PFDTD_SRL || d->scheme == PFDTD_IWB) ? d->scheme
                                                                       : PFDTD_SRL_FORWARD;
  const int form = scheme == PFDTD_SRL_FORWARD ? d->update_form : PFDTD_FORM_REFERENCE;
  if (!d->classes_dirty && d->class_scheme == scheme && d->class_form == form) return PFDTD_OK;
  if (!d->nodes_set) return fail(PFDTD_ERR_STATE, "node bytes not set");
  if (d->n_mat <= 0) return fail(PFDTD_ERR_STATE, "material table not set");
  if (form != PFDTD_FORM_REFERENCE) {
    for (int32_t f : d->dif_flags)
      if (f)
        return fail(PFDTD_ERR_UNSUPPORTED,
                    "the difference form is not built for frequency-dependent boundaries");
    if (d->precision != PFDTD_F32)
      return fail(PFDTD_ERR_UNSUPPORTED, "the difference form is built for FP32 fields");
  }
  cudaStream_t s = d->stream;
  uint8_t* d_present = nullptr;
  PFDTD_CK(cudaMallocAsync((void**)&d_present, 65536, s));
  PFDTD_CK(cudaMemsetAsync(d_present, 0, 65536, s));
  // IWB classes are keyed by the geometry code instead of the position byte.
  const uint8_t* key_bytes = d->d_pos;
  if (scheme == PFDTD_IWB) {
    if (!d->d_iwb_mask) {
      if (d->alloc((void**)&d->d_iwb_mask, (size_t)d->N * sizeof(uint32_t)) != cudaSuccess ||
          d->alloc((void**)&d->d_iwb_code, (size_t)d->N) != cudaSuccess)
        return fail(PFDTD_ERR_NOMEM, "IWB geometry allocation failed");
    }
    const int64_t gb = std::min<int64_t>((d->N + 255) / 256, kGridSMs * 32);
    k_iwb_geometry<<<(int)gb, 256, 0, s>>>(d->d_pos, d->N, d->X, d->XY, d->d_iwb_mask,
                                           d->d_iwb_code);
    count_launch();
    PFDTD_CK(cudaGetLastError());
    key_bytes = d->d_iwb_code;
  }
  const int64_t begin = d->XY, end = d->N - d->XY;
  if (end > begin) {
    const int64_t blocks = std::min<int64_t>((end - begin + 255) / 256, kGridSMs * 32);
    k_key_presence<<<(int)blocks, 256, 0, s>>>(key_bytes, d->d_mat, begin, end, d_present);
    count_launch();
    PFDTD_CK(cudaGetLastError());
  }
  std::vector<uint8_t> present(65536);
  PFDTD_CK(cudaMemcpyAsync(present.data(), d_present, 65536, cudaMemcpyDeviceToHost, s));
  PFDTD_CK(cudaStreamSynchronize(s));
  PFDTD_CK(cudaFreeAsync(d_present, s));
  std::vector<uint16_t> keys;
  std::vector<uint16_t> lut(65536, 0);
  for (int k = 0; k < 65536; ++k)
    if (present[k]) {
      lut[k] = (uint16_t)keys.size();
      keys.push_back((uint16_t)k);
    }
  if (keys.empty()) keys.push_back(0);  // grid without updated planes
  std::vector<uint8_t> tab;
  int rc = eval_class_coefs(d->precision, scheme, form, d->quirks, d->params, d->materials,
                            d->n_mat, d->n_coef, keys, tab);
  if (rc != PFDTD_OK) return rc;
  const int n_classes = (int)keys.size();
  const int cls_bytes = n_classes <= 256 ? 1 : 2;
  if (d->d_cls == nullptr || cls_bytes > d->cls_bytes) {
    d->release(d->d_cls);
    d->d_cls = nullptr;
    if (d->alloc(&d->d_cls, (size_t)d->N * cls_bytes + 64) != cudaSuccess)
      return fail(PFDTD_ERR_NOMEM, "class id allocation failed");
  }
  d->cls_bytes = cls_bytes;
  d->release(d->d_ctab);
  d->d_ctab = nullptr;
  PFDTD_CK(d->alloc(&d->d_ctab, tab.size()));
  PFDTD_CK(cudaMemcpyAsync(d->d_ctab, tab.data(), tab.size(), cudaMemcpyHostToDevice, s));
  uint16_t* d_lut = nullptr;
  PFDTD_CK(cudaMallocAsync((void**)&d_lut, 65536 * sizeof(uint16_t), s));
  PFDTD_CK(cudaMemcpyAsync(d_lut, lut.data(), 65536 * sizeof(uint16_t), cudaMemcpyHostToDevice, s));
  const int64_t blocks = std::min<int64_t>((d->N + 255) / 256, kGridSMs * 32);
  if (cls_bytes == 1)
    k_map_classes<uint8_t><<<(int)blocks, 256, 0, s>>>(key_bytes, d->d_mat, d->N, d_lut,
                                                        (uint8_t*)d->d_cls);
  else
    k_map_classes<uint16_t><<<(int)blocks, 256, 0, s>>>(key_bytes, d->d_mat, d->N, d_lut,
                                                         (uint16_t*)d->d_cls);
  count_launch();
  PFDTD_CK(cudaGetLastError());
  PFDTD_CK(cudaFreeAsync(d_lut, s));
  // The TMA kernels read the class ids through a 2-D tensor map whose row
  // stride must be a multiple of 16 bytes.  Where the field rows are 16-byte
  // aligned but the class-id rows (X ids) are not, they read a copy with each
  // row padded to 16 bytes.
  const int64_t cls_row = d->X * cls_bytes;
  if (cls_row % 16 != 0 && (d->X * d->K * (int64_t)d->esize) % 16 == 0) {
    const int64_t pitch = (cls_row + 15) / 16 * 16;
    const size_t need = (size_t)(pitch * d->Y * d->Z);
    if (!d->d_cls_tma || d->cls_tma_bytes < need) {
      d->release(d->d_cls_tma);
      d->d_cls_tma = nullptr;
      d->cls_tma_bytes = 0;
      if (d->alloc(&d->d_cls_tma, need) != cudaSuccess)
        return fail(PFDTD_ERR_NOMEM, "padded class-id allocation failed");
      d->cls_tma_bytes = need;
    }
    PFDTD_CK(cudaMemcpy2DAsync(d->d_cls_tma, (size_t)pitch, d->d_cls, (size_t)cls_row,
                               (size_t)cls_row, (size_t)(d->Y * d->Z), cudaMemcpyDeviceToDevice, s));
    d->cls_pitch = pitch / cls_bytes;
  } else {
    d->cls_pitch = 0;
  }
  PFDTD_CK(cudaStreamSynchronize(s));
  d->n_classes = n_classes;
  d->air_class = scheme == PFDTD_IWB            ? -1
                 : d->precision == PFDTD_F64 ? find_air<double>(scheme, keys, tab)
                                                : find_air<float>(scheme, keys, tab);
  d->iwb_open = scheme == PFDTD_IWB && d->precision != PFDTD_F64 &&
                iwb_open_classes(keys, tab, &d->iwb_open_b);
  // (1e-5 for a lambda rounded to float)
  d->passive = d->params[1] <= (1.0 / 3.0) * (1.0 + 1e-5) &&
               (d->precision == PFDTD_F64 ? passive_classes<double>(scheme, keys.size(), tab)
                                          : passive_classes<float>(scheme, keys.size(), tab));
  d->class_scheme = scheme;
  d->class_form = form;
  rc = build_dif(d, keys, tab);
  if (rc != PFDTD_OK) return rc;
  rc = build_iwb_closure(d, keys);
  if (rc != PFDTD_OK) return rc;
  rc = check_tb_faces(d);
  if (rc != PFDTD_OK) return rc;
  d->classes_dirty = false;
  d->class_version++;
  return PFDTD_OK;
}

}  // namespace pfdtd
