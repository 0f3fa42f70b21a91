// Burst stitching of burst interferograms into a frame (the reference's
// s1proc/interfere.py:81-180, NumPy on memmaps there).
//
// Per subswath, bursts in order of top + bottom as Subswath.sort
// (s1proc/sario.py:239-244) inside the union box of the first and last burst
// (sario.py:230-237): each burst after the first, when its pair of burst ids
// differs from the previous one, estimates the phase offset over its overlap
// with what the earlier bursts left there:
//   m = angle(mean(conj(old) new)),  m += median(angle(conj(old) new e^{-i m}))
// (float mode: differences of phases instead of products), and is written
// rotated by -m where that is still empty (real part 0).  The offset carries
// over to later bursts without an overlap, as in the reference.  Then the
// frame: subswaths 1..3 written in order where non-zero.
//
// No subswath mosaic is kept: what the earlier bursts left at a pixel is the
// first of them, in order, that is not empty there, rotated by its own offset
// (Rotated, fold_pixel), so both the overlaps and the frame are read straight
// from the bursts.  Every burst's overlap is measured at once against the
// unrotated earlier bursts; where its pixels all belong to one of them, which
// consecutive bursts' do, the chain of offsets is then a few additions, and
// only a burst over pixels of several is measured again, in order.  The mean
// is summed in FP64 in a fixed order; the median is exact, selected over the
// float angles (np.median: for an even count the mean of the middle two).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "s1b.h"
#include "s1b_device.cuh"
#include "s1b_internal.h"

namespace {

constexpr int ST_THREADS = 1024;

struct Swath {
  int32_t first, count;              // bursts [first, first + count) of the sorted table
  int32_t left, top, right, bottom;  // union box
};

struct Bst {
  int64_t off;
  int32_t left, top, right, bottom, group;  // the box clipped to the subswath's; off: its first pixel
  int32_t width;                            // pixels from row to row
  int32_t over_top, over_bottom;            // rows that earlier bursts reach
  int32_t measured;                         // 1: it takes an offset of its own from them
};

// A burst's offset and what rotates by it (written by the chain, read by the frame).
struct Turn {
  double phase;
  float c, s;
};

__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float keyf(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

template <bool kFloat>
struct Px;

template <>
struct Px<false> {
  using T = float2;
  __device__ static bool empty(T v) { return v.x == 0.f; }  // .real == 0, as the reference masks
  __device__ static bool nonzero(T v) { return v.x != 0.f || v.y != 0.f; }
};

template <>
struct Px<true> {
  using T = float;
  __device__ static bool empty(T v) { return v == 0.f; }
  __device__ static bool nonzero(T v) { return v != 0.f; }
};

// conj(old) new (complex) or exp(i (new - old)) (phase) of an overlap pixel.
__device__ __forceinline__ float2 pdiff(float2 o, float2 n) {
  return make_float2(o.x * n.x + o.y * n.y, o.x * n.y - o.y * n.x);
}
__device__ __forceinline__ float2 pdiff(float o, float n) {
  float s, c;
  sincosf(n - o, &s, &c);
  return make_float2(c, s);
}

// A cluster barrier: every thread of every CTA of the cluster arrives, and
// what they wrote before it (shared memory of the cluster, global memory) is
// visible to all of them after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Address of `p`, a variable in this CTA's shared memory, in CTA `rank`'s.
__device__ __forceinline__ uint32_t peer_smem(const void *p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void peer_store(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void peer_store(uint32_t a, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t peer_load(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void peer_add(uint32_t a, unsigned v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

constexpr int ST_CLUSTER = 16;      // most CTAs per burst (fewer where a device cannot place 16)
constexpr int ST_KEEP = 22 * 1024;  // overlap pixels a CTA keeps in shared memory
constexpr int ST_BINS = 2048;       // bins of the circle that the median is first sought in
constexpr int ST_CAND = 2048;       // angles of the median's bin that are gathered
constexpr int ST_TABLE = 64;        // bursts a launch takes by value
constexpr int ST_NEAR = 32;         // bursts under one burst, or in one block of the frame, that are listed

// The burst table: by value up to ST_TABLE bursts, else in the workspace.
struct Table {
  Swath swaths[3];
  int32_t n_swaths;
  Bst bursts[ST_TABLE];
  const Bst *more;
  __device__ __forceinline__ const Bst &burst(int i) const { return more ? more[i] : bursts[i]; }
};

// A burst as it lies in its subswath: its pixels rotated by -phase.
template <bool kFloat>
struct Rotated {
  const typename Px<kFloat>::T *src;  // its first pixel
  int left, top, right, bottom, width;
  float c, s;
  double phase;
  __device__ __forceinline__ void set(const Bst &b, const void *data, const Turn &t) {
    src = reinterpret_cast<const typename Px<kFloat>::T *>(data) + b.off;
    left = b.left;
    top = b.top;
    right = b.right;
    bottom = b.bottom;
    width = b.width;
    c = t.c;
    s = t.s;
    phase = t.phase;
  }
  __device__ __forceinline__ bool covers(int x, int y) const {
    return x >= left && x < right && y >= top && y < bottom;
  }
  __device__ __forceinline__ typename Px<kFloat>::T raw(int x, int y) const {
    return __ldg(src + (int64_t)(y - top) * width + (x - left));
  }
  __device__ __forceinline__ typename Px<kFloat>::T turned(typename Px<kFloat>::T v) const {
    if (phase == 0.0) return v;
    if constexpr (kFloat) {
      double w = (double)v - phase;
      if (w > kPiD) w -= 2 * kPiD;
      if (w < -kPiD) w += 2 * kPiD;
      return (float)w;
    } else {
      return make_float2(v.x * c + v.y * s, v.y * c - v.x * s);
    }
  }
};

// One more burst in order at a pixel: it shows where the earlier ones are empty.
template <bool kFloat>
__device__ __forceinline__ void fold_pixel(typename Px<kFloat>::T &cur, const Rotated<kFloat> &b, int x, int y) {
  if (!Px<kFloat>::empty(cur) || !b.covers(x, y)) return;
  const typename Px<kFloat>::T v = b.raw(x, y);
  if (!Px<kFloat>::empty(v)) cur = b.turned(v);
}

// A burst's overlap: pixels, the angle of the mean product, the median about
// it, and the burst of the subswath the old pixels belong to (-1: several).
struct Measured {
  double mean, median;
  uint32_t n;
  int32_t owner;
};

template <bool kFloat>
struct __align__(16) StSmem {
  double part[2][ST_CLUSTER][3];  // sums of every CTA of the cluster, alternating between bursts
  uint32_t owners[2][ST_CLUSTER][2];
  double red[3][ST_THREADS / 32];
  unsigned red_o[2][ST_THREADS / 32];
  unsigned hist[ST_BINS];         // this CTA's counts
  unsigned total[ST_BINS];        // the cluster's
  unsigned total8[3][256];        // the cluster's counts of a digit, in turn
  uint32_t cand[ST_CAND], sel[ST_CAND];  // keys of the median's bin: this CTA's, the cluster's
  unsigned n_cand, n_sel, sel_lo, sel_hi;
  unsigned digit, below, here, least;
  unsigned scan[ST_THREADS / 32];
  unsigned count, own_lo, own_hi;  // overlap pixels of the cluster; smallest and largest owner
  float cm, sm;                    // cosine and sine of the mean
  int mean_ok;
  Measured out;
  int n_near;                      // earlier bursts under this one (-1: more than ST_NEAR)
  Rotated<kFloat> near[ST_NEAR];
  int near_index[ST_NEAR];
};

// Which of `v` counts per lane position (8 consecutive per lane, one warp)
// holds rank rk: writes its index, the counts below it and its own count.
__device__ __forceinline__ void warp_find(const unsigned *counts, int per, int lane, unsigned rk, unsigned base,
                                          unsigned &index, unsigned &below, unsigned &here) {
  unsigned s = 0;
  for (int k = 0; k < per; ++k) s += counts[lane * per + k];
  unsigned inc = s;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned w = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += w;
  }
  unsigned cum = base + inc - s;
  for (int k = 0; k < per; ++k) {
    const unsigned v = counts[lane * per + k];
    if (cum <= rk && rk < cum + v) {
      index = lane * per + k;
      below = cum;
      here = v;
    }
    cum += v;
  }
}

// Bin of an angle's key on the circle: monotone in the key (the largest keys
// are no numbers and go to the last bin).
__device__ __forceinline__ unsigned angle_bin(uint32_t key) {
  const float a = keyf(key);
  return a == a ? min((unsigned)((a + 3.14159274f) * (float)(ST_BINS / 6.283185307179586)), (unsigned)ST_BINS - 1)
                : ST_BINS - 1;
}

// The offset of burst q of a subswath against the earlier ones, measured by
// one cluster.  turns: the earlier bursts' (null: unrotated).  An overlap is
// small (160 rows of 470 pixels for a frame's bursts at 4 x 20 looks), so what
// counts is the latency of a pass: products and then keys of the angles stay
// in shared memory, and the passes of the selection are separated by hardware
// cluster barriers.  The keys are counted in bins of the circle; the counts
// that are not zero are added into every CTA of the cluster; the keys of the
// median's bin are gathered in each CTA and ranked there, or, when one bin
// holds more than ST_CAND of them (equal angles), found digit by digit over
// the cluster.  The result is in sm.out of every CTA; the whole cluster calls.
template <bool kFloat, typename Idx>
__device__ __forceinline__ void measure(StSmem<kFloat> &sm, float2 *s_kept, const Table &tab, const Swath &sw,
                                        int q, int ot, int ob, const void *data, const Turn *turns, int keep,
                                        int &nsum, int &ndig) {
  using T = typename Px<kFloat>::T;
  const uint32_t rank = cluster_rank(), ncta = cluster_size();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Idx first = rank * ST_THREADS + tid, stride = ncta * ST_THREADS;
  const Bst b = tab.burst(sw.first + q);
  const Turn still{0.0, 1.f, 0.f};
  // the earlier bursts that reach into the overlap, in order
  if (warp == 0) {
    int n = 0;
    for (int p0 = 0; p0 < q && n >= 0; p0 += 32) {
      const int p = p0 + lane;
      bool hit = false;
      if (p < q) {
        const Bst &e = tab.burst(sw.first + p);
        hit = e.left < b.right && e.right > b.left && e.top < ob && e.bottom > ot;
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      const int at = n + __popc(m & ((1u << lane) - 1u));
      n += __popc(m);
      if (n > ST_NEAR) {
        n = -1;
      } else if (hit) {
        sm.near[at].set(tab.burst(sw.first + p), data, turns ? turns[sw.first + p] : still);
        sm.near_index[at] = p;
      }
    }
    if (lane == 0) {
      sm.n_near = n;
      sm.n_cand = sm.n_sel = sm.sel_hi = 0;
      sm.sel_lo = 0xffffffffu;
    }
  }
  __syncthreads();
  const int n_near = sm.n_near;
  const Idx ow = b.right - b.left, on = (Idx)(ob - ot) * ow;
  const Idx step_y = stride / ow, step_x = stride - step_y * ow, y0 = first / ow, x0 = first - y0 * ow;
  const T *src = reinterpret_cast<const T *>(data) + b.off + (int64_t)(ot - b.top) * b.width;
  // what the earlier bursts left at overlap pixel (x, y), and whose it is
  auto old_at = [&](Idx x, Idx y, int &owner) -> T {
    T o{};
    if (n_near >= 0) {
      for (int k = 0; k < n_near && Px<kFloat>::empty(o); ++k) {
        fold_pixel<kFloat>(o, sm.near[k], b.left + (int)x, ot + (int)y);
        owner = sm.near_index[k];
      }
    } else {
      for (int p = 0; p < q && Px<kFloat>::empty(o); ++p) {
        Rotated<kFloat> e;
        e.set(tab.burst(sw.first + p), data, turns ? turns[sw.first + p] : still);
        fold_pixel<kFloat>(o, e, b.left + (int)x, ot + (int)y);
        owner = p;
      }
    }
    return o;
  };
  // the CTA's overlap pixels (x, y), j their place in s_kept
  auto each = [&](auto &&f) {
    Idx x = x0, y = y0;
#pragma unroll 4
    for (Idx i = first, j = tid; i < on; i += stride, j += ST_THREADS) {
      f(x, y, j);
      x += step_x;
      y += step_y;
      if (x >= ow) {
        x -= ow;
        ++y;
      }
    }
  };
  const bool kept = (Idx)keep * ncta >= on;  // uniform over the cluster
  double sx = 0.0, sy = 0.0;
  unsigned sn = 0, own_lo = 0xffffffffu, own_hi = 0;
  auto product = [&](T o, T n, int owner, Idx j) {
    float2 d = make_float2(__uint_as_float(0xffffffffu), 0.f);  // no result of arithmetic has these bits
    if (!Px<kFloat>::empty(o) && Px<kFloat>::nonzero(n)) {
      d = pdiff(o, n);
      sx += d.x;
      sy += d.y;
      ++sn;
      own_lo = min(own_lo, (unsigned)owner);
      own_hi = max(own_hi, (unsigned)owner);
    }
    if (kept) s_kept[j] = d;
  };
  if (n_near == 1) {  // the usual overlap: the loads of four pixels in flight together
    const Rotated<kFloat> e = sm.near[0];
    const int owner = sm.near_index[0];
    Idx x = x0, y = y0;
    for (Idx i = first, j = tid; i < on; i += 4 * stride, j += 4 * ST_THREADS) {
      T o[4], n[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = i + k * stride < on;
        const int gx = b.left + (int)x, gy = ot + (int)y;
        o[k] = n[k] = T{};
        if (in && e.covers(gx, gy)) o[k] = e.raw(gx, gy);
        if (in) n[k] = __ldg(src + (int64_t)y * b.width + x);
        x += step_x;
        y += step_y;
        if (x >= ow) {
          x -= ow;
          ++y;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k * stride < on)
          product(Px<kFloat>::empty(o[k]) ? T{} : e.turned(o[k]), n[k], owner, j + k * ST_THREADS);
    }
  } else {
    each([&](Idx x, Idx y, Idx j) {
      const T n = __ldg(src + (int64_t)y * b.width + x);
      int owner = 0;
      const T o = old_at(x, y, owner);
      product(o, n, owner, j);
    });
  }
  // fixed-order reduction: warps by shuffles, warp sums, then CTA sums
  double sc = sn;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    sx += __shfl_down_sync(0xffffffffu, sx, off);
    sy += __shfl_down_sync(0xffffffffu, sy, off);
    sc += __shfl_down_sync(0xffffffffu, sc, off);
  }
  own_lo = __reduce_min_sync(0xffffffffu, own_lo);
  own_hi = __reduce_max_sync(0xffffffffu, own_hi);
  if (lane == 0) {
    sm.red[0][warp] = sx;
    sm.red[1][warp] = sy;
    sm.red[2][warp] = sc;
    sm.red_o[0][warp] = own_lo;
    sm.red_o[1][warp] = own_hi;
  }
  __syncthreads();
  const int half = nsum++ & 1;
  double(*part)[3] = sm.part[half];
  uint32_t(*owners)[2] = sm.owners[half];
  if (warp < 3) {
    double v = sm.red[warp][lane];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane < ncta) peer_store(peer_smem(&part[rank][warp], lane), v);
  } else if (warp < 5) {
    const unsigned w = sm.red_o[warp - 3][lane];
    const unsigned v = warp == 3 ? __reduce_min_sync(0xffffffffu, w) : __reduce_max_sync(0xffffffffu, w);
    if (lane < ncta) peer_store(peer_smem(&owners[rank][warp - 3], lane), v);
  }
  cluster_sync();
  double ax = 0.0, ay = 0.0, an = 0.0;  // warp 0: the overlap's sums
  if (warp == 0) {
    // one warp takes the FP64 functions (in every warp they would keep the
    // SM's FP64 unit busy for microseconds); the cosine and sine of the mean
    // come from the sums, its angle is needed only at the end
    own_lo = 0xffffffffu;
    own_hi = 0;
    if (lane < ncta) {
      ax = part[lane][0];
      ay = part[lane][1];
      an = part[lane][2];
      own_lo = owners[lane][0];
      own_hi = owners[lane][1];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, off);
      ay += __shfl_xor_sync(0xffffffffu, ay, off);
      an += __shfl_xor_sync(0xffffffffu, an, off);
    }
    own_lo = __reduce_min_sync(0xffffffffu, own_lo);
    own_hi = __reduce_max_sync(0xffffffffu, own_hi);
    const double len = sqrt(ax * ax + ay * ay);
    double c = 1.0, s = 0.0;
    if (len > 0.0 && len < INFINITY) {
      c = ax / len;
      s = ay / len;
    } else if (!(len == 0.0)) {  // infinite products among them, or no number
      sincos(atan2(ay, ax), &s, &c);
    }
    if (lane == 0) {
      sm.count = (unsigned)an;
      sm.cm = (float)c;
      sm.sm = (float)s;
      sm.mean_ok = !isnan(c);
      // no overlap, or a mean that is no number, as the median about it is then
      sm.out = Measured{c, 0.0, (unsigned)an, own_lo == own_hi ? (int32_t)own_lo : -1};
    }
  }
  __syncthreads();
  const unsigned n = sm.count;
  if (n == 0 || !sm.mean_ok) return;  // uniform over the cluster
  const float cm = sm.cm, smn = sm.sm;
  // key of an overlap pixel's angle about the mean; no pixel: all ones
  auto key_of = [&](float2 d) -> uint32_t {
    return min(fkey(atan2f(d.y * cm - d.x * smn, d.x * cm + d.y * smn)), 0xfffffffeu);
  };
  auto key_at = [&](Idx x, Idx y, Idx j) -> uint32_t {
    if (kept) return __float_as_uint(s_kept[j].x);
    int owner = 0;
    const T o = old_at(x, y, owner), v = __ldg(src + (int64_t)y * b.width + x);
    return !Px<kFloat>::empty(o) && Px<kFloat>::nonzero(v) ? key_of(pdiff(o, v)) : 0xffffffffu;
  };
  each([&](Idx x, Idx y, Idx j) {
    uint32_t k = 0xffffffffu;
    if (kept) {
      const float2 d = s_kept[j];
      if (__float_as_uint(d.x) != 0xffffffffu) {
        k = key_of(d);
        s_kept[j].x = __uint_as_float(k);
      }
    } else {
      k = key_at(x, y, j);
    }
    if (k != 0xffffffffu) atomicAdd(&sm.hist[angle_bin(k)], 1u);
  });
  __syncthreads();
  for (int i = tid; i < ST_BINS; i += ST_THREADS) {
    const unsigned c = sm.hist[i];
    if (c) {
      sm.hist[i] = 0;
      for (uint32_t k = 0; k < ncta; ++k) peer_add(peer_smem(&sm.total[i], k), c);
    }
  }
  cluster_sync();
  unsigned rk = (n - 1) / 2;
  {
    constexpr int PER = ST_BINS / ST_THREADS;
    unsigned s = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) s += sm.total[tid * PER + k];
    const unsigned w = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) sm.scan[warp] = w;
    __syncthreads();
    unsigned base = warp > lane ? sm.scan[lane] : 0;
    base = __reduce_add_sync(0xffffffffu, base);
    if (base <= rk && rk < base + w) warp_find(sm.total + warp * 32 * PER, PER, lane, rk, base, sm.digit, sm.below, sm.here);
    if (base <= rk && rk < base + w && lane == 0) sm.least = warp * 32 * PER;
    __syncthreads();
    for (int i = tid; i < ST_BINS; i += ST_THREADS) sm.total[i] = 0;  // added to again after the next barrier
  }
  const unsigned bin = sm.least + sm.digit;
  unsigned here = sm.here;
  rk -= sm.below;
  __syncthreads();
  uint32_t lower, upper;
  bool next = n % 2 == 0 && rk + 1 >= here;  // the upper middle value lies above the bin
  if (here <= ST_CAND) {
    each([&](Idx x, Idx y, Idx j) {
      const uint32_t k = key_at(x, y, j);
      if (k != 0xffffffffu && angle_bin(k) == bin) sm.cand[atomicAdd(&sm.n_cand, 1u)] = k;
    });
    cluster_sync();
    if (warp < ncta) {  // warp w takes CTA w's
      const unsigned m = peer_load(peer_smem(&sm.n_cand, warp));
      unsigned at = lane == 0 ? atomicAdd(&sm.n_sel, m) : 0;
      at = __shfl_sync(0xffffffffu, at, 0);
      unsigned lo = 0xffffffffu, hi = 0;
      for (unsigned i = lane; i < m; i += 32) {
        const uint32_t k = peer_load(peer_smem(&sm.cand[i], warp));
        sm.sel[at + i] = k;
        lo = min(lo, k);
        hi = max(hi, k);
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lane == 0 && m) {
        atomicMin(&sm.sel_lo, lo);
        atomicMax(&sm.sel_hi, hi);
      }
    }
    __syncthreads();
    // ranked in each CTA by 8-bit digits below the bits all of them share
    auto rank_key = [&](unsigned r) -> uint32_t {
      const uint32_t lo = sm.sel_lo, hi = sm.sel_hi;
      int bits = lo == hi ? 0 : 32 - __clz(lo ^ hi);
      uint32_t mask = bits >= 32 ? 0u : ~0u << bits, prefix = lo & mask;
      while (bits > 0) {
        const int shift = max(0, bits - 8);
        const unsigned dm = (1u << (bits - shift)) - 1u;
        for (unsigned i = tid; i < here; i += ST_THREADS) {
          const uint32_t k = sm.sel[i];
          if ((k & mask) == prefix) atomicAdd(&sm.hist[(k >> shift) & dm], 1u);
        }
        __syncthreads();
        if (warp == 0) warp_find(sm.hist, 8, lane, r, 0, sm.digit, sm.below, sm.least);
        __syncthreads();
        if (tid < 256) sm.hist[tid] = 0;
        prefix |= sm.digit << shift;
        mask |= dm << shift;
        r -= sm.below;
        bits = shift;
        __syncthreads();
      }
      return prefix;
    };
    lower = rank_key(rk);
    upper = n % 2 == 0 && !next ? rank_key(rk + 1) : lower;
  } else {
    // by 8-bit digits over the cluster
    unsigned prefix = 0, mask = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
      unsigned *total = sm.total8[ndig % 3], *spare = sm.total8[(ndig + 2) % 3];
      ++ndig;
      each([&](Idx x, Idx y, Idx j) {
        const uint32_t k = key_at(x, y, j);
        if (k != 0xffffffffu && (k & mask) == prefix && angle_bin(k) == bin) {
          const unsigned dig = (k >> shift) & 255u, same = __match_any_sync(__activemask(), dig);
          if (lane == __ffs(same) - 1) atomicAdd(&sm.hist[dig], (unsigned)__popc(same));
        }
      });
      __syncthreads();
      if (tid < 256) {
        const unsigned c = sm.hist[tid];
        if (c) {
          sm.hist[tid] = 0;
          for (uint32_t k = 0; k < ncta; ++k) peer_add(peer_smem(&total[tid], k), c);
        }
      }
      cluster_sync();
      // the counts read a digit ago are cleared for the digit after the next
      if (tid < 256) spare[tid] = 0;
      if (warp == 0) warp_find(total, 8, lane, rk, 0, sm.digit, sm.below, sm.here);
      __syncthreads();
      prefix |= sm.digit << shift;
      mask |= 255u << shift;
      rk -= sm.below;
      here = sm.here;  // keys equal to the prefix so far
      __syncthreads();
    }
    lower = upper = prefix;
    next = n % 2 == 0 && rk + 1 >= here;
  }
  if (next) {  // the smallest key above: of the cluster
    unsigned least = 0xffffffffu;
    each([&](Idx x, Idx y, Idx j) {
      const uint32_t k = key_at(x, y, j);
      if (k > lower) least = min(least, k);
    });
    least = __reduce_min_sync(0xffffffffu, least);
    if (tid == 0) sm.least = 0xffffffffu;
    __syncthreads();
    if (lane == 0) atomicMin(&sm.least, least);
    cluster_sync();
    if (warp == 0) {
      upper = lane < ncta ? peer_load(peer_smem(&sm.least, lane)) : 0xffffffffu;
      upper = __reduce_min_sync(0xffffffffu, upper);
    }
  }
  if (warp == 0) {
    const double lo = keyf(lower), hi = keyf(upper);
    const double mean = atan2(ay, ax);
    if (lane == 0) {
      sm.out.mean = mean;
      sm.out.median = n % 2 ? lo : 0.5 * (lo + hi);
    }
  }
  cluster_sync();  // the cluster has read this CTA's shared memory
}

// Every burst's overlap against the unrotated earlier bursts: one cluster per
// burst of the table.  27 bursts of 430 x 470 pixels in 3
// subswaths, 24 overlaps of 77 k pixels: 37 us here, 6 us for the chain, 31 us
// for the frame (75 us a call, its host work included); one CTA per subswath,
// which walked the bursts in order over a mosaic and formed the overlap's
// angles again for every digit of both middle ranks, took 5.08 ms.  What
// bounds it is instruction issue of the passes over the overlap (the angle
// is about 100 instructions a pixel) on 96 SMs.
template <bool kFloat, typename Idx>
__global__ __launch_bounds__(ST_THREADS, 1) void stitch_measure_kernel(const __grid_constant__ Table tab,
                                                                       const void *__restrict__ data,
                                                                       Measured *__restrict__ out, int keep) {
  extern __shared__ __align__(16) unsigned char st_raw[];
  StSmem<kFloat> &sm = *reinterpret_cast<StSmem<kFloat> *>(st_raw);
  float2 *s_kept = reinterpret_cast<float2 *>(st_raw + sizeof(StSmem<kFloat>));  // keep entries
  const int i = blockIdx.x / cluster_size(), tid = threadIdx.x;
  const Bst b = tab.burst(i);
  int s = 0;
  while (i >= tab.swaths[s].first + tab.swaths[s].count) ++s;
  const Swath sw = tab.swaths[s];
  if (!b.measured) {  // uniform over the cluster
    if (cluster_rank() == 0 && tid == 0) out[i] = Measured{0.0, 0.0, 0u, -1};
    return;
  }
  for (int k = tid; k < ST_BINS; k += ST_THREADS) sm.hist[k] = sm.total[k] = 0;
  for (int k = tid; k < 256; k += ST_THREADS) sm.total8[0][k] = sm.total8[1][k] = sm.total8[2][k] = 0;
  cluster_sync();  // every CTA of the cluster runs before its shared memory is written
  int nsum = 0, ndig = 0;
  measure<kFloat, Idx>(sm, s_kept, tab, sw, i - sw.first, b.over_top, b.over_bottom, data, nullptr, keep, nsum, ndig);
  __syncthreads();
  if (cluster_rank() == 0 && tid == 0) out[i] = sm.out;
  cluster_sync();  // no CTA leaves while another may still reach its shared memory
}

// The chain of offsets of one subswath (one cluster): an overlap
// that belongs to one earlier burst was measured against it as it lies, and
// that burst's own rotation adds to the mean; any other is measured here, in
// order, against the rotated bursts.
template <bool kFloat, typename Idx>
__global__ __launch_bounds__(ST_THREADS, 1) void stitch_chain_kernel(const __grid_constant__ Table tab,
                                                                     const void *__restrict__ data,
                                                                     const Measured *__restrict__ measured,
                                                                     Turn *turns, int keep) {
  extern __shared__ __align__(16) unsigned char st_raw[];
  StSmem<kFloat> &sm = *reinterpret_cast<StSmem<kFloat> *>(st_raw);
  float2 *s_kept = reinterpret_cast<float2 *>(st_raw + sizeof(StSmem<kFloat>));  // keep entries
  const Swath sw = tab.swaths[blockIdx.x / cluster_size()];
  const int tid = threadIdx.x;
  __shared__ int s_serial;
  __shared__ double s_phase;
  // without a burst over several others the chain is one thread's
  if (tid == 0) s_serial = 0;
  __syncthreads();
  for (int q = tid; q < sw.count; q += ST_THREADS) {
    const Measured m = measured[sw.first + q];
    if (m.n > 0 && m.owner < 0) s_serial = 1;
  }
  __syncthreads();
  auto phase_of = [&](const Measured &m, double carried) -> double {
    if (m.n == 0) return carried;
    const double owner = turns[sw.first + m.owner].phase, mean = owner + m.mean;
    // the mean's angle in [-pi, pi], as atan2 would give it
    return mean - 2 * kPiD * rint(mean / (2 * kPiD)) + m.median;
  };
  if (!s_serial) {  // uniform over the cluster: every CTA read the same table
    if (cluster_rank() == 0) {
      if (tid == 0) {
        double phase = 0.0;
        for (int q = 0; q < sw.count; ++q) {
          phase = phase_of(measured[sw.first + q], phase);
          turns[sw.first + q].phase = phase;
        }
      }
      __syncthreads();
      for (int q = tid; q < sw.count; q += ST_THREADS) {
        double sn, cs;
        sincos(turns[sw.first + q].phase, &sn, &cs);
        turns[sw.first + q].c = (float)cs;
        turns[sw.first + q].s = (float)sn;
      }
    }
    return;
  }
  for (int k = tid; k < ST_BINS; k += ST_THREADS) sm.hist[k] = sm.total[k] = 0;
  for (int k = tid; k < 256; k += ST_THREADS) sm.total8[0][k] = sm.total8[1][k] = sm.total8[2][k] = 0;
  cluster_sync();  // every CTA of the cluster runs before its shared memory is written
  double phase = 0.0;
  int nsum = 0, ndig = 0;
  for (int q = 0; q < sw.count; ++q) {
    const Measured m = measured[sw.first + q];
    if (m.n > 0 && m.owner < 0) {
      const Bst b = tab.burst(sw.first + q);
      measure<kFloat, Idx>(sm, s_kept, tab, sw, q, b.over_top, b.over_bottom, data, turns, keep, nsum, ndig);
      __syncthreads();
      if (sm.out.n > 0) phase = sm.out.mean + sm.out.median;
      __syncthreads();
    } else {
      if (tid == 0) s_phase = phase_of(m, phase);
      __syncthreads();
      phase = s_phase;
    }
    if (tid == 0) {  // every CTA writes the same entry, so each reads back what it wrote itself
      double sn, cs;
      sincos(phase, &sn, &cs);
      turns[sw.first + q] = Turn{phase, (float)cs, (float)sn};
    }
    __syncthreads();
  }
  cluster_sync();  // no CTA leaves while another may still reach its shared memory
}

// The frame: a block is 256 columns x ST_FROWS rows; the bursts that reach
// into it are listed once, so a pixel tests one or two instead of all.
constexpr int ST_FROWS = 16;

template <bool kFloat>
__global__ __launch_bounds__(256) void stitch_frame_kernel(const __grid_constant__ Table tab,
                                                           const void *__restrict__ data,
                                                           const Turn *__restrict__ turns,
                                                           typename Px<kFloat>::T *__restrict__ frame, int nrow0,
                                                           int ncol0) {
  using T = typename Px<kFloat>::T;
  __shared__ Rotated<kFloat> s_b[ST_NEAR];
  __shared__ int s_end[3];  // listed bursts of subswaths 0 .. s; -1: not listed
  const int xb = blockIdx.x * 256, yb = blockIdx.y * ST_FROWS, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    int n = 0;
    for (int s = 0; s < tab.n_swaths; ++s) {
      const Swath &sw = tab.swaths[s];
      for (int p0 = 0; p0 < sw.count; p0 += 32) {
        const int p = p0 + lane;
        bool hit = false;
        if (p < sw.count) {
          const Bst &e = tab.burst(sw.first + p);
          hit = e.left < xb + 256 && e.right > xb && e.top < yb + ST_FROWS && e.bottom > yb;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        const int at = n + __popc(m & ((1u << lane) - 1u));
        if (n >= 0) n = n + __popc(m) > ST_NEAR ? -1 : n + __popc(m);
        if (n >= 0 && hit) s_b[at].set(tab.burst(sw.first + p), data, turns[sw.first + p]);
      }
      if (lane == 0) s_end[s] = n;
    }
  }
  __syncthreads();
  const int x = xb + threadIdx.x, rows = min(ST_FROWS, nrow0 - yb);
  if (x >= ncol0) return;
  const int listed = s_end[tab.n_swaths - 1];
  T *dst = frame + (int64_t)yb * ncol0 + x;
  // written where real (or value) != 0, the last subswath on top
  if (listed >= 0 && listed <= 4) {  // nearly every block: the loads of four rows in flight together
    int swath_of[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) swath_of[k] = k < s_end[0] ? 0 : (tab.n_swaths > 1 && k < s_end[1] ? 1 : 2);
    for (int r0 = 0; r0 < rows; r0 += 4) {
      T c[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          c[r][k] = T{};
          if (k < listed && r0 + r < rows && s_b[k].covers(x, yb + r0 + r)) c[r][k] = s_b[k].raw(x, yb + r0 + r);
        }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r0 + r >= rows) break;
        T v{}, m{};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k >= listed) break;
          if (k > 0 && swath_of[k] != swath_of[k - 1]) {
            if (!Px<kFloat>::empty(m)) v = m;
            m = T{};
          }
          if (Px<kFloat>::empty(m) && !Px<kFloat>::empty(c[r][k])) m = s_b[k].turned(c[r][k]);
        }
        if (!Px<kFloat>::empty(m)) v = m;
        __stcs(dst + (int64_t)(r0 + r) * ncol0, v);
      }
    }
    return;
  }
  for (int r = 0; r < rows; ++r, dst += ncol0) {
    T v{};
    for (int s = tab.n_swaths - 1; s >= 0 && Px<kFloat>::empty(v); --s) {
      T m{};
      if (listed >= 0) {
        for (int k = s ? s_end[s - 1] : 0; k < s_end[s]; ++k) fold_pixel<kFloat>(m, s_b[k], x, yb + r);
      } else {
        const Swath &sw = tab.swaths[s];
        for (int p = 0; p < sw.count; ++p) {
          Rotated<kFloat> e;
          e.set(tab.burst(sw.first + p), data, turns[sw.first + p]);
          fold_pixel<kFloat>(m, e, x, yb + r);
        }
      }
      if (!Px<kFloat>::empty(m)) v = m;
    }
    __stcs(dst, v);
  }
}

struct Plan {
  std::vector<Bst> bursts;
  std::vector<int32_t> index;  // the caller's index of each burst
  std::vector<Swath> swaths;
  int64_t overlap = 0;         // pixels of the largest overlap
  int measured = 0;            // bursts that take an offset of their own
};

int make_plan(const s1b_stitch_burst_t *in, int32_t n, Plan &p) {
  for (int sw = 1; sw <= 3; ++sw) {
    std::vector<int> idx;
    for (int i = 0; i < n; ++i)
      if (in[i].subswath == sw) idx.push_back(i);
    if (idx.empty()) continue;
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) {
      return in[a].top + in[a].bottom < in[b].top + in[b].bottom;
    });
    Swath s;
    s.first = (int32_t)p.bursts.size();
    s.count = (int32_t)idx.size();
    const s1b_stitch_burst_t &f = in[idx.front()], &l = in[idx.back()];
    s.left = std::min(f.left, l.left);
    s.top = std::min(f.top, l.top);
    s.right = std::max(f.right, l.right);
    s.bottom = std::max(f.bottom, l.bottom);
    int hull_t = 0, hull_b = 0;
    for (int k = 0; k < s.count; ++k) {
      const s1b_stitch_burst_t &b = in[idx[k]];
      if (b.right <= b.left || b.bottom <= b.top) return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_stitch: empty burst");
      // the part inside the subswath's box; a burst outside it is empty there
      Bst c;
      c.width = b.right - b.left;
      c.group = b.group;
      c.left = std::min(std::max(b.left, s.left), s.right);
      c.top = std::min(std::max(b.top, s.top), s.bottom);
      c.right = std::max(std::min(b.right, s.right), c.left);
      c.bottom = std::max(std::min(b.bottom, s.bottom), c.top);
      c.off = b.offset + (int64_t)(c.top - b.top) * c.width + (c.left - b.left);
      c.over_top = k ? std::max(c.top, hull_t) : 0;
      c.over_bottom = k ? std::min(c.bottom, hull_b) : 0;
      c.measured = k && b.group != in[idx[k - 1]].group && c.left < c.right && c.over_bottom > c.over_top;
      if (c.measured) {
        p.overlap = std::max(p.overlap, (int64_t)(c.over_bottom - c.over_top) * (c.right - c.left));
        ++p.measured;
      }
      hull_t = k ? std::min(hull_t, c.top) : c.top;
      hull_b = k ? std::max(hull_b, c.bottom) : c.bottom;
      p.bursts.push_back(c);
      p.index.push_back(idx[k]);
    }
    p.swaths.push_back(s);
  }
  return S1B_OK;
}

// Workspace: the turns, the measured overlaps, then the burst table where it
// does not fit a launch.
size_t turns_bytes(size_t n) { return (n * sizeof(Turn) + 255) / 256 * 256; }
size_t measured_bytes(size_t n) { return (n * sizeof(Measured) + 255) / 256 * 256; }

template <bool kFloat>
size_t chain_smem(int keep) {
  static_assert(sizeof(StSmem<kFloat>) % 16 == 0 && sizeof(StSmem<kFloat>) + ST_KEEP * sizeof(float2) <= 227 * 1024,
                "kept products follow the block, within an SM's shared memory");
  return sizeof(StSmem<kFloat>) + (size_t)keep * sizeof(float2);
}

// CTAs per cluster that the current device can place with the kernels'
// largest shared memory (16 on a B200); the kernel attributes are set on the
// first call per device.
template <bool kFloat, typename Idx>
int cluster_limit(int *ncta) {
  static std::mutex mu;
  static int known[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return s1b_fail(S1B_ERR_UNSUPPORTED, "s1b_stitch: device ordinal above 63");
  std::lock_guard<std::mutex> lock(mu);
  if (!known[dev]) {
    int best = ST_CLUSTER;
    auto limit = [&](auto kernel) -> cudaError_t {
      cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)chain_smem<kFloat>(ST_KEEP));
      if (err != cudaSuccess) return err;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        best = std::min(best, 8);
      for (; best > 1; best /= 2) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = best;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(best, 3);
        cfg.blockDim = dim3(ST_THREADS);
        cfg.dynamicSmemBytes = chain_smem<kFloat>(ST_KEEP);
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0) break;
      }
      cudaGetLastError();
      return cudaSuccess;
    };
    e = limit(stitch_measure_kernel<kFloat, Idx>);
    if (e == cudaSuccess) e = limit(stitch_chain_kernel<kFloat, Idx>);
    if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
    known[dev] = best;
  }
  *ncta = known[dev];
  return S1B_OK;
}

template <bool kFloat, typename Idx>
int launch_chain(const Table &tab, const Plan &p, const void *data, Measured *measured, Turn *turns, cudaStream_t st) {
  int most = 0, dev = 0, sms = 148;
  const int s = cluster_limit<kFloat, Idx>(&most);
  if (s) return s;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  auto launch = [&](auto kernel, int ncta, int n, auto... args) -> cudaError_t {
    const int64_t per = (p.overlap + ncta - 1) / ncta;
    const int keep = (int)std::min<int64_t>((per + ST_THREADS - 1) / ST_THREADS * ST_THREADS, ST_KEEP);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ncta;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)ncta * n);
    cfg.blockDim = dim3(ST_THREADS);
    cfg.dynamicSmemBytes = chain_smem<kFloat>(keep);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, tab, data, args..., keep);
  };
  // all overlaps at once where the SMs allow it: the largest cluster that
  // leaves room for the others beside it, but one that keeps the largest
  // overlap in shared memory (a pass that forms the angles again costs more
  // than a second wave: 57 against 30 us for 24 overlaps of 77 k pixels)
  int ncta = most;
  while (ncta > 1 && (int64_t)ncta * p.measured > sms && (int64_t)ncta / 2 * ST_KEEP >= p.overlap) ncta /= 2;
  cudaError_t e = launch(stitch_measure_kernel<kFloat, Idx>, ncta, (int)p.bursts.size(), measured);
  if (e == cudaSuccess) e = launch(stitch_chain_kernel<kFloat, Idx>, most, tab.n_swaths, (const Measured *)measured, turns);
  if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
  return s1b_launch_status();
}

template <bool kFloat>
int launch_stitch(const Table &tab, const Plan &p, const void *data, Measured *measured, Turn *turns, void *frame,
                  int nrow0, int ncol0, cudaStream_t st) {
  const int s = p.overlap >= ((int64_t)1 << 30) ? launch_chain<kFloat, uint64_t>(tab, p, data, measured, turns, st)
                                                : launch_chain<kFloat, uint32_t>(tab, p, data, measured, turns, st);
  if (s) return s;
  const dim3 grid((ncol0 + 255) / 256, (nrow0 + ST_FROWS - 1) / ST_FROWS);
  stitch_frame_kernel<kFloat><<<grid, 256, 0, st>>>(tab, data, turns, (typename Px<kFloat>::T *)frame, nrow0, ncol0);
  return s1b_launch_status();
}

}  // namespace

extern "C" size_t s1b_stitch_workspace_bytes(const s1b_stitch_burst_t *bursts, int32_t n, int32_t out_float) {
  (void)out_float;
  Plan p;
  if (!bursts || n < 1 || make_plan(bursts, n, p)) return 0;
  const size_t nb = p.bursts.size();
  return turns_bytes(nb) + measured_bytes(nb) + nb * sizeof(Bst);
}

extern "C" int s1b_stitch(const s1b_stitch_burst_t *bursts, int32_t n, const void *data, int32_t out_float,
                          int32_t nrow0, int32_t ncol0, void *frame, double *offsets_host, void *workspace,
                          size_t workspace_bytes, void *stream) {
  if (!bursts || n < 1 || !data || !frame || !workspace)
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_stitch: null argument");
  if (nrow0 < 1 || ncol0 < 1) return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_stitch: empty frame");
  for (int i = 0; i < n; ++i) {
    const s1b_stitch_burst_t &b = bursts[i];
    if (b.subswath < 1 || b.subswath > 3)
      return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_stitch: subswath must be 1, 2 or 3");
    if (b.left < 0 || b.top < 0 || b.right > ncol0 || b.bottom > nrow0)
      return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_stitch: burst outside the frame");
  }
  Plan p;
  int s = make_plan(bursts, n, p);
  if (s) return s;
  if (workspace_bytes < s1b_stitch_workspace_bytes(bursts, n, out_float))
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_stitch: workspace too small");
  if (nrow0 > 65535) return s1b_fail(S1B_ERR_TOO_LARGE, "s1b_stitch: frame too tall");
  const size_t nb = p.bursts.size();
  Turn *turns = (Turn *)workspace;
  Measured *measured = (Measured *)((unsigned char *)workspace + turns_bytes(nb));
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e;
  Table tab = {};
  tab.n_swaths = (int32_t)p.swaths.size();
  std::copy(p.swaths.begin(), p.swaths.end(), tab.swaths);
  if (p.bursts.size() <= ST_TABLE) {
    std::copy(p.bursts.begin(), p.bursts.end(), tab.bursts);
  } else {
    Bst *d_b = (Bst *)((unsigned char *)measured + measured_bytes(nb));
    e = cudaMemcpyAsync(d_b, p.bursts.data(), p.bursts.size() * sizeof(Bst), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
    tab.more = d_b;
  }
  // The frame is written while bursts are still read: one that lies over any
  // of them is formed beside them and copied.
  const size_t es = out_float ? sizeof(float) : sizeof(float2), frame_bytes = (size_t)nrow0 * ncol0 * es;
  void *formed = frame;
  for (int i = 0; i < n && formed == frame; ++i) {
    const s1b_stitch_burst_t &b = bursts[i];
    const uintptr_t lo = (uintptr_t)data + (uintptr_t)(b.offset * (int64_t)es);
    const uintptr_t hi = lo + (size_t)(b.right - b.left) * (b.bottom - b.top) * es;
    if (lo < (uintptr_t)frame + frame_bytes && (uintptr_t)frame < hi) {
      e = cudaMallocAsync(&formed, frame_bytes, st);
      if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  s = out_float ? launch_stitch<true>(tab, p, data, measured, turns, formed, nrow0, ncol0, st)
                : launch_stitch<false>(tab, p, data, measured, turns, formed, nrow0, ncol0, st);
  if (formed != frame) {
    e = s ? cudaSuccess : cudaMemcpyAsync(frame, formed, frame_bytes, cudaMemcpyDeviceToDevice, st);
    const cudaError_t freed = cudaFreeAsync(formed, st);
    if (!s && (e != cudaSuccess || freed != cudaSuccess))
      s = s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e != cudaSuccess ? e : freed));
  }
  if (s) return s;
  if (offsets_host) {
    // offsets per burst in the caller's order (the kernel writes them in subswath order)
    std::vector<Turn> tmp(p.bursts.size());
    e = cudaMemcpyAsync(tmp.data(), turns, tmp.size() * sizeof(Turn), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
    for (size_t k = 0; k < tmp.size(); ++k) offsets_host[p.index[k]] = tmp[k].phase;
  }
  return S1B_OK;
}
