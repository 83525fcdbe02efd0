// bief_resident.cu -- the CG kernels that keep their search direction in
// shared memory (k_cg_res: GRACJG; k_mixed_res: its mixed-precision form).
//
// A block owns a fixed set of nodes for the whole solve, and the nodes its
// rows read besides are a fixed list, the halo.  The block keeps the search
// direction of both in shared memory and updates the halo's copy itself
// (D = R + BETA D needs only R of the halo nodes, one value per halo node and
// iteration instead of two per gather entry), so a row's neighbour values are
// shared-memory reads through 16-bit local indices, and what is streamed per
// iteration is the operator alone.  k_cg64 and k_mixed gather R and the old D
// of every neighbour through L1/L2 and were bound by that latency.
//
// The arithmetic is that of k_cg64 / k_mixed: the same operations per node
// and the same dot-product tree (G virtual blocks of 1024 threads, thread t
// of block b summing rows lo+t, lo+t+1024, ...), so the same bits.
//
// Two forms:
//   CL = false  one physical block per SM holding V virtual blocks (V = 2
//               when the tree has more blocks than SMs), grid barriers
//               through global memory;
//   CL = true   meshes of up to 12 virtual blocks (24,576 nodes) with at most
//               two rows per thread: one cluster of G*S <= 12 blocks, each holding 1/S of a virtual block's warps;
//               partial sums and halo values through distributed shared
//               memory.
#include <type_traits>

#include "bief_resident.h"

namespace bief {

// Virtual block that holds node j (blk_lo's ranges).
__device__ __forceinline__ int res_block_of(int j, int n, int G) {
  int b = (int)((long long)j * G / n);
  while (b + 1 < G && blk_lo(b + 1, n, G) <= j) ++b;
  while (b > 0 && blk_lo(b, n, G) > j) --b;
  return b;
}

// Physical block and local index of node j.
__device__ __forceinline__ void res_local(const ResPart &Q, int j, int &p, int &loc) {
  const int b = res_block_of(j, Q.n, Q.G);
  const int off = j - (int)blk_lo(b, Q.n, Q.G);
  const int k = off / RES_T, vt = off % RES_T;
  if (Q.V > 1) {
    p = b / Q.V;
    loc = ((b % Q.V) * Q.R + k) * Q.TP + vt;
  } else {
    p = b * Q.S + vt / Q.TP;
    loc = k * Q.TP + vt % Q.TP;
  }
}

// Node of the block's local row (kk, t), -1 where there is none.
__device__ __forceinline__ int res_node(const ResPart &Q, int p, int kk, int t) {
  int b, k, vt;
  if (Q.V > 1) {
    b = p * Q.V + kk / Q.R;
    k = kk % Q.R;
    vt = t;
  } else {
    b = p / Q.S;
    k = kk;
    vt = (p % Q.S) * Q.TP + t;
  }
  if (b >= Q.G) return -1;
  const int j = (int)blk_lo(b, Q.n, Q.G) + vt + RES_T * k;
  return j < (int)blk_lo(b + 1, Q.n, Q.G) ? j : -1;
}

// ---------------------------------------------------------------------------
// Halo lists and local indices, one block per physical block.  The nodes
// outside the block that its rows name are marked in a bitmap held in shared
// memory, PLAN_W * 32 nodes at a time; their ranks are the halo positions.
//   FILL = false: halo_n[p] = number of halo nodes;
//   FILL = true : the halo list when A.halo is given, and one list of 16-bit
//                 local indices: rec_li (a record's two vertices), seg_li,
//                 sg_li or sg_li2 (a slot's neighbour).
// ---------------------------------------------------------------------------
template <bool FILL>
__global__ void __launch_bounds__(1024, 1) k_res_plan(PlanP A) {
  extern __shared__ unsigned plan_sm[];
  unsigned *bits = plan_sm, *rank = plan_sm + PLAN_W;
  __shared__ int s_min, s_max, s_w[32], s_run;
  const int t = threadIdx.x, T = blockDim.x, p = blockIdx.x, lane = t & 31, w = t >> 5;
  const ResPart Q = A.Q;
  if (t == 0) {
    s_min = 0x7fffffff;
    s_max = -1;
    s_run = 0;
  }
  __syncthreads();
  // the block's own node ranges (res_node and res_local for this block,
  // without their 64-bit divisions)
  const int b0 = Q.V > 1 ? p * Q.V : p / Q.S, s0 = Q.V > 1 ? 0 : (p % Q.S) * Q.TP;
  const int L0 = (int)blk_lo(b0, Q.n, Q.G), L1 = (int)blk_lo(b0 + 1, Q.n, Q.G);
  const int L2 = Q.V > 1 && b0 + 1 < Q.G ? (int)blk_lo(b0 + 2, Q.n, Q.G) : L1;
  auto each_row = [&](auto f) {
#pragma unroll 1
    for (int a = t; a < Q.own; a += T) {
      const int kk = a / Q.TP, v = kk / Q.R;
      const int i = (v ? L1 : L0) + s0 + a % Q.TP + RES_T * (kk - v * Q.R);
      if (i < (v ? L2 : L1)) f(i);
    }
  };
  auto outside = [&](int j, int &loc) {
    int v = 0, off = j - L0;
    if (j >= L1) {
      v = 1;
      off = j - L1;
      if (j >= L2) return true;
    }
    if (off < 0) return true;
    const int k = off / RES_T, vt = off % RES_T - s0;
    loc = (v * Q.R + k) * Q.TP + vt;
    return vt < 0 || vt >= Q.TP;
  };
  int mn = 0x7fffffff, mx = -1;
  each_row([&](int i) {
    const int nn = A.nb_meta[i] >> 16, b = A.nb_off[i >> 5] + (i & 31);
#pragma unroll 1
    for (int m = 0; m < nn; ++m) {
      int loc;
      const int j = A.nb_col[b + 32 * m];
      if (outside(j, loc)) {
        mn = min(mn, j);
        mx = max(mx, j);
      }
    }
  });
  atomicMin(&s_min, mn);
  atomicMax(&s_max, mx);
  __syncthreads();
  const int first = s_min & ~31, last = s_max;
  bool own_done = false;
#pragma unroll 1
  for (long long lo = first; lo <= last || !own_done; lo += 32LL * PLAN_W) {
    const long long hi = lo + 32LL * PLAN_W;
    auto inside = [&](int j) { return j >= lo && j < hi; };
#pragma unroll 1
    for (int q = t; q < PLAN_W; q += T) bits[q] = 0;
    __syncthreads();
    each_row([&](int i) {
      const int nn = A.nb_meta[i] >> 16, b = A.nb_off[i >> 5] + (i & 31);
#pragma unroll 1
      for (int m = 0; m < nn; ++m) {
        int loc;
        const int j = A.nb_col[b + 32 * m];
        if (inside(j) && outside(j, loc)) atomicOr(&bits[(j - lo) >> 5], 1u << (j & 31));
      }
    });
    __syncthreads();
    // rank[q]: halo nodes before word q (chunk of words per thread, block scan)
    constexpr int PER = (PLAN_W + 1023) / 1024;
    int cnt = 0;
#pragma unroll 1
    for (int q = t * PER; q < min(PLAN_W, (t + 1) * PER); ++q) cnt += __popc(bits[q]);
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (w == 0) {
      int v = s_w[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      s_w[lane] = v;
    }
    __syncthreads();
    int run = s_run + inc - cnt + (w ? s_w[w - 1] : 0);
#pragma unroll 1
    for (int q = t * PER; q < min(PLAN_W, (t + 1) * PER); ++q) {
      rank[q] = run;
      run += __popc(bits[q]);
    }
    __syncthreads();
    if (t == 0) s_run += s_w[31];
    if (FILL) {
#pragma unroll 1
      for (int q = t; A.halo && q < PLAN_W; q += T) {
        unsigned m = bits[q];
        int r = rank[q];
        while (m) {
          const int bit = __ffs(m) - 1;
          m &= m - 1;
          const int j = (int)(lo + 32LL * q + bit);
          const int at = A.Q.halo_off[p] + r++;
          A.halo[at] = j;
          if (A.halo_loc) {
            int pp, loc;
            res_local(Q, j, pp, loc);
            A.halo_loc[at] = ((unsigned)pp << 16) | (unsigned)(loc & 0xffff);
          }
        }
      }
      auto local_of = [&](int j, int &loc) -> bool {  // true when this pass settles it
        if (!outside(j, loc)) return !own_done;
        if (!inside(j)) return false;
        const int q = (int)((j - lo) >> 5);
        loc = Q.own + (int)rank[q] + __popc(bits[q] & ((1u << (j & 31)) - 1u));
        return true;
      };
      each_row([&](int i) {
        int loc;
        // pairs of indices: slot m of a lane at word m / 2
        auto pair_at = [&](int b0, int m) {
          return 2 * (((b0 - (i & 31)) >> 1) + 32 * (m >> 1) + (i & 31)) + (m & 1);
        };
        if (A.rec_li) {
          const int deg = A.meta[i] & 0xffff, b = A.rec_off[i >> 5] + (i & 31);
#pragma unroll 1
          for (int m = 0; m < deg; ++m) {
            const int2 v = A.rec_idx[b + 32 * m];
            if (local_of(v.x, loc)) A.rec_li[b + 32 * m].x = (unsigned short)loc;
            if (local_of(v.y, loc)) A.rec_li[b + 32 * m].y = (unsigned short)loc;
          }
          return;
        }
        const bool mesh = A.seg_li != nullptr;  // the mesh's neighbours, else the segments'
        const int nn = (mesh ? A.meta : A.sg_meta)[i] >> 16;
        const int b = (mesh ? A.seg_off : A.sg_off)[i >> 5] + (i & 31);
        const int *col = mesh ? A.seg_col : A.sg_col;
        unsigned short *pairs = mesh ? A.seg_li : A.sg_li2;
#pragma unroll 1
        for (int m = 0; m < nn; ++m)
          if (local_of(col[b + 32 * m], loc)) {
            if (pairs) pairs[pair_at(b, m)] = (unsigned short)(loc << A.shift);
            else A.sg_li[b + 32 * m] = (unsigned short)loc;
          }
      });
    }
    own_done = true;
    __syncthreads();
    if (last < 0) break;
  }
  if (!FILL && t == 0) A.halo_n[p] = s_run;
}

// ---------------------------------------------------------------------------
// Reductions.  send() starts one, wait() ends it; work that no other block
// waits for goes between the two.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned mapa(unsigned a, unsigned cta) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta));
  return r;
}

// The zero-padded 32-value butterfly of block_tree's second stage over the
// first ns (<= 16) values, formed by every thread for itself.
template <typename T>
__device__ __forceinline__ T tree16(const T *u, int ns) {
  T z[16];
  if (ns <= 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] = i < ns ? add(T(0), u[i]) : T(0);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) z[i] = i < ns ? add(T(0), u[i]) : T(0);
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] = add(z[i], z[i + 8]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) z[i] = add(z[i], z[i + 4]);
  return add(add(z[0], z[2]), add(z[1], z[3]));
}

template <typename T>
__device__ __forceinline__ T warp_tree(T v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v = add(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// A value with the number of its reduction beside each 32 bits of it: one or
// two 64-bit words, each valid as soon as it shows the number waited for.
template <typename T>
__device__ __forceinline__ void tag_words(T u, unsigned tag, unsigned long long &x,
                                          unsigned long long &y) {
  if constexpr (sizeof(T) == 8) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong((double)u);
    x = (bits << 32) | tag;
    y = (bits & 0xffffffff00000000ull) | tag;
  } else {
    x = ((unsigned long long)__float_as_uint((float)u) << 32) | tag;
    y = tag;
  }
}
template <typename T>
__device__ __forceinline__ T tag_value(unsigned long long x, unsigned long long y) {
  if constexpr (sizeof(T) == 8)
    return __longlong_as_double((long long)((x >> 32) | (y & 0xffffffff00000000ull)));
  else
    return __uint_as_float((unsigned)(x >> 32));
}

// How the blocks of a solve talk to each other.
//   COM_CL   cluster: every warp's total goes straight to every block's shared
//            memory, each with an arrival on that block's mbarrier; halo values
//            are read from the owner's shared memory;
//   COM_TAG  grid: block totals as tagged words that all blocks poll;
//   COM_CNT  grid: block totals and an arrival counter.
// Measured per reduction in a loop of nothing else at 1024 threads (us):
// counter 2.5 (1 to 75 blocks) to 2.6 (148); tagged, without / with fences,
// 17 blocks 1.1 / 1.6, 44 blocks 2.5 / 2.5, 148 blocks 5.5 / 5.3, as polls
// queue at an L2 line and delay the write they wait for.  So tags up to
// RES_TAG blocks: binary64 / mixed us per iteration with tags against the
// counter, 13 blocks 8.95 / 7.19 against 9.53 / 8.17, 20 blocks (41,000 nodes)
// 8.98 / 7.75 against 9.55 / 8.18, 24 blocks 9.12 / 7.40 against 9.34 / 8.02.
//
// PUB: the reduction also publishes what the block wrote before it (R for
// its neighbours' halos).  Without it tagged words need no fence: what the
// block read before is already in the partial sums it sends.
enum : int { COM_CL = 0, COM_TAG = 1, COM_CNT = 2 };

// Communication state of one block.
template <int COM>
struct Comm {
  static constexpr bool CL = COM == COM_CL;
  Ctl *ctl;
  double *part;               // grid form: 2 halves of G partials
  long long timeout_ns;
  RedShared *sh;
  unsigned long long *box;    // tagged words, 2 halves: cluster 32 G (shared memory), grid G
  int G, V, S, NP, p;
  unsigned nbar;              // reductions so far

  // a publishing reduction made on a copy of this state
  __device__ __forceinline__ void done() { ++nbar; }

  // v: this thread's partial per virtual block of the block (V of them).
  template <bool PUB, typename T>
  __device__ __forceinline__ void send(const T *v) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    unsigned long long x, y;
    ++nbar;
    if constexpr (CL) {
      const T u = warp_tree(v[0]);
      __syncwarp();  // the warp's writes before its lanes' releases
      if (lane < NP) {
        const int vw = (p % S) * ((int)blockDim.x >> 5) + w;
        const int slot = (p / S) * 32 + vw;
        const unsigned a =
            mapa(smem_addr(box + (size_t)(nbar & 1) * 32 * G + slot), (unsigned)lane);
        if constexpr (sizeof(T) == 8)
          asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"((double)u)
                       : "memory");
        else
          asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"((float)u)
                       : "memory");
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                         mapa(smem_addr(&sh->mbar[nbar & 1]), (unsigned)lane))
                     : "memory");
      }
    } else {
#pragma unroll 1
      for (int q = 0; q < V; ++q) {
        const T u = warp_tree(v[q]);
        if (lane == 0) sh->ws[q][w] = (double)u;
      }
      __syncthreads();
      if (w == 0) {
        if (PUB && COM == COM_TAG) fence_gpu();
#pragma unroll 1
        for (int q = 0; q < V; ++q) {
          const T u = warp_tree((T)sh->ws[q][lane]);
          const int b = p * V + q;
          if (b >= G) break;
          if (lane) continue;
          if constexpr (COM == COM_TAG) {
            tag_words(u, nbar, x, y);
            asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(
                             box + 2 * ((size_t)(nbar & 1) * G + b)),
                         "l"(x), "l"(y)
                         : "memory");
          } else {
            part[(size_t)(nbar & 1) * G + b] = (double)u;
          }
        }
        if (COM == COM_CNT && lane == 0)
          asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&ctl->arrivals), "l"(1ull)
                       : "memory");
      }
    }
  }

  // The sum over all blocks; false when the bounded wait ran out.
  template <bool PUB, typename T>
  __device__ __forceinline__ bool wait(T &out) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    int ns, bad = 0;
    if constexpr (COM != COM_CNT) {
      // cluster: warp w sums the 32 warp totals of virtual block w; grid: the
      // totals of virtual blocks 32 w ..
      ns = CL ? G : (G + 31) >> 5;
      if (w < ns) {
        T u = T(0);
        if constexpr (CL) {
          const unsigned bar = smem_addr(&sh->mbar[nbar & 1]), par = ((nbar - 1) >> 1) & 1;
          unsigned ok = 0;
          unsigned long long t0 = 0;
#pragma unroll 1
          for (unsigned n = 1;; ++n) {  // each try waits in hardware, for a bounded time
            asm volatile(
                "{\n.reg .pred p;\n"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                "selp.u32 %0, 1, 0, p;\n}"
                : "=r"(ok)
                : "r"(bar), "r"(par)
                : "memory");
            if (ok) break;
            if ((n & 0xf) == 0) {
              if (!t0) t0 = global_ns();
              else if ((long long)(global_ns() - t0) > timeout_ns) { bad = 1; break; }
            }
          }
          u = *reinterpret_cast<const volatile T *>(box + (size_t)(nbar & 1) * 32 * G + t);
        } else if (t < G) {
          const unsigned long long *m = box + 2 * ((size_t)(nbar & 1) * G + t);
          unsigned long long x, y, t0 = 0;
#pragma unroll 1
          for (unsigned n = 1;; ++n) {
            asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                         : "=l"(x), "=l"(y)
                         : "l"(m)
                         : "memory");
            if ((unsigned)x == nbar && (unsigned)y == nbar) break;
            if ((n & 0xff) == 0) {
              if (!t0) t0 = global_ns();
              else if ((long long)(global_ns() - t0) > timeout_ns) { bad = 1; break; }
            }
          }
          u = add(T(0), tag_value<T>(x, y));
        }
        if (PUB && !CL) fence_gpu();
        __syncwarp();
        u = warp_tree(u);
        if (lane == 0) reinterpret_cast<T *>(sh->us[nbar & 1])[w] = u;
      }
      if (__syncthreads_or(bad)) {
        if (t == 0) atomicExch(&ctl->status, (int)ST_TIMEOUT);
        return false;
      }
    } else {
      if (t == 0) {
        const unsigned long long target = (unsigned long long)nbar * (unsigned long long)NP;
        unsigned long long t0 = 0, c;
#pragma unroll 1
        for (unsigned n = 1;; ++n) {
          asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
                       : "=l"(c)
                       : "l"(&ctl->arrivals)
                       : "memory");
          if (c >= target) break;
          if ((n & 0xff) == 0) {
            if (!t0) t0 = global_ns();
            else if ((long long)(global_ns() - t0) > timeout_ns) {
              bad = 1;
              atomicExch(&ctl->status, (int)ST_TIMEOUT);
              break;
            }
          }
        }
      }
      if (__syncthreads_or(bad)) return false;
      ns = (G + 31) >> 5;
      if (w < ns) {
        const double *buf = part + (size_t)(nbar & 1) * G;
        T u = t < G ? add(T(0), (T)__ldcg(buf + t)) : T(0);
        u = warp_tree(u);
        if (lane == 0) reinterpret_cast<T *>(sh->us[nbar & 1])[w] = u;
      }
      __syncthreads();
    }
    out = tree16(reinterpret_cast<const T *>(sh->us[nbar & 1]), ns);
    return true;
  }
};

__device__ __forceinline__ double td_term(int td, double yi, const double *da, int i) {
  return td == DIA_Q ? mul(yi, __ldg(da + i)) : (td == DIA_I ? yi : 0.0);
}

// Per slice of 32 own rows (local rows 32 sl .. 32 sl + 31, one warp's rows
// of one step): x = its first slot in the operator's arrays, y = width |
// smallest row length << 8 | first cached slot / U << 16, bit 31 set for the
// leading slices, whose slots are kept in shared memory (U = 32 slots, or 64
// for the binary32 slots, which lie in pairs).  s_deg: slots of each row.
__device__ __forceinline__ int sl_width(int2 o) { return o.y & 0xff; }
__device__ __forceinline__ int sl_least(int2 o) { return (o.y >> 8) & 0xff; }
__device__ __forceinline__ bool sl_cached(int2 o) { return o.y < 0; }
__device__ __forceinline__ int sl_at(int2 o) { return (o.y >> 16) & 0x7fff; }

// Shared-memory copies of the leading slots, C: coefficients of one unit
// lane (a slot, or a pair), I: its local indices.
template <typename C, typename I, int PER>
__device__ __forceinline__ void res_setup(const ResPart &Q, int p, const int *meta, int shift,
                                          const int *off, const C *gc, const I *gi, int cache,
                                          int2 *s_off, unsigned char *s_deg, C *s_c, I *s_i) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, W = Q.TP >> 5, nsl = Q.own >> 5;
  const int room = cache / (32 * PER);
#pragma unroll 1
  for (int sl = w; sl < nsl; sl += W) {
    const int a = sl * 32 + lane;
    const int node = res_node(Q, p, a / Q.TP, a % Q.TP);
    const int deg = node >= 0 ? (meta[node] >> shift) & 0xffff : 0;
    s_deg[a] = (unsigned char)deg;
    const int wd = __reduce_max_sync(0xffffffffu, deg), mn = __reduce_min_sync(0xffffffffu, deg);
    const int n0 = __shfl_sync(0xffffffffu, node, 0);
    if (lane == 0) s_off[sl] = make_int2(n0 >= 0 ? off[n0 >> 5] : 0, wd | (mn << 8));
  }
  __syncthreads();
  if (w == 0) {
    int run = 0;  // units cached so far
#pragma unroll 1
    for (int s0 = 0; s0 < nsl; s0 += 32) {
      const int sl = s0 + lane;
      // (single slots: an odd slice's last batch reads one slot past its width)
      const int ws = sl < nsl ? (sl_width(s_off[sl]) + 1) & ~1 : 0;
      const int wd = ws / PER;
      int inc = wd;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      if (sl < nsl && run + inc <= room && run + inc - wd < 0x7fff)
        s_off[sl].y |= (int)(0x80000000u | ((unsigned)(run + inc - wd) << 16));
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int sl = w; sl < nsl; sl += W) {
    const int2 o = s_off[sl];
    if (!sl_cached(o)) continue;
    const int wd = (sl_width(o) + PER - 1) / PER, c0 = 32 * sl_at(o) + lane, g0 = o.x / PER + lane;
#pragma unroll 1
    for (int m = 0; m < wd; ++m) {
      s_c[c0 + 32 * m] = gc[g0 + 32 * m];
      s_i[c0 + 32 * m] = gi[g0 + 32 * m];
    }
    if (PER == 1 && (wd & 1)) s_i[c0 + 32 * wd] = 0;  // a valid index, never added
  }
  __syncthreads();
}

// Operator loads: read once per product, so past L1, and in L2 by the policy
// given (evict-first for what streams through it).
__device__ __forceinline__ unsigned long long l2_policy(bool stream) {
  unsigned long long p;
  if (stream)
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  else
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
#define RES_LD "ld.global.nc.L1::no_allocate.L2::cache_hint."
__device__ __forceinline__ double2 ld_pol(const double2 *a, unsigned long long p) {
  double2 v;
  asm(RES_LD "v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(a), "l"(p));
  return v;
}
__device__ __forceinline__ double ld_pol(const double *a, unsigned long long p) {
  double v;
  asm(RES_LD "f64 %0, [%1], %2;" : "=d"(v) : "l"(a), "l"(p));
  return v;
}
__device__ __forceinline__ float2 ld_pol(const float2 *a, unsigned long long p) {
  float2 v;
  asm(RES_LD "v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(a), "l"(p));
  return v;
}
__device__ __forceinline__ float ld_pol(const float *a, unsigned long long p) {
  float v;
  asm(RES_LD "f32 %0, [%1], %2;" : "=f"(v) : "l"(a), "l"(p));
  return v;
}
__device__ __forceinline__ unsigned ld_pol(const unsigned *a, unsigned long long p) {
  unsigned v;
  asm(RES_LD "u32 %0, [%1], %2;" : "=r"(v) : "l"(a), "l"(p));
  return v;
}
__device__ __forceinline__ unsigned short ld_pol(const unsigned short *a, unsigned long long p) {
  unsigned short v;
  asm(RES_LD "u16 %0, [%1], %2;" : "=h"(v) : "l"(a), "l"(p));
  return v;
}
#undef RES_LD

// Rows of the binary64 operators, NB slots at a time: the slots' loads, then
// the window reads, then the additions in slot order.  Slots beyond a row's
// own count (the slice is as wide as its longest row; one slot past an odd
// width) are read and, when PRED, not added.  Few batch sizes: the solver's
// loop has to fit the instruction caches.
struct RecRow {  // acc + (XA(k,a) D(a) + XA(k,b) D(b)) per record
  using C = double2;
  using I = unsigned;  // two 16-bit local indices
  static __device__ __forceinline__ double term(C c, I j, const double *win) {
    return add(mul(c.x, win[j & 0xffffu]), mul(c.y, win[j >> 16]));
  }
};
struct SegRow {  // acc + XA D(other) per incident segment
  using C = double;
  using I = unsigned short;
  static __device__ __forceinline__ double term(C c, I j, const double *win) {
    return mul(c, win[j]);
  }
};

template <class ROW, int NB, bool PRED, class LC, class LI>
__device__ __forceinline__ void res_batch(double &acc, int m, int n, LC lc, LI li,
                                          const double *win) {
  typename ROW::C c[NB];
  typename ROW::I j[NB];
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    c[q] = lc(m + q);
    j[q] = li(m + q);
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const double s = add(acc, ROW::term(c[q], j[q], win));
    acc = !PRED || m + q < n ? s : acc;
  }
}

template <class ROW, class LC, class LI>
__device__ __forceinline__ double res_batches(double acc, int2 o, int n, LC lc, LI li,
                                              const double *win) {
  const int wd = sl_width(o);
  int m = 0;
  if (sl_least(o) >= 6) {
    res_batch<ROW, 6, false>(acc, 0, n, lc, li, win);
    m = 6;
  } else if (wd >= 6) {
    res_batch<ROW, 6, true>(acc, 0, n, lc, li, win);
    m = 6;
  }
#pragma unroll 1
  for (; m < wd; m += 2) res_batch<ROW, 2, true>(acc, m, n, lc, li, win);
  return acc;
}

template <class ROW>
__device__ __forceinline__ double res_row(double acc, int2 o, int n, const typename ROW::C *gc,
                                          const typename ROW::I *gi, unsigned long long pol,
                                          const typename ROW::C *s_c, const typename ROW::I *s_i,
                                          const double *win) {
  const int lane = threadIdx.x & 31;
  if (sl_cached(o)) {
    const typename ROW::C *c = s_c + 32 * sl_at(o) + lane;
    const typename ROW::I *j = s_i + 32 * sl_at(o) + lane;
    return res_batches<ROW>(
        acc, o, n, [&](int m) { return c[32 * m]; }, [&](int m) { return j[32 * m]; }, win);
  }
  const typename ROW::C *c = gc + o.x + lane;
  const typename ROW::I *j = gi + o.x + lane;
  return res_batches<ROW>(
      acc, o, n, [&](int m) { return ld_pol(c + 32 * m, pol); },
      [&](int m) { return ld_pol(j + 32 * m, pol); }, win);
}

// Binary32 rows: acc + c_ij (p_j - p_i) per neighbour.  The slots lie in
// pairs (float2 coefficients, two 16-bit indices in one word), so a pair
// costs two loads; the first three pairs of a row (a P1 node has about six
// neighbours) are loaded together, ahead of the row before them.
struct Pair3 {
  float2 c[3];
  unsigned j[3];
};

// SH = 0: the indices are byte offsets into the window; 2: element numbers.
template <int SH>
__device__ __forceinline__ float win_at(const float *win, unsigned j) {
  return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(win) + (j << SH));
}

__device__ __forceinline__ void pair_load(Pair3 &P, int2 o, const float2 *gc, const unsigned *gi,
                                          unsigned long long pol, const float2 *s_c,
                                          const unsigned *s_i) {
  const int lane = threadIdx.x & 31;
  if (sl_width(o) < 5) return;  // fewer than three pairs: pair_row loads them
  if (sl_cached(o)) {
    const int c0 = 32 * sl_at(o) + lane;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      P.c[q] = s_c[c0 + 32 * q];
      P.j[q] = s_i[c0 + 32 * q];
    }
  } else {
    const int b0 = (o.x >> 1) + lane;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      P.c[q] = ld_pol(gc + b0 + 32 * q, pol);
      P.j[q] = ld_pol(gi + b0 + 32 * q, pol);
    }
  }
}

template <int SH, bool PRED>
__device__ __forceinline__ float pair_add(float acc, float y0, float2 c, unsigned j, int m, int n,
                                          const float *win) {
  const float v0 = win_at<SH>(win, j & 0xffffu), v1 = win_at<SH>(win, j >> 16);
  const float s0 = add(acc, mul(c.x, sub(v0, y0)));
  acc = !PRED || m < n ? s0 : acc;
  const float s1 = add(acc, mul(c.y, sub(v1, y0)));
  return !PRED || m + 1 < n ? s1 : acc;
}

template <int SH>
__device__ __forceinline__ float pair_row(const Pair3 &P, float acc, float y0, int2 o, int n,
                                          const float2 *gc, const unsigned *gi,
                                          unsigned long long pol, const float2 *s_c,
                                          const unsigned *s_i, const float *win) {
  const int lane = threadIdx.x & 31, wd = sl_width(o);
  int m = 0;
  if (wd >= 5) {
    if (sl_least(o) >= 6) {
#pragma unroll
      for (int q = 0; q < 3; ++q) acc = pair_add<SH, false>(acc, y0, P.c[q], P.j[q], 0, 0, win);
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q) acc = pair_add<SH, true>(acc, y0, P.c[q], P.j[q], 2 * q, n, win);
    }
    m = 6;
  }
#pragma unroll 1
  for (; m < wd; m += 2) {
    float2 c;
    unsigned j;
    if (sl_cached(o)) {
      c = s_c[32 * (sl_at(o) + (m >> 1)) + lane];
      j = s_i[32 * (sl_at(o) + (m >> 1)) + lane];
    } else {
      c = ld_pol(gc + (o.x >> 1) + 16 * m + lane, pol);
      j = ld_pol(gi + (o.x >> 1) + 16 * m + lane, pol);
    }
    acc = pair_add<SH, true>(acc, y0, c, j, m, n, win);
  }
  return acc;
}

// First node (of this thread) and end of the block's virtual blocks: formed
// once, as the ranges' 64-bit divisions are dear.
struct Ranges {
  int lo0, hi0, lo1, hi1;
  __device__ __forceinline__ void init(const ResPart &Q, int p) {
    const int b0 = Q.V > 1 ? p * Q.V : p / Q.S, sh = (p % Q.S) * Q.TP + threadIdx.x;
    lo0 = (int)blk_lo(b0, Q.n, Q.G) + (Q.V > 1 ? (int)threadIdx.x : sh);
    hi0 = (int)blk_lo(b0 + 1, Q.n, Q.G);
    const bool two = Q.V > 1 && b0 + 1 < Q.G;
    lo1 = two ? hi0 + (int)threadIdx.x : 0;
    hi1 = two ? (int)blk_lo(b0 + 2, Q.n, Q.G) : 0;
  }
  __device__ __forceinline__ int lo(int v) const { return v == 0 ? lo0 : lo1; }
  __device__ __forceinline__ int hi(int v) const { return v == 0 ? hi0 : hi1; }
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}

// The halo's owners: the first HR halo nodes of a thread by their addresses
// in registers (cluster: the owner's copy of R in distributed shared memory;
// grid: node numbers), the others through the list.
template <typename T, bool CL>
struct Halo {
  static constexpr int HR = CL ? 4 : 2;
  unsigned at[HR];
  int nh, h0;
  __device__ __forceinline__ unsigned where(const ResPart &Q, const T *src, int h) const {
    if constexpr (CL) {
      const unsigned c = __ldg(Q.halo_loc + h0 + h);
      return mapa(smem_addr(src + (c & 0xffffu)), c >> 16);
    } else {
      return (unsigned)__ldg(Q.halo + h0 + h);
    }
  }
  __device__ __forceinline__ T read(const T *src, unsigned a) const {
    if constexpr (CL) {
      if constexpr (sizeof(T) == 8) {
        double v;
        asm volatile("ld.relaxed.cluster.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
        return v;
      } else {
        float v;
        asm volatile("ld.relaxed.cluster.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
        return v;
      }
    } else {
      return __ldcg(src + a);
    }
  }
  __device__ __forceinline__ void init(const ResPart &Q, int p, const T *src) {
    h0 = Q.halo_off[p];
    nh = Q.halo_off[p + 1] - h0;
#pragma unroll
    for (int q = 0; q < HR; ++q) {
      const int h = threadIdx.x + q * blockDim.x;
      at[q] = h < nh ? where(Q, src, h) : 0u;
    }
  }
  // f(h, R of halo node h) for this thread's halo nodes; src: the block's
  // own copy of R (CL) or R in global memory
  template <class F>
  __device__ __forceinline__ void each(const ResPart &Q, const T *src, F f) const {
    T v[HR];
#pragma unroll
    for (int q = 0; q < HR; ++q)
      if ((int)(threadIdx.x + q * blockDim.x) < nh) v[q] = read(src, at[q]);
#pragma unroll
    for (int q = 0; q < HR; ++q) {
      const int h = threadIdx.x + q * blockDim.x;
      if (h < nh) f(h, v[q]);
    }
    // the rest two at a time, each through the list
    int h = threadIdx.x + HR * blockDim.x;
#pragma unroll 1
    for (; h + (int)blockDim.x < nh; h += 2 * blockDim.x) {
      const unsigned a0 = where(Q, src, h), a1 = where(Q, src, h + blockDim.x);
      const T v0 = read(src, a0), v1 = read(src, a1);
      f(h, v0);
      f(h + blockDim.x, v1);
    }
    if (h < nh) f(h, read(src, where(Q, src, h)));
  }
};

// A reduction off the iteration's path (one copy of the code per type).
template <int COM, typename T>
__device__ __noinline__ bool cold_reduce(Comm<COM> M, T v0, T v1, T *out) {  // the caller counts it: done()
  const T v[2] = {v0, v1};
  M.template send<true>(v);
  return M.template wait<true>(*out);
}

template <int COM>
__device__ __forceinline__ void comm_init(Comm<COM> &M, const ResP &P, int V, unsigned char *red,
                                          unsigned char *box) {
  M.ctl = P.ctl;
  M.part = P.part;
  M.timeout_ns = P.timeout_ns;
  M.sh = reinterpret_cast<RedShared *>(red);
  M.box = COM == COM_CL ? reinterpret_cast<unsigned long long *>(box) : P.box;
  M.G = P.Q.G;
  M.V = V;
  M.S = P.Q.S;
  M.NP = P.Q.NP;
  M.p = blockIdx.x;
  M.nbar = 0;
  if (COM == COM_CL)
    if (threadIdx.x == 0) {
      // one arrival per warp of the cluster and reduction
      for (int q = 0; q < 2; ++q)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&M.sh->mbar[q])),
                     "r"(32 * M.G)
                     : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// ---------------------------------------------------------------------------
// GRACJG (gracjg.F:169-420), statement for statement k_cg64.  R and AD of the
// own rows are in shared memory when they fit (nvec >= 2), X too in the
// cluster form (nvec = 3), else in global memory; X is updated while the
// partial sums travel.  The three products (A X, A R, A D) are one piece of
// code, told apart by `phase`, and loops stay rolled: unrolled or repeated,
// the loop outgrew the instruction caches, and with most of the SM's memory
// taken as shared memory every register spill is an L2 access.
// Bound: the reductions and dependent binary64 chains on small meshes (1,681
// nodes 10.7 -> 3.5 us per iteration against k_cg64), window conflicts and two
// grid reductions at 150k (18 -> 12), the records' bytes at 1.0M (34 -> 26.8).
// ---------------------------------------------------------------------------
template <int STO, int COM, int MT>
__global__ void __launch_bounds__(MT, 1) k_cg_res(const __grid_constant__ ResP P) {
  constexpr bool CL = COM == COM_CL;
  using ROW = typename std::conditional<STO == 3, SegRow, RecRow>::type;
  using C = typename ROW::C;
  using I = typename ROW::I;
  extern __shared__ __align__(16) unsigned char res_sm[];
  const ResPart &Q = P.Q;
  const int t = threadIdx.x, TP = blockDim.x, lane = t & 31;
  const int p = blockIdx.x, V = CL ? 1 : Q.V, R = Q.R;
  const ResLayout L = res_layout(Q.own, P.halo_max, Q.G, CL, 8, P.nvec, sizeof(C), sizeof(I),
                                 P.cache);
  double *win = reinterpret_cast<double *>(res_sm + L.win);
  double *s_r = reinterpret_cast<double *>(res_sm + L.vec);
  double *s_ad = s_r + Q.own, *s_x = s_ad + Q.own;
  int2 *s_off = reinterpret_cast<int2 *>(res_sm + L.off);
  unsigned char *s_deg = res_sm + L.deg;
  C *s_c = reinterpret_cast<C *>(res_sm + L.ccoef);
  I *s_i = reinterpret_cast<I *>(res_sm + L.cidx);
  const C *gc;
  const I *gi;
  if constexpr (STO == 3) {
    gc = P.S.sg_c;
    gi = P.li;
  } else {
    gc = P.S.rec_c;
    gi = reinterpret_cast<const unsigned *>(P.rli);
  }
  Comm<COM> M;
  comm_init(M, P, V, res_sm + L.red, res_sm + L.box);
  res_setup<C, I, 1>(Q, p, P.S.meta, 0, P.S.rec_off, gc, gi, P.cache, s_off, s_deg, s_c, s_i);
  if constexpr (CL) cluster_sync();  // every block's mbarriers are set up
  const bool vs = CL || P.nvec >= 2;
  const unsigned long long pol_keep = l2_policy(false), pol_stream = l2_policy(true);
  Ranges N;
  N.init(Q, p);
  Halo<double, CL> H;
  const double *hsrc = CL ? s_r : P.r;
  H.init(Q, p, hsrc);
  double s[2], red;

  // f(step, virtual block of the block, local row, node, has): the thread's
  // rows, whole warps (lanes past the block's last row have has = false)
  auto steps = [&](auto f) {
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
      const int hi = N.hi(v);
      int k = v * R, a = v * R * TP + t;
#pragma unroll 1
      for (int i = N.lo(v); i - lane < hi; i += RES_T, ++k, a += TP) f(k, v, a, i, i < hi);
    }
  };
  auto rows = [&](auto f) {
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
      const int hi = N.hi(v);
      int a = v * R * TP + t;
#pragma unroll 1
      for (int i = N.lo(v); i < hi; i += RES_T, a += TP) f(v, a, i);
    }
  };
  auto dacc = [&](int v, double a, double c) {
    const double m = mul(a, c);
    if (CL || v == 0) s[0] = add(s[0], m); else s[1] = add(s[1], m);
  };
  auto put_r = [&](int a, int i, double v) {
    if (vs) s_r[a] = v;
    if (!CL) __stcg(P.r + i, v);
  };
  auto get_x = [&](int a, int i) { return CL ? s_x[a] : P.x[i]; };
  auto finish = [&](int status, int m, double rmrm, double xl, int relat) {
    rows([&](int, int a, int i) {
      const double v = get_x(a, i);
      P.x[i] = P.dsc ? mul(v, P.dsc[i]) : v;  // solve.f:637-641: X = X*D
    });
    if (p == 0 && t == 0) {
      set_status(P.ctl, status);
      P.ctl->nit = m;
      P.ctl->relres = __dsqrt_rn(__ddiv_rn(rmrm, xl));
      P.ctl->relat = relat;
    }
  };

  auto solve = [&]() {
    // XL = P_DOTS(B,B) (gracjg.F:189)
    s[0] = s[1] = 0.0;
    rows([&](int v, int a, int i) {
      dacc(v, P.b[i], P.b[i]);
      if constexpr (CL) s_x[a] = P.x[i];
    });
    double xl;
    {
      double got;
      if (!cold_reduce<COM, double>(M, s[0], s[1], &got)) return;
      M.done();
      xl = got;
    }
    int relat = 1, m = 0, phase = 0, status = ST_OK;
    double rmrm = 0.0, rmgm = 0.0, beta = 0.0;
    if (__dsqrt_rn(xl) < 1.0e-15) {  // gracjg.F:194-202: X = 0
      rows([&](int, int a, int i) {
        if constexpr (CL) s_x[a] = 0.0;
        else P.x[i] = 0.0;
      });
      finish(ST_OK, 0, 0.0, 1.0, 0);
      return;
    }
    if (xl < 1.0) { xl = 1.0; relat = 0; }  // gracjg.F:204-209
    const double tol = mul(xl, mul(P.eps, P.eps));
    // X staged through the window for the first product
#pragma unroll 1
    for (int h = t; h < H.nh; h += TP) win[Q.own + h] = P.x[__ldg(Q.halo + H.h0 + h)];
    rows([&](int, int a, int i) { win[a] = P.x[i]; });

#pragma unroll 1
    for (;;) {
      // phase 0: R = A X - B, R.R (gracjg.F:213-216)
      // phase 1: D = R, AD = A D, D.AD (:248-261)
      // phase 2: D = R + BETA D (:361) in the whole window (the halo's by the
      //          same operations as its owner's), AD = A D (:376), D.AD (:382)
      if (phase) {
        const bool first = phase == 1;
        H.each(Q, hsrc, [&](int h, double v) {
          win[Q.own + h] = first ? v : add(v, mul(beta, win[Q.own + h]));
        });
        rows([&](int, int a, int i) {
          const double v = vs ? s_r[a] : P.r[i];
          win[a] = first ? v : add(v, mul(beta, win[a]));
        });
      }
      __syncthreads();
      s[0] = s[1] = 0.0;
      steps([&](int k, int v, int a, int i, bool has) {
        const double d0 = has ? win[a] : 0.0;
        // the leading steps' slots stay in L2 (keep), the others stream through it
        const double acc =
            res_row<ROW>(has ? td_term(P.td, d0, P.da, i) : 0.0, s_off[a >> 5], s_deg[a], gc, gi,
                         k < P.keep ? pol_keep : pol_stream, s_c, s_i, win);
        if (!has) return;
        if (phase == 0) {
          const double r0 = sub(acc, P.b[i]);
          put_r(a, i, r0);
          dacc(v, r0, r0);
          return;
        }
        if (vs) s_ad[a] = acc;
        else P.ad[i] = acc;
        dacc(v, d0, acc);
      });
      // the first product's residual is published (the counter always does;
      // one reduction for every phase, as a call here costs the loop registers)
      if constexpr (COM == COM_CNT) {
        M.template send<true>(s);
        if (!M.template wait<true>(red)) return;
      } else if (phase == 0) {
        double got;
        if (!cold_reduce<COM, double>(M, s[0], s[1], &got)) return;
        M.done();
        red = got;
      } else {
        M.template send<false>(s);
        if (!M.template wait<false>(red)) return;
      }
      if (phase == 0) {
        rmrm = rmgm = red;
        if (isnan(rmrm)) { status = ST_NAN; break; }
        if (rmrm < mul(mul(P.eps, P.eps), xl)) break;
        phase = 1;
        continue;
      }
      if (!(red > 0.0)) { status = isnan(red) ? ST_NAN : ST_BREAKDOWN; break; }
      const double ro = __ddiv_rn(rmgm, red);  // :261, :383 (RMDM = RMGM)
      const double nro = -ro;
      const bool stop = phase == 2 && m >= P.nitmax;  // :406 -- last X update, unconverged
      phase = 2;
      if (!stop) {
        // R = R - RO*AD (:290), RMRM = P_DOTS(R,R) (:295)
        ++m;
        s[0] = s[1] = 0.0;
        rows([&](int v, int a, int i) {
          const double ri = add(vs ? s_r[a] : P.r[i], mul(nro, vs ? s_ad[a] : P.ad[i]));
          put_r(a, i, ri);
          dacc(v, ri, ri);
        });
        M.template send<true>(s);
      }
      // X = X - RO*D (:268 / :387) while the partial sums travel
      if constexpr (CL) {
        rows([&](int, int a, int) { s_x[a] = add(s_x[a], mul(nro, win[a])); });
      } else {
#pragma unroll 1
        for (int v = 0; v < V; ++v) {
          const int hi = N.hi(v);
          const double *wa = win + (size_t)v * R * TP + t;
          int i = N.lo(v);
#pragma unroll 1
          for (; i + 3 * RES_T < hi; i += 4 * RES_T, wa += 4 * RES_T) {
            double xv[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) xv[q] = P.x[i + q * RES_T];
#pragma unroll
            for (int q = 0; q < 4; ++q) P.x[i + q * RES_T] = add(xv[q], mul(nro, wa[q * RES_T]));
          }
#pragma unroll 1
          for (; i < hi; i += RES_T, wa += RES_T) P.x[i] = add(P.x[i], mul(nro, *wa));
        }
      }
      if (stop) { status = m; break; }
      if (!M.template wait<true>(red)) return;
      const double rm1gm1 = rmgm;
      rmrm = red;
      rmgm = rmrm;
      if (isnan(rmrm)) { status = ST_NAN; break; }
      if (rmrm <= tol) break;                 // :303
      beta = __ddiv_rn(rmgm, rm1gm1);         // :357
    }
    finish(status, m, rmrm, xl, relat);
  };
  solve();
  if constexpr (CL) cluster_sync();  // nobody leaves while another may reach its memory
}

// ---------------------------------------------------------------------------
// CGSTAB (cgstab.f:95-200), statement for statement k_cgstab, in the grid
// form with one tree block per physical block.  Q, S, R and V of the block's
// nodes and of its halo are in shared memory: the halo's copies follow by
// their owners' operations from one value per product (V, then T), where
// k_cgstab gathered three vectors per neighbour for A Q and two for A S.
// Bound: three grid reductions and two products (100k nodes 37.4 -> 27.0 us
// per iteration, 300k 29.8 -> 25.5).
// ---------------------------------------------------------------------------
template <int STO, bool COMP>
__global__ void __launch_bounds__(RES_T, 1) k_cgstab_res(const __grid_constant__ ResP P) {
  using ROW = typename std::conditional<STO == 3, SegRow, RecRow>::type;
  using C = typename ROW::C;
  using I = typename ROW::I;
  extern __shared__ __align__(16) unsigned char res_sm[];
  const ResPart &Q = P.Q;
  const int t = threadIdx.x, TP = RES_T, lane = t & 31, p = blockIdx.x;
  const ResLayout L = res_layout(Q.own, P.halo_max, Q.G, false, 32, 0, sizeof(C), sizeof(I),
                                 P.cache);
  const int W = Q.own + P.halo_max;
  double *wq = reinterpret_cast<double *>(res_sm + L.win), *ws = wq + W, *wr = ws + W, *wv = wr + W;
  int2 *s_off = reinterpret_cast<int2 *>(res_sm + L.off);
  unsigned char *s_deg = res_sm + L.deg;
  C *s_c = reinterpret_cast<C *>(res_sm + L.ccoef);
  I *s_i = reinterpret_cast<I *>(res_sm + L.cidx);
  const C *gc;
  const I *gi;
  if constexpr (STO == 3) {
    gc = P.S.sg_c;
    gi = P.li;
  } else {
    gc = P.S.rec_c;
    gi = reinterpret_cast<const unsigned *>(P.rli);
  }
  res_setup<C, I, 1>(Q, p, P.S.meta, 0, P.S.rec_off, gc, gi, P.cache, s_off, s_deg, s_c, s_i);
  const unsigned long long pol_keep = l2_policy(false), pol_stream = l2_policy(true);
  const int lo = (int)blk_lo(p, Q.n, Q.G) + t, hi = (int)blk_lo(p + 1, Q.n, Q.G);
  const int h0 = Q.halo_off[p], nh = Q.halo_off[p + 1] - h0;
  DotAcc<COMP, 2> sd;
  double rd[2];
  int nbar = 0;

  auto rows = [&](auto f) {
    int a = t;
#pragma unroll 1
    for (int i = lo; i < hi; i += RES_T, a += TP) f(a, i);
  };
  // f(window index, node) over the halo
  auto halo = [&](auto f) {
#pragma unroll 1
    for (int h = t; h < nh; h += TP) f(Q.own + h, __ldg(Q.halo + h0 + h));
  };
  auto finish = [&](int status, int m, double rmrm, double xl, int relat) {
    if (P.dsc) rows([&](int, int i) { P.x[i] = mul(P.x[i], P.dsc[i]); });  // solve.f:637-641
    if (p == 0 && t == 0) {
      set_status(P.ctl, status);
      P.ctl->nit = m;
      P.ctl->relres = __dsqrt_rn(__ddiv_rn(rmrm, xl));
      P.ctl->relat = relat;
    }
  };

  // XL (:105-111); SQRT(XL) < RMIN: X = 0 (:112-116)
  sd.zero();
  rows([&](int, int i) { sd.acc(0, P.b[i], P.b[i]); });
  if (!dred<COMP, 2>(P.ctl, P.part, P.timeout_ns, nbar, sd, rd)) return;
  double xl = rd[0];
  int relat = 1;
  if (xl < 1.0) { xl = 1.0; relat = 0; }
  if (__dsqrt_rn(xl) < 1.0e-15) {
    rows([&](int, int i) { P.x[i] = 0.0; });
    finish(ST_OK, 0, 0.0, xl, relat);
    return;
  }
  const double tol = mul(xl, mul(P.eps, P.eps));
  rows([&](int a, int i) { wq[a] = P.x[i]; });
  halo([&](int a, int j) { wq[a] = P.x[j]; });
  double rmrm = 0.0, beta1 = 0.0, alfa = 1.0, beta = 1.0, omeg1 = 1.0;
  int m = 0, phase = 0;
#pragma unroll 1
  for (;;) {
    // phase 0: R = B - A X (:120-123); 1: V = A Q, P.V (:163, :173);
    // phase 2: T = A S, T.S and T.T (:177, :186-187)
    const double *win = phase == 2 ? ws : wq;
    __syncthreads();
    sd.zero();
    {
      int a = t, k = 0;
#pragma unroll 1
      for (int i = lo; i - lane < hi; i += RES_T, a += TP, ++k) {
        const bool has = i < hi;
        const double d0 = has ? win[a] : 0.0;
        const double acc =
            res_row<ROW>(has ? td_term(P.td, d0, P.da, i) : 0.0, s_off[a >> 5], s_deg[a], gc, gi,
                         k < P.keep ? pol_keep : pol_stream, s_c, s_i, win);
        if (!has) continue;
        if (phase == 0) {
          const double r0 = sub(P.b[i], acc);
          wr[a] = r0;
          __stcg(P.r + i, r0);
          P.p0[i] = r0;
          sd.acc(0, r0, r0);
        } else if (phase == 1) {
          wv[a] = acc;
          __stcg(P.ad + i, acc);
          sd.acc(0, P.p0[i], acc);
        } else {
          __stcg(P.tv + i, acc);
          sd.acc(0, acc, d0);
          sd.acc(1, acc, acc);
        }
      }
    }
    if (!dred<COMP, 2>(P.ctl, P.part, P.timeout_ns, nbar, sd, rd)) return;
    if (phase == 1) {
      omeg1 = __ddiv_rn(beta1, rd[0]);  // :174
      const double nomeg1 = -omeg1;     // S = R - OMEG1 V (:176)
      halo([&](int a, int j) {
        const double v = __ldcg(P.ad + j);
        wv[a] = v;
        ws[a] = add(wr[a], mul(nomeg1, v));
      });
      rows([&](int a, int) { ws[a] = add(wr[a], mul(nomeg1, wv[a])); });
      phase = 2;
      continue;
    }
    if (phase == 2) {
      alfa = __ddiv_rn(rd[0], rd[1]);  // :188
      // X = X + OMEG1 Q + ALFA S (:190-191), R = S - ALFA T (:192), R.R and R.P
      const double nalfa = -alfa;
      sd.zero();
      rows([&](int a, int i) {
        const double si = ws[a];
        P.x[i] = add(add(P.x[i], mul(omeg1, wq[a])), mul(alfa, si));
        const double ri = add(si, mul(nalfa, __ldcg(P.tv + i)));
        wr[a] = ri;
        sd.acc(0, ri, ri);
        sd.acc(1, ri, P.p0[i]);
      });
      halo([&](int a, int j) { wr[a] = add(ws[a], mul(nalfa, __ldcg(P.tv + j))); });
      if (!dred<COMP, 2>(P.ctl, P.part, P.timeout_ns, nbar, sd, rd)) return;
      rmrm = rd[0];
      beta1 = rd[1];
      if (isnan(rmrm)) { finish(ST_NAN, m, rmrm, xl, relat); return; }
      if (rmrm <= tol) { finish(ST_OK, m, rmrm, xl, relat); return; }  // :194
      if (m >= P.nitmax) { finish(m, m, rmrm, xl, relat); return; }
    } else {
      rmrm = rd[0];
      if (isnan(rmrm)) { finish(ST_NAN, 0, rmrm, xl, relat); return; }
      if (rmrm < mul(mul(P.eps, P.eps), xl)) { finish(ST_OK, 0, rmrm, xl, relat); return; }
      beta1 = rmrm;  // R.P with P a copy of R: the same products and sum
      // V = Q = 0 (:144-147)
      rows([&](int a, int) { wq[a] = wv[a] = 0.0; });
      halo([&](int a, int j) {
        wq[a] = wv[a] = 0.0;
        wr[a] = __ldcg(P.r + j);
      });
    }
    ++m;
    const double omeg2 = __ddiv_rn(mul(omeg1, beta1), beta);  // :156
    const double omeg = __ddiv_rn(omeg2, alfa);
    beta = beta1;
    const double nomeg2 = -omeg2;
    // Q = R + OMEG Q - OMEG2 V (:161-162)
    rows([&](int a, int) { wq[a] = add(add(wr[a], mul(omeg, wq[a])), mul(nomeg2, wv[a])); });
    halo([&](int a, int) { wq[a] = add(add(wr[a], mul(omeg, wq[a])), mul(nomeg2, wv[a])); });
    phase = 1;
  }
}

// True residual of the mixed solve, r = b - A x in binary64, r32 = (float)r
// (to shared memory in the cluster form, else to ri; VS: both), with the
// thread's partial sums of r.r in both precisions.
struct ResidualSums {
  double d0, d1;
  float f0, f1;
};
template <int STO, bool CL, bool VS>
__device__ __noinline__ ResidualSums mixed_residual(const ResP &P, float *s_r) {
  Ranges N;
  N.init(P.Q, blockIdx.x);
  ResidualSums sum = {0.0, 0.0, 0.0f, 0.0f};
  const int V = CL ? 1 : P.Q.V, TP = blockDim.x;
#pragma unroll 1
  for (int v = 0; v < V; ++v) {
    const int hi = N.hi(v);
    int a = v * P.Q.R * TP + threadIdx.x;
    double d = 0.0;
    float f = 0.0f;
#pragma unroll 1
    for (int i = N.lo(v); i < hi; i += RES_T, a += TP) {
      double a0 = td_term(P.td, __ldcg(P.x + i), P.da, i), a1 = 0.0;
      op_row2<STO>(i, i, false, a0, a1, P.S, [&](int j) { return __ldcg(P.x + j); });
      const double r0 = sub(P.b[i], a0);
      d = add(d, mul(r0, r0));
      const float q0 = (float)r0;
      if (VS) s_r[a] = q0;
      if (!CL) __stcg(P.ri + i, q0);
      f = add(f, mul(q0, q0));
    }
    if (v == 0) {
      sum.d0 = d;
      sum.f0 = f;
    } else {
      sum.d1 = d;
      sum.f1 = f;
    }
  }
  return sum;
}

// ---------------------------------------------------------------------------
// Mixed precision, statement for statement k_mixed.  VS: r, q and z of the
// own rows and their row sums in shared memory (always in the cluster form);
// else in global memory.  SH = 0: local indices as byte offsets.
// Bound: reductions (5.2 of 12.7 us per iteration at 1.0M nodes; k_mixed 16.4)
// and the latency of the slots that are not in shared memory; at 4.0M nodes
// HBM, about 200 MB per iteration (78 -> 53 us).
// ---------------------------------------------------------------------------
template <int STO, int COM, bool VS, int SH, int MT>
__global__ void __launch_bounds__(MT, 1) k_mixed_res(const __grid_constant__ ResP P) {
  constexpr bool CL = COM == COM_CL;
  extern __shared__ __align__(16) unsigned char res_sm[];
  const ResPart &Q = P.Q;
  const int t = threadIdx.x, TP = blockDim.x, lane = t & 31;
  const int p = blockIdx.x, V = CL ? 1 : Q.V, R = Q.R;
  const ResLayout L = res_layout(Q.own, P.halo_max, Q.G, CL, 4, P.nvec, 4, 2, P.cache);
  float *win = reinterpret_cast<float *>(res_sm + L.win);
  float *s_r = reinterpret_cast<float *>(res_sm + L.vec);
  float *s_q = s_r + Q.own, *s_z = s_q + Q.own, *s_s = s_z + Q.own;
  int2 *s_off = reinterpret_cast<int2 *>(res_sm + L.off);
  unsigned char *s_deg = res_sm + L.deg;
  float2 *s_c = reinterpret_cast<float2 *>(res_sm + L.ccoef);
  unsigned *s_i = reinterpret_cast<unsigned *>(res_sm + L.cidx);
  const float2 *gc = reinterpret_cast<const float2 *>(P.S.seg_c);
  const unsigned *gi = reinterpret_cast<const unsigned *>(P.li);
  Comm<COM> M;
  comm_init(M, P, V, res_sm + L.red, res_sm + L.box);
  res_setup<float2, unsigned, 2>(Q, p, P.S.meta, 16, P.S.seg_off, gc, gi, P.cache, s_off, s_deg,
                                 s_c, s_i);
  if constexpr (CL) cluster_sync();
  const float *hsrc = CL ? s_r : P.ri;

  // f(v, local row, node) over the thread's rows
  auto rows_of = [&](const Ranges &N, auto f) {
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
      const int hi = N.hi(v);
      int a = v * R * TP + t;
#pragma unroll 1
      for (int i = N.lo(v); i < hi; i += RES_T, a += TP) f(v, a, i);
    }
  };
  float sf[2], rho = 0.0f;
  int inner = 0, outer = 0;
  auto acc32 = [&](int v, float c) {
    if (CL || v == 0) sf[0] = add(sf[0], c); else sf[1] = add(sf[1], c);
  };
  // ||D.B||^2, the outer tolerance and the last true residual: shared memory,
  // as registers are what this kernel runs out of (thread 0 writes them)
  double *cold = M.sh->cold;
  auto rows_once = [&](auto f) {
    Ranges N;
    N.init(Q, p);
    rows_of(N, f);
  };
  auto finish = [&](int status, double rr, double xl) {
    if (P.dsc) rows_once([&](int, int, int i) { P.x[i] = mul(P.x[i], P.dsc[i]); });
    if (p == 0 && t == 0) {
      set_status(P.ctl, status);
      P.ctl->nit = inner;
      P.ctl->outer = outer;
      P.ctl->relres = __dsqrt_rn(__ddiv_rn(rr, xl));
    }
  };

  auto solve = [&]() {
    double xl;
    {
      double sd[2] = {0.0, 0.0}, got;
      rows_once([&](int v, int a, int i) {
        const double m = mul(P.b[i], P.b[i]);
        if (v == 0) sd[0] = add(sd[0], m); else sd[1] = add(sd[1], m);
        if constexpr (VS) {
          s_s[a] = P.S.s32[i];
          s_z[a] = 0.0f;
        } else {
          P.z[i] = 0.0f;
        }
      });
      if (!cold_reduce<COM, double>(M, sd[0], sd[1], &got)) return;
      M.done();
      xl = got;
    }
    if (__dsqrt_rn(xl) < 1.0e-15) {
      rows_once([&](int, int, int i) { P.x[i] = 0.0; });
      finish(ST_OK, 0.0, 1.0);
      return;
    }
    if (xl < 1.0) xl = 1.0;
    if (t == 0) {
      cold[0] = xl;
      cold[1] = mul(xl, mul(P.outer_tol, P.outer_tol));
    }
    const float itol2 = (float)mul(P.inner_tol, P.inner_tol);
    float rmax = 0.0f, beta = 0.0f, rho_rec = 0.0f, rho_old = 0.0f;
    bool start = true, last = false;
#pragma unroll 1
    for (;;) {
      // the true residual, then CG iterations up to the next update.  Nothing
      // but a few scalars lives across these calls: values held over them
      // would be spilled, and read back inside the iteration.
      double got64;
      float got32;
      const ResidualSums sum = mixed_residual<STO, CL, VS>(P, s_r);
      if (!cold_reduce<COM, double>(M, sum.d0, sum.d1, &got64)) return;
      M.done();
      if (!cold_reduce<COM, float>(M, sum.f0, sum.f1, &got32)) return;
      M.done();
      const double rr = got64;
      rho = got32;
      if (t == 0) cold[2] = rr;
      if (!start) ++outer;
      if (isnan(rr)) { finish(ST_NAN, rr, cold[0]); return; }
      if (rr <= cold[1]) { finish(ST_OK, rr, cold[0]); return; }
      if (!start && (last || outer >= P.max_outer)) { finish(inner, rr, cold[0]); return; }
      rmax = rho;
      const unsigned long long pol = l2_policy(P.S.cs_seg != 0);
      Ranges N;
      N.init(Q, p);
      Halo<float, CL> H;
      H.init(Q, p, hsrc);
      auto rows = [&](auto f) { rows_of(N, f); };
#pragma unroll 1
      for (;;) {
      if (!start) beta = __fdiv_rn(rho_rec, rho_old);
      // p = r + beta p in the whole window; q = A32 p; p.q
      H.each(Q, hsrc, [&](int h, float rv) {
        win[Q.own + h] = start ? rv : add(rv, mul(beta, win[Q.own + h]));
      });
      if constexpr (VS) {
        rows([&](int, int a, int) {
          win[a] = start ? s_r[a] : add(s_r[a], mul(beta, win[a]));
        });
      } else {
#pragma unroll 1
        for (int v = 0; v < V; ++v) {
          const int hi = N.hi(v);
          int i = N.lo(v);
          float *wa = win + (size_t)v * R * TP + t;
#pragma unroll 1
          for (; i + 3 * RES_T < hi; i += 4 * RES_T, wa += 4 * RES_T) {
            float rv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) rv[c] = P.ri[i + c * RES_T];
#pragma unroll
            for (int c = 0; c < 4; ++c)
              wa[c * RES_T] = start ? rv[c] : add(rv[c], mul(beta, wa[c * RES_T]));
          }
#pragma unroll 1
          for (; i < hi; i += RES_T, wa += RES_T)
            *wa = start ? P.ri[i] : add(P.ri[i], mul(beta, *wa));
        }
      }
      __syncthreads();
      start = false;
      sf[0] = sf[1] = 0.0f;
#pragma unroll 1
      for (int v = 0; v < V; ++v) {
        const int hi = N.hi(v);
        int i = N.lo(v), a = v * R * TP + t;
        if (i - lane >= hi) continue;
        auto use = [&](const Pair3 &A, float sm) {
          const float y0 = i < hi ? win[a] : 0.0f;
          const float a0 = pair_row<SH>(A, mul(y0, sm), y0, s_off[a >> 5], s_deg[a], gc, gi, pol,
                                        s_c, s_i, win);
          if (i >= hi) return;
          if constexpr (VS) s_q[a] = a0;
          else P.q[i] = a0;
          acc32(v, mul(y0, a0));
        };
        Pair3 A;
        if constexpr (VS) {
#pragma unroll 1
          for (; i - lane < hi; i += RES_T, a += TP) {
            pair_load(A, s_off[a >> 5], gc, gi, pol, s_c, s_i);
            use(A, s_s[a]);
          }
        } else {
          // streamed from HBM: the next step's slots are loaded before this
          // one's are used
          Pair3 B;
          float sa, sb = 0.0f;
          pair_load(A, s_off[a >> 5], gc, gi, pol, s_c, s_i);
          sa = i < hi ? ld_pol(P.S.s32 + i, pol) : 0.0f;
#pragma unroll 1
          for (;;) {
            const bool more = i + RES_T - lane < hi;
            if (more) {
              pair_load(B, s_off[(a + TP) >> 5], gc, gi, pol, s_c, s_i);
              sb = i + RES_T < hi ? ld_pol(P.S.s32 + i + RES_T, pol) : 0.0f;
            }
            use(A, sa);
            if (!more) break;
            A = B;
            sa = sb;
            i += RES_T;
            a += TP;
          }
        }
      }
      float pq;
      M.template send<false>(sf);
      if (!M.template wait<false>(pq)) return;
      if (!(pq > 0.0f)) {
        finish(isnan(pq) ? ST_NAN : ST_BREAKDOWN, cold[2], cold[0]);
        return;
      }
      const float alpha = __fdiv_rn(rho, pq);
      // r = r - alpha q, r.r; z = z + alpha p while the partial sums travel
      sf[0] = sf[1] = 0.0f;
      if constexpr (VS) {
        rows([&](int v, int a, int i) {
          const float rv = sub(s_r[a], mul(alpha, s_q[a]));
          s_r[a] = rv;
          if (!CL) __stcg(P.ri + i, rv);
          acc32(v, mul(rv, rv));
        });
      } else {
#pragma unroll 1
        for (int v = 0; v < V; ++v) {
          const int hi = N.hi(v);
          int i = N.lo(v);
#pragma unroll 1
          for (; i + 3 * RES_T < hi; i += 4 * RES_T) {
            float rv[4], qv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              rv[c] = P.ri[i + c * RES_T];
              qv[c] = P.q[i + c * RES_T];
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              rv[c] = sub(rv[c], mul(alpha, qv[c]));
              __stcg(P.ri + i + c * RES_T, rv[c]);
              acc32(v, mul(rv[c], rv[c]));
            }
          }
#pragma unroll 1
          for (; i < hi; i += RES_T) {
            const float rv = sub(P.ri[i], mul(alpha, P.q[i]));
            __stcg(P.ri + i, rv);
            acc32(v, mul(rv, rv));
          }
        }
      }
      M.template send<true>(sf);
      if constexpr (VS) {
        rows([&](int, int a, int) { s_z[a] = add(s_z[a], mul(alpha, win[a])); });
      } else {
#pragma unroll 1
        for (int v = 0; v < V; ++v) {
          const int hi = N.hi(v);
          int i = N.lo(v);
          const float *wa = win + (size_t)v * R * TP + t;
#pragma unroll 1
          for (; i + 3 * RES_T < hi; i += 4 * RES_T, wa += 4 * RES_T) {
            float zv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) zv[c] = P.z[i + c * RES_T];
#pragma unroll
            for (int c = 0; c < 4; ++c)
              P.z[i + c * RES_T] = add(zv[c], mul(alpha, wa[c * RES_T]));
          }
#pragma unroll 1
          for (; i < hi; i += RES_T, wa += RES_T) P.z[i] = add(P.z[i], mul(alpha, *wa));
        }
      }
      rho_old = rho;
      if (!M.template wait<true>(rho_rec)) return;
      rho = rho_rec;
      ++inner;
      last = inner >= P.max_inner;
      if (last || rho_rec <= mul(itol2, rmax) || (double)rho_rec <= cold[1]) break;
      }
      // reliable update: x += z in binary64
      rows([&](int, int a, int i) {
        if constexpr (VS) {
          P.x[i] = add(P.x[i], (double)s_z[a]);
          s_z[a] = 0.0f;
        } else {
          P.x[i] = add(P.x[i], (double)P.z[i]);
          P.z[i] = 0.0f;
        }
      });
      if (CL) fence_gpu();  // x is read at neighbours through global memory
      float dummy;
      if (!cold_reduce<COM, float>(M, 0.0f, 0.0f, &dummy)) return;
      M.done();
      if (CL) fence_gpu();
    }
  };
  solve();
  if constexpr (CL) cluster_sync();
}

// ---------------------------------------------------------------------------
// Self-test of the bounded waits: one block of 1024 threads in a reduction
// that never completes, as if a warp (cluster form) or another block had
// stopped.  Every thread must come back with false, after the time limit and
// with the timeout recorded; ctl->nit counts them.  The cluster form makes a
// complete reduction first, ctl->relres is its sum.
// ---------------------------------------------------------------------------
template <int COM>
__global__ void __launch_bounds__(RES_T, 1) k_res_wait_test(const __grid_constant__ ResP P) {
  __shared__ RedShared red;
  __shared__ unsigned long long box[2 * 32];
  Comm<COM> M;
  comm_init(M, P, 1, reinterpret_cast<unsigned char *>(&red),
            reinterpret_cast<unsigned char *>(box));
  __syncthreads();
  const double one = 1.0;
  double sum = 0.0;
  if constexpr (COM == COM_CL) {
    M.template send<true>(&one);
    if (!M.template wait<true>(sum)) return;
    if (threadIdx.x == 0) P.ctl->relres = sum;
    if (threadIdx.x < RES_T - 32) M.template send<true>(&one);
    else M.done();
  } else {
    M.template send<true>(&one);
  }
  if (!M.template wait<true>(sum)) atomicAdd(&P.ctl->nit, 1);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
namespace {

// The kernel's limit of dynamic shared memory is state of the context, shared
// by every thread that launches the kernel: it is set to P.smem_limit, the
// same for every mesh, and never to what one launch needs, which another
// thread's launch might find too low (measured with three threads and two
// sizes in a loop: 72 of 20,000 launches refused).
template <class K>
cudaError_t launch(K k, bool cl, const ResP &P, size_t smem, cudaStream_t st) {
  cudaError_t e =
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, P.smem_limit);
  if (e != cudaSuccess) return e;
  if (cl && (e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) !=
                cudaSuccess)
    return e;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(P.Q.NP);
  c.blockDim = dim3(P.Q.TP);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at[1];
  if (cl) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = P.Q.NP;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  c.attrs = at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, P);
}

}  // namespace

cudaError_t res_launch_plan(bool fill, const PlanP &A, cudaStream_t st) {
  const size_t smem = 2 * sizeof(unsigned) * PLAN_W;
  cudaError_t e;
  if (fill) {
    e = cudaFuncSetAttribute(k_res_plan<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    k_res_plan<true><<<A.Q.NP, 1024, smem, st>>>(A);
  } else {
    e = cudaFuncSetAttribute(k_res_plan<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    k_res_plan<false><<<A.Q.NP, 1024, smem, st>>>(A);
  }
  return cudaGetLastError();
}

template <int STO>
static cudaError_t launch_cg(bool cl, const ResP &P, size_t smem, cudaStream_t st) {
  if (cl)
    return P.Q.TP <= RES_T / 2 ? launch(k_cg_res<STO, COM_CL, RES_T / 2>, cl, P, smem, st)
                               : launch(k_cg_res<STO, COM_CL, RES_T>, cl, P, smem, st);
  return P.Q.G <= RES_TAG ? launch(k_cg_res<STO, COM_TAG, RES_T>, cl, P, smem, st)
                          : launch(k_cg_res<STO, COM_CNT, RES_T>, cl, P, smem, st);
}

cudaError_t res_launch_cg(int sto, bool cl, const ResP &P, size_t smem, cudaStream_t st) {
  return sto == 3 ? launch_cg<3>(cl, P, smem, st) : launch_cg<1>(cl, P, smem, st);
}

cudaError_t res_launch_cgstab(int sto, bool comp, const ResP &P, size_t smem, cudaStream_t st) {
  if (sto == 3)
    return comp ? launch(k_cgstab_res<3, true>, false, P, smem, st)
                : launch(k_cgstab_res<3, false>, false, P, smem, st);
  return comp ? launch(k_cgstab_res<1, true>, false, P, smem, st)
              : launch(k_cgstab_res<1, false>, false, P, smem, st);
}

template <int STO, int COM>
static cudaError_t launch_mixed_grid(bool vs, int shift, const ResP &P, size_t smem,
                                     cudaStream_t st) {
  if (!vs) return launch(k_mixed_res<STO, COM, false, 2, RES_T>, false, P, smem, st);
  return shift ? launch(k_mixed_res<STO, COM, true, 2, RES_T>, false, P, smem, st)
               : launch(k_mixed_res<STO, COM, true, 0, RES_T>, false, P, smem, st);
}

template <int STO>
static cudaError_t launch_mixed(bool cl, bool vs, int shift, const ResP &P, size_t smem,
                                cudaStream_t st) {
  if (cl)
    return P.Q.TP <= RES_T / 2
               ? launch(k_mixed_res<STO, COM_CL, true, 0, RES_T / 2>, cl, P, smem, st)
               : launch(k_mixed_res<STO, COM_CL, true, 0, RES_T>, cl, P, smem, st);
  // (vectors in global memory: meshes of far more than RES_TAG blocks)
  return vs && P.Q.G <= RES_TAG ? launch_mixed_grid<STO, COM_TAG>(vs, shift, P, smem, st)
                                : launch_mixed_grid<STO, COM_CNT>(vs, shift, P, smem, st);
}

cudaError_t res_launch_mixed(int sto, bool cl, bool vs, int shift, const ResP &P, size_t smem,
                             cudaStream_t st) {
  return sto == 3 ? launch_mixed<3>(cl, vs, shift, P, smem, st)
                  : launch_mixed<1>(cl, vs, shift, P, smem, st);
}

cudaError_t res_wait_test(int form, Ctl *ctl, double *part, unsigned long long *box,
                          long long timeout_ns) {
  ResP P = {};
  P.Q.S = 1;
  P.Q.G = P.Q.NP = form == COM_CL ? 1 : 2;
  P.ctl = ctl;
  P.part = part;
  P.box = box;
  P.timeout_ns = timeout_ns;
  if (form == COM_CL) k_res_wait_test<COM_CL><<<1, RES_T>>>(P);
  else if (form == COM_TAG) k_res_wait_test<COM_TAG><<<1, RES_T>>>(P);
  else k_res_wait_test<COM_CNT><<<1, RES_T>>>(P);
  return cudaGetLastError();
}

cudaError_t res_smem_limit(int *bytes) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, k_cg_res<1, COM_CL, RES_T / 2>);
  *bytes = e == cudaSuccess ? a.maxDynamicSharedSizeBytes : 0;
  return e;
}

bool res_cluster_fits(int np, int tp, size_t smem) {
  auto k = k_cg_res<1, COM_CL, RES_T>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(np);
  c.blockDim = dim3(tp);
  c.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = np;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  c.attrs = at;
  c.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k, &c) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n >= 1;
}

}  // namespace bief
