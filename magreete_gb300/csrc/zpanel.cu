// Panel factorisation of the complex128 LU: m rows x 32 columns, partial
// pivoting (largest |re|+|im|, lowest row on ties).
//
// What bounds it: the FP64 pipe.  One FP64 instruction holds a warp for about
// 72 clocks whatever its independence from its neighbours (measured: 65 clocks
// dependent, 73 for 16 independent chains; 19 clocks per warp instruction and
// SM with every sub-partition busy), so the layout spreads a row over four
// threads and the panel over as many SMs as the exchange allows.
//
// Layout: thread (r, g) = (tid / 4, tid % 4) holds columns g, g + 4, ... of
// its row in registers, a[k] = column 4 (j + k) + g after j shifts, so that
// register indices stay compile-time constants.  Rows never move: a row keeps
// its LAPACK position in `pos`; the row chosen at column c takes position c and
// retires, the row that was there takes the chosen row's position, and
// every row is written to its position at the end.  Only the chosen row is
// therefore exchanged between CTAs.
//
// Exchange per column: every CTA publishes its candidate's key at once; one more
// warp per CTA gathers the keys and picks the same pivot everywhere.  The
// chosen row and its reciprocal follow as soon as they are ready (a cluster's
// chosen CTA sends them to the others; through global memory every CTA
// publishes its own and the chosen one is read).
// There is no fence, barrier or flag: every 64-bit word of a message carries the
// column's tag (zpanel_msg.cuh), so a reader that sees the tag has the data.
// Messages alternate by column parity; what a buffer held before never carries
// the current tag, however long its CTA had no row, and it is overwritten only by
// a CTA that has every key of the column in between, when nobody reads it any more.
//   CLUSTER: one thread-block cluster (at most 16 CTAs), messages in
//     distributed shared memory (tables cleared before a first cluster barrier);
//   otherwise records in global memory, cleared when a factorisation starts.
// The update of a column is split: the next column first, so that its keys go
// out; the other columns while the exchange is in flight.  The pivot's
// reciprocal is made by a warp of its own beside them.
// Every wait is bounded (MGT_ERR_TIMEOUT).
//
// The arithmetic per element (multiplier, then one complex multiply-subtract
// per column, in column order) is that of lu_panel_kernel: bit-identical factors.
#include <algorithm>

#include "zpanel.cuh"
#include "zpanel_msg.cuh"
#include "diag.cuh"

namespace mgt {
namespace zp {

constexpr int NB = kZNB;
constexpr int LD = NB + 1;
constexpr int kMaxCluster = 16;

// |re|+|im| as an ordered integer: bits + 1, 0 for a NaN
__device__ __forceinline__ unsigned long long pivot_key(double2 v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(cabs1(v));
  return u <= 0x7FF0000000000000ull ? u + 1ull : 0ull;
}

// Warp-wide choice: largest key, lowest position on ties.  Returns the lane
// that holds it (-1: no lane bids); key and pos become the winner's.
__device__ __forceinline__ int warp_choose(unsigned long long& key, int& pos) {
  const bool bids = pos != kNoPos;
  const unsigned hi = bids ? (unsigned)(key >> 32) : 0u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = bids && hi == mh ? (unsigned)key : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  const bool top = bids && hi == mh && (unsigned)key == ml;
  const unsigned mp = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : (unsigned)kNoPos);
  const unsigned who = __ballot_sync(0xffffffffu, top && (unsigned)pos == mp);
  key = ((unsigned long long)mh << 32) | ml;
  pos = (int)mp;
  return __ffs(who) - 1;
}

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Messages of 64-bit words that carry the column's tag.
using Word = unsigned long long;
__device__ __forceinline__ void encode(Word tag, double2 v, Word* w) {
  uint64_t q[3];
  pack_number(tag, (uint64_t)__double_as_longlong(v.x), (uint64_t)__double_as_longlong(v.y), q);
#pragma unroll
  for (int t = 0; t < 3; ++t) w[t] = q[t];
}
__device__ __forceinline__ double2 decode(const Word* w) {
  const uint64_t q[3] = {w[0], w[1], w[2]};
  uint64_t x, y;
  unpack_number(q, &x, &y);
  return make_double2(__longlong_as_double((long long)x), __longlong_as_double((long long)y));
}
__device__ __forceinline__ bool tagged(Word tag, const Word* w) {
  return has_tag(tag, w[0]) && has_tag(tag, w[1]) && has_tag(tag, w[2]);
}
// Row message, laid out so that a warp reads it in few sectors: per column the
// first two words, then the third ones, then the reciprocal's three words.
constexpr int kWordB = 2 * NB, kWordInv = 3 * NB, kMsgWords = 3 * NB + 4;

// words of a message in global memory
struct Mail {
  unsigned long long* g;
  __device__ void put(int i, unsigned long long v) const {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(g + i), "l"(v) : "memory");
  }
  __device__ void put2(int i, unsigned long long v, unsigned long long w) const {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(g + i), "l"(v), "l"(w) : "memory");
  }
  __device__ unsigned long long get(int i) const {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(g + i) : "memory");
    return v;
  }
  __device__ void get2(int i, unsigned long long& v, unsigned long long& w) const {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v), "=l"(w) : "l"(g + i) : "memory");
  }
};
// words stored into the shared memory of a CTA of the cluster
__device__ __forceinline__ void st_cluster1(uint32_t a, unsigned long long v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void st_cluster2(uint32_t a, unsigned long long v, unsigned long long w) {
  asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(a), "l"(v), "l"(w) : "memory");
}
// the CTA chosen at column c, as the exchange warp finds it (bounded; -1 on expiry)
__device__ __forceinline__ int wait_chosen(const volatile int* s, int c) {
  for (unsigned it = 0; it < kSpinLimit; ++it) {
    const int v = *s;
    if (v >> 8 == c + 1) return v & 255;
  }
  return -1;
}

// a[k] -= l U[4 k] for 1 <= k < live.  One piece of code per length: an FP64
// instruction that is predicated off still takes its 72 clocks.
template <int LIVE>
__device__ __forceinline__ void update_rest(double2* a, double2 l, const double2* U) {
#pragma unroll
  for (int k = 1; k < LIVE; ++k) cfms(a[k], l, U[4 * k]);
}

template <int ROWS>
struct Smem {
  static constexpr int WARPS = ROWS / 8;
  double2 sL[ROWS][LD];                            // finished columns (L, then the retired row's U part)
  double2 cand[NB];                                // the CTA's candidate row
  double2 U[2][NB];                                // the chosen row, by column parity
  double2 inv;                                     // 1 / pivot
  double2 pv[2][WARPS];                            // each warp's candidate pivot
  __align__(16) unsigned long long msg[2][kMsgWords];   // (cluster) this CTA's row message
  unsigned long long keys[2][kMaxCluster][2];      // (cluster) every CTA's key message
  unsigned long long key[2][WARPS];
  int pos[2][WARPS];
  int fin[ROWS];                                   // final position of each row
  int piv[NB];
  int slot_pos[2 * NB], slot_src[2 * NB];
  int nslot, p, nz, fail;
  int chosen[2];                                   // (cluster) column + 1 and rank of the chosen CTA
};

template <int ROWS, bool CLUSTER>
__global__ void __launch_bounds__(4 * ROWS + 64, 1)
zpanel_kernel(double2* __restrict__ A, int64_t lda, int m, int w, int j0, int rows_per_cta,
              int32_t* __restrict__ perm, ZPanelWs ws) {
  early_start();
  constexpr int WARPS = ROWS / 8, THREADS = 4 * ROWS + 64, KR = NB / 4;
  extern __shared__ __align__(16) unsigned char zp_smem[];
  Smem<ROWS>& S = *reinterpret_cast<Smem<ROWS>*>(zp_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool worker = warp < WARPS;              // warp WARPS: exchange, warp WARPS + 1: reciprocals
  const int r = worker ? tid >> 2 : 0, g = tid & 3;
  const int G = gridDim.x, bid = blockIdx.x;     // CLUSTER: one cluster spans the grid, rank = blockIdx.x
  const int r0 = bid * rows_per_cta, nr = max(0, min(m, r0 + rows_per_cta) - r0);

  for (int i = tid; i < ROWS * NB; i += THREADS) {
    const int rr = i / NB, k = i % NB;
    S.sL[rr][k] = (rr < nr && k < w) ? A[(int64_t)(r0 + rr) * lda + k] : make_double2(0.0, 0.0);
  }
  if (tid == 0) S.fail = S.chosen[0] = S.chosen[1] = 0;
  if constexpr (CLUSTER) {
    for (int i = tid; i < 2 * kMsgWords; i += THREADS) (&S.msg[0][0])[i] = 0ull;
    for (int i = tid; i < 4 * kMaxCluster; i += THREADS) (&S.keys[0][0][0])[i] = 0ull;
    cluster_sync();
  } else {
    __syncthreads();
  }
  double2 a[KR];
#pragma unroll
  for (int k = 0; k < KR; ++k) a[k] = S.sL[r][4 * k + g];
  bool active = worker && r < nr;
  int pos = active ? r0 + r : kNoPos;
  auto keys_of = [&](int buf) { return ws.records + (size_t)buf * ws.max_ctas * 2; };
  auto msg_of = [&](int buf, int q) {
    return ws.records + (size_t)ws.max_ctas * 4 + ((size_t)buf * ws.max_ctas + q) * kMsgWords;
  };

  int j = 0;                                     // shifts of a[]: a[k] is column 4 (j + k) + g
  double2 l = make_double2(0.0, 0.0);            // multiplier of the column before
  bool pending = false;                          // its columns beyond the next one still to be updated
  for (int c = 0; c < w; ++c) {
    const int buf = c & 1, u = c & 3, live = KR - j;
    const unsigned long long tag = column_tag(j0 + c);
    // ---- the warps' candidates
    int who = -1;
    if (worker) {
      unsigned long long key = 0;
      int bpos = kNoPos;
      if (active && g == u) {
        key = pivot_key(a[0]);
        bpos = pos;
      }
      who = warp_choose(key, bpos);
      if (lane == 0) {
        S.key[buf][warp] = key;
        S.pos[buf][warp] = bpos;
      }
      if (lane == who) S.pv[buf][warp] = a[0];
    }
    __syncthreads();
    // ---- the CTA's candidate, known to every warp
    unsigned long long ckey = 0;
    int cpos = kNoPos;
    if (lane < WARPS) {
      ckey = S.key[buf][lane];
      cpos = S.pos[buf][lane];
    }
    const int cw = warp_choose(ckey, cpos);
    Mail mine;                                   // this CTA's row message in global memory
    if constexpr (!CLUSTER) mine.g = msg_of(buf, bid);
    if (worker) {
      // ---- the rest of the column before, then the candidate's row goes out
      if (pending && active) {
        const double2* U = &S.U[buf ^ 1][4 * j + g];
        switch (live) {
          case 8: update_rest<8>(a, l, U); break;
          case 7: update_rest<7>(a, l, U); break;
          case 6: update_rest<6>(a, l, U); break;
          case 5: update_rest<5>(a, l, U); break;
          case 4: update_rest<4>(a, l, U); break;
          case 3: update_rest<3>(a, l, U); break;
          case 2: update_rest<2>(a, l, U); break;
          default: break;
        }
      }
      if (warp == cw) {
        if ((lane >> 2) == (who >> 2)) {
#pragma unroll
          for (int k = 0; k < KR; ++k)
            if (k < live) S.cand[4 * (j + k) + g] = a[k];
        }
        __syncwarp();
        unsigned long long q[3];
        encode(tag, (lane >= c && lane < w) ? S.cand[lane] : make_double2(0.0, 0.0), q);
        if constexpr (CLUSTER) {
          if (wait_chosen(&S.chosen[buf], c) == bid)
            for (int t = 0; t < G; ++t) {
              const uint32_t to = map_rank(saddr(&S.msg[buf][0]), (uint32_t)t);
              st_cluster2(to + 16u * (uint32_t)lane, q[0], q[1]);
              st_cluster1(to + 8u * (uint32_t)(kWordB + lane), q[2]);
            }
        } else {
          mine.put2(2 * lane, q[0], q[1]);
          mine.put(kWordB + lane, q[2]);
        }
      }
    } else if (warp == WARPS + 1) {
      if (cw >= 0) {
        const double2 pv = S.pv[buf][cw];
        unsigned long long q[3];
        encode(tag, (pv.x != 0 || pv.y != 0) ? crecip(pv) : make_double2(0.0, 0.0), q);
        if constexpr (CLUSTER) {
          if (wait_chosen(&S.chosen[buf], c) == bid && lane < G) {
            const uint32_t to = map_rank(saddr(&S.msg[buf][kWordInv]), (uint32_t)lane);
#pragma unroll
            for (int t = 0; t < 3; ++t) st_cluster1(to + 8u * t, q[t]);
          }
        } else if (lane == 0) {
#pragma unroll
          for (int t = 0; t < 3; ++t) mine.put(kWordInv + t, q[t]);
        }
      }
    } else {
      // ---- exchange warp: publish the key, gather all keys, fetch the chosen row
      uint64_t kw[2];
      pack_key(tag, ckey, cpos, kw);
      if constexpr (CLUSTER) {
        if (lane < G) {
          st_cluster2(map_rank(saddr(&S.keys[buf][bid][0]), (uint32_t)lane), kw[0], kw[1]);
        }
      } else if (lane == 0) {
        Mail to;
        to.g = keys_of(buf);
        to.put2(2 * bid, kw[0], kw[1]);
      }
      unsigned seen = 0, it = 0;
      const int per = (G + 31) / 32;
      const unsigned want = (1u << per) - 1u;
      unsigned long long bk = 0;
      int bp = kNoPos, bb = 0;
      bool ok = true;
      while (true) {
        for (int t = 0; t < per; ++t) {
          const int q = lane + 32 * t;
          if (seen & (1u << t)) continue;
          if (q >= G) { seen |= 1u << t; continue; }
          unsigned long long h0, h1;
          if constexpr (CLUSTER) {
            volatile unsigned long long* from = &S.keys[buf][q][0];
            h0 = from[0];
            h1 = from[1];
          } else {
            Mail from;
            from.g = keys_of(buf);
            from.get2(2 * q, h0, h1);
          }
          if (!has_tag(tag, h0) || !has_tag(tag, h1)) continue;
          seen |= 1u << t;
          uint64_t k2;
          int p2;
          unpack_key(h0, h1, &k2, &p2);
          if (p2 != kNoPos && (bp == kNoPos || k2 > bk || (k2 == bk && p2 < bp))) { bk = k2; bp = p2; bb = q; }
        }
        if (__all_sync(0xffffffffu, seen == want)) break;
        if (++it > kSpinLimit) { ok = false; break; }
      }
      ok = __all_sync(0xffffffffu, ok);
      const int p = c;
      int chosen = p;
      double2 uv = make_double2(0.0, 0.0), iv = uv;
      if (ok) {
        const int rank_lane = warp_choose(bk, bp);
        chosen = bp;
        const int rank = __shfl_sync(0xffffffffu, bb, max(rank_lane, 0));
        unsigned long long q[3], v[3];
        it = 0;
        if constexpr (CLUSTER) {
          // the chosen CTA's row and reciprocal warps send them to every CTA: poll the local copy
          if (lane == 0) S.chosen[buf] = (c + 1) << 8 | rank;
          const volatile unsigned long long* from = &S.msg[buf][0];
          while (true) {
            q[0] = from[2 * lane];
            q[1] = from[2 * lane + 1];
            q[2] = from[kWordB + lane];
#pragma unroll
            for (int t = 0; t < 3; ++t) v[t] = from[kWordInv + t];
            if (__all_sync(0xffffffffu, tagged(tag, q) && tagged(tag, v))) break;
            if (++it > kSpinLimit) { ok = false; break; }
          }
        } else {
          Mail from;
          from.g = msg_of(buf, rank);
          while (true) {
            from.get2(2 * lane, q[0], q[1]);
            q[2] = from.get(kWordB + lane);
#pragma unroll
            for (int t = 0; t < 3; ++t) v[t] = from.get(kWordInv + t);
            if (__all_sync(0xffffffffu, tagged(tag, q) && tagged(tag, v))) break;
            if (++it > kSpinLimit) { ok = false; break; }
          }
        }
        uv = decode(q);
        iv = decode(v);
      }
      const double px = __shfl_sync(0xffffffffu, uv.x, c), py = __shfl_sync(0xffffffffu, uv.y, c);
      S.U[buf][lane] = uv;
      if (lane == 0) {
        const bool nz = px != 0 || py != 0;
        S.inv = iv;
        S.p = chosen;
        S.nz = nz;
        if (!ok) {
          S.fail = 1;
          atomicExch(ws.status, MGT_ERR_TIMEOUT);
        }
        if (bid == 0) {
          S.piv[c] = nz ? chosen : c;
          if (!nz && ws.status[1] == 0) ws.status[1] = j0 + c + 1;
        }
      }
    }
    __syncthreads();
    if (S.fail) break;
    const int p = S.p;
    const bool nz = S.nz;
    // ---- positions: the chosen row retires at c, the row at c moves to p
    if (active && pos == p) {
      active = false;
      pos = c;
#pragma unroll
      for (int k = 0; k < KR; ++k)
        if (k < live && 4 * (j + k) + g >= c) S.sL[r][4 * (j + k) + g] = a[k];
    } else if (active && pos == c) {
      pos = p;
    }
    // ---- multiplier, then the next column
    pending = false;
    if (worker && __any_sync(0xffffffffu, active)) {
      if (nz) {
        l = make_double2(0.0, 0.0);
        if (g == u) l = cmul(a[0], S.inv);
        l.x = __shfl_sync(0xffffffffu, l.x, (lane & ~3) | u);
        l.y = __shfl_sync(0xffffffffu, l.y, (lane & ~3) | u);
        if (active && g == u) S.sL[r][c] = l;
        pending = true;
      } else if (active && g == u) {
        S.sL[r][c] = a[0];
      }
    }
    if (u == 3) {
#pragma unroll
      for (int k = 0; k + 1 < KR; ++k) a[k] = a[k + 1];
      ++j;
    }
    if (pending && active && 4 * j + g < NB) cfms(a[0], l, S.U[buf][4 * j + g]);
  }
  if (worker && g == 0) S.fin[r] = pos;
  __syncthreads();
  if (!S.fail)
    for (int i = tid; i < nr * NB; i += THREADS) {
      const int rr = i / NB, k = i % NB;
      if (k < w) A[(int64_t)S.fin[rr] * lda + k] = S.sL[rr][k];
    }
  // ---- net interchanges of the panel: row slot_pos[q] holds what was at slot_src[q]
  if (bid == 0 && warp == 0 && !S.fail) {
    for (int s2 = lane; s2 < NB; s2 += 32) { S.slot_pos[s2] = s2; S.slot_src[s2] = s2; }
    if (lane == 0) S.nslot = NB;
    __syncwarp();
    for (int s2 = 0; s2 < w; ++s2) {
      const int pv = S.piv[s2];
      if (pv == s2) continue;
      int slot = -1;
      if (pv < NB) {
        slot = pv;
      } else {
        const int ns = S.nslot;
        const int q = NB + lane;
        const unsigned hit = __ballot_sync(0xffffffffu, q < ns && S.slot_pos[q] == pv);
        if (hit) slot = NB + __ffs(hit) - 1;
        if (slot < 0) {
          slot = ns;
          if (lane == 0) { S.slot_pos[ns] = pv; S.slot_src[ns] = pv; S.nslot = ns + 1; }
        }
      }
      __syncwarp();
      if (lane == 0) { const int t = S.slot_src[s2]; S.slot_src[s2] = S.slot_src[slot]; S.slot_src[slot] = t; }
      __syncwarp();
    }
    const int ns = S.nslot;
    for (int q = lane; q < ns; q += 32) ws.slots[q] = make_int2(S.slot_pos[q], S.slot_src[q]);
    if (lane == 0) *ws.nslot = ns;
    int32_t pv[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int q = lane + 32 * t;
      if (q < ns) pv[t] = perm[j0 + S.slot_src[q]];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int q = lane + 32 * t;
      if (q < ns) perm[j0 + S.slot_pos[q]] = pv[t];
    }
  }
  if constexpr (CLUSTER) {
    __syncwarp();
    cluster_sync();   // no CTA leaves while another may still read its shared memory
  }
}

// largest cluster (16, 8 or 0 CTAs) of zpanel_kernel<ROWS, true> the device schedules
template <int ROWS>
static int max_cluster() {
  static int cmax_dev[kMaxDevices];
  static OncePerDevice once;
  const int dev = current_device();
  once([dev] {
    int& cmax = cmax_dev[dev];
    cmax = 0;
    auto* kern = zpanel_kernel<ROWS, true>;
    cudaFuncSetAttribute(zpanel_kernel<ROWS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(Smem<ROWS>));
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<ROWS>)) !=
        cudaSuccess) {
      cudaGetLastError();
      return;
    }
    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int size : {kMaxCluster, 8}) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(size);
      cfg.blockDim = dim3(4 * ROWS + 64);
      cfg.dynamicSmemBytes = sizeof(Smem<ROWS>);
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = size;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0) {
        cmax = size;
        break;
      }
    }
    cudaGetLastError();
  });
  return cmax_dev[dev];
}

template <int ROWS, bool CLUSTER>
static int launch(double2* P, int64_t lda, int m, int w, int j0, int32_t* perm, const ZPanelWs& ws, int G, int rpc,
                  bool cooperative, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3(4 * ROWS + 64);
  cfg.dynamicSmemBytes = sizeof(Smem<ROWS>);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  if (CLUSTER) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // early_start
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.numAttrs = cooperative ? 1 : 0;
  }
  cfg.attrs = at;
  if (cudaLaunchKernelEx(&cfg, zpanel_kernel<ROWS, CLUSTER>, P, lda, m, w, j0, rpc, perm, ws) != cudaSuccess)
    return MGT_ERR_CUDA;
  count_launch();
  return MGT_OK;
}

}  // namespace zp

int zpanel_factor(double2* P, int64_t lda, int m, int w, int j0, int32_t* perm, const ZPanelWs& ws, int rows_target,
                  int max_ctas, bool cooperative, bool allow_cluster, bool allow_wide, cudaStream_t s) {
  using namespace zp;
  if (m <= 0 || w <= 0 || w > NB || m >= kNoPos || j0 + w > kMaxColumns) return MGT_ERR_UNSUPPORTED;
  const int c64 = max_cluster<64>();
  max_cluster<128>();   // sets its kernels' attributes
  const int cap = std::max(1, std::min(max_ctas, ws.max_ctas));
  if (!zpanel_fits(m, rows_target, cap)) return MGT_ERR_UNSUPPORTED;
  // Up to 64 rows a CTA one cluster is fastest (1000 rows: 3.4 us a column against 4.5 through global
  // memory); with 128 rows its 16 SMs' FP64 pipes take longer than the wider exchange (5.6 against 4.8).
  if (allow_cluster) {
    const int g64 = std::min(c64, cap);
    if (g64 > 0 && m <= 64 * g64) {
      const int G = std::min(g64, (m + rows_target - 1) / rows_target), rpc = (m + G - 1) / G;
      if (rpc <= 64)
        return launch<64, true>(P, lda, m, w, j0, perm, ws, (m + rpc - 1) / rpc, rpc, cooperative, s);
    }
  }
  if (!allow_wide) return MGT_ERR_UNSUPPORTED;
  int G = std::min(cap, (m + rows_target - 1) / rows_target);
  const int rpc = (m + G - 1) / G;
  G = (m + rpc - 1) / rpc;
  if (rpc <= 64) return launch<64, false>(P, lda, m, w, j0, perm, ws, G, rpc, cooperative, s);
  if (rpc <= 128) return launch<128, false>(P, lda, m, w, j0, perm, ws, G, rpc, cooperative, s);
  return MGT_ERR_UNSUPPORTED;
}

}  // namespace mgt
