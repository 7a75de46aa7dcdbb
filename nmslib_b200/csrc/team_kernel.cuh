// The team kernel: one block (a team of warps) per query, instantiated per distance by team_l2.cu,
// team_dot.cu, team_lp.cu and team_sift.cu. See the comment at search_team_kernel, at the end.
#pragma once

#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include "engine.h"
#include "search_device.cuh"
#include "../../include/nmslib_b200.h"

namespace nmsg {
namespace {

// Distance policies of the team kernel.
enum TeamDist { kTeamL2 = 0, kTeamCos = 1, kTeamNeg = 2, kTeamL1 = 3, kTeamLInf = 4, kTeamSift = 5 };

constexpr uint32_t kTabEmpty = 0xffffffffu;
constexpr uint32_t kTabVisited = 0x80000000u;  // the id has been passed to the beam (or dropped by it)
constexpr uint32_t kTabNew = 0x40000000u;      // and is kept by the expansions under way (ids are below 2^30)
constexpr uint32_t kTabIdMask = 0x3fffffffu;
constexpr int kNoEntry = 0xffff;
constexpr int kPlanFlush = -1;  // plans other than a number of lists: empty the table,
constexpr int kPlanAgain = -2;  // expand on (the front candidate's list is evaluated already),
constexpr int kPlanRestart = -3;  // or search anew with heaps

// What a block knows of its query between phases (shared memory; warp 0 writes).
struct TeamState {
  int plan;                // lists to evaluate next: 0 ends the search, or one of the above
  int work;                // table entries this round computes
  int item, epoch;
  int curr, num;           // V1Merge: SortArrBI position and size
  int qsize, csize, rsize; // SearchOld: candidate heap, closest heap, results
  int tcount;              // entries of the table
  int st_dist, st_expand, st_greedy, st_list_ints;
  int overflow;
  int line, ready;           // V1Merge: candidates in line (at most 16), how many of the first are evaluated
  int tied;                  // equal keys met where SearchOld's order among them would matter
  float edge_in, edge_out;   // SearchOld's walk: the last key that stays in the array, the first that falls off,
  float edge_tie;            // the key at the array's end that another like it fell off or was rejected at,
  uint32_t late_tie;         // and the largest (ordered) key of an expanded candidate that had an equal beside it
  int kept, first;           // the expansions under way: kept neighbours, their smallest position
  int cnt[kTeamSlots];       // list lengths of the evaluated lists
  int slot_node[kTeamSlots]; // whose lists they are, or negative
  int plan_node[kTeamSlots]; // candidates whose lists this round evaluates
  int plan_slot[kTeamSlots]; // and where they go
  int line_node[16];         // the candidates in line,
  int line_slot[16];         // their evaluated lists (or -1),
  int line_pos[16];          // and V1Merge's array positions and (ordered) keys
  uint32_t line_key[16];
  uint32_t near[16];         // the nearest unvisited neighbour in each one's list
};
static_assert(sizeof(TeamState) == kTeamStateBytes, "team_layout reserves the state");

// A block's shared-memory pieces, at the offsets of its launch.
struct TeamView {
  const TeamLayout& l;
  int mpad, table_log2;
  template <class T>
  __device__ __forceinline__ T* at(int off) const {
    extern __shared__ __align__(16) char smem[];
    return reinterpret_cast<T*>(smem + off);
  }
  __device__ __forceinline__ TeamState& st() const { return *at<TeamState>(0); }
  // the query, permuted (l2sqr_sift: 128 bytes and the norm)
  __device__ __forceinline__ float* q() const { return at<float>(l.q); }
  // V1Merge's sorted array, or SearchOld's closest heap and results
  __device__ __forceinline__ uint2* items() const { return at<uint2>(l.items); }
  // table of evaluated ids (id | kTabVisited, open addressing) and their distances
  __device__ __forceinline__ uint32_t* tkey() const { return at<uint32_t>(l.tkey); }
  __device__ __forceinline__ float* tdist() const { return at<float>(l.tdist); }
  // batch merge scratch
  __device__ __forceinline__ float* sk() const { return at<float>(l.merge); }
  __device__ __forceinline__ int* sv() const { return at<int>(l.merge) + mpad; }
  __device__ __forceinline__ float* nb_d() const { return at<float>(l.merge) + 2 * mpad; }
  __device__ __forceinline__ int* nb_id() const { return at<int>(l.merge) + 3 * mpad; }
  // SearchOld: the head of the candidate heap
  __device__ __forceinline__ uint2* heap() const { return at<uint2>(l.heap); }
  // [kTeamSlots][lcap]: an evaluated list as table entries, in list order
  __device__ __forceinline__ uint16_t* tix() const { return at<uint16_t>(l.tix); }
  // kept neighbours of the expansions under way: table entries (keys in sk, ids in sv)
  __device__ __forceinline__ uint16_t* ste() const { return at<uint16_t>(l.ste); }
  // table entries whose distance this round computes
  __device__ __forceinline__ uint16_t* work() const { return at<uint16_t>(l.work); }
  __device__ __forceinline__ int tsize() const { return 1 << table_log2; }
  __device__ __forceinline__ int tlimit() const { return tsize() - tsize() / 5; }
};

// A distance as an integer of the same order, the two zeros as one.
__device__ __forceinline__ uint32_t order_of(float d) { return ordered_key(__fadd_rn(d, 0.0f)); }

// Finds or inserts id; *fresh is set when this call inserted it. The table always keeps free
// entries (tlimit), so the probe ends.
__device__ __forceinline__ int team_insert(const TeamView& v, uint32_t id, bool* fresh) {
  uint32_t* tkey = v.tkey();
  uint32_t h = (id * 2654435761u) >> (32 - v.table_log2);
  while (true) {
    uint32_t k = tkey[h];
    if (k == kTabEmpty) {
      k = atomicCAS(tkey + h, kTabEmpty, id);
      if (k == kTabEmpty) {
        *fresh = true;
        return (int)h;
      }
    }
    if ((k & kTabIdMask) == id) return (int)h;
    h = (h + 1) & (v.tsize() - 1);
  }
}

// ------------------------------------------------------------------ distances
template <int D>
__device__ __forceinline__ float team_term(float q, float x, float acc) {
  if constexpr (D == kTeamL2) {
    const float d = __fsub_rn(q, x);
    return __fmaf_rn(d, d, acc);
  } else if constexpr (D == kTeamL1) {
    return __fadd_rn(acc, fabsf(__fsub_rn(q, x)));
  } else if constexpr (D == kTeamLInf) {
    return fmaxf(acc, fabsf(__fsub_rn(q, x)));
  } else {
    return __fmaf_rn(q, x, acc);
  }
}

template <int D>
constexpr int team_group_lanes() {
  return D >= kTeamL1 ? 4 : 8;
}
// Rows one group holds in flight: two where four warps' groups are fewer than a round's rows (about
// 30), or a row is small; else one, with more of its pieces in flight.
template <int D, int NF, int NW>
constexpr int team_rows() {
  return D == kTeamSift || (D < kTeamL1 && NF > 0 && NW == 4) ? 2 : 1;
}

// Distances from the query to rows id[0..R) (act[r] false: not read, value meaningless), by the
// lanes of a group; every lane of the warp calls it and every lane of the group gets the values.
// Rows go from memory to registers, every 16-byte piece of up to four (wide rows: eight) 32-float
// blocks in flight at once. The arithmetic is combine() / lp_group_dist() / the l2sqr_sift branch of compute_dists()
// in hnsw_search.cu, order included:
//  * l2, cosine, dot: lane j of 8 holds the reference's accumulator j (the permuted layout gives it
//    its elements as one float4 per block); the 4-wide remainder and the scalar tail follow;
//  * L1, LInf: lane a of 4 reads the pieces at positions a and a + 4 of a block, whose elements
//    interleave to e == a (mod 4) in order: the reference's accumulator a without shuffles;
//  * l2sqr_sift: byte dot products, exact in any order.
// NF: 32-float blocks per row when known at compile time, else 0.
template <int D, int NF, int R>
__device__ __forceinline__ void team_dists(const DevIndex& ix, const float* __restrict__ q, const int (&id)[R],
                                           const bool (&act)[R], float (&d)[R]) {
  const int lane = lane_id();
  if constexpr (D == kTeamSift) {
    const int j = lane & 3;
    const uint4* qv = reinterpret_cast<const uint4*>(q) + 2 * j;
    const uint4 qa = qv[0], qb = qv[1];
    const int qn = reinterpret_cast<const int*>(q)[kSiftDim / 4];
    uint4 xa[R], xb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint4* row = reinterpret_cast<const uint4*>(ix.vecs_u8 + (int64_t)id[r] * kSiftDim) + 2 * j;
      xa[r] = act[r] ? __ldg(row) : make_uint4(0u, 0u, 0u, 0u);
      xb[r] = act[r] ? __ldg(row + 1) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t x[8] = {xa[r].x, xa[r].y, xa[r].z, xa[r].w, xb[r].x, xb[r].y, xb[r].z, xb[r].w};
      const uint32_t y[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
      unsigned dot = 0, xx = 0;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        dot = __dp4a(x[t], y[t], dot);
        xx = __dp4a(x[t], x[t], xx);
      }
      dot += __shfl_xor_sync(kFull, dot, 1);
      xx += __shfl_xor_sync(kFull, xx, 1);
      dot += __shfl_xor_sync(kFull, dot, 2);
      xx += __shfl_xor_sync(kFull, xx, 2);
      const int xn = ix.norms ? (act[r] ? __ldg(ix.norms + id[r]) : 0) : (int)xx;
      d[r] = __int2float_rn(qn + xn - 2 * (int)dot);
    }
  } else {
    const int nfull = NF > 0 ? NF : ix.n16 >> 5;
    const bool half = (ix.n16 & 31) != 0;
    const bool tail = ix.dim != ix.n16;
    const float* row[R];
#pragma unroll
    for (int r = 0; r < R; ++r) row[r] = ix.vecs + (int64_t)id[r] * ix.pitch;
    if constexpr (D >= kTeamL1) {
      const int a = lane & 3, gb = lane & ~3;
      float s[R];
      float4 t[R];
      float2 h0[R], h1[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        s[r] = 0.0f;
        t[r] = tail && act[r] ? __ldg(reinterpret_cast<const float4*>(row[r] + ix.n16) + a) : make_float4(0.f, 0.f, 0.f, 0.f);
        h0[r] = h1[r] = make_float2(0.f, 0.f);
        if (half && act[r]) {
          h0[r] = __ldg(reinterpret_cast<const float2*>(row[r] + nfull * 32) + a);
          h1[r] = __ldg(reinterpret_cast<const float2*>(row[r] + nfull * 32) + 4 + a);
        }
      }
      constexpr int U = 4;
      for (int c0 = 0; c0 < nfull; c0 += U) {
        float4 x[R][U][2];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const bool on = act[r] && c0 + u < nfull;
            const float4* p = reinterpret_cast<const float4*>(row[r] + (c0 + u) * 32) + a;
            x[r][u][0] = on ? __ldg(p) : make_float4(0.f, 0.f, 0.f, 0.f);
            x[r][u][1] = on ? __ldg(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (c0 + u >= nfull) break;
          const float4 p0 = reinterpret_cast<const float4*>(q + (c0 + u) * 32)[a];
          const float4 p1 = reinterpret_cast<const float4*>(q + (c0 + u) * 32)[a + 4];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            s[r] = team_term<D>(p0.x, x[r][u][0].x, s[r]);
            s[r] = team_term<D>(p1.x, x[r][u][1].x, s[r]);
            s[r] = team_term<D>(p0.y, x[r][u][0].y, s[r]);
            s[r] = team_term<D>(p1.y, x[r][u][1].y, s[r]);
            s[r] = team_term<D>(p0.z, x[r][u][0].z, s[r]);
            s[r] = team_term<D>(p1.z, x[r][u][1].z, s[r]);
            s[r] = team_term<D>(p0.w, x[r][u][0].w, s[r]);
            s[r] = team_term<D>(p1.w, x[r][u][1].w, s[r]);
          }
        }
      }
      if (half) {
        const float2 p0 = reinterpret_cast<const float2*>(q + nfull * 32)[a];
        const float2 p1 = reinterpret_cast<const float2*>(q + nfull * 32)[a + 4];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          s[r] = team_term<D>(p0.x, h0[r].x, s[r]);
          s[r] = team_term<D>(p1.x, h1[r].x, s[r]);
          s[r] = team_term<D>(p0.y, h0[r].y, s[r]);
          s[r] = team_term<D>(p1.y, h1[r].y, s[r]);
        }
      }
      if constexpr (D == kTeamL1) {
        const int n4 = (ix.dim >> 2) << 2, blocks = (n4 - ix.n16) >> 2;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          // tail element o (from n16) is component o & 3 of lane o >> 2
          for (int i = 0; i < blocks; ++i) {
            const float vx = __shfl_sync(kFull, t[r].x, gb + i), vy = __shfl_sync(kFull, t[r].y, gb + i);
            const float vz = __shfl_sync(kFull, t[r].z, gb + i), vw = __shfl_sync(kFull, t[r].w, gb + i);
            const float x = a == 0 ? vx : a == 1 ? vy : a == 2 ? vz : vw;
            s[r] = team_term<D>(q[ix.n16 + 4 * i + a], x, s[r]);
          }
          float sum = __fadd_rn(__shfl_sync(kFull, s[r], gb), __shfl_sync(kFull, s[r], gb + 1));
          sum = __fadd_rn(sum, __shfl_sync(kFull, s[r], gb + 2));
          sum = __fadd_rn(sum, __shfl_sync(kFull, s[r], gb + 3));
          if (n4 < ix.dim) {  // the reference adds the last dim % 4 elements in double
            double w = (double)sum;
            for (int e = n4; e < ix.dim; ++e) {
              const int o = e & 3;
              const float m = o == 0 ? t[r].x : o == 1 ? t[r].y : t[r].z;
              w = __dadd_rn(w, (double)fabsf(__fsub_rn(q[e], __shfl_sync(kFull, m, gb + blocks))));
            }
            sum = __double2float_rn(w);
          }
          d[r] = sum;
        }
      } else {
        if (tail) {  // both paddings are zeros, which leave a maximum of magnitudes as it is
          const float4 p = reinterpret_cast<const float4*>(q + ix.n16)[a];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (!act[r]) continue;
            s[r] = team_term<D>(p.x, t[r].x, s[r]);
            s[r] = team_term<D>(p.y, t[r].y, s[r]);
            s[r] = team_term<D>(p.z, t[r].z, s[r]);
            s[r] = team_term<D>(p.w, t[r].w, s[r]);
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          s[r] = fmaxf(s[r], __shfl_xor_sync(kFull, s[r], 2));
          d[r] = fmaxf(s[r], __shfl_xor_sync(kFull, s[r], 1));
        }
      }
    } else {
      const int j = lane & 7, gb = lane & ~7;
      float acc[R];
      float2 h[R], t[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        acc[r] = 0.0f;
        h[r] = half && act[r] ? __ldg(reinterpret_cast<const float2*>(row[r] + nfull * 32) + j) : make_float2(0.f, 0.f);
        t[r] = tail && act[r] ? __ldg(reinterpret_cast<const float2*>(row[r] + ix.n16) + j) : make_float2(0.f, 0.f);
      }
      constexpr int U = NF > 0 ? NF : 8;
      if (NF == 0) {  // the rest of a wide row on its way to L2 while its first blocks are read
        for (int c = U + j; c < nfull; c += 8) {
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (act[r]) prefetch_l2(row[r] + c * 32);
        }
      }
      for (int c0 = 0; c0 < nfull; c0 += U) {
        float4 x[R][U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int r = 0; r < R; ++r)
            x[r][u] = act[r] && (NF > 0 || c0 + u < nfull)
                          ? __ldg(reinterpret_cast<const float4*>(row[r] + (c0 + u) * 32) + j)
                          : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (NF == 0 && c0 + u >= nfull) break;
          const float4 p = reinterpret_cast<const float4*>(q + (c0 + u) * 32)[j];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            acc[r] = team_term<D>(p.x, x[r][u].x, acc[r]);
            acc[r] = team_term<D>(p.y, x[r][u].y, acc[r]);
            acc[r] = team_term<D>(p.z, x[r][u].z, acc[r]);
            acc[r] = team_term<D>(p.w, x[r][u].w, acc[r]);
          }
        }
      }
      if (half) {
        const float2 p = reinterpret_cast<const float2*>(q + nfull * 32)[j];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          acc[r] = team_term<D>(p.x, h[r].x, acc[r]);
          acc[r] = team_term<D>(p.y, h[r].y, acc[r]);
        }
      }
      if (D == kTeamL2 && ix.dist_type == kL2Sqr16Ext) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float s = __shfl_sync(kFull, acc[r], gb);
#pragma unroll
          for (int i = 1; i < 8; ++i) s = __fadd_rn(s, __shfl_sync(kFull, acc[r], gb + i));
          d[r] = s;
        }
      } else {
        const int blocks = (ix.n4 - ix.n16) >> 2;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float t4 = __fadd_rn(acc[r], __shfl_down_sync(kFull, acc[r], 4, 8));
          // tail element o (from n16) is component o & 1 of lane o >> 1
          for (int i = 0; i < blocks; ++i) {
            const int src = gb + ((j & 3) >> 1) + 2 * i;
            const float vx = __shfl_sync(kFull, t[r].x, src), vy = __shfl_sync(kFull, t[r].y, src);
            if (j < 4) t4 = team_term<D>(q[ix.n16 + 4 * i + j], (j & 1) ? vy : vx, t4);
          }
          float s = __fadd_rn(__shfl_sync(kFull, t4, gb), __shfl_sync(kFull, t4, gb + 1));
          s = __fadd_rn(s, __shfl_sync(kFull, t4, gb + 2));
          s = __fadd_rn(s, __shfl_sync(kFull, t4, gb + 3));
          for (int e = ix.n4; e < ix.dim; ++e) {
            const int o = e - ix.n16;
            s = team_term<D>(q[e], __shfl_sync(kFull, (o & 1) ? t[r].y : t[r].x, gb + (o >> 1)), s);
          }
          if constexpr (D == kTeamCos) {
            const float mn = (s < 1.0f) ? s : 1.0f;
            const float mx = (-1.0f < mn) ? mn : -1.0f;
            const float w = __fsub_rn(1.0f, mx);
            s = (0.0f < w) ? w : 0.0f;
          } else if constexpr (D == kTeamNeg) {
            s = -s;
          }
          d[r] = s;
        }
      }
    }
  }
}

// Distances of n rows by the whole block: row w's id is get(w), its distance goes to put(w, d).
template <int D, int NF, int NW, class Get, class Put>
__device__ __forceinline__ void team_eval(const DevIndex& ix, const float* q, int n, Get get, Put put) {
  constexpr int GL = team_group_lanes<D>(), R = team_rows<D, NF, NW>(), kGroups = NW * 32 / GL;
  const int group = threadIdx.x / GL;
  const int warp_first = warp_index() * (32 / GL);
  for (int base = 0; base + warp_first < n; base += kGroups * R) {
    int id[R];
    bool act[R];
    float d[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int w = base + r * kGroups + group;
      act[r] = w < n;
      id[r] = act[r] ? get(w) : 0;
    }
    team_dists<D, NF, R>(ix, q, id, act, d);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (act[r] && (lane_id() & (GL - 1)) == 0)  // cosine, LInf and bytes have no NaN
        put(base + r * kGroups + group, D == kTeamL2 || D == kTeamNeg || D == kTeamL1 ? kept_dist(d[r]) : d[r]);
  }
}

// The query into shared memory in the permuted layout, normalised for cosine as hnsw.h:486-497
// does (sequential, unfused sum of squares).
template <int D, int NW>
__device__ void team_load_query(const SearchArgs& a, float* q, int64_t qi) {
  const DevIndex& ix = a.ix;
  const int lane = lane_id();
  if constexpr (D == kTeamSift) {
    if (threadIdx.x < 32) {
      const uint32_t word = __ldg(reinterpret_cast<const uint32_t*>(a.queries_u8 + qi * kSiftDim) + lane);
      reinterpret_cast<uint32_t*>(q)[lane] = word;
      int s = (int)__dp4a(word, word, 0u);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
      if (lane == 0) reinterpret_cast<int*>(q)[kSiftDim / 4] = s;
    }
  } else {
    const float* src = a.queries + qi * ix.dim;
    float s = 1.0f;
    bool scale = false;
    if constexpr (D == kTeamCos) {  // every warp forms the sum for itself
      float sum = 0.0f;
      for (int e0 = 0; e0 < ix.dim; e0 += 32) {
        const float x = e0 + lane < ix.dim ? __ldg(src + e0 + lane) : 0.0f;
        const float x2 = __fmul_rn(x, x);
        const int m = min(32, ix.dim - e0);
        for (int i = 0; i < m; ++i) sum = __fadd_rn(sum, __shfl_sync(kFull, x2, i));
      }
      if (sum != 0.0f) {
        s = __fdiv_rn(1.0f, __fsqrt_rn(sum));
        scale = true;
      }
    }
    for (int e = threadIdx.x; e < ix.pitch; e += NW * 32) {
      float x = e < ix.dim ? __ldg(src + e) : 0.0f;
      if (scale) x = __fmul_rn(x, s);
      q[e < ix.dim ? permuted_pos(e, ix.dim) : e] = x;
    }
  }
}

// ------------------------------------------------------------------ SearchOld's candidate heap
// The head of the heap in shared memory, the rest in the slot's area in HBM.
struct TeamHeap {
  uint2* s;
  uint2* g;
  int ns;
  __device__ __forceinline__ uint2 get(int i) const { return i < ns ? s[i] : g[i]; }
  __device__ __forceinline__ void set(int i, uint2 x) const {
    if (i < ns)
      s[i] = x;
    else
      g[i] = x;
  }
};

// libstdc++'s push_heap / pop_heap by distance (the order of std::priority_queue over
// EvaluatedMSWNodeInt, hnsw.h:410-431). Single lane.
__device__ void team_heap_push(const TeamHeap& h, int& size, float key, int id) {
  int hole = size++;
  while (hole > 0) {
    const int parent = (hole - 1) / 2;
    const uint2 p = h.get(parent);
    if (!(key_of(p) < key)) break;
    h.set(hole, p);
    hole = parent;
  }
  h.set(hole, make_uint2(__float_as_uint(key), (uint32_t)id));
}

__device__ void team_heap_pop(const TeamHeap& h, int& size) {
  if (size > 1) {
    const int len = size - 1;
    const uint2 value = h.get(len);
    int hole = 0, child = 0;
    while (child < (len - 1) / 2) {
      child = 2 * (child + 1);
      uint2 c = h.get(child);
      const uint2 l = h.get(child - 1);
      if (key_of(c) < key_of(l)) {
        c = l;
        child--;
      }
      h.set(hole, c);
      hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
      child = 2 * (child + 1);
      h.set(hole, h.get(child - 1));
      hole = child - 1;
    }
    while (hole > 0) {
      const int parent = (hole - 1) / 2;
      const uint2 p = h.get(parent);
      if (!(key_of(p) < key_of(value))) break;
      h.set(hole, p);
      hole = parent;
    }
    h.set(hole, value);
  }
  --size;
}

// The k-bounded result queue (knnqueue.h:55-64 + knnquery.cc:67-75) as an array sorted by
// (distance, node). Single lane.
__device__ void team_result_offer(uint2* res, int& size, int k, float d, int node) {
  if (size >= k) {
    if (!(key_of(res[size - 1]) > d)) return;
    --size;
  }
  int pos = size;
  while (pos > 0) {
    const uint2 p = res[pos - 1];
    if (key_of(p) < d || (key_of(p) == d && (int)p.y < node)) break;
    res[pos] = p;
    --pos;
  }
  res[pos] = make_uint2(__float_as_uint(d), (uint32_t)node);
  ++size;
}

// ------------------------------------------------------------------ beam merge
// Kept neighbours sk/sv[0..qty) inserted the general way (equal keys, more of them than threads):
// the batch merge when nothing ties, else std::sort's order and one insertion after another. Returns
// the smallest insertion position; *num_io is the array's size.
__device__ __noinline__ int team_insert_general(uint2* items, int* num_io, int cap, float* sk, int* sv, int qty,
                                                float* tk, int* tv, int* tied) {
  const int lane = lane_id();
  int num = *num_io, p0 = 0x7fffffff;
  if (!merge_unsorted_batch(items, num, cap, sk, sv, qty, tk, tv, &p0)) {
    if (lane == 0) *tied = 1;
    sort_like_std(sk, sv, qty, tk, tv);
    p0 = 0x7fffffff;
    for (int i = 0; i < qty; ++i) p0 = min(p0, sorted_insert(items, num, cap, sk[i], sv[i]));
  }
  __syncwarp();
  if (lane == 0) *num_io = num;
  __syncwarp();
  return p0;
}

// ------------------------------------------------------------------ the query
// Warp 0: the slot whose list is candidate `node`'s, or -1 (slot_node: lane 16 + f holds slot f's).
__device__ __forceinline__ int team_slot_of(int slot_node, int node) {
  const unsigned m = __ballot_sync(kFull, lane_id() >= 16 && slot_node == node);
  return m ? __ffs(m) - 17 : -1;
}

// Warp 0: which lists the next round evaluates. `cand`: lane i < 16 holds the i-th candidate in
// line (or a negative value). Lists already in a slot stay; the first `spec` candidates without
// one get the slots whose candidates are no longer in line.
__device__ __forceinline__ void team_plan(const SearchArgs& a, const TeamView& v, int slot_node, int cand) {
  const int lane = lane_id();
  TeamState& st = v.st();
  // lanes 0..15 hold candidates, lanes 16..31 slots: one match finds the evaluated ones
  const int key = lane < 16 ? (cand >= 0 ? cand : -2 - lane) : (slot_node >= 0 ? slot_node : -2 - lane);
  const unsigned same = __match_any_sync(kFull, key);
  const bool want = lane < 16 && cand >= 0 && !(same & 0xffff0000u);
  const bool unused = lane >= 16 && !(same & 0x0000ffffu);
  const unsigned wm = __ballot_sync(kFull, want), um = __ballot_sync(kFull, unused);
  int n = min(min(__popc(wm), __popc(um)), a.team.spec);
  const int room = v.tlimit() - uni(st.tcount);
  if (n * a.ix.maxM0 > room) {
    n = room / a.ix.maxM0;
    if (n < 1) n = kPlanFlush;
  }
  if (n == 0 && __shfl_sync(kFull, cand, 0) >= 0) n = kPlanAgain;
  const int i = __popc((lane < 16 ? wm : um) & lanemask_lt());
  const bool mine = (want || unused) && i < n;
  if (mine && lane < 16) st.plan_node[i] = cand;
  if (mine && lane >= 16) st.plan_slot[i] = lane - 16;
  __syncwarp();
  if (lane < 16)
    st.line_slot[lane] = mine ? st.plan_slot[i] : (cand >= 0 && !want) ? 31 - __clz(same) - 16 : -1;
  else
    st.slot_node[lane - 16] = mine ? st.plan_node[i] : slot_node;
  // evaluated candidates at the front of the line after this round's evaluation
  const unsigned behind = __ballot_sync(kFull, lane < 16 && (cand < 0 || (want && !mine)));
  if (lane == 0) {
    st.plan = n;
    st.work = 0;
    st.ready = behind ? __ffs(behind) - 1 : 16;
    st.kept = 0;
    st.first = 0x7fffffff;
    st.tied = 0;
    st.edge_in = 0.0f;
    st.edge_out = __int_as_float(0x7fffffff);  // NaN: equal to nothing
  }
}

// Entry t of the evaluated list in slot f: its table entry when it is not visited yet (an id listed
// twice: at its first place in the 32), else -1; its distance and id.
__device__ __forceinline__ int team_peek(const SearchArgs& a, const TeamView& v, int f, int t, int cnt, float* d,
                                         int* id) {
  const int ti = t < cnt ? v.tix()[f * a.team.lcap + t] : kNoEntry;
  const uint32_t key = ti != kNoEntry ? v.tkey()[ti] : kTabVisited;
  *d = ti != kNoEntry ? v.tdist()[ti] : 0.0f;
  bool fresh = !(key & kTabVisited);
  if (!a.ix.l0_unique) {
    const unsigned same = __match_any_sync(kFull, fresh ? ti : -1 - lane_id());
    fresh = fresh && (__ffs(same) - 1) == lane_id();
  }
  *id = (int)(key & kTabIdMask);
  return fresh ? ti : -1;
}

// Warp 0, V1Merge: the line (the unused among the items that may be expanded, from the first on, up
// to 16) and the next round's plan. kth: SearchOld's walk, the length of its result; else past any array.
__device__ __forceinline__ void team_line_v1(const SearchArgs& a, const TeamView& v, int ef, int kth) {
  const int lane = lane_id();
  TeamState& st = v.st();
  const uint2* items = v.items();
  const int end = min(uni(st.num), ef);
  int curr = uni(st.curr), found = 0;
  for (int t0 = curr; t0 < end && found < 16 && t0 < curr + 128; t0 += 32) {
    const int t = t0 + lane;
    const uint2 it = t < end ? items[t] : make_uint2(0u, kUsedBit);
    const bool open = !(it.y & kUsedBit);
    const unsigned m = __ballot_sync(kFull, open);
    const int p = found + __popc(m & lanemask_lt());
    if (open && p < 16) {
      st.line_node[p] = (int)it.y;
      st.line_pos[p] = t;
      st.line_key[p] = order_of(key_of(it));
    }
    found += __popc(m);
    if (!found) curr = min(t0 + 32, end);
  }
  found = min(found, 16);
  if (lane == 0) {
    st.curr = curr;
    st.line = found;
  }
  __syncwarp();
  team_plan(a, v, lane >= 16 ? st.slot_node[lane - 16] : -1, lane < found ? st.line_node[lane] : -1);
  // over: SearchOld's walk, see team_expand_v1
  if (lane == 0 && found == 0) {
    const float last = key_of(items[st.num - 1]);
    if (last == st.edge_tie || (st.num >= ef && order_of(last) <= st.late_tie) ||
        (kth < st.num && key_of(items[kth - 1]) == key_of(items[kth])))
      st.plan = kPlanRestart;
  }
}

// Warp 0: the kept neighbours of the expansions 0..n under way, inserted expansion after expansion in
// list order, each held against its own expansion's threshold. They are the table entries marked
// kTabNew, each first listed where the serial walk meets it.
__device__ __noinline__ void team_insert_ordered(const TeamView& v, int n, int ef, int cap, int lcap, int* line_slot) {
  const int lane = lane_id();
  TeamState& st = v.st();
  for (int i = 0; i < n; ++i) {
    const int f = line_slot[i];
    const int cnt = st.cnt[f];
    const float top_key = key_of(v.items()[st.num - 1]);
    const bool open = st.num < ef;
    int qty = 0;
    for (int b = 0; b < cnt; b += 32) {
      const int ti = b + lane < cnt ? v.tix()[f * lcap + b + lane] : kNoEntry;
      const uint32_t key = ti != kNoEntry ? v.tkey()[ti] : 0u;
      const bool is_new = (key & kTabNew) != 0;
      const unsigned same = __match_any_sync(kFull, is_new ? ti : -1 - lane);
      const bool mine = is_new && (__ffs(same) - 1) == lane;
      const float d = mine ? v.tdist()[ti] : 0.0f;
      const bool take = mine && ((d < top_key) || open);
      const unsigned m = __ballot_sync(kFull, take);
      if (mine) v.tkey()[ti] = key & ~kTabNew;
      if (take) {
        const int p = qty + __popc(m & lanemask_lt());
        v.sk()[p] = d;
        v.sv()[p] = (int)(key & kTabIdMask);
      }
      qty += __popc(m);
      __syncwarp();
    }
    if (qty) {
      const int p0 = team_insert_general(v.items(), &st.num, cap, v.sk(), v.sv(), qty, v.nb_d(), v.nb_id(),
                                         &st.tied);
      if (lane == 0) st.first = min(st.first, p0);
      __syncwarp();
    }
  }
}

// V1Merge's expansions (hnsw_distfunc_opt.cc:200-283), by the whole block. The candidates at the
// front of the line are expanded for as long as their lists are evaluated and none of the neighbours
// brought so far is nearer than the next one in line (it would be expanded before it). Within such a
// run the array is not needed between expansions, so their kept neighbours are merged together: with
// k <= ef the array after a run is the best ef of everything, whichever expansion's threshold a
// neighbour is held against (k > ef: one expansion at a time).
//
// The merge: push_or_replace_non_empty_exp (sort_arr_bi.h:159-199) inserts at the lower bound, before
// an equal key, unless its exponential probe can meet one of several equals or the equal key is the
// last at that moment. So a kept item lands at (array keys below it) + (kept keys below it) and an
// array item moves right by the number of kept keys not above it. Where that may not hold (equal
// kept keys, two equal array keys, an equal one at the array's end, more kept than threads) the
// kept ones are inserted one by one in the reference's order instead.
//
// `old`: SearchOld (hnsw_distfunc_opt.cc:285-381) with k <= ef, which is this walk too. Its candidates
// leave the heap nearest first until one is past the closest set's largest, so the expanded ones are
// the array's unused; its closest set is the best ef of everything, as the array is; its results are
// the k nearest of them. Equal keys leave its heaps in an order of their own, which matters in three
// places, and there the query is searched anew with heaps:
//  * of two equal candidates the one expanded first may bring neighbours that cut the other off. Both
//    are expanded in either order if the final largest lies past them (it only ever shrinks), and then
//    all that either brings is seen; so the largest such key is held against the final largest;
//  * where the array's end has one key of several equal ones, and the rest fell off or were rejected,
//    SearchOld would still expand them if it came to them with that key as its largest: the walk must
//    not expand a candidate of that key, nor end with it as the last;
//  * a result queue that holds k rejects an equal distance whatever its node (knnqueue.h:55-64), so of
//    equal keys on both sides of the k-th place those found first are the results, an order the array
//    does not keep: the walk must not end with such a pair.
template <int NW>
__device__ __forceinline__ void team_expand_v1(const SearchArgs& a, const TeamView& v, int k, int ef, bool old) {
  constexpr int kThreads = 32 * NW;
  const DevIndex& ix = a.ix;
  const int lane = lane_id(), warp = warp_index();
  const int cap = max(ef, k);
  TeamState& st = v.st();
  uint2* items = v.items();
  const int num = uni(st.num), ready = uni(st.ready);
  const float top_key = key_of(items[num - 1]);
  const bool open = num < ef;  // keep d < topKey || size < ef
  const uint32_t edge = order_of(st.edge_tie);
  // ---- the nearest unvisited neighbour of every evaluated candidate at the front; a warp holds on to
  // the entries of its (first) list when they are one to a lane
  int my_cnt = 0, my_ti = kNoEntry;
  uint32_t my_key = kTabVisited;
  float my_d = 0.0f;
  for (int i = warp; i < ready; i += NW) {
    const int f = uni(st.line_slot[i]);
    const int cnt = uni(st.cnt[f]);
    uint32_t near_key = 0xffffffffu;
    for (int b = 0; b < cnt; b += 32) {
      const int ti = b + lane < cnt ? v.tix()[f * a.team.lcap + b + lane] : kNoEntry;
      const uint32_t key = ti != kNoEntry ? v.tkey()[ti] : kTabVisited;
      const float d = ti != kNoEntry ? v.tdist()[ti] : 0.0f;
      if (!(key & kTabVisited)) near_key = min(near_key, order_of(d));
      if (i == warp && cnt <= 32) {
        my_cnt = cnt;
        my_ti = ti;
        my_key = key;
        my_d = d;
      }
    }
    near_key = __reduce_min_sync(kFull, near_key);
    if (lane == 0) st.near[i] = near_key;
  }
  __syncthreads();
  // ---- how many are expanded: candidate i if it is nearer than every neighbour of those before it
  int n;
  {
    uint32_t least = lane < ready ? st.near[lane & 15] : 0xffffffffu;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t up = __shfl_up_sync(kFull, least, o);
      if (lane >= o) least = min(least, up);
    }
    least = __shfl_up_sync(kFull, least, 1);
    const bool stop = lane > 0 && (lane >= ready || !(st.line_key[lane & 15] < least));
    n = __ffs(__ballot_sync(kFull, stop)) - 1;
    if (k > ef) n = 1;
    if (old && __any_sync(kFull, lane < n && st.line_key[lane & 15] == edge)) {
      __syncthreads();  // every warp has seen it
      if (threadIdx.x == 0) st.plan = kPlanRestart;
      return;
    }
  }
  // ---- their lists: unvisited neighbours are marked, those that pass are kept
  for (int i = warp; i < n; i += NW) {
    const bool held = i == warp && my_cnt > 0;
    const int f = held ? 0 : uni(st.line_slot[i]);
    const int cnt = held ? my_cnt : uni(st.cnt[f]);
    int fresh_n = 0;
    for (int b = 0; b < cnt; b += 32) {
      int ti = my_ti;
      uint32_t key = my_key;
      float d = my_d;
      if (!held) {
        ti = b + lane < cnt ? v.tix()[f * a.team.lcap + b + lane] : kNoEntry;
        key = ti != kNoEntry ? v.tkey()[ti] : kTabVisited;
        d = ti != kNoEntry ? v.tdist()[ti] : 0.0f;
      }
      const bool pass = (d < top_key) || open;
      bool fresh = !(key & kTabVisited);  // of equal ids in one or several lists, one finds it unvisited
      if (fresh) fresh = !(atomicOr(v.tkey() + ti, pass ? kTabVisited | kTabNew : kTabVisited) & kTabVisited);
      if (old && fresh && !pass && d == top_key) st.edge_tie = top_key;
      const unsigned km = __ballot_sync(kFull, fresh && pass);
      fresh_n += __popc(__ballot_sync(kFull, fresh));
      if (km) {
        int at = 0;
        if (lane == 0) at = atomicAdd(&st.kept, __popc(km));
        at = uni(at);
        if (fresh && pass) {
          const int p = at + __popc(km & lanemask_lt());
          if (p < kThreads) {
            v.sk()[p] = d;
            v.sv()[p] = (int)key;
            v.ste()[p] = (uint16_t)ti;
          }
          // a kept neighbour is usually expanded later: pull its list into L2
          const int32_t* lst = ix.l0 + (int64_t)(int)key * ix.l0_pitch;
          prefetch_l2(lst);
          if (ix.l0_pitch > 32) prefetch_l2(lst + 32);
        }
      }
    }
    if (lane == 0) {
      const int p = st.line_pos[i];
      items[p].y = (uint32_t)st.line_node[i] | kUsedBit;
      if (old && p + 1 < num && key_of(items[p + 1]) == key_of(items[p])) atomicMax(&st.late_tie, st.line_key[i]);
      atomicAdd(&st.st_dist, fresh_n);
      atomicAdd(&st.st_list_ints, 1 + cnt);
    }
  }
  if (threadIdx.x == 0) st.st_expand += n;
  __syncthreads();
  const int m = uni(st.kept);
  bool general = m > kThreads;
  if (m && !general) {
    // the last threads take the kept items, the first ones the array's: different warps when both are few
    const int u = kThreads - 1 - threadIdx.x;
    const bool mine = u < m;
    const float* sk = v.sk();
    float d = 0.0f;
    int id = 0, pos = 0;
    bool hard = false;
    if (mine) {
      d = sk[u];
      id = v.sv()[u];
      int lo = 0, hi = num;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (key_of(items[mid]) < d)
          lo = mid + 1;
        else
          hi = mid;
      }
      int rank = 0, equal = 0;
      for (int w = 0; w < m; w += 4) {
        const float4 s4 = *reinterpret_cast<const float4*>(sk + w);
        rank += (s4.x < d) + (w + 1 < m && s4.y < d) + (w + 2 < m && s4.z < d) + (w + 3 < m && s4.w < d);
        equal += (s4.x == d) + (w + 1 < m && s4.y == d) + (w + 2 < m && s4.z == d) + (w + 3 < m && s4.w == d);
      }
      if (old && equal > 1)  // in the order they were kept
        for (int w = 0; w < u; ++w) rank += sk[w] == d;
      if (!old) {
        const bool twin = lo < num && key_of(items[lo]) == d;
        hard = equal != 1;  // itself
        hard |= twin && (lo + 1 >= num || lo + rank + 1 >= cap || key_of(items[lo + 1 < num ? lo + 1 : lo]) == d);
      }
      pos = lo + rank;
      atomicMin(&st.first, lo);
      if (old && pos == cap - 1) st.edge_in = d;
      if (old && pos == cap) st.edge_out = d;
    }
    // the array in runs of one item a thread, from its tail: a run is read before it is written, and
    // what it writes lies below what the runs above it have moved
    for (int top = num; top > 0; top -= kThreads) {
      const int t = top - 1 - threadIdx.x;
      uint2 it = make_uint2(0u, 0u);
      int c = 0;
      if (t >= 0) {
        it = items[t];
        const float key = key_of(it);
        for (int w = 0; w < m; w += 4) {
          const float4 s4 = *reinterpret_cast<const float4*>(sk + w);
          c += (s4.x <= key) + (w + 1 < m && s4.y <= key) + (w + 2 < m && s4.z <= key) + (w + 3 < m && s4.w <= key);
        }
        if (old && t + c == cap - 1) st.edge_in = key;
        if (old && t + c == cap) st.edge_out = key;
      }
      if (top == num)
        general = __syncthreads_or(hard);
      else
        __syncthreads();
      if (general) break;
      if (c && t + c < cap) items[t + c] = it;
    }
    if (!general) {
      if (mine) {
        if (pos < cap) items[pos] = make_item(d, id, false);
        v.tkey()[v.ste()[u]] = (uint32_t)id | kTabVisited;
      }
      if (threadIdx.x == 0) st.num = min(num + m, cap);
    }
  }
  if (general) {
    __syncthreads();
    // the walk follows no ties here: neither those that made it general nor those among what falls off
    if (old && (m <= kThreads || num + m > cap)) {
      if (threadIdx.x == 0) st.plan = kPlanRestart;
      return;
    }
    if (threadIdx.x == 0) st.first = 0x7fffffff;
    __syncwarp();
    if (warp == 0) team_insert_ordered(v, n, ef, cap, a.team.lcap, st.line_slot);
  }
  __syncthreads();
  if (old) {
    if (uni(st.tied)) {
      if (threadIdx.x == 0) st.plan = kPlanRestart;
      return;
    }
    if (threadIdx.x == 0 && st.edge_in == st.edge_out) st.edge_tie = st.edge_in;
  }
  if (warp == 0) {
    if (lane == 0) st.curr = min(st.line_pos[n - 1] + 1, st.first);  // everything before it is used
    __syncwarp();
    team_line_v1(a, v, ef, old ? k : INT_MAX);
  }
}

// Warp 0, SearchOld (hnsw_distfunc_opt.cc:285-381): pops candidates for as long as their lists are
// evaluated, then plans the next round from the top five levels of the candidate heap.
__device__ __forceinline__ void team_commit_old(const SearchArgs& a, const TeamView& v, const TeamHeap& heap, int k,
                                                int ef) {
  const int lane = lane_id();
  TeamState& st = v.st();
  uint2* closest = v.items();
  uint2* res = closest + (ef + 1);
  const TeamHeap near{closest, closest, 0x7fffffff};
  int qsize = uni(st.qsize), csize = uni(st.csize), rsize = uni(st.rsize);
  int slot_node = lane >= 16 ? st.slot_node[lane - 16] : -1;
  int dist = 0, expand = 0, list_ints = 0;
  bool over = false, overflow = false;
  while (true) {
    float lb = 0.0f;
    int node = -1;
    if (qsize > 0) {
      const uint2 top = heap.get(0);
      lb = key_of(closest[0]);
      if (!(-key_of(top) > lb)) node = (int)top.y;
    }
    node = uni(node);
    over = node < 0;
    if (over) break;
    const int f = team_slot_of(slot_node, node);
    if (f < 0) break;
    const int cnt = uni(st.cnt[f]);
    if (lane == 16 + f) slot_node = -1;
    expand += 1;
    list_ints += 1 + cnt;
    __syncwarp();
    if (lane == 0) team_heap_pop(heap, qsize);
    // while the closest heap is full its largest only shrinks: a distance not below it now is
    // never taken
    const bool full = csize >= ef;
    int qty = 0;
    for (int b = 0; b < cnt; b += 32) {
      float d;
      int id;
      const int ti = team_peek(a, v, f, b + lane, cnt, &d, &id);
      if (ti >= 0) v.tkey()[ti] = (uint32_t)id | kTabVisited;
      dist += __popc(__ballot_sync(kFull, ti >= 0));
      const bool may = ti >= 0 && (!full || lb > d);
      const unsigned km = __ballot_sync(kFull, may);
      if (may) {
        const int p = qty + __popc(km & lanemask_lt());
        v.sk()[p] = d;
        v.sv()[p] = id;
      }
      qty += __popc(km);
      __syncwarp();
    }
    __syncwarp();
    if (lane == 0) {
      for (int i = 0; i < qty; ++i) {
        const float d = v.sk()[i];
        const int id = v.sv()[i];
        if (key_of(closest[0]) > d || csize < ef) {
          if (qsize >= a.old_heap_cap) {
            overflow = true;
            break;
          }
          team_heap_push(heap, qsize, -d, id);
          team_result_offer(res, rsize, k, d, id);
          team_heap_push(near, csize, d, id);
          if (csize > ef) team_heap_pop(near, csize);
        }
      }
    }
    qsize = __shfl_sync(kFull, qsize, 0);
    csize = __shfl_sync(kFull, csize, 0);
    rsize = __shfl_sync(kFull, rsize, 0);
    overflow = __shfl_sync(kFull, (int)overflow, 0) != 0;
    __syncwarp();
    if (overflow) break;
  }
  if (lane == 0) {
    st.qsize = qsize;
    st.csize = csize;
    st.rsize = rsize;
    st.overflow = overflow;
    st.st_dist += dist;
    st.st_expand += expand;
    st.st_list_ints += list_ints;
  }
  if (over || overflow) {
    if (lane == 0) st.plan = 0;
    return;
  }
  // the heap's first 31 entries, nearest first
  __syncwarp();
  const float lb = key_of(closest[0]);
  const bool in = lane < 31 && lane < qsize;
  const uint2 c = in ? heap.get(lane) : make_uint2(0u, 0u);
  const bool open = in && !(-key_of(c) > lb);
  const unsigned om = __ballot_sync(kFull, open);
  int rank = 0;
  for (unsigned mm = om; mm; mm &= mm - 1) {
    const int u = __ffs(mm) - 1;
    const float ku = __shfl_sync(kFull, key_of(c), u);
    rank += ku > key_of(c) || (ku == key_of(c) && u < lane);
  }
  if (lane < 16) st.line_node[lane] = -1;
  __syncwarp();
  if (open && rank < 16) st.line_node[rank] = (int)c.y;
  __syncwarp();
  team_plan(a, v, slot_node, lane < 16 ? st.line_node[lane] : -1);
}

// The upper levels (hnsw_distfunc_opt.cc:168-198): at each level, move to the earliest list entry
// whose distance is strictly below every earlier one while one is below the current distance. Every
// warp takes the same decisions from the distances the block computed.
template <int D, int NF, int NW>
__device__ __forceinline__ void team_descent(const SearchArgs& a, const TeamView& v, int* cur_out, float* dist_out) {
  const DevIndex& ix = a.ix;
  const int lane = lane_id();
  int cur = ix.enterpoint, lev = ix.maxlevel + 1;  // level maxlevel + 1: the entry point's own distance
  float curdist = 0.0f;
  int st_dist = 0, st_greedy = 0, st_list_ints = 0;
  bool flip = false;
  while (lev > 0) {
    const bool first = lev > ix.maxlevel;
    const int32_t* lst = first ? nullptr : ix.up_links + __ldg(ix.up_off + cur) + (int64_t)(ix.maxM + 1) * (lev - 1);
    const int cnt = first ? 1 : uni(__ldg(lst));
    float* out = flip ? v.nb_d() : v.sk();  // a step's distances are read while the next step's are written
    flip = !flip;
    team_eval<D, NF, NW>(ix, v.q(), cnt, [&](int w) { return first ? cur : __ldg(lst + 1 + w); },
                         [&](int w, float d) { out[w] = d; });
    __syncthreads();
    st_dist += cnt;
    if (first) {
      curdist = out[0];
      --lev;
      continue;
    }
    st_greedy += 1;
    st_list_ints += 1 + cnt;
    float best = curdist;
    int bpos = 0x7fffffff;
    for (int t = lane; t < cnt; t += 32) {
      const float d = out[t];
      if (d < best) {
        best = d;
        bpos = t;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(kFull, best, o);
      const int op = __shfl_xor_sync(kFull, bpos, o);
      if (ob < best || (ob == best && op < bpos)) {
        best = ob;
        bpos = op;
      }
    }
    if (!uni(bpos != 0x7fffffff && best < curdist)) {
      --lev;
      continue;
    }
    cur = __ldg(lst + 1 + bpos);
    curdist = best;
  }
  if (threadIdx.x == 0) {
    TeamState& st = v.st();
    st.st_dist = st_dist;
    st.st_greedy = st_greedy;
    st.st_list_ints = st_list_ints;
  }
  __syncthreads();
  *cur_out = cur;
  *dist_out = curdist;
}

template <int D, int NF, int NW, bool OLD>
__device__ __forceinline__ void team_query(const SearchArgs& a, const TeamView& v, int64_t qi) {
  const DevIndex& ix = a.ix;
  const int lane = lane_id(), warp = warp_index(), slot = blockIdx.x;
  const int k = a.k_per_q ? uni(a.k_per_q[qi]) : a.k_default;
  const int ef = a.ef_per_q ? uni(a.ef_per_q[qi]) : a.ef_default;
  const bool use_old = OLD && (a.algo == NMSG_ALGO_OLD || (a.algo == NMSG_ALGO_HYBRID && ef >= 1000));
  TeamState& st = v.st();
  for (int t = threadIdx.x; t < v.tsize() / 4; t += NW * 32)
    reinterpret_cast<uint4*>(v.tkey())[t] = make_uint4(kTabEmpty, kTabEmpty, kTabEmpty, kTabEmpty);
  team_load_query<D, NW>(a, v.q(), qi);
  __syncthreads();
  int cur;
  float curdist;
  if (a.split == 2) {  // level 0 from where the descent pass ended, with its counts
    cur = __ldg(a.entry_node + qi);
    curdist = __ldg(a.entry_dist + qi);
    if (cur < 0 || cur >= ix.n) {  // the descent pass gave up on this query
      if (threadIdx.x == 0) {
        set_status(a.status, NMSG_ERR_TIMEOUT);
        a.counts[qi] = 0;
      }
      return;
    }
    if (threadIdx.x == 0) {
      st.st_dist = __ldg(a.entry_stats + 3 * qi + 0);
      st.st_greedy = __ldg(a.entry_stats + 3 * qi + 1);
      st.st_list_ints = __ldg(a.entry_stats + 3 * qi + 2);
    }
  } else {
    team_descent<D, NF, NW>(a, v, &cur, &curdist);
  }
  // ---- level 0: the entry point is visited and first in line
  const TeamHeap heap{v.heap(), OLD ? a.old_heap + (int64_t)slot * a.old_heap_cap : nullptr, a.team.heap_items};
  // SearchOld with heaps, or (k <= ef, unless equal distances count, see team_expand_v1) as V1Merge's walk
  bool heaps = OLD && use_old && k > ef;
  const int kth = OLD && use_old ? k : INT_MAX;
  const int walk_dist = uni(st.st_dist), walk_ints = uni(st.st_list_ints);
  bool restart = false;
  bool spilled = false;
  int epoch = 0;
  uint8_t* vis = a.visited + (int64_t)slot * a.visited_pitch;
  while (true) {
    if (restart) {
      for (int t = threadIdx.x; t < v.tsize() / 4; t += NW * 32)
        reinterpret_cast<uint4*>(v.tkey())[t] = make_uint4(kTabEmpty, kTabEmpty, kTabEmpty, kTabEmpty);
      heaps = true;
      spilled = false;
      __syncthreads();
    }
    if (warp == 0) {
      if (lane == 0) {
        bool fresh = false;
        const int ti = team_insert(v, (uint32_t)cur, &fresh);
        v.tkey()[ti] = (uint32_t)cur | kTabVisited;
        st.curr = st.line = 0;
        st.num = 1;
        st.tcount = 1;
        st.st_expand = 0;
        st.overflow = 0;
        st.edge_tie = __int_as_float(0x7fffffff);
        st.late_tie = 0;
        st.st_dist = walk_dist;
        st.st_list_ints = walk_ints;
        if (!heaps) {
          v.items()[0] = make_item(curdist, cur, false);
        } else {
          const uint2 e = make_uint2(__float_as_uint(curdist), (uint32_t)cur);
          heap.set(0, make_uint2(__float_as_uint(-curdist), (uint32_t)cur));
          v.items()[0] = v.items()[ef + 1] = e;
          st.qsize = st.csize = st.rsize = 1;
        }
      }
      if (lane < kTeamSlots) st.slot_node[lane] = -1;
      __syncwarp();
    }
    if (warp == 0) {
      if (heaps)
        team_commit_old(a, v, heap, k, ef);
      else
        team_line_v1(a, v, ef, kth);
    }
    while (true) {
      __syncthreads();
      const int plan = uni(st.plan);
      restart = OLD && plan == kPlanRestart;
      if (plan == 0 || restart) break;
      if (plan == kPlanFlush) {
        // the table is full: its visited ids move to the slot's epoch bytes in HBM, which every later
        // insertion checks, and the lists evaluated ahead are dropped
        if (!spilled) {
          if (threadIdx.x == 0) st.epoch = a.epochs[slot] + 1;
          __syncthreads();
          epoch = st.epoch;
          if (epoch == 256) {  // the byte wraps: clear (hnsw.h:582-589)
            uint4* p = reinterpret_cast<uint4*>(vis);
            for (int64_t t = threadIdx.x; t < a.visited_pitch / 16; t += NW * 32) p[t] = make_uint4(0, 0, 0, 0);
            epoch = 1;
            __syncthreads();
          }
          if (threadIdx.x == 0) a.epochs[slot] = (uint8_t)epoch;
          spilled = true;
        }
        for (int t = threadIdx.x; t < v.tsize(); t += NW * 32) {
          const uint32_t key = v.tkey()[t];
          if (key != kTabEmpty && (key & kTabVisited)) vis[key & kTabIdMask] = (uint8_t)epoch;
          v.tkey()[t] = kTabEmpty;
        }
        if (threadIdx.x < kTeamSlots) st.slot_node[threadIdx.x] = -1;
        if (threadIdx.x == 0) st.tcount = 0;
        __syncthreads();
        if (warp == 0) {
          if (heaps)
            team_commit_old(a, v, heap, k, ef);
          else
            team_line_v1(a, v, ef, kth);
        }
        continue;
      }
      if (plan > 0) {
        // ---- lists: one warp per candidate; ids not evaluated yet join the round's work
        for (int i = warp; i < plan; i += NW) {
          const int32_t* lst = ix.l0 + (int64_t)st.plan_node[i] * ix.l0_pitch;
          const int f = uni(st.plan_slot[i]);
          uint16_t* tix = v.tix() + f * a.team.lcap;
          const int cnt = __ldg(lst);
          for (int b = 0; b < ix.maxM0; b += 32) {
            const int t = b + lane;
            const int id = t < ix.maxM0 ? __ldg(lst + 1 + t) : 0;
            bool valid = t < cnt;
            if (spilled && valid) valid = vis[id] != (uint8_t)epoch;
            bool fresh = false;
            int ti = kNoEntry;
            if (valid) ti = team_insert(v, (uint32_t)id, &fresh);
            if (t < cnt) tix[t] = (uint16_t)ti;
            const unsigned m = __ballot_sync(kFull, fresh);
            int at = 0;
            if (lane == 0 && m) at = atomicAdd(&st.work, __popc(m));
            at = __shfl_sync(kFull, at, 0);
            if (fresh) v.work()[at + __popc(m & lanemask_lt())] = (uint16_t)ti;
          }
          if (lane == 0) st.cnt[f] = cnt;
        }
        __syncthreads();
        // ---- rows
        team_eval<D, NF, NW>(
            ix, v.q(), uni(st.work), [&](int w) { return (int)(v.tkey()[v.work()[w]] & kTabIdMask); },
            [&](int w, float d) { v.tdist()[v.work()[w]] = d; });
        __syncthreads();
        if (threadIdx.x == 0) st.tcount += st.work;
      }
      // ---- expansions, then the next round's lists
      if (heaps) {
        if (warp == 0) team_commit_old(a, v, heap, k, ef);
      } else {
        team_expand_v1<NW>(a, v, k, ef, OLD && use_old);
      }
    }
    if (!OLD || !restart) break;
  }
  if (warp == 0) {
    if (heaps) {
      if (st.overflow) set_status(a.status, NMSG_ERR_CAPACITY);
      write_result_row(a, qi, v.items() + (ef + 1), st.overflow ? 0 : st.rsize, true);
    } else {
      write_result_row(a, qi, v.items(), min(k, st.num), false);
    }
    if (a.stats && lane == 0) {
      a.stats[qi * 4 + 0] = st.st_dist;
      a.stats[qi * 4 + 1] = st.st_expand;
      a.stats[qi * 4 + 2] = st.st_greedy;
      a.stats[qi * 4 + 3] = (int64_t)ix.row_bytes * st.st_dist + 4LL * st.st_list_ints;
    }
    __syncwarp();
  }
}

// search_team_kernel<D, NF, NW, OLD>: one block of NW warps per query, for batches that leave the
// one-warp-per-query kernels waiting: there a query is a chain of expansions (list, visited bytes,
// rows, merge: 6-7 us each on an otherwise idle GPU, 1M x 128), and below some thousand queries the
// longest chain is the whole call. Here the next `spec` candidates in line have their lists read and
// their new neighbours' rows measured in one round by all warps, ahead of their turn, and a round's
// expansions then follow one another without a memory access (about 4 per round on clustered data;
// a candidate that drops out of the beam before its turn wasted its rows, 5-20 % of them). Results
// and counts are those of the sequential walk: a distance does not depend on when it is computed, a
// neighbour joins the beam only at its candidate's turn, and only then is it visited.
//
// The visited set and the distances computed ahead share one open-addressing table in shared memory
// (visited bytes in HBM cost the other kernels a dependent read per expansion); a full table moves to
// the slot's epoch bytes. Bound by latency: a round is about 10K cycles, a quarter of them the two
// memory accesses (list, rows), the rest dependent shared-memory and vote instructions in six
// barrier-separated phases. Eight warps (4 blocks per SM) while the batch leaves SMs idle, four
// (8 blocks per SM) beyond. Measured against the one-warp kernels (kernel time, one B200): one query,
// 10K x 128 l2, efSearch 100: 242 -> 115 us; 16 queries, 1M x 128, efSearch 100: 766 -> 370 us; 300
// and 1,000 queries at efSearch 64: 919 -> 598 and 1,006 -> 802 us; 600 queries, 1M x 100 cosine,
// efSearch 200: 2,389 -> 940 us; 3,001 queries, 200K x 100 L1: 2,254 -> 1,476 us.
template <int D, int NF, int NW, bool OLD>
__global__ void __launch_bounds__(32 * NW, 32 / NW) search_team_kernel(const __grid_constant__ SearchArgs a) {
  const TeamView v{a.team.l, a.team.mpad, a.team.table_log2};
  if ((int)blockIdx.x >= a.num_slots) return;
  int item = blockIdx.x;  // the first queries go to the blocks in order, the rest as blocks come free
  while (item < a.nq) {
    team_query<D, NF, NW, OLD>(a, v, a.order ? a.order[item] : item);
    if (threadIdx.x == 0) v.st().item = gridDim.x + atomicAdd(a.work_counter, 1);
    __syncthreads();
    item = uni(v.st().item);
  }
}

}  // namespace
}  // namespace nmsg
