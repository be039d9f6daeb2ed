// route_block.cuh -- the whole routing stage of a decode / verify call (T <= 16, T*k <= 256) by the 512 threads of
// one block: router top-k (a warp per token), stable bucketing of the pairs by expert, offsets, run and tile
// lists. Used by k_route_block (route.cu) and by the gate/up GEMV (expert_gemv.cu), whose blocks each repeat it for
// themselves: 4.3 us of every block at T = 1, 5.8 at T = 13 (a chain of latencies: loads of the logits, shuffles, five
// barriers), against a launch of its own, 6.3 us at T = 1 and 12.7 at T = 5 (one block for all tokens in double
// arithmetic: 15 us for 16 tokens of 64 experts), and lists that travelled through memory.
//   * Selection. "Largest probability, ties to the lowest id" is "largest logit, ties to the lowest id" unless two
//     different logits round to one float probability (exp and the division by the sum are monotone): the ids come
//     from the logits' order. Where two of a token's k+1 largest differ by less than 1e-6 (equal ones have equal probabilities),
//     the k-th is so far below the largest that its probability might not be a normal float (kMaxSpread), or a logit is NaN or
//     +inf, the token's warp takes the general body instead (router_one_token: the reference's arithmetic to the letter, out of
//     line, so that calls without such tokens do not fetch it).
//   * Weights: double exponentials of the k selected logits over their sum in rank order; the sum over all experts
//     cancels and is not formed.
//   * With a router weight the logits are double tree sums (k_router_dots) and the warp first does what
//     k_router_flag / k_router_pairs do for longer calls: where two of the leaders are closer than 5e-7 of the
//     magnitude, all that can be in or next to the top-k are formed again in the reference's arithmetic.
//   * Bucketing: a thread per pair, ranks inside a warp by match, over warps and experts by prefix sums.
#pragma once
#include "kernels.h"
#include "route_small.cuh"
#include "router_exact.cuh"

namespace b200moe {

constexpr int kPairWarps = kSmallPairs / 32;

struct alignas(16) RouteBlock {
  int key[kSmallPairs];      // expert of pair t*k + s; kMaxExperts: dropped
  float w[kSmallPairs];
  uint16_t before[kPairWarps][kMaxExperts + 8];  // pairs of an expert: per warp, then in the warps before; [kMaxExperts]: dropped pairs
  int start[kMaxExperts + 1];
  int wsum[16], wmore[16];
  float floor[16];           // a token's logits from here on are to be refined first (+inf: none)
  int unsure;
  float row[4][kMaxExperts];  // near-tied tokens' logits
  double prod[256];           // products of one of them
  float cand[16][128];       // per warp
};
constexpr int kRouteBlockBytes = (int)sizeof(RouteBlock);

// The same by n rounds of arg-max, n <= 32: for the rare token with more candidates than warp_leaders ranks (a few residues
// mod 32 hold most of its leaders, or many logits are equal). Value and id.
static __device__ __noinline__ float2 warp_leaders_rounds(const float* lg, int E, int n, int lane) {
  float v[16], last = INFINITY;
  int last_id = -1;
  float2 mine = make_float2(-INFINITY, 0.f);
#pragma unroll
  for (int j = 0; j < 16; j++) v[j] = j * 32 + lane < E ? lg[j * 32 + lane] : -INFINITY;
  for (int r = 0; r < n; r++) {
    float bv = -INFINITY;
    int bi = kMaxExperts;  // none
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const int e = j * 32 + lane;
      if (e < E && (v[j] < last || (v[j] == last && e > last_id)) && (v[j] > bv || bi == kMaxExperts)) {
        bv = v[j];
        bi = e;
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) {
        bv = ov;
        bi = oi;
      }
    }
    last = bv;
    last_id = bi;
    if (lane == r) mine = make_float2(bv, __int_as_float(bi));
  }
  return mine;
}

// The k+1 largest of E <= 512 logits in order (value descending, id ascending), by one warp: lane i gets the i-th.
// s: 128 floats of the warp. Returns how many lanes have one, at least min(k+1, E); 0: a logit is NaN or +inf.
__device__ __forceinline__ int warp_leaders(const float* lg, int E, int k, int lane, float* s, float& vr, int& id) {
  float v[16];
  float lm = -INFINITY;  // the lane's largest
  bool odd = false;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    const int e = j * 32 + lane;
    v[j] = e < E ? lg[e] : -INFINITY;
    odd |= e < E && !(v[j] <= 3.0e38f);  // (-inf, a masked expert, has its place in the order)
    lm = fmaxf(lm, v[j]);
  }
  if (__any_sync(0xffffffffu, odd)) return 0;
  // the (k+1)-th largest of the lanes' maxima is a lower bound of the (k+1)-th largest logit
  int rank = 0;
#pragma unroll
  for (int i = 0; i < 32; i++) {
    const float o = __shfl_sync(0xffffffffu, lm, i);
    rank += (o > lm) || (o == lm && i < lane);
  }
  const float bound = __shfl_sync(0xffffffffu, lm, __ffs(__ballot_sync(0xffffffffu, rank == k)) - 1);
  float *cv = s, *sv = s + 64;
  int *ci = (int*)s + 32, *si = (int*)s + 96;
  int C = 0;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    const bool c = j * 32 + lane < E && v[j] >= bound;
    const unsigned bal = __ballot_sync(0xffffffffu, c);
    const int pos = C + __popc(bal & ((1u << lane) - 1u));
    if (c && pos < 32) {
      cv[pos] = v[j];
      ci[pos] = j * 32 + lane;
    }
    C += __popc(bal);
  }
  if (C > 32) {
    const float2 mine = warp_leaders_rounds(lg, E, min(k + 1, E), lane);
    vr = mine.x;
    id = __float_as_int(mine.y);
    return min(k + 1, E);
  }
  __syncwarp();
  if (lane < C) {
    const float mv = cv[lane];
    const int mi = ci[lane];
    int r = 0;
    for (int i = 0; i < C; i++) r += (cv[i] > mv) || (cv[i] == mv && ci[i] < mi);
    sv[r] = mv;
    si[r] = mi;
  }
  __syncwarp();
  vr = lane < C ? sv[lane] : -INFINITY;
  id = lane < C ? si[lane] : 0;
  __syncwarp();
  return C;
}

// Several equal logits in the last places: the next smaller one is none of the leaders, and might share their probability.
static __device__ __noinline__ bool warp_near_below(const float* lg, int E, float vk, int lane) {
  bool near = false;
  for (int e = lane; e < E; e += 32) near |= lg[e] < vk && !(vk - lg[e] > 1e-6f * fmaxf(1.f, fabsf(vk)));
  return __any_sync(0xffffffffu, near);
}

// Top-k ids and weights from the order of the logits: lane r < k gets the r-th (weights only if asked for). False where
// that does not decide.
__device__ __forceinline__ bool warp_topk(const float* lg, int E, int C, float vr, int k, int lane, bool weights, float& wv) {
  const float vn = __shfl_down_sync(0xffffffffu, vr, 1), mx = __shfl_sync(0xffffffffu, vr, 0), vk = __shfl_sync(0xffffffffu, vr, k - 1);
  // neighbours in the order closer than 1e-6, but not equal: their probabilities might round to one float
  if (__any_sync(0xffffffffu, lane < k && lane + 1 < C && vr != vn && !(vr - vn > 1e-6f * fmaxf(1.f, fabsf(vr)))) || C < k ||
      !(mx - vk <= kMaxSpread))
    return false;
  if (k < C && vk == __shfl_sync(0xffffffffu, vr, k) && warp_near_below(lg, E, vk, lane)) return false;
  if (!weights) return true;
  const double e = lane < k ? exp((double)vr - (double)mx) : 0.0;
  double kept = 0;
#pragma unroll 1
  for (int r = 0; r < k; r++) kept += shfl_f64(e, r);  // rank order, as the reference adds
  wv = lane < k ? (float)(e / kept) : 0.f;
  return true;
}

// ids and weights of one token whose logits are final: lane r < k gets the r-th.
__device__ __forceinline__ void warp_select(const float* lg, int C, int E, int k, int lane, bool exact, bool weights, float vr, int& id, float& wv) {
  if (C == 0 || exact || !warp_topk(lg, E, C, vr, k, lane, weights, wv)) {
    const float2 r = router_one_token(lg, E, k, lane);
    wv = r.x;
    id = __float_as_int(r.y);
  }
}

// The near-tied tokens of a call (bits of `left`): k_router_pairs' arithmetic for their logits from sc.floor on, then their
// selection. Four tokens at a time in the block's own copy (other blocks read the same logits at the same time and have to
// come to the same answer), the (token, expert) pairs dealt out to the 16 warps. One warp and one token at a time took 950 us
// for 16 tokens of 512 experts whose router rows are equal in pairs, this 210 (a call without near-ties: 93). Separate kernels
// would spread them over all SMs (180 and 172); 512 identical rows, where every pair is refined by every block, take 2.9 ms.
static __device__ __noinline__ void refine_tied(const RouteIn& q, RouteBlock& sc, unsigned left, bool write) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, E = q.E, k = q.k, d = q.d;
  while (left) {
    int tok[4], n = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      tok[i] = __ffs(left) - 1;
      n += left != 0;
      left &= left - 1;
      if (i < n && tid < E) sc.row[i][tid] = q.logits[(size_t)tok[i] * E + tid];
    }
    if (tid == 0) sc.unsure = 0;
    rs_sync();
    int at = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (i >= n) break;
      const float* lg = q.logits + (size_t)tok[i] * E;
      const uint16_t* x = q.x + (size_t)tok[i] * d;
      const float floor = sc.floor[tok[i]];
      for (int e0 = 0; e0 < E; e0 += 32)
        for (unsigned m = __ballot_sync(0xffffffffu, e0 + lane < E && lg[min(e0 + lane, E - 1)] >= floor); m; m &= m - 1)
          if ((at++ & 15) == warp) {
            const int e = e0 + __ffs(m) - 1;
            const float v = exact_logit(x, q.router + (size_t)e * d, d, nullptr, lane);
            if (lane == 0) {
              sc.row[i][e] = v;
              if (v != v) sc.unsure = 1;
            }
          }
    }
    rs_sync();
    if (sc.unsure) {  // sums on a rounding boundary: replayed one after the other
      if (warp == 0)
        for (int i = 0; i < n; i++)
          for (int e0 = 0; e0 < E; e0 += 32)
            for (unsigned m = __ballot_sync(0xffffffffu, e0 + lane < E && sc.row[i][e0 + lane] != sc.row[i][e0 + lane]); m; m &= m - 1) {
              const int e = e0 + __ffs(m) - 1, t = i == 0 ? tok[0] : i == 1 ? tok[1] : i == 2 ? tok[2] : tok[3];
              const float v = exact_logit(q.x + (size_t)t * d, q.router + (size_t)e * d, d, sc.prod, lane);
              if (lane == 0) sc.row[i][e] = v;
            }
      rs_sync();
    }
    if (warp < n) {
      const int t = warp == 0 ? tok[0] : warp == 1 ? tok[1] : warp == 2 ? tok[2] : tok[3];
      float vr, wv = 0.f;
      int id;
      const int C = warp_leaders(sc.row[warp], E, k, lane, sc.cand[warp], vr, id);
      warp_select(sc.row[warp], C, E, k, lane, q.exact, write, vr, id, wv);
      if (lane < k) {
        sc.key[t * k + lane] = id;
        sc.w[t * k + lane] = wv;
      }
    }
    rs_sync();
  }
}

// Threads 0..511 of a block, sc and the scratch behind it in shared memory. write: leave everything in q.rb, too.
// row_token (shared memory, [T*k]): the token of every permuted row. Calls emit(expert, first, count, at) for
// every non-empty expert from one thread; at: passes of `rows` rows of the experts before. Returns their number.
template <typename Emit>
__device__ __forceinline__ int route_block(const RouteIn& q, RouteBlock& sc, bool write, int rows, uint8_t* row_token, Emit emit) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = q.T, E = q.E, k = q.k, P = T * k;
  for (int i = tid; i < (int)sizeof(sc.before) / 4; i += 512) ((uint32_t*)sc.before)[i] = 0;
  if (q.logits) {
    if (warp < T) {
      const float* lg = q.logits + (size_t)warp * E;
      float vr, wv = 0.f;
      int id;
      const int C = warp_leaders(lg, E, k, lane, sc.cand[warp], vr, id);
      float floor = INFINITY;
      if (q.router && C > 0) {
        // (Leaders that are all exactly 0 -- a token or a router of zeros -- stay: an index-order sum that differs from
        // the tree's is too close to 0 for its probability to differ, and equal ones go to the lowest id.)
        const float top = __shfl_sync(0xffffffffu, vr, 0), margin = 5e-7f * fmaxf(1.f, fabsf(top));
        const float vn = __shfl_down_sync(0xffffffffu, vr, 1), kth = __shfl_sync(0xffffffffu, vr, min(k, E) - 1);
        if (__any_sync(0xffffffffu, lane < k && lane + 1 < C && vr - vn < margin) && (top != 0.f || kth != 0.f)) floor = kth - 2.f * margin;
      }
      if (floor == INFINITY) {
        warp_select(lg, C, E, k, lane, q.exact, write, vr, id, wv);
        if (lane < k) {
          sc.key[warp * k + lane] = id;
          sc.w[warp * k + lane] = wv;
        }
      }
      if (lane == 0) sc.floor[warp] = floor;
    }
    rs_sync();
    if (q.router) {
      const unsigned tied = __ballot_sync(0xffffffffu, lane < T && sc.floor[lane & 15] < INFINITY);
      if (tied) refine_tied(q, sc, tied, write);  // (uniform for the block)
    }
  } else {
    for (int p = tid; p < P; p += 512) {
      // a caller-supplied id outside [0, E) must never index anything: the pair is dropped (it sorts behind
      // every expert) and the status word records it
      int id = q.ids[(size_t)(p / k) * q.stride + p % k];
      if ((unsigned)id >= (unsigned)E) {
        if (write && q.rb.status && atomicCAS(q.rb.status, 0, kStatusBadId) == 0) q.rb.status[1] = id;
        id = kMaxExperts;
      }
      sc.key[p] = id;
      sc.w[p] = q.w[(size_t)(p / k) * q.stride + p % k];
    }
    rs_sync();
  }
  // ---- bucketing ----
  const bool live = tid < P;
  const int key = live ? sc.key[tid] : -1, pt = live ? tid / k : 0;
  unsigned same = 0;
  if (warp < kPairWarps) {
    same = __match_any_sync(0xffffffffu, key);
    if (live && lane == __ffs(same) - 1) sc.before[warp][key] = (uint16_t)__popc(same);
  }
  if (write && q.logits)
    for (int i = tid; i < T * kIdStride; i += 512) {
      const int t = i / kIdStride, s = i % kIdStride;
      q.rb.topids[i] = s < k ? sc.key[t * k + s] : 0;
      q.rb.topw[i] = s < k ? sc.w[t * k + s] : 0.f;
    }
  rs_sync();
  // a thread per expert (the first one also for the dropped pairs): its pairs before each warp's, its count
  int cnt = 0;
#pragma unroll
  for (int v = 0; v < kPairWarps; v++) {
    const int n = sc.before[v][tid];
    sc.before[v][tid] = (uint16_t)cnt;
    cnt += n;
  }
  if (tid == 0) {
    int c = 0;
    for (int v = 0; v < kPairWarps; v++) {
      const int n = sc.before[v][kMaxExperts];
      sc.before[v][kMaxExperts] = (uint16_t)c;
      c += n;
    }
  }
  // Ids may repeat within a token (a caller's, or the selection's on non-finite logits), so an expert can have
  // up to T*k rows: the first tile_cap of them stand at the expert's place among the non-empty ones, the tiles
  // cut from the rest behind all of those.
  const int more = cnt > q.tile_cap ? (cnt - 1) / q.tile_cap : 0, passes = (cnt + rows - 1) / rows;
  int a = cnt | (cnt > 0) << 16, b = more | passes << 16;  // sums of counts and of non-empty experts; of further tiles and of passes
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, a, o), v = __shfl_up_sync(0xffffffffu, b, o);
    if (lane >= o) {
      a += u;
      b += v;
    }
  }
  if (lane == 31) {
    sc.wsum[warp] = a;
    sc.wmore[warp] = b;
  }
  rs_sync();
  int all = 0, all_more = 0;
#pragma unroll
  for (int w2 = 0; w2 < 16; w2++) {
    const int u = sc.wsum[w2], v = sc.wmore[w2];
    if (w2 < warp) {
      a += u;
      b += v;
    }
    all += u;
    all_more += v;
  }
  const int n_rows = all & 0xffff, n_active = all >> 16;
  const int first = (a & 0xffff) - cnt, at = (a >> 16) - 1;
  sc.start[tid] = first;
  if (cnt > 0) emit(tid, first, cnt, (b >> 16) - passes);
  if (tid == 0) sc.start[kMaxExperts] = n_rows;
  if (write) {
    if (tid < E) q.rb.eoff[tid] = first;
    if (cnt > 0) {
      q.rb.runs[at] = Run{tid, first, cnt};
      q.rb.tiles[at] = Tile{tid, first, min(cnt, q.tile_cap)};
      for (int j = 1; j <= more; j++)
        q.rb.tiles[n_active + ((b & 0xffff) - more) + j - 1] = Tile{tid, first + j * q.tile_cap, min(cnt - j * q.tile_cap, q.tile_cap)};
    }
    if (tid == 0) {
      q.rb.eoff[E] = n_rows;  // pairs actually placed
      q.rb.n_runs[0] = n_active;
      q.rb.n_runs[1] = 1;
      q.rb.runs[kMaxExperts] = Run{0, P, T};
      q.rb.n_tiles[0] = n_active + (all_more & 0xffff);
      q.rb.n_tiles[1] = 1;
      q.rb.tiles_sh[0] = Tile{0, P, T};
    }
  }
  rs_sync();
  if (live) {
    const int row = sc.start[key] + sc.before[warp][key] + __popc(same & ((1u << lane) - 1u));
    row_token[row] = (uint8_t)pt;
    if (write) {
      // slot of the pair in the token's reduce order: ascending expert id; equal ids (a caller's duplicate, or
      // two dropped pairs) keep their slot order, so every slot is written
      int rank = 0;
#pragma unroll 4
      for (int p = pt * k; p < pt * k + k; p++) rank += (sc.key[p] < key) || (sc.key[p] == key && p < tid);
      q.rb.tokidx[row] = pt;
      q.rb.pw[row] = sc.w[tid];
      q.rb.pairids[(size_t)pt * k + rank] = key == kMaxExperts ? -1 : row;  // the combine skips negative rows
    }
  }
  return all_more >> 16;
}

// Scalar sigmoid gate of the shared expert (src/ref.cpp:623-626) of the tokens t0, t0 + step, ...: d-long dot products
// in double by 512 threads (tid: their number), gpart: [16][16] doubles of shared memory, sync: their barrier.
template <typename Sync>
__device__ __forceinline__ void gate_block(const RouteIn& q, int t0, int step, int tid, double* gpart, Sync sync) {
  const int lane = tid & 31, T = q.T, d = q.d, P = q.T * q.k;
#pragma unroll 1
  for (int t = t0; t < T; t += step) {
    double a = 0;
    const uint4* xv = (const uint4*)(q.x + (size_t)t * d);
    const uint4* gv = (const uint4*)q.gate_w;
#pragma unroll 1
    for (int c = tid; c < d / 8; c += 512) {
      const uint4 xa = xv[c], ga = __ldg(gv + c);
      const uint32_t xw[4] = {xa.x, xa.y, xa.z, xa.w}, gq[4] = {ga.x, ga.y, ga.z, ga.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        a += (double)__uint_as_float(gq[i] << 16) * (double)__uint_as_float(xw[i] << 16);
        a += (double)__uint_as_float(gq[i] & 0xFFFF0000u) * (double)__uint_as_float(xw[i] & 0xFFFF0000u);
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1)
      a += __hiloint2double(__shfl_xor_sync(0xffffffffu, __double2hiint(a), o),
                            __shfl_xor_sync(0xffffffffu, __double2loint(a), o));
    if (lane == 0) gpart[t * 16 + (tid >> 5)] = a;
  }
  sync();
  if (tid < T && tid >= t0 && (tid - t0) % step == 0) {
    double tot = 0;
#pragma unroll 1
    for (int w2 = 0; w2 < 16; w2++) tot += gpart[tid * 16 + w2];
    const float gate = sigmoid_f32((float)tot);
    q.rb.sgate[tid] = gate;
    q.rb.tokidx[P + tid] = tid;
    q.rb.pw[P + tid] = gate;
  }
}

}  // namespace b200moe
