// pair_rows.cuh — the explicit reduced camera system S from camera pairs.
//
// Write W_o = A_o^T Jp_o and E_o = W_o Vhat_p^-1 (A the 2 x 9 camera columns of an observation's record,
// Jp its 2 x 3 point columns). The point coupling of cameras c <= c' is
//   K(c, c') = sum over points p seen by both, over their observations a (of c) and b (of c'): W_a E_b^T,
// a 9 x 9 block over the cameras' own parameters (pose columns, then intrinsic columns), and
//   S_XY = U_XY - (the rows of X and columns of Y of K, summed over the cameras that own them).
// Only the pairs c <= c' are formed and S_YX is S_XY's transpose: half the products of a build by rows.
// The inverse stays on the side of the later camera, as in a row of the lower triangle (the triangle
// the factorization reads), so weakly conditioned points enter the factor as they do in a build by
// rows. U_XY (diagonal blocks and pose/intrinsic edges) is taken from the camera-side assembly records.
//
// The pair lists (which observations meet in each camera pair) depend only on the topology: they are
// built on the device at a solver's first build and kept with it. A build is three kernels:
//   k_pair_operands  W and E of every observation, observation-major, from the record tiles (streaming);
//   k_pair_products  one warp per item, an item being at most `chunk` entries of one pair's list: the
//                    entries' W and E are concatenated along k into FP64 m8n8k4 tensor products, so
//                    four entries take three k-steps with nothing but the 9th row and column padded;
//   k_pair_gather    one warp per block S_XY (one CTA where a shared intrinsic group collects more
//                    than kPairHeavy pairs): the items of its pairs in list order, plus U.
// Every list is in a fixed order (ascending camera, then observation) and every sum runs in it, so the
// rows are the same bits run to run.
//
// Bound: the gather of W and E through L2 (2 x 27 doubles per entry), then the FP64 pipe. Splitting lists
// into items keeps the chip busy whatever the shape: 20 cameras that share one intrinsic group have
// 210 pairs, where a CTA per block row left one CTA walking every observation of the group.
// Measured on a B200, build by block rows -> by pairs: 3,000 cameras / 12M observations (FP32 records)
// 81 -> 6.6 ms (operands 1.3, products 4.9), 500 cameras / 1.2M observations 9.1 -> 0.7 ms, a 20-camera
// window of 8,000 observations 0.34 -> 0.04 ms, the same window with one shared intrinsic group
// 12.8 -> 0.1 ms.
#pragma once

#include <cstdint>

namespace omvgba {

constexpr int kPairDim = 9;                      // parameters of a camera: pose (<= 6), intrinsics (<= 3)
constexpr int kPairPart = kPairDim * kPairDim;   // doubles of one item's product
constexpr uint32_t kPairHeavy = 64;              // contributions from which a block takes a whole CTA

struct CamPairs {
  int ncam, segs, gw;            // gw: doubles per observation in W and in E (3 x the widest camera)
  uint32_t npairs, nitems, chunk;
  const uint32_t* pt_off;        // P + 1
  const uint32_t* obs_cam;       // N
  const uint32_t* obs_point;     // N
  const uint8_t* fixed_points;   // P
  const int* unit_dim;           // free parameters of each camera, 0: the camera has no unit
  const uint32_t* cam_begin;     // ncam + 1: each camera's range in cam_obs
  const uint32_t* cam_obs;       // N: observations of each camera, ascending
  const uint32_t* adj_begin;     // ncam + 1: each camera's range in adj
  const uint32_t* adj;           // cameras sharing a free point with it (itself included), ascending
  const uint32_t* up_begin;      // ncam + 1: first pair of each camera (its neighbours >= itself)
  const uint64_t* list_begin;    // npairs x segs + 1: entries of each pair, by segment of its camera
  const uint2* entries;          // (observation of c, observation of c')
  const uint32_t* item_begin;    // npairs + 1
  const uint32_t* item_pair;     // nitems
};

__device__ __forceinline__ uint32_t pair_adj_first_up(const CamPairs& t, uint32_t c) {
  return t.adj_begin[c + 1] - (t.up_begin[c + 1] - t.up_begin[c]);
}
// Pair (c, c2), c <= c2: its index, or 0xFFFFFFFF when the cameras share no free point.
__device__ __forceinline__ uint32_t pair_find(const CamPairs& t, uint32_t c, uint32_t c2) {
  const uint32_t first = pair_adj_first_up(t, c), end = t.adj_begin[c + 1];
  uint32_t lo = first, hi = end;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (t.adj[mid] < c2)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < end && t.adj[lo] == c2 ? t.up_begin[c] + (lo - first) : 0xFFFFFFFFu;
}

// ---- topology (once per solver) ---------------------------------------------------------------
__global__ void k_pair_units(int ncam, const int* __restrict__ pose_dim, const uint32_t* __restrict__ cam_group,
                             const int* __restrict__ intr_dim, int self_cal, int* __restrict__ unit_dim) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < ncam) unit_dim[c] = pose_dim[c] + (self_cal ? intr_dim[cam_group[c]] : 0);
}

__global__ void k_pair_obs_point(int P, const uint32_t* __restrict__ pt_off, uint32_t* __restrict__ obs_point) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  for (uint32_t o = pt_off[p]; o < pt_off[p + 1]; ++o) obs_point[o] = (uint32_t)p;
}

// Observations of each camera, ascending (a stable counting sort): one warp per chunk of consecutive
// observations counts its cameras into counts[chunk][camera]; with cam_obs non-null the counters
// hold the chunk's offsets inside each camera's range and the warp places its observations.
__global__ void __launch_bounds__(32) k_pair_cam_sort(uint32_t n, uint32_t per, int ncam,
                                                      const uint32_t* __restrict__ obs_cam, uint32_t* counts,
                                                      const uint32_t* __restrict__ cam_begin, uint32_t* cam_obs) {
  uint32_t* cnt = counts + (size_t)blockIdx.x * ncam;
  const uint32_t b = blockIdx.x * per, e = min(n, b + per), lane = threadIdx.x;
  for (uint32_t base = b; base < e; base += 32) {
    const uint32_t o = base + lane;
    const uint32_t c = o < e ? obs_cam[o] : 0xFFFFFFFFu;
    const uint32_t same = __match_any_sync(0xffffffffu, c);
    const uint32_t rank = __popc(same & ((1u << lane) - 1u));
    uint32_t at = 0;
    if (o < e && rank == 0) {
      at = cnt[c];
      cnt[c] = at + __popc(same);
    }
    at = __shfl_sync(0xffffffffu, at, __ffs(same) - 1);
    if (cam_obs && o < e) cam_obs[cam_begin[c] + at + rank] = o;
    __syncwarp();  // the counters written above are read by other lanes next round
  }
}
__global__ void k_pair_cam_prefix(int ncam, int nchunks, uint32_t* counts, uint32_t* total) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncam) return;
  uint32_t run = 0;
  for (int k = 0; k < nchunks; ++k) {
    const uint32_t v = counts[(size_t)k * ncam + c];
    counts[(size_t)k * ncam + c] = run;
    run += v;
  }
  total[c] = run;
}

// out[0..n] = exclusive prefix sums of in[0..n), one CTA: each thread its contiguous share. total: the sum
// itself, where it may be past TOut.
template <typename TOut>
__global__ void __launch_bounds__(1024) k_pair_scan(const uint32_t* __restrict__ in, size_t n, TOut* __restrict__ out,
                                                    unsigned long long* total) {
  __shared__ unsigned long long warp_tot[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t per = (n + blockDim.x - 1) / blockDim.x, b = min(n, per * tid), e = min(n, b + per);
  unsigned long long sum = 0;
  for (size_t i = b; i < e; ++i) sum += in[i];
  unsigned long long inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  unsigned long long run = inc - sum;
  for (int w = 0; w < warp; ++w) run += warp_tot[w];
  for (size_t i = b; i < e; ++i) {
    out[i] = (TOut)run;
    run += in[i];
  }
  if (tid == (int)blockDim.x - 1) {
    out[n] = (TOut)run;
    if (total) *total = run;
  }
}

// Neighbours of each camera: one CTA per camera marks them in a bitmap (dynamic shared memory, a bit
// per camera). Without adj: their number, and the number at or above the camera itself. With adj:
// the ascending list.
__global__ void __launch_bounds__(256) k_pair_neighbours(CamPairs t, uint32_t* full, uint32_t* upper, uint32_t* adj) {
  extern __shared__ uint32_t bits[];
  __shared__ uint32_t s_full, s_up;
  const uint32_t c = blockIdx.x;
  const int words = (t.ncam + 31) >> 5, tid = threadIdx.x, lane = tid & 31;
  for (int w = tid; w < words; w += blockDim.x) bits[w] = 0;
  if (tid == 0) s_full = s_up = 0;
  __syncthreads();
  if (t.unit_dim[c] > 0)
    for (uint32_t i = t.cam_begin[c] + tid; i < t.cam_begin[c + 1]; i += blockDim.x) {
      const uint32_t p = t.obs_point[t.cam_obs[i]];
      if (t.fixed_points[p]) continue;
      for (uint32_t k = t.pt_off[p]; k < t.pt_off[p + 1]; ++k) {
        const uint32_t c2 = t.obs_cam[k];
        if (t.unit_dim[c2] > 0) atomicOr(&bits[c2 >> 5], 1u << (c2 & 31));
      }
    }
  __syncthreads();
  if (!adj) {
    uint32_t nf = 0, nu = 0;
    for (int w = tid; w < words; w += blockDim.x) {
      const uint32_t b = bits[w];
      nf += __popc(b);
      const int lo = (int)c - 32 * w;  // bits from lo up belong to cameras >= c
      nu += lo <= 0 ? __popc(b) : (lo < 32 ? __popc(b & (0xFFFFFFFFu << lo)) : 0);
    }
    atomicAdd(&s_full, nf);
    atomicAdd(&s_up, nu);
    __syncthreads();
    if (tid == 0) {
      full[c] = s_full;
      upper[c] = s_up;
    }
    return;
  }
  if (tid >= 32) return;
  uint32_t at = t.adj_begin[c];
  for (int w0 = 0; w0 < words; w0 += 32) {
    uint32_t b = w0 + lane < words ? bits[w0 + lane] : 0;
    const uint32_t n = __popc(b);
    uint32_t inc = n;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    uint32_t q = at + inc - n;
    while (b) {
      adj[q++] = 32 * (w0 + lane) + __ffs(b) - 1;
      b &= b - 1;
    }
    at += __shfl_sync(0xffffffffu, inc, 31);
  }
}

// Entries of the pair lists: warp (camera c, segment) walks its share of c's observations in order,
// 32 at a time, their tracks flattened over the lanes. Without entries it counts into
// counts[pair x segs + segment]; with entries the counters hold list offsets and the warp places
// (observation of c, observation of c') in (observation, track) order.
template <typename TCnt>
__global__ void __launch_bounds__(32) k_pair_lists(CamPairs t, TCnt* counts, uint2* entries) {
  const uint32_t c = blockIdx.x, seg = blockIdx.y, lane = threadIdx.x;
  if (t.unit_dim[c] == 0) return;
  const uint32_t c0 = t.cam_begin[c], len = t.cam_begin[c + 1] - c0;
  const uint32_t b = c0 + (uint32_t)((uint64_t)len * seg / t.segs), e = c0 + (uint32_t)((uint64_t)len * (seg + 1) / t.segs);
  for (uint32_t base = b; base < e; base += 32) {
    uint32_t o = 0, first = 0, n = 0;
    if (base + lane < e) {
      o = t.cam_obs[base + lane];
      const uint32_t p = t.obs_point[o];
      if (!t.fixed_points[p]) {
        first = t.pt_off[p];
        n = t.pt_off[p + 1] - first;
      }
    }
    uint32_t inc = n;
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, s);
      if (lane >= s) inc += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    for (uint32_t k0 = 0; k0 < total; k0 += 32) {
      const uint32_t k = k0 + lane;
      uint32_t src = 0;  // the lane whose track holds position k: the first with inc > k
      for (int s = 16; s > 0; s >>= 1) {
        const uint32_t v = __shfl_sync(0xffffffffu, inc, src + s - 1);
        if (v <= k) src += s;
      }
      src = min(src, 31u);
      const uint32_t so = __shfl_sync(0xffffffffu, o, src), sf = __shfl_sync(0xffffffffu, first, src),
                     se = __shfl_sync(0xffffffffu, inc - n, src);
      uint32_t pair = 0xFFFFFFFFu, ob = 0;
      if (k < total) {
        ob = sf + (k - se);
        const uint32_t c2 = t.obs_cam[ob];
        if (c2 >= c && t.unit_dim[c2] > 0) pair = pair_find(t, c, c2);
      }
      const uint32_t same = __match_any_sync(0xffffffffu, pair);
      const uint32_t rank = __popc(same & ((1u << lane) - 1u));
      const bool have = pair != 0xFFFFFFFFu;
      TCnt* cell = counts + (size_t)(have ? pair : 0) * t.segs + seg;
      const TCnt at = have ? *cell : 0;
      __syncwarp();  // every lane has read the counters before one of them moves on
      if (have && rank == 0) *cell = at + (TCnt)__popc(same);
      if (have && entries) entries[at + rank] = make_uint2(so, ob);
      __syncwarp();
    }
  }
}

__global__ void k_pair_item_count(CamPairs t, uint32_t* count) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= t.npairs) return;
  const uint64_t n = t.list_begin[(size_t)(p + 1) * t.segs] - t.list_begin[(size_t)p * t.segs];
  count[p] = (uint32_t)((n + t.chunk - 1) / t.chunk);
}
__global__ void k_pair_item_fill(CamPairs t, uint32_t* item_pair) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= t.npairs) return;
  for (uint32_t i = t.item_begin[p]; i < t.item_begin[p + 1]; ++i) item_pair[i] = p;
}

// Contributions of the camera pairs to each block S_XY, one warp per block: the cameras that own X
// (a pose block's camera, every camera of an intrinsic group), ascending, and for each its neighbours
// that own Y; from Y's side when Y has fewer cameras. A contribution is (pair | transposed << 31,
// first row of X | first column of Y << 8) in the pair's 9 x 9 product. Without out: the number.
struct BlockCams {
  const uint32_t* begin;      // nb + 1
  const uint32_t* cams;       // cameras that own each block, ascending
  const int* blk_pose;        // camera of a pose block, -1 for an intrinsic block
  const int* blk_group;       // group of an intrinsic block, -1 for a pose block
  const uint32_t* cam_group;  // ncam
  const int* pose_dim;        // ncam
};
__global__ void __launch_bounds__(256) k_pair_slots(CamPairs t, BlockCams bc, uint32_t slots,
                                                    const int* __restrict__ nbr, const int* __restrict__ nbr_row,
                                                    uint32_t* count, const uint32_t* __restrict__ begin, uint2* out,
                                                    uint32_t* heavy_n, uint32_t* heavy) {
  const uint32_t q = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (q >= slots) return;
  int X = nbr_row[q], Y = nbr[q];
  const bool swap = bc.begin[Y + 1] - bc.begin[Y] < bc.begin[X + 1] - bc.begin[X];
  if (swap) {
    const int s = X;
    X = Y;
    Y = s;
  }
  uint32_t at = out ? begin[q] : 0, n = 0;
  for (uint32_t i = bc.begin[X]; i < bc.begin[X + 1]; ++i) {
    const uint32_t cx = bc.cams[i];
    for (uint32_t k0 = t.adj_begin[cx]; k0 < t.adj_begin[cx + 1]; k0 += 32) {
      uint32_t cy = 0;
      bool hit = false;
      if (k0 + lane < t.adj_begin[cx + 1]) {
        cy = t.adj[k0 + lane];
        hit = bc.blk_pose[Y] >= 0 ? (int)cy == bc.blk_pose[Y] : (int)bc.cam_group[cy] == bc.blk_group[Y];
      }
      const uint32_t mask = __ballot_sync(0xffffffffu, hit);
      if (hit && out) {
        const uint32_t ox = bc.blk_pose[X] >= 0 ? 0 : bc.pose_dim[cx], oy = bc.blk_pose[Y] >= 0 ? 0 : bc.pose_dim[cy];
        // the block's row side is the smaller camera of the pair unless the pair is transposed
        const uint32_t row = swap ? cy : cx, col = swap ? cx : cy;
        // (a camera with itself: transposed, so that the row side carries the inverse)
        const uint32_t tr = row >= col ? 1u : 0u;
        const uint32_t pair = tr ? pair_find(t, col, row) : pair_find(t, row, col);
        out[at + __popc(mask & ((1u << lane) - 1u))] =
            make_uint2(pair | tr << 31, (swap ? oy : ox) | (swap ? ox : oy) << 8);
      }
      at += __popc(mask);
      n += __popc(mask);
    }
  }
  if (lane == 0) {
    if (!out)
      count[q] = n;
    else if (n > kPairHeavy)
      heavy[atomicAdd(heavy_n, 1u)] = q;  // the order of this list does not matter
  }
}

// ---- a build ------------------------------------------------------------------------------------
// W and E of every observation of a tile (thread per observation), gw doubles each,
// observation-major, through shared memory so the stores are coalesced.
template <typename R>
__global__ void __launch_bounds__(mv_tile_obs<R>()) k_pair_operands(MvTiles mt, LinOut<R> lin, int gw,
                                                                    const uint32_t* __restrict__ pt_off,
                                                                    double* __restrict__ W, double* __restrict__ E) {
  constexpr int TILE = mv_tile_obs<R>();
  extern __shared__ double g_sh[];  // TILE x gw
  const int t = blockIdx.x, tid = threadIdx.x;
  const uint4 hdr = mt.tile_hdr[t];
  const uint32_t nobs = hdr.x, p0 = hdr.w;
  const unsigned char* slot = mt.slots + (size_t)t * MvSlot::bytes(TILE);
  const size_t o0 = pt_off[p0];
  const bool live = (uint32_t)tid < nobs;
  double w[3 * kPairDim], P[6];
  double* mine = g_sh + (size_t)tid * gw;
  if (live) {
    const R* r = lin.rec + (size_t)t * TILE * kRec + tid;
    double jp[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) jp[c] = (double)r[(size_t)(kJp + c) * TILE];
    const uint32_t lp = reinterpret_cast<const uint16_t*>(slot + MvSlot::lpt(TILE))[tid];
    const double* vi = lin.vinv + 6 * (size_t)(p0 + lp);
#pragma unroll
    for (int c = 0; c < 6; ++c) P[c] = vi[c];
#pragma unroll
    for (int c = 0; c < kPairDim; ++c)
      if (3 * c < gw) {
        const double a0 = (double)r[(size_t)c * TILE], a1 = (double)r[(size_t)(9 + c) * TILE];
#pragma unroll
        for (int d = 0; d < 3; ++d) mine[3 * c + d] = w[3 * c + d] = a0 * jp[d] + a1 * jp[3 + d];
      }
  }
  __syncthreads();
  for (uint32_t i = tid; i < nobs * (uint32_t)gw; i += TILE) W[o0 * gw + i] = g_sh[i];
  __syncthreads();
  if (live) {
#pragma unroll
    for (int c = 0; c < kPairDim; ++c)
      if (3 * c < gw) sym3_apply(P, w + 3 * c, mine + 3 * c);
  }
  __syncthreads();
  for (uint32_t i = tid; i < nobs * (uint32_t)gw; i += TILE) E[o0 * gw + i] = g_sh[i];
}

// Item products: K = sum over the item's entries of W_a E_b^T. Lane l holds A(l / 4, l % 4),
// B(l % 4, l / 4) and C(l / 4, 2 (l % 4) + i); k runs over (entry, component of the point), four
// entries in three steps. WIDE: cameras with 9 parameters, whose 9th row and column take three more
// products.
template <bool WIDE>
__global__ void __launch_bounds__(256) k_pair_products(CamPairs t, const double* __restrict__ W,
                                                       const double* __restrict__ E, double* __restrict__ part) {
  const uint32_t item = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31, g = lane >> 2, f = lane & 3;
  if (item >= t.nitems) return;
  const uint32_t pair = t.item_pair[item];
  const uint64_t l0 = t.list_begin[(size_t)pair * t.segs], l1 = t.list_begin[(size_t)(pair + 1) * t.segs];
  const uint64_t b = l0 + (uint64_t)(item - t.item_begin[pair]) * t.chunk;
  const uint32_t n = (uint32_t)min((uint64_t)t.chunk, l1 - b);
  const int gw = t.gw, rows = gw / 3;
  const bool live = g < rows;  // rows of a narrow camera end here
  // k-step s: this lane's entry of the four and its component
  int ej[3], ed[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int kk = 4 * s + f;
    ej[s] = kk / 3;
    ed[s] = kk - 3 * ej[s];
  }
  double c00[2] = {0, 0}, c01[2] = {0, 0}, c10[2] = {0, 0}, c11[2] = {0, 0};
  for (uint32_t base = 0; base < n; base += 32) {
    const uint32_t m = min(32u, n - base);
    const uint2 mine = lane < (int)m ? t.entries[b + base + lane] : make_uint2(0u, 0u);
#pragma unroll 2
    for (uint32_t q = 0; q < m; q += 4) {
      double a0[3], b0[3], a1[3], b1[3];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const uint32_t j = q + ej[s];
        const uint32_t oa = __shfl_sync(0xffffffffu, mine.x, j & 31), ob = __shfl_sync(0xffffffffu, mine.y, j & 31);
        const bool in = j < m;
        const double* pa = W + (size_t)oa * gw + ed[s];
        const double* pb = E + (size_t)ob * gw + ed[s];
        a0[s] = in && live ? __ldg(pa + 3 * g) : 0.0;
        b0[s] = in && live ? __ldg(pb + 3 * g) : 0.0;
        if (WIDE) {
          a1[s] = in && g == 0 ? __ldg(pa + 24) : 0.0;
          b1[s] = in && g == 0 ? __ldg(pb + 24) : 0.0;
        }
      }
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        dmma_m8n8k4(a0[s], b0[s], c00[0], c00[1]);
        if (WIDE) {
          dmma_m8n8k4(a0[s], b1[s], c01[0], c01[1]);
          dmma_m8n8k4(a1[s], b0[s], c10[0], c10[1]);
          dmma_m8n8k4(a1[s], b1[s], c11[0], c11[1]);
        }
      }
    }
  }
  double* out = part + (size_t)item * kPairPart;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    out[g * kPairDim + 2 * f + i] = c00[i];
    if (WIDE && g == 0) out[8 * kPairDim + 2 * f + i] = c10[i];
  }
  if (WIDE && f == 0) {
    out[g * kPairDim + 8] = c01[0];
    if (g == 0) out[8 * kPairDim + 8] = c11[0];
  }
}

// U_XY of block q from the camera-side records: the diagonal block (symmetric, packed lower) and the
// edge between a pose block and its camera's intrinsic block.
__device__ __forceinline__ double pair_u(const double* __restrict__ blk_out, const int* __restrict__ blk_edge, int X,
                                         int Y, int m, int k) {
  if (X == Y) {
    const int r = max(m, k), c = min(m, k);
    return blk_out[(size_t)kAsmRec * X + r * (r + 1) / 2 + c];
  }
  if (blk_edge[X] == Y) return blk_out[(size_t)kAsmRec * X + 39 + 3 * m + k];
  if (blk_edge[Y] == X) return blk_out[(size_t)kAsmRec * Y + 39 + 3 * k + m];
  return 0.0;
}

// Sum of element (m, k) over contributions [i, e) of a block, every `step`-th, items in order.
__device__ __forceinline__ double pair_sum(const CamPairs& t, const uint2* __restrict__ cont, uint32_t i, uint32_t e,
                                           uint32_t step, int m, int k, const double* __restrict__ part) {
  double acc = 0.0;
  for (; i < e; i += step) {
    const uint2 c = cont[i];
    const uint32_t pair = c.x & 0x7FFFFFFFu;
    const int r = (int)(c.y & 0xFF) + m, col = (int)(c.y >> 8) + k;
    const double* p = part + ((c.x >> 31) ? col * kPairDim + r : r * kPairDim + col);
    const uint32_t i1 = t.item_begin[pair + 1];
    for (uint32_t it = t.item_begin[pair]; it < i1; ++it) acc += p[(size_t)it * kPairPart];
  }
  return acc;
}

__global__ void __launch_bounds__(256) k_pair_gather(CamPairs t, RowTables rt, const uint32_t* __restrict__ cont_begin,
                                                     const uint2* __restrict__ cont, const double* __restrict__ part,
                                                     const double* __restrict__ blk_out, const int* __restrict__ blk_edge,
                                                     double* __restrict__ rows) {
  const uint32_t q = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (q >= rt.entries) return;
  const uint32_t i0 = cont_begin[q], i1 = cont_begin[q + 1];
  if (i1 - i0 > kPairHeavy) return;  // k_pair_gather_heavy's
  const int X = rt.nbr_row[q], Y = rt.nbr[q], dX = rt.blk_dim[X], dY = rt.blk_dim[Y];
  for (int e = lane; e < dX * dY; e += 32) {
    const int m = e / dY, k = e - m * dY;
    rows[rt.slot_off[q] + e] = pair_u(blk_out, blk_edge, X, Y, m, k) - pair_sum(t, cont, i0, i1, 1, m, k, part);
  }
}

// The blocks with many contributions: one CTA per block, thread = (element, share of the contributions),
// the shares combined in order.
constexpr int kPairShares = 16;
__global__ void __launch_bounds__(36 * kPairShares) k_pair_gather_heavy(
    CamPairs t, RowTables rt, const uint32_t* __restrict__ cont_begin, const uint2* __restrict__ cont,
    const double* __restrict__ part, const double* __restrict__ blk_out, const int* __restrict__ blk_edge,
    const uint32_t* __restrict__ heavy_n, const uint32_t* __restrict__ heavy, double* __restrict__ rows) {
  __shared__ double sh[kPairShares][36];
  const int e = threadIdx.x % 36, share = threadIdx.x / 36;
  for (uint32_t h = blockIdx.x; h < *heavy_n; h += gridDim.x) {
    const uint32_t q = heavy[h];
    const int X = rt.nbr_row[q], Y = rt.nbr[q], dX = rt.blk_dim[X], dY = rt.blk_dim[Y];
    const int m = e / dY, k = e - m * dY;
    if (e < dX * dY) sh[share][e] = pair_sum(t, cont, cont_begin[q] + share, cont_begin[q + 1], kPairShares, m, k, part);
    __syncthreads();
    if (share == 0 && e < dX * dY) {
      double acc = 0.0;
      for (int s = 0; s < kPairShares; ++s) acc += sh[s][e];
      rows[rt.slot_off[q] + e] = pair_u(blk_out, blk_edge, X, Y, m, k) - acc;
    }
    __syncthreads();
  }
}

}  // namespace omvgba
