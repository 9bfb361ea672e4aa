// explicit_s.cuh — the explicit reduced camera system S and its banded tiled FP64 Cholesky factor.
//
// S = U - W Vhat^-1 W^T over the free camera parameters (schur/assembly.rs:832-1069 assembles the same
// matrix into faer's sparse pattern, sparse/direct_assembly.rs:371-687). It is built from camera
// pairs (pair_rows.cuh), or, where their lists do not fit the caller's workspace budget, by block rows:
// one CTA per parameter block X computes every block S_XY of its row (all co-visible blocks Y, both
// triangles), walking X's entities in a fixed order and the entities of each entity's point, so the
// row is the same bits run to run, needs no atomics and no storage beyond the rows. The rows serve as
// a block-sparse (BSR) operator directly (the PCG product and the model reduction) and are scattered
// into a banded tiled matrix for the factorization.
//
// Factorization. The parameter blocks are permuted so that each camera's pose block is followed by
// the intrinsic blocks it introduces; with cameras in their native order the co-visibility graph of
// a survey is banded, so the factor fits in a band of tiles (64 x 64 FP64, column-major) and a
// right-looking tiled Cholesky (POTRF of the diagonal tile, TRSM of the tiles below it, SYRK/GEMM
// update of the trailing band) never leaves the band. faer's sparse LLT with an AMD ordering
// (numerics/sparse.rs:119-250) factors the same matrix; the factors agree to rounding and the
// positive-definiteness decision is the same away from rounding-level pivots. Every tile update
// runs in a fixed order, so the factor is bitwise reproducible.
//
// Uses of the factor: the direct camera step (sparse/direct.rs:259-288), the camera rank test of the
// final undamped system (sparse/direct.rs:288-455: the spectral test after Jacobi equilibration
// when D <= 2048, a factorization otherwise), and the self-calibration intrinsic marginal
// covariances (sparse/covariance.rs:564-587) from the selected inverse of S inside the band.
#pragma once

#include <cooperative_groups.h>

#include <cstdint>

namespace omvgba {

// ---- block rows ---------------------------------------------------------------------------------
struct RowTables {
  int nblocks;
  const int* blk_dim;
  const int* blk_off;
  const uint32_t* blk_ent;    // nb + 1: each block's range in ent
  const uint32_t* ent;        // entity list (observation * 2 + segment), block-major
  const uint32_t* ent_point;  // point of each entity (same order)
  const int* seg_col;         // per entity id: column of its segment in the observation's record
  const int* ent_block;       // per entity id: parameter block, -1 when absent
  const uint32_t* pt_off;     // P + 1
  const uint32_t* nbr_begin;  // nb + 1: each block's range in nbr / slot_off
  const int* nbr;             // neighbour blocks of each block (ascending; the block itself included)
  const int* nbr_row;         // block owning each neighbour entry
  const uint64_t* slot_off;   // entries + 1: offset of block S_XY (dX x dY, row-major) in the rows
  uint32_t entries;           // neighbour entries in total
};


// D = A B + C for 8 x 8 FP64 tiles with k = 4 (mma.sync.m8n8k4 f64): each lane passes one element
// of A, one of B and two of C, updated in place.
__device__ __forceinline__ void dmma_m8n8k4(double a, double b, double& c0, double& c1) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ int find_slot(const int* __restrict__ nbr, uint32_t n0, uint32_t n1, int Y) {
  uint32_t lo = n0, hi = n1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (nbr[mid] < Y)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (lo < n1 && nbr[lo] == Y) ? (int)(lo - n0) : -1;
}

// Row X of S. Each entity e of X (observation o of point p, camera columns cX..cX+dX of its
// record) meets every entity e' of p's track in a block Y (observation k, columns cY..cY+dY):
//   S_XY += [k == o] A_o,X^T A_o,Y - E_e W_k,Y^T,   E_e = A_o,X^T Jp_o Vhat_p^-1 (dX x 3),
//   W_k,Y = A_k,Y^T Jp_k (dY x 3),
// U, the pose/intrinsic edges and the point coupling in one sum (A = the 2 x 9 camera columns and
// Jp the 2 x 3 point columns of a record).
//
// One CTA per row, kRowWarps warps. The row's entities are taken kRowWarps at a time, one per warp:
// the warp computes E of its entity and W of every observation of the track (a chunk of at most
// kRowStage observations per round; longer tracks take several rounds) into shared memory, and the
// slot of each target. After a barrier every warp adds the batch's contributions to the slots it
// owns (slot index mod kRowWarps), entity by entity in batch order and target by target in track
// order, one tensor-pipe product per target. Each element therefore has one writer and a fixed
// summation order: the row is the same bits run to run, without atomics. The row accumulates in
// shared memory when it has at most row_smem doubles (else in place in global memory) and is
// stored once at the end. Each warp fetches the indices of its next entity a batch ahead.
constexpr int kRowWarps = 8;
constexpr int kRowThreads = 32 * kRowWarps;
constexpr int kRowStage = 16;           // track observations per round (2 targets each: 32 lanes)
constexpr int kRowNbr = 1024;           // neighbour lists up to this length sit in shared memory
constexpr int kRowSmemDoubles = 8192;   // rows up to 64 KB accumulate in shared memory
template <typename R>
__global__ void __launch_bounds__(kRowThreads, 2) k_block_rows(RowTables rt, LinOut<R> lin, int row_smem,
                                                               double* __restrict__ rows) {
  extern __shared__ double row_sh[];
  __shared__ int nbr_s[kRowNbr];                       // neighbour blocks
  __shared__ uint32_t ninf_s[kRowNbr];                 // (offset in the row) << 3 | dY
  __shared__ double Wsh[kRowWarps][kRowStage][27];     // W of each chunk observation, 9 x 3 row-major
  __shared__ double Osh[kRowWarps][32];                // the entity's record: A (18), Jp (6), Vhat^-1 (6)
  __shared__ double Esh[kRowWarps][18];                // E (dX x 3)
  __shared__ int tsl[kRowWarps][2 * kRowStage];        // per target: slot or -1
  __shared__ uint32_t tinf[kRowWarps][2 * kRowStage];  // per target: offset << 3 | dY
  __shared__ int tcd[kRowWarps][2 * kRowStage];        // per target: cY | own << 8 | chunk obs << 9
  __shared__ int item_n[kRowWarps], item_cx[kRowWarps];
  const int X = blockIdx.x, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  if (X >= rt.nblocks) return;
  const int dX = rt.blk_dim[X];
  const uint32_t n0 = rt.nbr_begin[X], n1 = rt.nbr_begin[X + 1], nn = n1 - n0;
  const bool nbr_local = nn <= (uint32_t)kRowNbr;
  const uint64_t r0 = rt.slot_off[n0], r1 = rt.slot_off[n1];
  if (nbr_local)
    for (uint32_t k = tid; k < nn; k += kRowThreads) {
      const int Y = rt.nbr[n0 + k];
      nbr_s[k] = Y;
      ninf_s[k] = (uint32_t)(rt.slot_off[n0 + k] - r0) << 3 | (uint32_t)rt.blk_dim[Y];
    }
  const uint32_t rlen = (uint32_t)(r1 - r0);
  double* row = rlen <= (uint32_t)row_smem ? row_sh : rows + r0;
  for (uint32_t k = tid; k < rlen; k += kRowThreads) row[k] = 0.0;
  const uint32_t i0 = rt.blk_ent[X], i1 = rt.blk_ent[X + 1];
  const int rs = lin.rs;
  // this warp's entity in the current batch (ce, cp, ca = first observation of the track, cl =
  // track length; cl = 0: none) and the next batch's entity and point
  uint32_t ce = 0, cp = 0, ca = 0, cl = 0, xe = 0, xp = 0;
  if (i0 + w < i1) {
    ce = rt.ent[i0 + w];
    cp = rt.ent_point[i0 + w];
    ca = rt.pt_off[cp];
    cl = rt.pt_off[cp + 1] - ca;
  }
  if (i0 + kRowWarps + w < i1) {
    xe = rt.ent[i0 + kRowWarps + w];
    xp = rt.ent_point[i0 + kRowWarps + w];
  }
  for (uint32_t base = i0; base < i1; base += kRowWarps) {
    // indices a batch ahead: the track of the next entity, the entity and point after it
    const uint32_t inext = base + kRowWarps + w, iafter = base + 2 * kRowWarps + w;
    uint32_t xa = 0, xl = 0, ye = 0, yp = 0;
    if (inext < i1) {
      xa = rt.pt_off[xp];
      xl = rt.pt_off[xp + 1] - xa;
    }
    if (iafter < i1) {
      ye = rt.ent[iafter];
      yp = rt.ent_point[iafter];
    }
    const uint32_t o = ce >> 1, ke = o - ca;
    const int cX = cl ? rt.seg_col[ce] : 0;
    for (uint32_t k0 = 0; __syncthreads_or(k0 < cl); k0 += kRowStage) {
      // ---- this warp's chunk: E (first round), targets, W ----
      // Loads are issued in two rounds: first every index (record offsets, target blocks and
      // columns, the point inverse), then every record value, so a chunk costs two memory latencies.
      const uint32_t Lc = k0 < cl ? min((uint32_t)kRowStage, cl - k0) : 0;
      const bool first = Lc && k0 == 0;
      const uint32_t rec_k = lane < Lc ? lin.obs_rec[ca + k0 + lane] : 0;  // record of chunk observation lane
      const uint32_t rec_o = first ? lin.obs_rec[o] : 0;
      int Y = -1, tcol = 0;
      uint32_t eid = 0;
      if (lane < 2 * Lc) {
        eid = 2 * (ca + k0 + (lane >> 1)) + (lane & 1);
        Y = rt.ent_block[eid];
        tcol = rt.seg_col[eid];
      }
      const double vi = (first && lane < 6) ? lin.vinv[6 * (size_t)cp + lane] : 0.0;
      // the entity's own record (E and the U term)
      double own = 0.0;
      if (first && lane < kRec) own = (double)lin.rec[rec_o + (size_t)lane * rs];
      // W of the chunk: lane kk + 16 h holds observation kk, columns 5h .. 5h + 4 (h = 1: 5 .. 8)
      const uint32_t kk = lane & 15, h = lane >> 4;
      const uint32_t rk_off = __shfl_sync(0xffffffffu, rec_k, (int)kk);
      const int c0 = h ? 5 : 0, nc = h ? 4 : 5;
      double jp[6], a0[5], a1[5];
      if (kk < Lc) {
        const R* rk = lin.rec + rk_off;
#pragma unroll
        for (int c = 0; c < 6; ++c) jp[c] = (double)rk[(size_t)(kJp + c) * rs];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          a0[j] = j < nc ? (double)rk[(size_t)(c0 + j) * rs] : 0.0;
          a1[j] = j < nc ? (double)rk[(size_t)(9 + c0 + j) * rs] : 0.0;
        }
      }
      if (first) {
        if (lane < kRec) Osh[w][lane] = own;
        if (lane < 6) Osh[w][kRec + lane] = vi;
      }
      if (kk < Lc) {
#pragma unroll
        for (int j = 0; j < 5; ++j)
          if (j < nc) {
            double* wq = Wsh[w][kk] + 3 * (c0 + j);
#pragma unroll
            for (int c = 0; c < 3; ++c) wq[c] = a0[j] * jp[c] + a1[j] * jp[3 + c];
          }
      }
      if (lane < 2 * Lc) {
        int sl = -1;
        uint32_t inf = 0;
        if (Y >= 0) {
          sl = nbr_local ? find_slot(nbr_s, 0, nn, Y) : find_slot(rt.nbr, n0, n1, Y);
          if (sl >= 0)
            inf = nbr_local ? ninf_s[sl]
                            : (uint32_t)(rt.slot_off[n0 + sl] - r0) << 3 | (uint32_t)rt.blk_dim[Y];
        }
        tsl[w][lane] = sl;
        tinf[w][lane] = inf;
        tcd[w][lane] = tcol | (k0 + (lane >> 1) == ke ? 1 << 8 : 0) | (int)(lane >> 1) << 9;
      }
      __syncwarp();
      if (first && lane < 3 * dX) {
        const int m = lane / 3, c = lane - 3 * m;
        const double* A = Osh[w];
        const double* P = Osh[w] + kRec;
        double wm[3];
        for (int d = 0; d < 3; ++d) wm[d] = A[cX + m] * A[kJp + d] + A[9 + cX + m] * A[kJp + 3 + d];
        const double v0 = c == 0 ? P[0] : (c == 1 ? P[1] : P[3]);
        const double v1 = c == 0 ? P[1] : (c == 1 ? P[2] : P[4]);
        const double v2 = c == 0 ? P[3] : (c == 1 ? P[4] : P[5]);
        Esh[w][lane] = wm[0] * v0 + wm[1] * v1 + wm[2] * v2;
      }
      if (lane == 0) {
        item_n[w] = 2 * (int)Lc;
        item_cx[w] = cX;
      }
      __syncthreads();
      // ---- every warp adds the batch's contributions to the slots it owns ----
      // One target is one FP64 m8n8k4 product on the tensor pipe, C (the slot, 8 x 8 with rows >= dX
      // and columns >= dY masked) += (-E) W_k,Y^T, plus A_o,X^T A_o,Y for the entity's own
      // observation. Fragments: lane l holds A(l / 4, l % 4), B(l % 4, l / 4) and C(l / 4, 2 (l % 4)
      // + i), i = 0, 1.
      const int fg = lane >> 2, ft = lane & 3;
      for (int b = 0; b < kRowWarps; ++b) {
        const int nt = item_n[b];
        if (nt == 0) continue;
        const int sl = lane < nt ? tsl[b][lane] : -1;
        unsigned mask = __ballot_sync(0xffffffffu, sl >= 0 && sl % kRowWarps == w);
        if (mask == 0u) continue;
        const int cxb = item_cx[b];
        const double* A = Osh[b];
        const double aE = (fg < dX && ft < 3) ? -Esh[b][3 * fg + ft] : 0.0;  // -E (dX x 3)
        const double aU = (fg < dX && ft < 2) ? A[9 * ft + cxb + fg] : 0.0;  // A_o,X^T (dX x 2)
        while (mask) {
          const int t = __ffs(mask) - 1;
          mask &= mask - 1;
          const uint32_t inf = tinf[b][t];
          const int cd = tcd[b][t], cY = cd & 0xff, own = (cd >> 8) & 1, dY = (int)(inf & 7);
          const double* Wk = Wsh[b][cd >> 9];
          double* out = row + (inf >> 3) + fg * dY;
          const double bW = (fg < dY && ft < 3) ? Wk[3 * (cY + fg) + ft] : 0.0;  // W_k,Y^T (3 x dY)
          const bool in0 = fg < dX && 2 * ft < dY, in1 = fg < dX && 2 * ft + 1 < dY;
          double c0 = in0 ? out[2 * ft] : 0.0, c1 = in1 ? out[2 * ft + 1] : 0.0;
          dmma_m8n8k4(aE, bW, c0, c1);
          if (own) {  // the same target in every lane
            const double bU = (fg < dY && ft < 2) ? A[9 * ft + cY + fg] : 0.0;  // A_o,Y (2 x dY)
            dmma_m8n8k4(aU, bU, c0, c1);
          }
          if (in0) out[2 * ft] = c0;
          if (in1) out[2 * ft + 1] = c1;
        }
      }
    }
    ce = xe;
    cp = xp;
    ca = xa;
    cl = inext < i1 ? xl : 0;
    xe = ye;
    xp = yp;
  }
  __syncthreads();
  if (row == row_sh)
    for (uint32_t k = tid; k < rlen; k += kRowThreads) rows[r0 + k] = row_sh[k];
}

// acc[m] += row m of block row X of S times x, a block per lane, over the row's blocks from `first` in
// steps of `stride`; xs gives x by parameter.
template <typename FX>
__device__ __forceinline__ void row_times(const RowTables& rt, const double* __restrict__ rows, int X, int dX,
                                          uint32_t first, uint32_t stride, FX xs, double acc[6]) {
  const uint32_t n1 = rt.nbr_begin[X + 1];
  for (uint32_t q = rt.nbr_begin[X] + first; q < n1; q += stride) {
    const int Y = rt.nbr[q], dY = rt.blk_dim[Y], oY = rt.blk_off[Y];
    const double* S = rows + rt.slot_off[q];
    double xv[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) xv[c] = c < dY ? xs(oY + c) : 0.0;
#pragma unroll
    for (int m = 0; m < 6; ++m)
      if (m < dX) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c)
          if (c < dY) s += S[m * dY + c] * xv[c];
        acc[m] += s;
      }
  }
}

// y = (S + lambda diag) x from the block rows: SPLIT warps per block row, the row's blocks dealt over
// their lanes in a fixed assignment, then a fixed shuffle tree and the warps in order. With xy non-null,
// xy[CTA] = sum of x_b . y_b over the CTA's blocks in block order. With ctl the damping is the control
// block's.
// Bound: L2 where S fits it (500 cameras: 30 MB), HBM above, latency below. SPLIT: while one warp per row
// leaves an SM fewer than eight warps (row_split) its loads do not cover the latency; measured on block
// rows of 61 cameras (one / two / four warps, back to back): 120 cameras 12.3 / 8.3 / 6.2 us, 500 12.4 /
// 10.3 / 10.3 us, 1,000 14.4 / 14.7 / 16.1 us, 3,000 37.9 / 39.1 / 43.2 us.
constexpr int kRowProductWarps = 8;
inline int row_split(int nblocks) { return nblocks <= 592 ? 4 : (nblocks <= 1184 ? 2 : 1); }
template <int SPLIT>
__global__ void __launch_bounds__(32 * kRowProductWarps) k_rows_matvec(RowTables rt, const double* __restrict__ rows,
                                                                       const double* __restrict__ diag, double lambda,
                                                                       const double* __restrict__ x,
                                                                       double* __restrict__ y, double* __restrict__ xy,
                                                                       const PcgCtl* ctl) {
  constexpr int ROWS = kRowProductWarps / SPLIT;
  __shared__ double s_part[kRowProductWarps][6];
  __shared__ double s_dot[ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int X = blockIdx.x * ROWS + warp / SPLIT;
  const bool have = X < rt.nblocks;
  pdl_trigger();
  pdl_wait();
  if (pcg_stopped(ctl)) return;
  if (ctl) lambda = ctl->lambda;
  const int dX = have ? rt.blk_dim[X] : 0;
  if (have) {
    double acc[6] = {0, 0, 0, 0, 0, 0};
    row_times(rt, rows, X, dX, 32u * (warp % SPLIT) + lane, 32u * SPLIT, [&](int i) { return x[i]; }, acc);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      acc[m] = warp_sum(acc[m]);
      if (lane == 0) s_part[warp][m] = acc[m];
    }
  }
  if (SPLIT > 1)
    __syncthreads();
  else
    __syncwarp();
  if (warp % SPLIT == 0) {
    double dot = 0.0;
    if (lane < dX) {
      const int o = rt.blk_off[X] + lane;
      double v = 0.0;
#pragma unroll
      for (int s = 0; s < SPLIT; ++s) v += s_part[warp + s][lane];
      const double xv = x[o];
      v += lambda * diag[o] * xv;
      y[o] = v;
      dot = xv * v;
    }
    dot = warp_sum(dot);
    if (lane == 0) s_dot[warp / SPLIT] = dot;
  }
  if (xy) {
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < ROWS; ++w) t += s_dot[w];
      xy[blockIdx.x] = t;
    }
  }
}

// Diagonal of S (no damping) from the rows: thread per block, its own slot.
__global__ void k_rows_diag(RowTables rt, const double* __restrict__ rows, double* __restrict__ out) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x;
  if (X >= rt.nblocks) return;
  const int dX = rt.blk_dim[X], oX = rt.blk_off[X];
  const int s = find_slot(rt.nbr, rt.nbr_begin[X], rt.nbr_begin[X + 1], X);
  const double* S = s >= 0 ? rows + rt.slot_off[rt.nbr_begin[X] + s] : nullptr;
  for (int m = 0; m < dX; ++m) out[oX + m] = S ? S[m * dX + m] : 0.0;
}

__global__ void k_set_int(int* p, int v) { *p = v; }

// ---- banded tiled matrix -----------------------------------------------------------------------
constexpr int kCT = 64;  // tile edge
constexpr int kCTT = kCT * kCT;

// Lower band of tiles of an n x n symmetric matrix in the permuted order: tile (i, j), 0 <= i - j <=
// bwt, at t + (i (bwt + 1) + (i - j)) kCTT, column-major inside the tile. Rows past n are padding
// (identity on the diagonal).
struct TileBand {
  int n, nt, bwt;
  double* t;
  double* w;  // nt tiles: the inverse of each diagonal tile of the factor (column-major)
};
__host__ __device__ __forceinline__ size_t tile_at(const TileBand& b, int i, int j) {
  return ((size_t)i * (b.bwt + 1) + (size_t)(i - j)) * kCTT;
}

// Scatter of the rows into the band: element (m, n) of block S_XY lands at permuted (P, Q) =
// (perm_off[X] + m, perm_off[Y] + n) when P >= Q. With scale non-null the stored value is
// scale_P S_PQ scale_Q; the diagonal gets + lambda diag_P, then - shift. A warp per four blocks, eight
// lanes a block (an element of its 36 each, in turn). The last CTA writes the identity on the padding
// rows of the last diagonal tile and sets the factorization's status word.
__global__ void __launch_bounds__(128) k_rows_to_tiles(RowTables rt, const double* __restrict__ rows,
                                                       const int* __restrict__ perm_off, const double* __restrict__ diag,
                                                       double lambda, const double* __restrict__ scale, double shift,
                                                       TileBand tb, int* status) {
  if (blockIdx.x == gridDim.x - 1) {
    if (threadIdx.x == 0) status[0] = 1;
    const int r = tb.n + threadIdx.x, i = tb.nt - 1;
    if (r < tb.nt * kCT) tb.t[tile_at(tb, i, i) + (size_t)(r % kCT) * kCT + (r % kCT)] = 1.0;
  }
  const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (q >= rt.entries) return;
  const int X = rt.nbr_row[q], Y = rt.nbr[q];
  const int dX = rt.blk_dim[X], dY = rt.blk_dim[Y];
  const int pX = perm_off[X], pY = perm_off[Y], oX = rt.blk_off[X], oY = rt.blk_off[Y];
  const double* S = rows + rt.slot_off[q];
  for (int e = threadIdx.x & 7; e < dX * dY; e += 8) {
    const int m = e / dY, n = e - m * dY;
    const int P = pX + m, Q = pY + n;
    if (P < Q) continue;
    double v = S[e];
    if (scale) v *= scale[oX + m] * scale[oY + n];
    if (P == Q) v += lambda * diag[oX + m] - shift;
    tb.t[tile_at(tb, P / kCT, Q / kCT) + (size_t)(Q % kCT) * kCT + (P % kCT)] = v;
  }
}

// Scatter of lower-triangle entries (row >= col) given as triplets into the band.
__global__ void k_triplets_to_tiles(uint32_t count, const int* __restrict__ rows, const int* __restrict__ cols,
                                    const double* __restrict__ vals, TileBand tb) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= count) return;
  const int P = rows[q], Q = cols[q];
  if (P < Q || P >= tb.n || Q < 0 || (P / kCT) - (Q / kCT) > tb.bwt) return;
  tb.t[tile_at(tb, P / kCT, Q / kCT) + (size_t)(Q % kCT) * kCT + (P % kCT)] = vals[q];
}

// Identity on the padding rows of the last diagonal tile.
__global__ void k_tiles_pad(TileBand tb) {
  const int r = tb.n + threadIdx.x;
  if (r >= tb.nt * kCT) return;
  const int i = tb.nt - 1;
  tb.t[tile_at(tb, i, i) + (size_t)(r % kCT) * kCT + (r % kCT)] = 1.0;
}

// Tiles in shared memory keep their column-major order with a column stride of kTS doubles: 4 modulo 16,
// so that the FP64 tensor fragments below read 16 different 8-byte banks per half warp both along a
// tile's columns and along its rows. Every operand is therefore staged by plain 16-byte asynchronous
// copies, transposed or not.
constexpr int kTS = 68;
constexpr size_t kStagedTile = sizeof(double) * kCT * kTS;

// Copies the column-major tile g into T (256 threads); complete after stage_wait() and a barrier.
__device__ __forceinline__ void stage_tile(const double* __restrict__ g, double* T) {
#pragma unroll
  for (int i = 0; i < kCTT / 2 / 256; ++i) {
    const int w = threadIdx.x + 256 * i, c = w >> 5, r = (w & 31) * 2;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(T + c * kTS + r);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(g + 2 * (size_t)w) : "memory");
  }
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A 64 x 64 product on the FP64 tensor pipe (m8n8k4), 8 warps: warp w owns rows 16 (w / 2) .. + 15 and
// columns 32 (w % 2) .. + 31 of the result, acc[i][j][e] being element (8 i + g, 8 j + 2 t + e) of
// that part for lane 4 g + t. The sum over the tile's 64 columns runs in order, four at a time.
// Against the 4 x 4-outputs-per-thread loop on the FP64 cores and the transposing copies it replaced
// (500-camera survey, 14 tiles a column, per launch): trsm 15.0 -> 6.2 us, update 17.4 -> 7.0 us,
// Takahashi partial sums 41.6 -> 16.0 us, off-diagonal tiles 34.3 -> 21.2 us.
struct TileAcc {
  double v[2][4][2];
};
__device__ __forceinline__ void zero_acc(TileAcc& acc) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc.v[i][j][0] = acc.v[i][j][1] = 0.0;
}
// acc += op(Ta) op(Tb), op the transpose when AT / BT is set.
template <bool AT, bool BT>
__device__ __forceinline__ void tile_mma_acc(const double* Ta, const double* Tb, TileAcc& acc) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int r0 = 16 * (w >> 1) + g, c0 = 32 * (w & 1) + g;
#pragma unroll 4
  for (int k0 = 0; k0 < kCT; k0 += 4) {
    const int k = k0 + t;
    double a[2], b[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) a[i] = AT ? Ta[(r0 + 8 * i) * kTS + k] : Ta[k * kTS + r0 + 8 * i];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = BT ? Tb[k * kTS + c0 + 8 * j] : Tb[(c0 + 8 * j) * kTS + k];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dmma_m8n8k4(a[i], b[j], acc.v[i][j][0], acc.v[i][j][1]);
  }
}
// f(row, column, value) over this thread's elements of the result.
template <typename F>
__device__ __forceinline__ void acc_each(const TileAcc& acc, F f) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int r0 = 16 * (w >> 1) + g, c0 = 32 * (w & 1) + 2 * t;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) f(r0 + 8 * i, c0 + 8 * j + e, acc.v[i][j][e]);
}
__device__ __forceinline__ void acc_store(const TileAcc& acc, double* g) {
  acc_each(acc, [&](int r, int c, double v) { g[(size_t)c * kCT + r] = v; });
}

// C (8 x 8, column-major at stride kTS) += sign * A B for one warp, A and B read through the lambdas
// a(row, k) and b(k, column), k < depth.
template <typename FA, typename FB>
__device__ __forceinline__ void mma8(int depth, FA a, FB b, double& c0, double& c1) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int k0 = 0; k0 < depth; k0 += 4) dmma_m8n8k4(a(g, k0 + t), b(k0 + t, g), c0, c1);
}

// POTRF of diagonal tile k and the inverse W_k = L_kk^-1 of its factor, one CTA of 8 warps, blocked by
// 8 columns. Warp 0 factors a panel (all rows, 8 columns) in registers, two rows per lane. Each lane also
// holds the panel's 8 x 8 diagonal block, so a pivot step is a reciprocal root, a product and a fused
// multiply-add, with no shuffle and no barrier in the chain. Then every warp subtracts the panel's rank-8
// product from one 8 x 8 block of the next panel's columns on the FP64 tensor pipe; the rest of the
// trailing triangle, the panel's columns of the factor and its row of the inverse,
// W_q. = -W_qq (L_q. W), are done by warps 1 to 7 while warp 0 factors the next panel (the pivots' roots
// and reciprocals, which only these need, among them). Bound: the 64 dependent pivot steps. A right-looking
// factor with one barrier per column and a second sweep of 64 barriers for the inverse took 64 us per tile;
// with shuffled pivots, every block of the triangle between two panels and the inverse afterwards it took
// 18.5; this takes 13.6.
// status[0] = 0 when a pivot is not finite and positive; later launches of the factorization then
// return at once.
constexpr size_t kPotrfSmem = 2 * kStagedTile;
// A: the tile in shared memory (visible to the CTA), then L below its diagonal; W: a second staged tile,
// the inverse on and below its diagonal, the products L_q. W above it.
__device__ void potrf_tile(const TileBand& tb, int k, double* A, double* W, int* status) {
  __shared__ double pivots[kCT];
  __shared__ int s_bad;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  double* gt = tb.t + tile_at(tb, k, k);
  // C(bi, bj) -= panel p's product, one warp
  auto trailing = [&](int p, int bi, int bj) {
    double* C = A + (8 * bj + 2 * t) * kTS + 8 * bi + g;
    double c0 = C[0], c1 = C[kTS];
    mma8(8, [&](int r, int kk) { return -A[(8 * p + kk) * kTS + 8 * bi + r]; },
         [&](int kk, int c) { return A[(8 * p + kk) * kTS + 8 * bj + c]; }, c0, c1);
    C[0] = c0;
    C[kTS] = c1;
  };
  // Columns of the factor and row of the inverse of panel q, warps 1 to 7.
  auto finish = [&](int q) {
    for (int i = tid - 32; i < 8 * kCT; i += 224) {  // the factor (zero above the diagonal)
      const int c = 8 * q + (i >> 6), r = i & 63;
      if (r != c) gt[c * kCT + r] = r > c ? A[c * kTS + r] : 0.0;
    }
    if (w == 7) {  // W_qq, lane c its column c
      const int col = lane & 7;
      const double sd = sqrt(pivots[8 * q + col]), rd = 1.0 / sd;
      if (lane < 8) gt[(8 * q + lane) * (kCT + 1)] = sd;
      double x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        double v = i == col ? 1.0 : 0.0;
#pragma unroll
        for (int z = 0; z < i; ++z) v -= A[(8 * q + z) * kTS + 8 * q + i] * x[z];
        const double r = __shfl_sync(0xffffffffu, rd, i);
        x[i] = i >= col ? v * r : 0.0;
        if (lane < 8) W[(8 * q + lane) * kTS + 8 * q + i] = x[i];
      }
    }
    // block column j: warp j + 1, warp 7 those left after W_qq
    const int j = w - 1;
    double* T = W + (8 * q + 2 * t) * kTS + 8 * j + g;
    if (j < q) {
      double c0 = 0.0, c1 = 0.0;
      mma8(8 * (q - j), [&](int r, int kk) { return A[(8 * j + kk) * kTS + 8 * q + r]; },
           [&](int kk, int c) { return W[(8 * j + c) * kTS + 8 * j + kk]; }, c0, c1);
      T[0] = c0;
      T[kTS] = c1;
    }
    asm volatile("bar.sync 1, 224;" ::: "memory");  // warps 1 to 7: W_qq and the products are there
    if (j < q) {
      double c0 = 0.0, c1 = 0.0;
      mma8(8, [&](int r, int kk) { return -W[(8 * q + kk) * kTS + 8 * q + r]; },
           [&](int kk, int c) { return W[(8 * q + c) * kTS + 8 * j + kk]; }, c0, c1);
      double* O = W + (8 * j + 2 * t) * kTS + 8 * q + g;
      O[0] = c0;
      O[kTS] = c1;
    }
  };
  if (tid == 0) s_bad = 0;
  __syncthreads();
  for (int p = 0; p < 8; ++p) {
    const int j0 = 8 * p;
    if (w == 0) {
      double lo[8], hi[8];  // rows lane and lane + 32 of the panel
      double d[8][8];       // its diagonal block, d[c][r]
#pragma unroll
      for (int c = 0; c < 8; ++c) {
#pragma unroll
        for (int r = c & ~1; r < 8; r += 2) {
          const double2 v = *reinterpret_cast<const double2*>(A + (j0 + c) * kTS + j0 + r);
          d[c][r] = v.x;
          d[c][r + 1] = v.y;
        }
        lo[c] = A[(j0 + c) * kTS + lane];
        hi[c] = A[(j0 + c) * kTS + lane + 32];
      }
      bool bad = false;
      double pivot = 1.0;  // lane c < 8: column c's
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        bad = bad || !(isfinite(d[c][c]) && d[c][c] > 0.0);
        if (lane == c) pivot = d[c][c];
        const double rs = rsqrt(d[c][c]);
        lo[c] *= rs;
        hi[c] *= rs;
#pragma unroll
        for (int r = c + 1; r < 8; ++r) d[c][r] *= rs;
#pragma unroll
        for (int c2 = c + 1; c2 < 8; ++c2) {
#pragma unroll
          for (int r = c2; r < 8; ++r) d[c2][r] -= d[c][r] * d[c][c2];
          lo[c2] -= lo[c] * d[c][c2];
          hi[c2] -= hi[c] * d[c][c2];
        }
      }
      __syncwarp();  // every lane has read the panel
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (lane > j0 + c) A[(j0 + c) * kTS + lane] = lo[c];
        if (lane + 32 > j0 + c) A[(j0 + c) * kTS + lane + 32] = hi[c];
      }
      if (lane < 8) pivots[j0 + lane] = pivot;
      if (bad && lane == 0) s_bad = 1;
    } else if (p > 0) {
      // blocks (bi >= bj > p) of the panel before, column by column of blocks
      const int m = 7 - p;
      for (int q = w - 1; q < m * (m + 1) / 2; q += 7) {
        int col = 0, at = q;
        while (at >= m - col) at -= m - col++;
        trailing(p - 1, p + 1 + col + at, p + 1 + col);
      }
      finish(p - 1);
    }
    __syncthreads();
    if (s_bad) {
      if (tid == 0) status[0] = 0;
      return;
    }
    if (p + 1 + w < 8) trailing(p, p + 1 + w, p + 1);
    __syncthreads();
  }
  if (w > 0) finish(7);
  __syncthreads();
  double* wk = tb.w + (size_t)k * kCTT;
  for (int i = tid; i < kCTT; i += 256) {
    const int c = i >> 6, r = i & 63;
    wk[i] = r >= c ? W[c * kTS + r] : 0.0;
  }
}

__global__ void __launch_bounds__(256) k_tile_potrf(TileBand tb, int k, int* status) {
  extern __shared__ __align__(16) double sh[];
  pdl_trigger();
  if (status[0] == 0) return;
  stage_tile(tb.t + tile_at(tb, k, k), sh);
  stage_wait();
  __syncthreads();
  potrf_tile(tb, k, sh, sh + kCT * kTS, status);
}

// TRSM as a product: the tiles below diagonal tile k, L_ik = A_ik W_k^T (CTA per tile). Dynamic shared
// memory: two staged operands.
constexpr size_t kTrsmSmem = 2 * kStagedTile;
__global__ void __launch_bounds__(256) k_tile_trsm(TileBand tb, int k, const int* status) {
  extern __shared__ __align__(16) double shm[];
  pdl_trigger();
  pdl_wait();
  if (status[0] == 0) return;
  double* Ta = shm;
  double* Tb = shm + kCT * kTS;
  const int i = k + 1 + blockIdx.x;
  double* bi = tb.t + tile_at(tb, i, k);
  stage_tile(bi, Ta);                        // A_ik
  stage_tile(tb.w + (size_t)k * kCTT, Tb);   // W_k
  stage_wait();
  __syncthreads();
  TileAcc acc;
  zero_acc(acc);
  tile_mma_acc<false, true>(Ta, Tb, acc);
  acc_store(acc, bi);
}

// Trailing update of step k: A_ij -= L_ik L_jk^T for k < j <= i <= min(k + bwt, nt - 1), one CTA per
// tile; the sum over the tile's 64 columns runs in order. CTA 0 has the next diagonal tile: it goes on to
// factor it (potrf_tile) while the other CTAs update theirs, so a column costs its factorization and its
// trsm, and the update runs in the factorization's shadow (500-camera survey, per column: 13.6 us of potrf,
// 6.1 of trsm and 7.0 of update become 6.1 + 17.2).
constexpr size_t kUpdateSmem = 2 * kStagedTile;
__global__ void __launch_bounds__(256) k_tile_update(TileBand tb, int k, int* status) {
  extern __shared__ __align__(16) double sh[];
  pdl_trigger();
  pdl_wait();
  if (status[0] == 0) return;
  double* Ta = sh;
  double* Tb = sh + kCT * kTS;
  int idx = blockIdx.x;
  int ii = (int)((sqrtf(8.0f * (float)idx + 1.0f) - 1.0f) * 0.5f);
  while ((ii + 1) * (ii + 2) / 2 <= idx) ++ii;
  while (ii * (ii + 1) / 2 > idx) --ii;
  const int jj = idx - ii * (ii + 1) / 2;
  const int i = k + 1 + ii, j = k + 1 + jj;
  stage_tile(tb.t + tile_at(tb, i, k), Ta);  // L_ik
  stage_tile(tb.t + tile_at(tb, j, k), Tb);  // L_jk
  double* cij = tb.t + tile_at(tb, i, j);
  TileAcc acc, old;
  zero_acc(acc);
  {  // the tile's own values, requested with the operands
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const double* c = cij + (size_t)(32 * (w & 1) + 2 * t) * kCT + 16 * (w >> 1) + g;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) old.v[a][b][e] = c[(8 * b + e) * kCT + 8 * a];
  }
  stage_wait();
  __syncthreads();
  tile_mma_acc<false, true>(Ta, Tb, acc);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) acc.v[a][b][e] = old.v[a][b][e] - acc.v[a][b][e];
  if (idx > 0) {
    acc_store(acc, cij);
    return;
  }
  __syncthreads();  // the operands are read: their place takes the diagonal tile
  acc_each(acc, [&](int r, int c, double v) { Ta[c * kTS + r] = v; });
  __syncthreads();
  potrf_tile(tb, k + 1, Ta, Tb, status);
}

// Forward (L y = -g) and backward (L^T x = y) substitution with the banded tiled factor, on the vector v in
// the factor's order (n entries; the padding is not touched), gathered from g and scattered to step_out in
// the parameters' order; one cluster of up to kSolveCtas CTAs.
// Right-looking: CTA i mod size owns rows of tile i. In step k every CTA has the 64 finished results of
// tile k in its shared memory. The owner of tile k + 1 subtracts their product with T(k + 1, k), multiplies
// by the inverse of the diagonal tile (W, from the factorization) and hands the results to every CTA; then
// it signals the cluster barrier of step k + 1, and only then does each CTA subtract the products of its
// other tiles of the column (forward) or row (backward), which no later step but k + 2 and on waits for.
// Both tiles of a CTA's next turn are loaded into registers a turn ahead and the next of its other tiles one
// product ahead, so no load lies in the chain. A CTA may thus still read the results of tile k while those
// of tile k + 2 are being written: three buffers. Each entry of v is only ever touched by one thread, in
// step order. Bound: 2 nt steps of two products, their CTA barriers and a cluster barrier, or the band's
// tiles from L2 through 8 SMs where the band is wide. One CTA that walked each row of the band with an
// in-tile triangular solve by one warp took 12.8 ms for 71 tiles in a band of 14; with every load and every
// product of a step between two cluster barriers it took 0.93 ms; this takes 0.31.
constexpr int kSolveCtas = 8;
constexpr int kSolveBuffers = 3;
struct SolveShared {
  double part[2][4 * kCT], u[kCT];
  double step[kSolveBuffers][kCT];  // finished parts of the vector, from their owners
};
// One sweep over the tiles: k-th tile is tile k of the factor (FORWARD) or tile nt - 1 - k.
template <bool FORWARD>
__device__ __forceinline__ void solve_sweep(const TileBand& tb, double* v, const int* __restrict__ perm_to_orig,
                                            double* __restrict__ step_out, SolveShared& sh) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int size = (int)cluster.num_blocks(), tid = threadIdx.x, r = tid & (kCT - 1), qtr = tid >> 6;
  const int nt = tb.nt;
  auto actual = [&](int k) { return FORWARD ? k : nt - 1 - k; };
  // the CTA's tiles are first, first + size, ...
  const int rank = (int)cluster.block_rank(), first = FORWARD ? rank : ((nt - 1 - rank) % size + size) % size;
  const int base = FORWARD ? 0 : nt;  // results are numbered on from the forward sweep's
  auto step = [&](int k) { return sh.step[(base + k) % kSolveBuffers]; };
  // A thread's 16 entries of a tile: of row r (columns 16 qtr ...), or of column tid / 4 (every fourth row).
  auto load = [&](const double* __restrict__ M, double m[16]) {
    if (FORWARD) {
#pragma unroll
      for (int c = 0; c < 16; ++c) m[c] = M[(size_t)(16 * qtr + c) * kCT + r];
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) m[j] = M[(size_t)(tid >> 2) * kCT + 4 * j + (tid & 3)];
    }
  };
  auto load_t = [&](int i, int k, double m[16]) {  // T of the i-th and the k-th tile, i > k
    load(tb.t + (FORWARD ? tile_at(tb, actual(i), actual(k)) : tile_at(tb, actual(k), actual(i))), m);
  };
  auto load_w = [&](int k, double m[16]) { load(tb.w + (size_t)actual(k) * kCTT, m); };
  auto partial = [&](const double m[16], const double* x) {
    if constexpr (FORWARD) {
      double s = 0.0;
#pragma unroll
      for (int c = 0; c < 16; ++c) s += m[c] * x[16 * qtr + c];
      return s;
    } else {
      double s[8];  // rows i and i + 32, then a balanced sum
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = m[j] * x[4 * j + (tid & 3)] + m[j + 8] * x[4 * j + (tid & 3) + 32];
#pragma unroll
      for (int h = 4; h > 0; h >>= 1)
#pragma unroll
        for (int j = 0; j < h; ++j) s[j] += s[j + h];
      return s[0];
    }
  };
  int used = 0;
  auto total = [&](double s) {  // entry r of the product, in every thread
    double* part = sh.part[used];
    used ^= 1;  // the buffer's next use lies after the next barrier
    if constexpr (FORWARD) {
      part[tid] = s;
      __syncthreads();
      return ((part[r] + part[kCT + r]) + part[2 * kCT + r]) + part[3 * kCT + r];
    } else {
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if ((tid & 3) == 0) part[tid >> 2] = s;
      __syncthreads();
      return part[r];
    }
  };
  // The entry of the i-th tile that this thread keeps (threads 0 to 63).
  auto own = [&](int i) { return tid < kCT && actual(i) * kCT + tid < tb.n; };
  auto entry = [&](int i) { return own(i) ? v[actual(i) * kCT + tid] : 0.0; };
  // Tile k's results from u = its right-hand side less all products, and to every CTA.
  auto finish = [&](int k, double u, const double w[16]) {
    if (tid < kCT) sh.u[tid] = u;
    __syncthreads();
    const double y = total(partial(w, sh.u));
    double* to = step(k) + r;
    for (int c = qtr; c < size; c += 4) *cluster.map_shared_rank(to, c) = y;
    if (own(k)) {
      const int P = actual(k) * kCT + tid;
      v[P] = y;
      if (!FORWARD) step_out[perm_to_orig[P]] = y;
    }
  };
  double mt[16], mw[16], mn[16];
  if (first == 0) {
    load_w(0, mw);
    finish(0, entry(0), mw);
  }
  cluster.barrier_arrive();
  int turn = first == 0 ? size : first;  // the CTA's next tile to finish
  auto load_turn = [&] {
    if (turn >= nt) return;
    if (tb.bwt > 0) load_t(turn, turn - 1, mt);
    load_w(turn, mw);
  };
  load_turn();
  int ik = -1, i = nt;  // the next of the CTA's other products, tile i in step ik
  auto next = [&] {
    i += size;
    while (ik < nt && i > min(nt - 1, ik + tb.bwt)) {
      ++ik;
      i = first + (max(0, ik + 2 - first) + size - 1) / size * size;
    }
    if (ik < nt) load_t(i, ik, mn);
  };
  next();
  for (int k = 0; k < nt; ++k) {
    const bool mine = turn == k + 1 && turn < nt;
    const double rhs = mine ? entry(turn) : 0.0;
    cluster.barrier_wait();
    if (mine) {
      const double x = tb.bwt > 0 ? total(partial(mt, step(k))) : 0.0;
      finish(turn, own(turn) ? rhs - x : 0.0, mw);
    }
    if (k + 1 < nt) cluster.barrier_arrive();
    if (mine) {
      turn += size;
      load_turn();
    }
    while (ik == k) {
      const int at = i;
      const double before = entry(at), s = partial(mn, step(k));
      next();
      const double x = total(s);
      if (own(at)) v[actual(at) * kCT + tid] = before - x;
    }
  }
}
__global__ void __launch_bounds__(256) k_tile_solve(TileBand tb, double* v, const int* status,
                                                    const int* __restrict__ perm_to_orig, const double* __restrict__ g,
                                                    double* __restrict__ step_out) {
  namespace cg = cooperative_groups;
  __shared__ __align__(16) SolveShared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks(), tid = threadIdx.x;
  const bool factored = status[0] != 0;  // the same value in every CTA of the cluster
  // the right-hand side -g in the factor's order, each CTA its own tiles
  for (int tile = rank; tile < tb.nt; tile += size)
    if (tid < kCT && tile * kCT + tid < tb.n) {
      const int o = perm_to_orig[tile * kCT + tid];
      v[tile * kCT + tid] = -g[o];
      if (!factored) step_out[o] = -g[o];  // a step that the host refuses, but one of defined values
    }
  if (!factored) return;
  cluster.sync();  // every CTA runs before any of them is written to
  solve_sweep<true>(tb, v, perm_to_orig, step_out, sh);
  solve_sweep<false>(tb, v, perm_to_orig, step_out, sh);
  cluster.sync();  // no CTA leaves while another may still write to it
}

// ---- selected inverse within the band (intrinsic marginal covariances) -----------------------
// Z = S^-1 restricted to the band of the factor, by the Takahashi recurrence on tiles, from the last
// tile column to the first: with Z L = L^-T, W_j = L_jj^-1 and M_kj = L_kj W_j,
//   Z_ij = -sum_{k=j+1}^{j+bwt} Z_ik M_kj                      (i > j)
//   Z_jj = W_j^T W_j - sum_{k=j+1}^{j+bwt} Z_kj^T M_kj
// where Z_ik for i < k is Z_ki^T; every Z_ik needed lies in the band. The marginal covariance of a
// group is the block of Z at its parameters' positions (sparse/covariance.rs:564-587 gets the same
// block by solving S x = e_p column by column).
//
// The products with W_j lie outside the chain of columns, in one launch over all tiles; column j then runs
// as three launches, each in place when the one before ends, so that the column's 64 x 64 products spread
// over the GPU:
//  k_takahashi_scale    CTA per tile of the band, in place of the factor: M_kj, and W_j^T W_j on the diagonal
//  k_takahashi_partial  CTA (b, s): part(b, s) = sum over k in chunk s of Z_ik M_kj, i = j + 1 + b,
//                       chunks of kTakahashiChunk consecutive k in order
//  k_takahashi_offdiag  CTA b: Z_ij = -sum_s part(b, s), and its share of the diagonal sum,
//                       q(b) = Z_ij^T M_ij
//  k_takahashi_diag     Z_jj = W_j^T W_j - sum_b q(b), an element per thread
// Every sum runs in a fixed order, so Z does not depend on scheduling. Dynamic shared memory:
// kTakahashiSmem (two staged operands). Bound: the chain of columns, each the latency of three launches and
// two tile products (at a band of 35 tiles the partial sums' products on the tensor pipe). With the products
// with W_j inside the columns these took, at a band of 14 tiles, 16 + 21 + 9 us a column, and 35 + 29 + 14 at
// a band of 35; now 16 + 11 + 6.5 and 34 + 18 + 7.5.
constexpr size_t kTakahashiSmem = 2 * kStagedTile;
constexpr int kTakahashiChunk = 4;
constexpr int kTakahashiDiagThreads = 64;

__global__ void __launch_bounds__(256) k_takahashi_scale(TileBand L, const int* status) {
  extern __shared__ __align__(16) double sh[];
  if (status[0] == 0) return;
  const int j = blockIdx.x, i = j + blockIdx.y;
  if (i >= L.nt) return;
  double* Ta = sh;
  double* Tb = sh + kCT * kTS;
  double* out = L.t + tile_at(L, i, j);
  stage_tile(L.w + (size_t)j * kCTT, Tb);
  if (i > j) stage_tile(out, Ta);
  stage_wait();
  __syncthreads();
  TileAcc acc;
  zero_acc(acc);
  if (i > j)
    tile_mma_acc<false, false>(Ta, Tb, acc);
  else
    tile_mma_acc<true, false>(Tb, Tb, acc);
  acc_store(acc, out);
}
__global__ void __launch_bounds__(256) k_takahashi_partial(TileBand L, TileBand Z, int j, double* part,
                                                           const int* status) {
  extern __shared__ __align__(16) double sh[];
  pdl_trigger();
  double* Ta = sh;
  double* Tb = sh + kCT * kTS;
  const int i = j + 1 + blockIdx.x;
  const int kmax = min(L.nt - 1, j + L.bwt);
  const int k0 = j + 1 + kTakahashiChunk * blockIdx.y, k1 = min(kmax, k0 + kTakahashiChunk - 1);
  TileAcc acc;
  zero_acc(acc);
  stage_tile(L.t + tile_at(L, k0, j), Tb);  // M is there before the column loop begins
  pdl_wait();
  if (status[0] == 0) {
    stage_wait();
    return;
  }
  for (int k = k0; k <= k1; ++k) {
    __syncthreads();
    stage_tile(Z.t + (i >= k ? tile_at(Z, i, k) : tile_at(Z, k, i)), Ta);  // Z_ik, or Z_ki for its transpose
    if (k > k0) stage_tile(L.t + tile_at(L, k, j), Tb);
    stage_wait();
    __syncthreads();
    if (i >= k)
      tile_mma_acc<false, false>(Ta, Tb, acc);
    else
      tile_mma_acc<true, false>(Ta, Tb, acc);
  }
  acc_store(acc, part + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * kCTT);
}

__global__ void __launch_bounds__(256) k_takahashi_offdiag(TileBand L, TileBand Z, int j, int nsplit,
                                                           const double* __restrict__ part, double* q,
                                                           const int* status) {
  extern __shared__ __align__(16) double sh[];
  pdl_trigger();
  double* Ta = sh;
  double* Tb = sh + kCT * kTS;
  const int i = j + 1 + blockIdx.x;
  stage_tile(L.t + tile_at(L, i, j), Tb);  // M_ij, there before the column loop begins
  pdl_wait();
  if (status[0] == 0) {
    stage_wait();
    return;
  }
  // Z_ij = -(sum of the partial tiles, in order)
  const double* pb = part + (size_t)blockIdx.x * nsplit * kCTT;
  double* z = Z.t + tile_at(Z, i, j);
  double v[kCTT / 256];
#pragma unroll
  for (int e = 0; e < kCTT / 256; ++e) v[e] = 0.0;
  for (int s = 0; s < nsplit; ++s)
#pragma unroll
    for (int e = 0; e < kCTT / 256; ++e) v[e] += pb[(size_t)s * kCTT + 256 * e + threadIdx.x];
#pragma unroll
  for (int e = 0; e < kCTT / 256; ++e) {
    const int w = 256 * e + threadIdx.x;
    Ta[(w >> 6) * kTS + (w & 63)] = -v[e];
    z[w] = -v[e];
  }
  stage_wait();
  __syncthreads();
  TileAcc acc;
  zero_acc(acc);
  tile_mma_acc<true, false>(Ta, Tb, acc);  // Z_ij^T M_ij
  acc_store(acc, q + (size_t)blockIdx.x * kCTT);
}
__global__ void __launch_bounds__(kTakahashiDiagThreads) k_takahashi_diag(TileBand L, TileBand Z, int j, int m,
                                                                          const double* __restrict__ q,
                                                                          const int* status) {
  pdl_trigger();
  pdl_wait();
  if (status[0] == 0) return;
  const int w = blockIdx.x * kTakahashiDiagThreads + threadIdx.x;
  double v = 0.0;
#pragma unroll 8
  for (int b = 0; b < m; ++b) v += q[(size_t)b * kCTT + w];
  Z.t[tile_at(Z, j, j) + w] = L.t[tile_at(L, j, j) + w] - v;
}

// (S^-1)_gg of each free group from Z: 9 values per group (row-major), thread per group.
__global__ void k_z_marginals(TileBand Z, int ngroups, const int* __restrict__ pos, const int* __restrict__ dims,
                              double* __restrict__ out, const int* status) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ngroups || status[0] == 0) return;
  const int dim = dims[g];
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b) {
      double v = 0.0;
      if (a < dim && b < dim) {
        int P = pos[3 * g + a], Q = pos[3 * g + b];
        if (P < Q) {
          const int t = P;
          P = Q;
          Q = t;
        }
        v = Z.t[tile_at(Z, P / kCT, Q / kCT) + (size_t)(Q % kCT) * kCT + (P % kCT)];
      }
      out[9 * (size_t)g + 3 * a + b] = v;
    }
}

// ---- loops over S inside one cluster -------------------------------------------------------------
// One cluster of kLoopCtas CTAs runs a whole iteration (power iteration, PCG), so the host waits once and
// no launch lies between two products. CTA r owns the block rows X = r mod kLoopCtas; a task is 32 blocks
// of one row, a block per lane. Every CTA keeps the whole iterate in shared memory; a row's results go to
// all CTAs' shared memory and one cluster barrier ends the product. Every row has a block, its own at least,
// and so a task that writes its results. While a CTA's tasks fit (kLoopTasks, a warp each) their blocks
// stay in shared memory too, element by element with the lanes side by side: the cluster barrier drops L1, so
// each iteration would otherwise wait for L2 three times over.
constexpr int kLoopCtas = 8;
constexpr int kLoopThreads = 512;
constexpr int kLoopWarps = kLoopThreads / 32;
constexpr int kLoopTasks = kLoopWarps;
constexpr size_t kLoopTaskDoubles = 36 * 32;

struct LoopTasks {
  int row[kLoopTasks], off[kLoopTasks][32];  // row; per lane first parameter << 3 | dimension
  int count;                                 // above kLoopTasks: not cached
  double part[kLoopWarps][6];
};
__host__ __device__ __forceinline__ int loop_row_tasks(uint32_t blocks) { return (int)((blocks + 31) / 32); }

// The CTA's tasks in row order (thread 0, before a barrier).
__device__ __forceinline__ void loop_list(const RowTables& rt, int rank, LoopTasks& t) {
  int nt = 0;
  for (int X = rank; X < rt.nblocks; X += kLoopCtas) {
    const int m = loop_row_tasks(rt.nbr_begin[X + 1] - rt.nbr_begin[X]);
    for (int q = 0; q < m && nt + q < kLoopTasks; ++q) t.row[nt + q] = X;
    nt += m;
    if (nt > kLoopTasks) break;
  }
  t.count = nt;
}
// Their blocks into `cache`, columns times scale when it is given (all warps).
__device__ __forceinline__ void loop_load(const RowTables& rt, const double* __restrict__ rows,
                                          const double* __restrict__ scale, LoopTasks& t, double* cache) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w >= t.count) return;
  const int X = t.row[w], dX = rt.blk_dim[X];
  int first = w;
  while (first > 0 && t.row[first - 1] == X) --first;
  const uint32_t q = rt.nbr_begin[X] + 32 * (w - first) + lane;
  const bool have = q < rt.nbr_begin[X + 1];
  const int Y = have ? rt.nbr[q] : 0, dY = have ? rt.blk_dim[Y] : 0, oY = have ? rt.blk_off[Y] : 0;
  t.off[w][lane] = oY << 3 | dY;
  const double* S = rows + (have ? rt.slot_off[q] : 0);
#pragma unroll
  for (int m = 0; m < 6; ++m)
#pragma unroll
    for (int c = 0; c < 6; ++c)
      cache[w * kLoopTaskDoubles + (6 * m + c) * 32 + lane] =
          m < dX && c < dY ? S[m * dY + c] * (scale ? scale[oY + c] : 1.0) : 0.0;
}
// The cached tasks' products with v (shared memory) into t.part, a barrier, then put(X, m, sum) by the
// warp of a row's first task: element e = lane, lane + 32, ... of dX x kLoopCtas, m = e / kLoopCtas, for
// CTA e % kLoopCtas.
template <typename F>
__device__ __forceinline__ void loop_product(const RowTables& rt, LoopTasks& t, const double* cache, const double* v,
                                             F put) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w < t.count) {
    const double* C = cache + w * kLoopTaskDoubles + lane;
    const int at = t.off[w][lane], dY = at & 7;
    double xv[6], acc[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) xv[c] = c < dY ? v[(at >> 3) + c] : 0.0;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      acc[m] = 0.0;
#pragma unroll
      for (int c = 0; c < 6; ++c) acc[m] += C[(6 * m + c) * 32] * xv[c];
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      acc[m] = warp_sum(acc[m]);
      if (lane == 0) t.part[w][m] = acc[m];
    }
  }
  __syncthreads();
  if (w < t.count && (w == 0 || t.row[w - 1] != t.row[w])) {
    const int X = t.row[w], dX = rt.blk_dim[X];
    int count = 1;
    while (w + count < t.count && t.row[w + count] == X) ++count;
    for (int e = lane; e < dX * kLoopCtas; e += 32) {
      const int m = e / kLoopCtas;
      double r = 0.0;
      for (int q = 0; q < count; ++q) r += t.part[w + q][m];
      put(rt.blk_off[X] + m, e % kLoopCtas, r);
    }
  }
}
// The CTA-wide sum of v in a fixed order, the same value in every thread; red: kLoopWarps doubles that no
// thread still reads.
__device__ __forceinline__ double loop_sum(double v, double* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < kLoopWarps; ++q) s += red[q];
  return s;
}

// Largest |eigenvalue| of the equilibrated D S D by power iteration (Rayleigh quotient of the
// normalized iterate): out[0] = lambda, out[1] = 1 when it settled (|rq - lambda| <= 1e-10 |rq| after
// the 8th iteration) or ran its 200 iterations with finite values, 0 otherwise. n <= kPowerMax. The iterate
// is not normalized (the products are scaled by the last norm); every CTA forms the same norm and
// quotient in the same order, so all leave the loop together.
// Bound: 200 dependent iterations of a barrier and a reduction. One CTA that kept the iterate in global
// memory took 1.80 ms at n = 113, the cluster without the blocks in shared memory 1.04 ms, this 0.56 ms.
constexpr int kPowerMax = 2048;
constexpr size_t power_smem(int n) { return sizeof(double) * (3 * (size_t)n + kLoopTasks * kLoopTaskDoubles); }
__global__ void __launch_bounds__(kLoopThreads) k_power_iteration(RowTables rt, const double* __restrict__ rows,
                                                                  const double* __restrict__ scale, int n, double* out) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) double sh[];  // three iterates in turn, then the cached tasks
  __shared__ double red[2][kLoopWarps];
  __shared__ LoopTasks t;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* cache = sh + 3 * (size_t)n;
  if (tid == 0) loop_list(rt, rank, t);
  const double v0 = 1.0 / sqrt((double)n);
  for (int i = tid; i < n; i += kLoopThreads) sh[i] = v0;
  __syncthreads();
  const bool cached = t.count <= kLoopTasks;
  if (cached) loop_load(rt, rows, scale, t, cache);
  cluster.sync();  // every CTA runs before any of them is written to; the cache is in place
  double lam = 0.0, inv = 1.0;
  int ok = 0;
  for (int it = 0; it < 200; ++it) {
    const double* v = sh + (it % 3) * (size_t)n;  // times inv: the normalized iterate
    double* w = sh + ((it + 1) % 3) * (size_t)n;
    if (cached) {
      loop_product(rt, t, cache, v, [&](int i, int cta, double r) { *cluster.map_shared_rank(w + i, cta) = r * inv * scale[i]; });
    } else {
      for (int x0 = 0; x0 * kLoopCtas + rank < rt.nblocks; x0 += kLoopWarps / 2) {  // two warps a row
        const int X = (x0 + warp / 2) * kLoopCtas + rank;
        const bool have = X < rt.nblocks;
        const int dX = have ? rt.blk_dim[X] : 0;
        if (have) {
          double acc[6] = {0, 0, 0, 0, 0, 0};
          row_times(rt, rows, X, dX, 32u * (warp % 2) + lane, 64u, [&](int i) { return scale[i] * v[i]; }, acc);
#pragma unroll
          for (int m = 0; m < 6; ++m) {
            acc[m] = warp_sum(acc[m]);
            if (lane == 0) t.part[warp][m] = acc[m];
          }
        }
        __syncthreads();
        if (have && warp % 2 == 0)
          for (int e = lane; e < dX * kLoopCtas; e += 32) {
            const int m = e / kLoopCtas, o = rt.blk_off[X] + m;
            *cluster.map_shared_rank(w + o, e % kLoopCtas) = (t.part[warp][m] + t.part[warp + 1][m]) * inv * scale[o];
          }
        __syncthreads();
      }
    }
    cluster.sync();
    double nn = 0.0, rq = 0.0;
    for (int i = tid; i < n; i += kLoopThreads) {
      nn += w[i] * w[i];
      rq += v[i] * w[i];
    }
    const double nrm = sqrt(loop_sum(nn, red[0])), quot = loop_sum(rq, red[1]) * inv;
    if (!(isfinite(nrm) && nrm > 0.0)) {
      ok = 0;
      break;
    }
    const bool settled = it > 8 && fabs(quot - lam) <= 1e-10 * fabs(quot);
    lam = quot;
    inv = 1.0 / nrm;
    ok = 1;
    if (settled) break;
  }
  cluster.sync();  // no CTA leaves while another may still write to it
  if (rank == 0 && tid == 0) {
    out[0] = lam;
    out[1] = ok;
  }
}

// The whole PCG run of a small system (sparse/pcg.rs:23-119) for (S + lambda diag) x = -g with x0 = 0: n
// at most kLoopThreads and every CTA's tasks cached, so thread i of every CTA keeps x_i, r_i and row i of
// the inverse of its preconditioner block, the products go over the cluster, and every CTA forms the same
// scalars in the same order. When the recursive residual meets the tolerance it is confirmed by the true
// residual g + S x, and the iteration starts over from it where it is not. fail: the preconditioner's
// per-block flags; any of them ends the run without a step.
// Bound: a cluster barrier, six CTA barriers and their reductions per iteration. A solve of 12 runs of about
// 27 iterations each at n = 185 (32 spherical cameras) went from 15.2 to 10.1 ms; the four kernels of a
// graph iteration take 19 us.
struct LoopPcgResult {
  int accepted, exhausted, terms, pad;
  double rel;
};
constexpr size_t pcg_loop_smem(int n) { return sizeof(double) * (4 * (size_t)n + kLoopTasks * kLoopTaskDoubles); }
__global__ void __launch_bounds__(kLoopThreads) k_pcg_loop(RowTables rt, const double* __restrict__ rows,
                                                           const double* __restrict__ diag, double lambda,
                                                           const double* __restrict__ factor, const int* __restrict__ fail,
                                                           const double* __restrict__ g, int n, int max_it, double tol,
                                                           double* __restrict__ x_out, LoopPcgResult* out) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) double sh[];  // the product's vector, r, the product in two buffers, the tasks
  __shared__ double red[4][kLoopWarps];
  __shared__ LoopTasks t;
  __shared__ int s_block[kLoopThreads];  // element's block
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x;
  double *vec = sh, *rs = sh + n, *qbuf = sh + 2 * (size_t)n, *cache = sh + 4 * (size_t)n;
  if (tid == 0) loop_list(rt, rank, t);
  int bad = 0;
  for (int b = tid; b < rt.nblocks; b += kLoopThreads) {
    bad |= fail[b];
    for (int k = 0; k < rt.blk_dim[b]; ++k) s_block[rt.blk_off[b] + k] = b;
  }
  bad = __syncthreads_or(bad);
  loop_load(rt, rows, nullptr, t, cache);
  const bool live = tid < n;
  const int blk = live ? s_block[tid] : 0, base = live ? rt.blk_off[blk] : 0, dim = live ? rt.blk_dim[blk] : 0;
  const double dg = live ? lambda * diag[tid] : 0.0, b = live ? -g[tid] : 0.0;
  double inv[6] = {0, 0, 0, 0, 0, 0};  // row of the inverse of the block (factor F and scales): F F^T scaled
  if (live && !bad) {
    const double* F = factor + 42 * (size_t)blk;
    const int me = tid - base;
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i < dim) {
        double v = i == me ? 1.0 / F[36 + i] : 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
          if (k < i) v -= F[6 * i + k] * inv[k];
        inv[i] = v / F[6 * i + i];
      }
#pragma unroll
    for (int i = 5; i >= 0; --i)
      if (i < dim) {
        double v = inv[i];
#pragma unroll
        for (int k = 0; k < 6; ++k)
          if (k > i && k < dim) v -= F[6 * k + i] * inv[k];
        inv[i] = v / F[6 * i + i];
      }
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i < dim) inv[i] /= F[36 + i];
  }
  int parity = 0;
  auto product = [&](double mine) {  // (S + lambda diag) vec, this thread's element; mine = vec[tid]
    double* q = qbuf + parity * (size_t)n;
    parity ^= 1;
    loop_product(rt, t, cache, vec, [&](int i, int cta, double r) { *cluster.map_shared_rank(q + i, cta) = r; });
    cluster.sync();
    return live ? q[tid] + dg * mine : 0.0;
  };
  auto precond = [&]() {  // row tid of the preconditioner times rs (visible to the CTA)
    double z = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (k < dim) z += inv[k] * rs[base + k];
    return z;
  };
  cluster.sync();  // every CTA runs before any of them is written to; the cache is in place
  LoopPcgResult res{0, 0, 0, 0, NAN};
  double x = 0.0, r = b;
  if (live) rs[tid] = r;
  const double n0 = sqrt(loop_sum(r * r, red[0]));  // its barrier makes rs visible
  double z = precond();
  double rho = loop_sum(r * z, red[1]);
  if (bad || !isfinite(n0)) {
    // no step
  } else if (n0 == 0.0) {
    res.accepted = 1;
    res.rel = 0.0;
  } else if (isfinite(rho) && rho > 0.0 && max_it > 0) {
    double d = z;
    for (;;) {  // one iteration, all threads of all CTAs together
      if (live) vec[tid] = d;
      __syncthreads();
      const double q = product(d);
      const double curv = loop_sum(d * q, red[0]);
      if (!(isfinite(curv) && curv > 0.0)) break;
      const double alpha = rho / curv;
      if (!isfinite(alpha)) break;
      x += alpha * d;
      r -= alpha * q;
      if (live) rs[tid] = r;
      const double rr = loop_sum(r * r, red[1]);
      z = precond();
      const double rz = loop_sum(r * z, red[2]);
      ++res.terms;
      const double ratio = sqrt(rr) / n0;
      if (!isfinite(ratio)) break;
      bool over = res.terms >= max_it;
      if (ratio <= tol) {  // confirm with the true residual
        if (live) vec[tid] = x;
        __syncthreads();
        const double sx = product(x);  // every thread: the product holds barriers
        r = live ? b - sx : 0.0;
        if (live) rs[tid] = r;
        const double tr = sqrt(loop_sum(r * r, red[3])) / n0;
        if (!isfinite(tr)) break;
        if (tr <= tol) {
          res.accepted = 1;
          res.rel = tr;
          break;
        }
        z = precond();
        rho = loop_sum(r * z, red[0]);
        if (!(isfinite(rho) && rho > 0.0)) {
          res.rel = tr;
          break;
        }
        d = z;
      } else {
        if (!(isfinite(rz) && rz > 0.0)) break;
        const double beta = rz / rho;
        if (!isfinite(beta)) break;
        d = z + beta * d;
        rho = rz;
      }
      if (over) {  // the iteration limit: the residual the step is left with
        if (live) vec[tid] = x;
        __syncthreads();
        const double sx = product(x);  // every thread: the product holds barriers
        r = live ? b - sx : 0.0;
        res.rel = sqrt(loop_sum(r * r, red[3])) / n0;
        res.terms = max_it;
        res.exhausted = 1;
        break;
      }
    }
  }
  cluster.sync();  // no CTA leaves while another may still write to it
  if (rank == 0) {
    if (live) x_out[tid] = x;
    if (tid == 0) *out = res;
  }
}

}  // namespace omvgba
