// Leaf evaluation of depth-limited solves. A depth-limited flop solve ends
// its tree at the turn deal (N_LEAF nodes); every traversal values those
// leaves with the leaf-value network instead of the turn and river subtrees:
//
//   prepare: the opponent's reach arriving at each leaf is kept per player
//            (the network takes both players' ranges; the traverser's own
//            range is the one its opponent's latest traversal delivered);
//   inputs:  one network row per (leaf, dealt card): both ranges in combo
//            order with the hands holding the card removed, scaled to a
//            maximum of 1, the board and dealt card one-hot, pot and stack;
//   values:  the network gives every combo's EV (in pots) after that card;
//            the leaf's counterfactual value of traverser hand h is
//              norm * factor * pot * sum_c [c not in h] EV_c(h) * m_c(h),
//            the same sum a chance node forms over its children
//            (cfr.rs:435-479), after a zero-sum correction of each card's
//            network values (see leaf_shift_kernel), where m_c(h) is the
//            opponent reach
//            compatible with h and c: with T the total, A[x] the reach of
//            hands holding card x and R{x,y} the reach of combo {x,y},
//              m_c(h) = T - A[h1] - A[h2] + R{h1,h2} - (A[c] - R{c,h1} - R{c,h2}).
#include <cuda_runtime.h>

#include <cstdint>

#include "engine.hpp"
#include "pdl.cuh"

namespace dcfr {

namespace {

constexpr float LEAF_SCALE = 10000.0f;

__device__ __forceinline__ int combo_of(int a, int b) {
  const int hi = a > b ? a : b, lo = a > b ? b : a;
  return hi * (hi - 1) / 2 + lo;
}

// Block (leaf task, side): side 0 also keeps the opponent's reach at the leaf;
// both leave their side's reach (0: opponent, 1: traverser) in combo order with
// its total and the reach of the hands holding each card: what every mass m_c
// is made of, summed once per leaf and traversal.
constexpr int PREPARE_WARPS = 16;
__global__ void __launch_bounds__(PREPARE_WARPS * 32) leaf_prepare_kernel(LeafArgs A,
                                                                          const LeafTask* __restrict__ tasks,
                                                                          const uint8_t* __restrict__ hc1_p,
                                                                          const uint8_t* __restrict__ hc2_p,
                                                                          const uint8_t* __restrict__ hc1_o,
                                                                          const uint8_t* __restrict__ hc2_o) {
  __shared__ float R[DCFR_NUM_COMBOS];      // combo order
  __shared__ float rs[DCFR_NUM_COMBOS + 8]; // hand order
  __shared__ uchar2 cs[DCFR_NUM_COMBOS + 8];
  __shared__ double red[PREPARE_WARPS];
  const int p = A.p, o = p ^ 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int side = blockIdx.y, q = side ? p : o, n = A.n[q];
  const uint8_t* c1 = side ? hc1_p : hc1_o;
  const uint8_t* c2 = side ? hc2_p : hc2_o;
  const LeafTask T = tasks[blockIdx.x];
  for (int j = tid; j < n; j += blockDim.x) cs[j] = make_uchar2(c1[j], c2[j]);
  for (int i = tid; i < DCFR_NUM_COMBOS; i += blockDim.x) R[i] = 0.0f;
  pdl_wait();
  pdl_trigger();
  const float* src = A.reach + (size_t)T.slot * A.stride;
  const bool live = A.alive[T.slot] != 0;
  if (side == 0) {
    float* kept = A.leaf_reach[o] + (size_t)T.leaf * A.stride;
    for (int h = tid; h < A.stride; h += blockDim.x) kept[h] = live ? src[h] : 0.0f;
  }
  if (!live) return;
  const float* r = side ? A.leaf_reach[p] + (size_t)T.leaf * A.stride : src;
  LeafMass& M = A.mass[T.leaf * 2 + side];
  __syncthreads();
  double t = 0.0;
  for (int j = tid; j < n; j += blockDim.x) {
    const float v = r[j];
    rs[j] = v;
    R[A.combos[q][j]] = v;
    t += (double)v;
  }
  for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
  if (lane == 0) red[warp] = t;
  __syncthreads();
  // A warp per card.
  for (int c = warp; c < 52; c += PREPARE_WARPS) {
    double s = 0.0;
    for (int j = lane; j < n; j += 32)
      if (cs[j].x == c || cs[j].y == c) s += (double)rs[j];
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0) M.card[c] = s;
  }
  if (tid == 0) {
    double sum = 0.0;
    for (int w = 0; w < PREPARE_WARPS; w++) sum += red[w];
    M.total = sum;
  }
  for (int i = tid; i < DCFR_NUM_COMBOS; i += blockDim.x) M.reach[i] = R[i];
}

// Block (leaf task, card index): one input row, as the network packs it (bf16,
// zeros past the network's inputs).
__global__ void __launch_bounds__(256) leaf_inputs_kernel(LeafArgs A, const LeafTask* __restrict__ tasks,
                                                          const uint8_t* __restrict__ hc1_0,
                                                          const uint8_t* __restrict__ hc2_0,
                                                          const uint8_t* __restrict__ hc1_1,
                                                          const uint8_t* __restrict__ hc2_1) {
  extern __shared__ __align__(16) __nv_bfloat16 row[];
  __shared__ float red[2][8];
  pdl_wait();
  pdl_trigger();
  const LeafTask T = tasks[blockIdx.x];
  const int ci = blockIdx.y, tid = threadIdx.x;
  const int card = A.cards[ci];
  __nv_bfloat16* x = A.x + ((size_t)T.leaf * A.nc + ci) * A.ldx;
  for (int i = tid; i < A.ldx / 8; i += blockDim.x) reinterpret_cast<uint4*>(row)[i] = make_uint4(0u, 0u, 0u, 0u);
  float mx[2] = {0.0f, 0.0f};
  for (int q = 0; q < 2; q++) {
    const float* r = A.leaf_reach[q] + (size_t)T.leaf * A.stride;
    const uint8_t* c1 = q ? hc1_1 : hc1_0;
    const uint8_t* c2 = q ? hc2_1 : hc2_0;
    for (int h = tid; h < A.n[q]; h += blockDim.x)
      if (c1[h] != card && c2[h] != card) mx[q] = fmaxf(mx[q], r[h]);
    for (int d = 16; d > 0; d >>= 1) mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], d));
    if ((tid & 31) == 0) red[q][tid >> 5] = mx[q];
  }
  __syncthreads();
  for (int q = 0; q < 2; q++) {
    const float* r = A.leaf_reach[q] + (size_t)T.leaf * A.stride;
    const uint8_t* c1 = q ? hc1_1 : hc1_0;
    const uint8_t* c2 = q ? hc2_1 : hc2_0;
    float m = 0.0f;
    for (int w = 0; w < 8; w++) m = fmaxf(m, red[q][w]);
    const float inv = m > 0.0f ? 1.0f / m : 0.0f;
    for (int h = tid; h < A.n[q]; h += blockDim.x)
      row[q * DCFR_NUM_COMBOS + A.combos[q][h]] =
          __float2bfloat16((c1[h] != card && c2[h] != card) ? r[h] * inv : 0.0f);
  }
  if (tid == 0) {
    for (int k = 0; k < 3; k++) row[2 * DCFR_NUM_COMBOS + A.board[k]] = __float2bfloat16(1.0f);
    row[2 * DCFR_NUM_COMBOS + card] = __float2bfloat16(1.0f);
    row[2 * DCFR_NUM_COMBOS + 52] = __float2bfloat16(T.pot / LEAF_SCALE);
    row[2 * DCFR_NUM_COMBOS + 53] = __float2bfloat16(T.stack / LEAF_SCALE);
  }
  __syncthreads();
  for (int i = tid; i < A.ldx / 8; i += blockDim.x)
    reinterpret_cast<uint4*>(x)[i] = reinterpret_cast<const uint4*>(row)[i];
}

// m_c for a hand: the other side's reach compatible with it and card c.
__device__ __forceinline__ double leaf_mass(double total, const double* card, const float* R, int h1, int h2, int ch,
                                            int c) {
  return total - card[h1] - card[h2] + (double)R[ch] - (card[c] - (double)R[combo_of(c, h1)] - (double)R[combo_of(c, h2)]);
}

// Block (leaf task, card index): the shift that makes the card's network
// values zero-sum (as the subgame is): with S_q = sum over q's hands of
// r_q(h) m_c(h) EV_q,c(h) and M the joint compatible mass, both sides are
// shifted by (S_p + S_o) / (2 M), so the corrected values satisfy
// S_p + S_o = 0.
__global__ void __launch_bounds__(256) leaf_shift_kernel(LeafArgs A, const LeafTask* __restrict__ tasks,
                                                         const uint8_t* __restrict__ hc1_p,
                                                         const uint8_t* __restrict__ hc2_p,
                                                         const uint8_t* __restrict__ hc1_o,
                                                         const uint8_t* __restrict__ hc2_o) {
  __shared__ float R[2][DCFR_NUM_COMBOS];
  __shared__ double card[2][52];
  __shared__ double red[3][8];
  pdl_wait();
  pdl_trigger();
  const LeafTask T = tasks[blockIdx.x];
  if (A.alive[T.slot] == 0) return;
  const int p = A.p, o = p ^ 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const LeafMass* M = A.mass + T.leaf * 2;
  for (int i = tid; i < 2 * DCFR_NUM_COMBOS; i += blockDim.x)
    (&R[0][0])[i] = M[i / DCFR_NUM_COMBOS].reach[i % DCFR_NUM_COMBOS];
  for (int i = tid; i < 104; i += blockDim.x) (&card[0][0])[i] = M[i / 52].card[i % 52];
  const double total[2] = {M[0].total, M[1].total};
  __syncthreads();
  const int ci = blockIdx.y, c = A.cards[ci];
  const float* y = A.y + ((size_t)T.leaf * A.nc + ci) * A.ldy;
  double sp = 0.0, so = 0.0, mm = 0.0;
  for (int h = tid; h < A.n[p]; h += blockDim.x) {
    const int h1 = hc1_p[h], h2 = hc2_p[h];
    if (h1 == c || h2 == c) continue;
    const int ch = A.combos[p][h];
    const double w = (double)R[1][ch] * leaf_mass(total[0], card[0], R[0], h1, h2, ch, c);
    sp += w * (double)y[(size_t)p * DCFR_NUM_COMBOS + ch];
    mm += w;
  }
  for (int j = tid; j < A.n[o]; j += blockDim.x) {
    const int h1 = hc1_o[j], h2 = hc2_o[j];
    if (h1 == c || h2 == c) continue;
    const int ch = A.combos[o][j];
    so += (double)R[0][ch] * leaf_mass(total[1], card[1], R[1], h1, h2, ch, c) *
          (double)y[(size_t)o * DCFR_NUM_COMBOS + ch];
  }
  for (int d = 16; d > 0; d >>= 1) {
    sp += __shfl_xor_sync(0xffffffffu, sp, d);
    so += __shfl_xor_sync(0xffffffffu, so, d);
    mm += __shfl_xor_sync(0xffffffffu, mm, d);
  }
  if (lane == 0) {
    red[0][warp] = sp;
    red[1][warp] = so;
    red[2][warp] = mm;
  }
  __syncthreads();
  if (tid == 0) {
    double a = 0.0, b = 0.0, m = 0.0;
    for (int w = 0; w < 8; w++) {
      a += red[0][w];
      b += red[1][w];
      m += red[2][w];
    }
    A.shift[T.leaf * A.nc + ci] = m > 0.0 ? 0.5 * (a + b) / m : 0.0;
  }
}

// Block (leaf task, LEAF_HANDS hands): the traverser's value row at the leaf.
// One block per leaf for the masses, the 49 shifts one after another and the
// values took 181 us of a traversal (14 leaves, 470 hands); the masses, the
// shifts and the values by blocks of their own take 3, 10 and 9 us.
constexpr int LEAF_HANDS = 64;
__global__ void __launch_bounds__(LEAF_HANDS) leaf_values_kernel(LeafArgs A, const LeafTask* __restrict__ tasks,
                                                                 const uint8_t* __restrict__ hc1_p,
                                                                 const uint8_t* __restrict__ hc2_p, int hp) {
  __shared__ float R[DCFR_NUM_COMBOS];
  __shared__ double card[52];
  pdl_wait();
  pdl_trigger();
  const LeafTask T = tasks[blockIdx.x];
  if (A.alive[T.slot] == 0) return;  // dead subtree (cfr.rs:267-274): row untouched
  const int p = A.p, tid = threadIdx.x;
  const LeafMass& M = A.mass[T.leaf * 2];
  for (int i = tid; i < DCFR_NUM_COMBOS; i += LEAF_HANDS) R[i] = M.reach[i];
  for (int i = tid; i < 52; i += LEAF_HANDS) card[i] = M.card[i];
  const double total = M.total;
  __syncthreads();
  const int h = blockIdx.y * LEAF_HANDS + tid;
  if (h >= hp) return;
  float v = 0.0f;
  if (h < A.n[p]) {
    const int h1 = hc1_p[h], h2 = hc2_p[h];
    const int ch = A.combos[p][h];
    const float* y = A.y + (size_t)T.leaf * A.nc * A.ldy + (size_t)p * DCFR_NUM_COMBOS + ch;
    const double* shift = A.shift + T.leaf * A.nc;
    double acc = 0.0;
#pragma unroll 7
    for (int ci = 0; ci < A.nc; ci++) {
      const int c = A.cards[ci];
      const double ev = (double)y[(size_t)ci * A.ldy] - shift[ci];
      if (c == h1 || c == h2) continue;
      acc += ev * leaf_mass(total, card, R, h1, h2, ch, c);
    }
    v = (float)(A.norm * (double)A.factor * (double)T.pot * acc);
  }
  A.vals[(size_t)T.row * A.stride + h] = v;
}

}  // namespace

// Before the network: the masses and its inputs.
void launch_leaf_inputs(const LeafArgs& A, const LeafTask* tasks, int ntasks, const uint8_t* hc1_0,
                        const uint8_t* hc2_0, const uint8_t* hc1_1, const uint8_t* hc2_1, cudaStream_t s) {
  if (ntasks <= 0) return;
  const uint8_t *p1 = A.p ? hc1_1 : hc1_0, *p2 = A.p ? hc2_1 : hc2_0, *o1 = A.p ? hc1_0 : hc1_1,
                *o2 = A.p ? hc2_0 : hc2_1;
  launch_dependent(leaf_prepare_kernel, dim3((unsigned)ntasks, 2), PREPARE_WARPS * 32, 0, s, A, tasks, p1, p2, o1, o2);
  launch_dependent(leaf_inputs_kernel, dim3((unsigned)ntasks, (unsigned)A.nc), 256,
                   (size_t)A.ldx * sizeof(__nv_bfloat16), s, A, tasks, hc1_0, hc2_0, hc1_1, hc2_1);
}

// After it: the leaves' value rows.
void launch_leaf_values(const LeafArgs& A, const LeafTask* tasks, int ntasks, const uint8_t* hc1_p,
                        const uint8_t* hc2_p, const uint8_t* hc1_o, const uint8_t* hc2_o, int hp, cudaStream_t s) {
  if (ntasks <= 0) return;
  launch_dependent(leaf_shift_kernel, dim3((unsigned)ntasks, (unsigned)A.nc), 256, 0, s, A, tasks, hc1_p, hc2_p, hc1_o,
                   hc2_o);
  launch_dependent(leaf_values_kernel, dim3((unsigned)ntasks, (unsigned)((hp + LEAF_HANDS - 1) / LEAF_HANDS)),
                   LEAF_HANDS, 0, s, A, tasks, hc1_p, hc2_p, hp);
}

}  // namespace dcfr
