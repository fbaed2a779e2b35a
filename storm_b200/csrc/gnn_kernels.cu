// gnn_kernels.cu -- warm-start network on the cell-dual graph: fused two-layer MLP
// kernels on the sm_100a tensor cores (tcgen05 MMA, TMEM accumulators), their
// backward passes, and the gather/scatter, loss and optimiser kernels around them.
//
// The network has no counterpart in the reference (SToRM starts steady runs from the
// user's initial condition); it predicts an initial h, hu, hv for the solver, which
// then runs on to its own stop test.
//
// Graph layout.  Cells are padded to Tp (a multiple of 128).  Every cell c owns three
// directed edge rows, one per local face k: row k*Tp + c carries the message from the
// neighbour nbr[k*Tp + c] (-1: no neighbour) into c.  An MLP input row is the
// concatenation of up to three 128-wide segments, each read from a bf16 matrix
// through an optional row map, or summed over the three edge rows of a cell
// (the message aggregation), so the edge update [e, h_src, h_dst] and the node
// update [h, sum_k e_k] need no materialised concatenation.
//
// One CTA per SM works through tiles of 128 rows (64 in the weight gradients) with its warps
// in fixed roles: copies, MMA issue, epilogues, rows that TMA cannot fetch.  Forward:
// D1 = A W1^T over the segments, bias + ReLU into a shared-memory tile, D2 = a1 W2^T,
// bias (+ residual).  Weights stay resident in shared memory for the CTA's lifetime.
#include <cstdint>
#include <cstdio>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "umma.cuh"

namespace storm {
namespace gnn {

using bf16 = __nv_bfloat16;

constexpr int kRows = 128;     // rows per tile (MMA M)
constexpr int kHid = 128;      // hidden width
constexpr int kMaxSeg = 3;

struct Seg {
  const bf16* src;       // [*, width] row-major
  const int32_t* idx;    // row map (nullptr: identity); a negative entry reads zeros
  int32_t width;         // 64 or 128
  int32_t agg;           // 1: sum of rows r + k*agg_stride (k < 3) whose nbr entry is >= 0
  int32_t agg_stride;
  const int32_t* nbr;    // [3*agg_stride] neighbour table (mask of the aggregation)
};

struct MlpFwd {
  int32_t rows, nseg, k_in, n_out;
  Seg seg[kMaxSeg];
  const bf16* w1;   // [128][k_in]
  const float* b1;  // [128]
  const bf16* w2;   // [n_out][128]
  const float* b2;  // [n_out]
  const bf16* res;  // [rows][n_out] residual added to the output, or nullptr
  bf16* out;        // [rows][n_out]
  float* out_f32;   // optional fp32 copy of the output
  bf16* a1_save;    // [rows][128] hidden activation (training), or nullptr
  int32_t* err;
};

// Backward, data part: da1 = dy W2, dz1 = da1 * (a1 > 0), dA = dz1 W1 split per segment.
struct SegGrad {
  float* out;         // [rows][width] fp32, or nullptr (segment gradient not needed)
  const float* add;   // added to the result (the residual path), or nullptr
};
struct MlpBwdData {
  int32_t rows, nseg, k_in, n_out;
  int32_t seg_width[kMaxSeg];
  SegGrad dseg[kMaxSeg];
  const float* dy;    // [rows][n_out]
  const bf16* a1;     // [rows][128]
  const bf16* w1;     // [128][k_in]
  const bf16* w2;     // [n_out][128]
  bf16* dz1_save;     // [rows][128]
  int32_t* err;
};

// Backward, weight part: per-CTA partial dW1 = dz1^T A, dW2 = dy^T a1, db1, db2.
struct MlpBwdWeight {
  int32_t rows, nseg, k_in, n_out;
  Seg seg[kMaxSeg];
  const float* dy;    // [rows][n_out]
  const bf16* a1;     // [rows][128]
  const bf16* dz1;    // [rows][128]
  float* part;        // [grid][128*k_in + 128 + n_out*128 + n_out]
  int32_t* err;
};

__device__ __forceinline__ void set_err(int32_t* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// ---- shared-memory staging -------------------------------------------------------

// 16 bytes, or zeros without touching memory: a predicated load, so that a batch of them
// is issued together (branches around loads made each wait for the one before).
__device__ __forceinline__ uint4 ld_if(const void* p, bool want) {
  uint4 v = make_uint4(0, 0, 0, 0);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.s32 p, %5, 0;\n\t"
      "@p ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}\n"
      : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
      : "l"(p), "r"(want ? 1 : 0));
  return v;
}

// The aggregation segment: rows r + k*agg_stride, k = 0, 1, 2, whose nbr entry is >= 0, added
// in that order in fp32.  Eight threads take a row, kThr / 8 rows at a time, four times over.
// Which of a thread's twelve rows count (bit 3 i + k), asked for ahead of the rows ...
template <int kThr>
__device__ __forceinline__ uint32_t agg_mask(const Seg& s, int row0, int tid) {
  int32_t e[4][3];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int k = 0; k < 3; k++)
      e[i][k] = s.nbr[static_cast<size_t>(k) * s.agg_stride + row0 + (tid >> 3) + i * (kThr / 8)];
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) m |= (e[i][k] >= 0 ? 1u : 0u) << (3 * i + k);
  return m;
}
// ... and 64 columns (from col0) of kThr / 2 rows into one block, all loads in flight together.
template <int kThr>
__device__ __forceinline__ void stage_agg_block(const Seg& s, uint32_t mask, int row0, int col0, uint8_t* dst, int tid) {
  uint4 w[4][3];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int k = 0; k < 3; k++)
      w[i][k] = ld_if(s.src + (static_cast<size_t>(k) * s.agg_stride + row0 + (tid >> 3) + i * (kThr / 8)) * s.width + col0 +
                          (tid & 7) * 8,
                      (mask >> (3 * i + k)) & 1);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = 0.f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if (!((mask >> (3 * i + k)) & 1)) continue;
      const uint32_t x[4] = {w[i][k].x, w[i][k].y, w[i][k].z, w[i][k].w};
#pragma unroll
      for (int u = 0; u < 4; u++) {
        acc[2 * u] += __uint_as_float(x[u] << 16);
        acc[2 * u + 1] += __uint_as_float(x[u] & 0xffff0000u);
      }
    }
    *reinterpret_cast<uint4*>(dst + umma::sw128_offset((tid >> 3) + i * (kThr / 8), (tid & 7) * 8)) =
        make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
  }
}

// Asynchronous copy of one 16-byte chunk global -> shared (zero-filled when `valid` is
// false); the copies of a thread are grouped with commit / wait_group.
__device__ __forceinline__ void cp_async16(uint8_t* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_addr(dst)), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A lane's four of 128 row-map entries, loaded a tile ahead; by a whole warp, the first
// entry if they are consecutive rows, else -1.
__device__ __forceinline__ int4 map_entries(const int32_t* idx, int lane) {
  const int32_t* e = idx + 4 * lane;
  return make_int4(e[0], e[1], e[2], e[3]);
}
__device__ __forceinline__ int consecutive(int4 e, int lane) {
  const int first = __shfl_sync(0xffffffffu, e.x, 0), want = first + 4 * lane;
  return __all_sync(0xffffffffu, e.x == want && e.y == want + 1 && e.z == want + 2 && e.w == want + 3) ? first : -1;
}

// The same for 64 rows, two entries a lane.
__device__ __forceinline__ int2 slab_entries(const int32_t* idx, int lane) {
  return make_int2(idx[2 * lane], idx[2 * lane + 1]);
}
__device__ __forceinline__ int consecutive(int2 e, int lane) {
  const int first = __shfl_sync(0xffffffffu, e.x, 0), want = first + 2 * lane;
  return __all_sync(0xffffffffu, e.x == want && e.y == want + 1) ? first : -1;
}

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

// Issue D (+)= A B^T over K (a multiple of 16), A and B K-major tiles with blocks of 64
// columns: a_blk / b_blk are the byte strides between their 64-column blocks.  Descriptors
// count 16 bytes.
template <int K>
__device__ __forceinline__ void mma_kmajor(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc, bool accumulate) {
  static_assert(K <= 64, "one block of columns");
  const uint64_t ad = umma::desc_kmajor(a), bd = umma::desc_kmajor(b);
#pragma unroll
  for (int k = 0; k < K; k += 16)
    umma::mma_bf16(tmem_d, ad + k / 8, bd + k / 8, idesc, (accumulate || k > 0) ? 1u : 0u);
}

// ---- forward ----------------------------------------------------------------------

// Shared memory: W1 (128 x k_in), W2 (n_out x 128), the ring of input blocks (128 rows x
// 64 columns, 16 KB), the output tile, half a hidden tile (training), biases, barriers.
constexpr int kBlk = kRows * 128;  // bytes of a block
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kMaxStages = 8;
__host__ __device__ constexpr size_t fwd_fixed_bytes(int k_in, int n_out, bool save) {
  return 1024 + static_cast<size_t>(kHid) * k_in * 2 + static_cast<size_t>(n_out) * kHid * 2 + (n_out / 64 + save) * kBlk +
         4 * (kHid + 128) + 512;
}
__host__ __device__ constexpr int fwd_stages(int k_in, int n_out, bool save) {
  const int n = static_cast<int>((kSmemMax - fwd_fixed_bytes(k_in, n_out, save)) / kBlk);
  return n < kMaxStages ? n : kMaxStages;
}
__host__ __device__ constexpr size_t fwd_smem_bytes(int k_in, int n_out, bool save) {
  return fwd_fixed_bytes(k_in, n_out, save) + static_cast<size_t>(fwd_stages(k_in, n_out, save)) * kBlk;
}
static_assert(fwd_stages(384, 128, false) == 4 && fwd_stages(384, 128, true) == 3, "ring stages of the widest input");

struct FwdMaps {  // boxes of 64 columns x 128 rows (w2: n_out rows)
  CUtensorMap seg[kMaxSeg], w1, w2, out, a1, res;
};
constexpr int kAnyRows = 1 << 30;  // rows of a mapped segment's matrix: the caller does not say

// A place in a ring of n stages: the stage and the parity of its present use.
struct RingPos {
  int st = 0;
  uint32_t par = 0;
  __device__ __forceinline__ void next(int n) {
    if (++st == n) {
      st = 0;
      par ^= 1;
    }
  }
};

// Warp roles of the forward kernel (512 or 640 threads):
//   warp 0      one thread hands out the ring's stages in the order of the blocks, and fills
//               by TMA (the weights with the first tile's) each 64-column block of the CTA's
//               tiles whose rows follow one another (unmapped segments, and mapped ones where
//               the map is a run, as the receiver's is);
//   warp 1      one thread issues the MMAs: D1[slot] = A W1^T block by block as the ring
//               fills, D2[slot] = a1 W2^T one tile behind, so the hidden tile's epilogue
//               is hidden by the next tile's first products;
//   warp 2      looks through the row maps, up to two tiles ahead of warps 0 and 12 on;
//   warps 4-7   epilogue 1: D1 -> bias + ReLU -> hidden tile as bf16 in the first half of D1's
//               own columns, which D2's MMAs read from TMEM (in training also out by TMA);
//   warps 8-11  epilogue 2: D2 -> residual + bias -> output; the residual comes into the
//               output tile's shared memory by TMA while D2 is computed, the sum leaves from
//               there by TMA (direct loads and stores, a row to a thread, take the L1 32
//               lines an instruction, and every other wait on that path with them);
//   the warps from 12 on the other blocks: mapped rows by cp.async (a negative entry reads zeros;
//               TMA's gather4 took about 130 cycles per four half rows, 135 us for the
//               edge update below), and the aggregation's sums of three edge rows.
// One warp alone waits on `empty`, for every block in turn: a parity tells a phase only
// from the one beside it, so a role that waited for its own blocks alone could take a stage
// two uses early.  The warps from 12 on get theirs from it through `grant`, which holds no phase
// but their own.
// D1 and D2 are double-buffered in TMEM (slot = tile parity); the MMAs of one thread run in
// order, so D1 of a tile may overwrite the hidden tile that D2 two tiles before has read.
// Every wait is bounded; a wait that runs out raises the abort flag, which every role polls.
//
// What bounds it: the latency of a block's way from L2 or HBM to its stage, with three (in
// training) or four stages at k_in = 384 next to 96 KB of W1.  Every role's loops stay rolled:
// unrolled over columns and segments, the roles' code no longer fitted the instruction cache
// and 6 of 17 stall cycles an instruction went on fetching it (0.7 now).  Measured (us;
// before, unrolled, the hidden tile in shared memory and the residual read a row to a thread):
// edge update 58 (90) at 300,000 rows, with saved hidden rows 73 (96), at 75,000 rows 22 (29),
// at 9,000 12 (14); node update 57 (68) at 100,000 rows, encoder 15 (17) at 75,000.
//
// Threads that gather: 128 where rows are only copied (256 took 65 us instead of 58 for the
// edge update of 300,000 rows), 256 where a segment is summed over three edge rows, so that
// twelve 16-byte loads a thread cover a block (node update of 100,000 rows: 57 us; 128 threads
// in two rounds 68 us).
__host__ __device__ constexpr int fwd_gather(bool agg) { return agg ? 256 : 128; }
__host__ __device__ constexpr int fwd_threads(bool agg) { return 384 + fwd_gather(agg); }
__device__ __forceinline__ bool aborted(const int* flag) { return *reinterpret_cast<const volatile int*>(flag) != 0; }

template <bool kAgg>
__global__ void __launch_bounds__(fwd_threads(kAgg), 1) k_mlp_fwd(const __grid_constant__ MlpFwd p,
                                                              const __grid_constant__ FwdMaps maps) {
  constexpr int kGather = fwd_gather(kAgg), kRowsEach = kRows * 8 / kGather;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = align1024(smem_raw);
  const bool save = p.a1_save != nullptr;
  const int nst = fwd_stages(p.k_in, p.n_out, save);
  uint8_t* w1s = base;
  uint8_t* w2s = w1s + kHid * p.k_in * 2;
  uint8_t* ring = w2s + p.n_out * kHid * 2;
  uint8_t* ios = ring + nst * kBlk;               // [n_out / 64] residual in, output out
  uint8_t* a1s = ios + (p.n_out >> 6) * kBlk;     // half a hidden tile (training)
  float* b1s = reinterpret_cast<float*>(a1s + (save ? kBlk : 0));
  float* b2s = b1s + kHid;
  uint64_t* bars = reinterpret_cast<uint64_t*>(b2s + 128);
  uint64_t* full = bars;          // [8] ring stage filled
  uint64_t* empty = bars + 8;     // [8] MMAs reading the stage done (commit)
  uint64_t* grant = bars + 16;    // [8] ring stage given to the warps from 12 on
  uint64_t* d1full = bars + 24;   // [2] D1[slot] complete (commit)
  uint64_t* a1full = bars + 26;   // [2] hidden tile written over D1[slot]
  uint64_t* d2full = bars + 28;   // [2] D2[slot] complete (commit)
  uint64_t* d2free = bars + 30;   // [2] epilogue 2 has read D2[slot]
  uint64_t* w1full = bars + 32;   // [6] W1 block loaded
  uint64_t* w2full = bars + 38;   // W2 loaded
  uint64_t* resfull = bars + 39;  // residual tile loaded
  uint64_t* runfull = bars + 40;  // [2] row maps of a tile looked through
  uint64_t* runfree = bars + 42;  // [2] ... and read by warps 0 and 12 on
  int* runs = reinterpret_cast<int*>(bars + 44);  // [2][4] first row of a segment whose 128 rows are consecutive, else -1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 48);
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < nst; i++) {
      umma::mbar_init(&full[i], 1);
      umma::mbar_init(&empty[i], 1);
      umma::mbar_init(&grant[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      umma::mbar_init(&d1full[i], 1);
      umma::mbar_init(&a1full[i], kRows);
      umma::mbar_init(&d2full[i], 1);
      umma::mbar_init(&d2free[i], kRows);
      umma::mbar_init(&runfull[i], 1);
      umma::mbar_init(&runfree[i], 1 + kGather / 32);
    }
    for (int i = 0; i < 6; i++) umma::mbar_init(&w1full[i], 1);
    umma::mbar_init(w2full, 1);
    umma::mbar_init(resfull, 1);
    umma::mbar_fence_init();
    umma::fence_async_smem();
    s_abort = 0;
  }
  if (warp == 1) umma::tmem_alloc(tmem_slot, 512);
  umma::grid_launch_next();
  umma::grid_wait();
  if (threadIdx.x >= 128 && threadIdx.x < 128 + kHid) b1s[threadIdx.x - 128] = p.b1[threadIdx.x - 128];
  if (threadIdx.x >= 256 && static_cast<int>(threadIdx.x) < 256 + p.n_out) b2s[threadIdx.x - 256] = p.b2[threadIdx.x - 256];
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const int ntiles = p.rows / kRows;
  const int mine = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int nblk = p.k_in >> 6;
  auto row_of = [&](int t) { return static_cast<int>(blockIdx.x + t * gridDim.x) * kRows; };

  if (warp == 0) {
    // ---- ring and TMA
    if (umma::elect_one()) {
      int nw = 0;  // W1 blocks asked for
      auto load_w1 = [&]() {
        umma::mbar_expect(&w1full[nw], kHid * 128);
        umma::tma_load(w1s + nw * (kHid * 128), &maps.w1, nw * 64, 0, &w1full[nw]);
        nw++;
      };
      RingPos r, last;  // the next block; the oldest whose copy may still be in flight
      int g = 0;        // blocks handed out
      bool ok = true;
      for (int t = 0; t < mine && ok; t++) {
        if (!umma::mbar_wait(&runfull[t & 1], (t >> 1) & 1)) {
          ok = false;
          break;
        }
#pragma unroll 1
        for (int s = 0; s < p.nseg; s++) {
          const int nb = p.seg[s].width >> 6, run = runs[(t & 1) * 4 + s];
#pragma unroll 1
          for (int b = 0; b < nb && ok; b++) {
            if (g >= nst) {
              ok = umma::mbar_wait(&empty[r.st], r.par ^ 1) && !aborted(&s_abort);
              if (!ok) break;
              last.next(nst);
            }
            if (nw < nblk) load_w1();
            if (run < 0) {
              umma::mbar_arrive(&grant[r.st]);
            } else {
              umma::mbar_expect(&full[r.st], kBlk);
              umma::tma_load(ring + r.st * kBlk, &maps.seg[s], b * 64, run, &full[r.st]);
            }
            r.next(nst);
            if (++g == (nst < nblk ? nst : nblk)) {  // the first stages are taken: the other weights
              while (nw < nblk) load_w1();
              umma::mbar_expect(w2full, p.n_out * kHid * 2);
              for (int x = 0; x < kHid; x += 64) umma::tma_load(w2s + (x >> 6) * (p.n_out * 128), &maps.w2, x, 0, w2full);
            }
          }
        }
        umma::mbar_arrive(&runfree[t & 1]);
      }
      if (!ok) s_abort = 1;
      // the copies still in flight land before the block's shared memory is given up
      for (int k = g < nst ? g : nst; k > 0; k--, last.next(nst)) umma::mbar_wait(&full[last.st], last.par);
      for (int k = 0; k < nw; k++) umma::mbar_wait(&w1full[k], 0);
      if (nw == nblk) umma::mbar_wait(w2full, 0);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issuer
    if (umma::elect_one()) {
      const uint32_t w1a = umma::smem_addr(w1s), ra = umma::smem_addr(ring);
      const uint64_t w2d = umma::desc_kmajor(umma::smem_addr(w2s));
      const uint32_t w2blk = p.n_out * 128 / 16;
      const uint32_t idesc1 = umma::idesc_bf16(kRows, kHid, false, false);
      const uint32_t idesc2 = umma::idesc_bf16(kRows, p.n_out, false, false);
      RingPos r;
      bool ok = true;
      for (int t = 0; t <= mine && ok; t++) {
        const int slot = t & 1;
        if (t < mine) {  // D1 of tile t
#pragma unroll 1
          for (int b = 0; b < nblk; b++) {
            if ((t == 0 && !umma::mbar_wait(&w1full[b], 0)) || !umma::mbar_wait(&full[r.st], r.par)) {
              ok = false;
              break;
            }
            umma::fence_after_sync();
            mma_kmajor<64>(tmem + slot * 128, ra + r.st * kBlk, w1a + b * (kHid * 128), idesc1, b > 0);
            umma::commit(&empty[r.st]);
            r.next(nst);
          }
          if (!ok) break;
          umma::commit(&d1full[slot]);
        }
        if (t > 0) {  // D2 of tile t - 1
          const int u = t - 1, us = u & 1;
          if ((u == 0 && !umma::mbar_wait(w2full, 0)) || (u >= 2 && !umma::mbar_wait(&d2free[us], ((u >> 1) - 1) & 1)) ||
              !umma::mbar_wait(&a1full[us], (u >> 1) & 1)) {
            ok = false;
            break;
          }
          umma::fence_after_sync();
#pragma unroll
          for (int k = 0; k < kHid; k += 16)
            umma::mma_bf16_ts(tmem + 256 + us * 128, tmem + us * 128 + k / 2, w2d + (k >> 6) * w2blk + (k & 63) / 8, idesc2,
                              k > 0 ? 1u : 0u);
          umma::commit(&d2full[us]);
        }
      }
      // the last commit (of them all, in order), before shared memory and TMEM are given up
      if (ok && mine > 0) ok = umma::mbar_wait(&d2full[(mine - 1) & 1], ((mine - 1) >> 1) & 1);
      if (!ok) s_abort = 1;
    }
    __syncwarp();
  } else if (warp == 2) {
    // ---- row maps
    for (int t = 0; t < mine; t++) {
      int4 ent[kMaxSeg];
      int run[kMaxSeg];
#pragma unroll
      for (int s = 0; s < kMaxSeg; s++)
        if (s < p.nseg && p.seg[s].idx && !p.seg[s].agg) ent[s] = map_entries(p.seg[s].idx + row_of(t), lane);
#pragma unroll
      for (int s = 0; s < kMaxSeg; s++) {
        run[s] = row_of(t);
        if (s >= p.nseg) continue;
        if (p.seg[s].agg) run[s] = -1;
        else if (p.seg[s].idx) run[s] = consecutive(ent[s], lane);
      }
      if ((t >= 2 && !umma::warp_wait(&runfree[t & 1], ((t >> 1) - 1) & 1)) || aborted(&s_abort)) {
        s_abort = 1;
        break;
      }
      if (lane == 0) {
        int* o = runs + (t & 1) * 4;
        o[0] = run[0];
        o[1] = run[1];
        o[2] = run[2];
        umma::mbar_arrive(&runfull[t & 1]);
      }
      __syncwarp();
    }
  } else if (warp >= 4 && warp < 8) {
    // ---- epilogue 1
    const int r = (warp & 3) * 32 + lane;  // row of the tile = TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool leader = warp == 4 && lane == 0;
    for (int t = 0; t < mine; t++) {
      const int slot = t & 1;
      const uint32_t d1 = tmem + slot * 128 + lane_off;
      const bool ok = umma::warp_wait(&d1full[slot], (t >> 1) & 1) && !aborted(&s_abort);
      if (save && leader) umma::tma_store_wait_read();  // the half tile before has been read
      if (!umma::bar_all(1, kRows, ok)) {  // the four warps go on, or stop, together
        s_abort = 1;
        break;
      }
      umma::fence_after_sync();
#pragma unroll 1
      for (int q = 0; q < 4; q++) {  // 32 columns into 16, over columns already read
        float v[32];
        uint32_t o[16];
        umma::tmem_ld32(d1 + q * 32, v);
        const float4* bp = reinterpret_cast<const float4*>(b1s + q * 32);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float4 x = bp[j];
          o[2 * j] = pack_bf16(fmaxf(v[4 * j] + x.x, 0.f), fmaxf(v[4 * j + 1] + x.y, 0.f));
          o[2 * j + 1] = pack_bf16(fmaxf(v[4 * j + 2] + x.z, 0.f), fmaxf(v[4 * j + 3] + x.w, 0.f));
        }
        umma::tmem_st16(d1 + q * 16, o);
        if (q == 3) {
          umma::tmem_st_wait();
          umma::fence_before_sync();
          umma::mbar_arrive(&a1full[slot]);
        }
        if (!save) continue;
        if (q == 2) {  // the first half has been read
          if (leader) umma::tma_store_wait_read();
          umma::bar_sync(1, kRows);
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
          *reinterpret_cast<uint4*>(a1s + umma::sw128_offset(r, (q & 1) * 32 + j * 8)) =
              make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        if (q & 1) {
          umma::fence_async_smem();
          umma::bar_sync(1, kRows);
          if (leader) umma::tma_store(&maps.a1, (q >> 1) * 64, row_of(t), a1s);
          __syncwarp();
        }
      }
    }
    if (save && leader) umma::tma_store_wait();
  } else if (warp >= 8 && warp < 12) {
    // ---- epilogue 2
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool leader = warp == 8 && lane == 0;
    for (int t = 0; t < mine; t++) {
      const int slot = t & 1;
      const size_t row = static_cast<size_t>(row_of(t)) + r;
      if (leader) {
        umma::tma_store_wait_read();  // the tile before has been read
        if (p.res) {
          umma::mbar_expect(resfull, p.n_out * 2 * kRows);
          for (int x = 0; x < p.n_out; x += 64) umma::tma_load(ios + (x >> 6) * kBlk, &maps.res, x, row_of(t), resfull);
        }
      }
      __syncwarp();
      bool ok = umma::warp_wait(&d2full[slot], (t >> 1) & 1);
      if (p.res) ok = umma::warp_wait(resfull, t & 1) && ok;
      if (!umma::bar_all(2, kRows, ok && !aborted(&s_abort))) {
        s_abort = 1;
        break;
      }
      umma::fence_after_sync();
#pragma unroll 1
      for (int col0 = 0; col0 < p.n_out; col0 += 32) {
        uint8_t* io = ios + (col0 >> 6) * kBlk;
        float v[32];
        umma::tmem_ld32(tmem + 256 + slot * 128 + lane_off + col0, v);
        if (p.res) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const uint4 w = *reinterpret_cast<const uint4*>(io + umma::sw128_offset(r, (col0 & 32) + j * 8));
            const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
              v[8 * j + 2 * u] += __uint_as_float(x[u] << 16);
              v[8 * j + 2 * u + 1] += __uint_as_float(x[u] & 0xffff0000u);
            }
          }
        }
        const float4* bp = reinterpret_cast<const float4*>(b2s + col0);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float4 x = bp[j];
          v[4 * j] += x.x;
          v[4 * j + 1] += x.y;
          v[4 * j + 2] += x.z;
          v[4 * j + 3] += x.w;
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
          *reinterpret_cast<uint4*>(io + umma::sw128_offset(r, (col0 & 32) + j * 8)) =
              make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                         pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
        if (p.out_f32) {
          float4* fp = reinterpret_cast<float4*>(p.out_f32 + row * p.n_out + col0);
#pragma unroll
          for (int j = 0; j < 8; j++) fp[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        if (!(col0 & 32)) continue;
        if (col0 + 32 == p.n_out) {
          umma::fence_before_sync();
          umma::mbar_arrive(&d2free[slot]);
        }
        umma::fence_async_smem();
        umma::bar_sync(2, kRows);
        if (leader) umma::tma_store(&maps.out, col0 - 32, row_of(t), io);
        __syncwarp();
      }
    }
    if (leader) umma::tma_store_wait();
  } else if (warp >= 12) {
    // ---- mapped rows and aggregation
    const int tid = threadIdx.x - 384;
    RingPos r;
    uint32_t granted = 0;  // (bit: parity of a stage's next grant)
    bool ok = true;
    for (int t = 0; t < mine && ok; t++) {  // (the gathering warps go on, or stop, together)
      const int row0 = row_of(t);
      ok = umma::bar_all(4, kGather, umma::warp_wait(&runfull[t & 1], (t >> 1) & 1) && !aborted(&s_abort));
#pragma unroll 1
      for (int s = 0; s < p.nseg && ok; s++) {
        const Seg& sg = p.seg[s];
        const int nb = sg.width >> 6;
        if (runs[(t & 1) * 4 + s] >= 0) {
          r.next(nst);
          if (nb > 1) r.next(nst);
          continue;
        }
        // (these loads are on their way while the stage is waited for)
        const bool agg = kAgg && sg.agg;
        uint32_t mask = 0;
        int src[kRowsEach];
        if constexpr (kAgg) {
          if (agg) mask = agg_mask<kGather>(sg, row0, tid);
        }
        if (!agg) {
#pragma unroll
          for (int i = 0; i < kRowsEach; i++) src[i] = sg.idx[row0 + (tid >> 3) + i * (kGather / 8)];
        }
        // the segment's one or two blocks in flight together
        RingPos w = r;
#pragma unroll 1
        for (int b = 0; b < nb; b++) {
          const bool given = umma::warp_wait(&grant[r.st], (granted >> r.st) & 1);
          granted ^= 1u << r.st;
          ok = umma::bar_all(4, kGather, given && !aborted(&s_abort));
          if (!ok) break;
          uint8_t* dst = ring + r.st * kBlk;
          if constexpr (kAgg) {
            if (agg) stage_agg_block<kGather>(sg, mask, row0, b * 64, dst, tid);
          }
          if (!agg) {
#pragma unroll
            for (int i = 0; i < kRowsEach; i++)
              cp_async16(dst + umma::sw128_offset((tid >> 3) + i * (kGather / 8), (tid & 7) * 8),
                         sg.src + static_cast<size_t>(src[i] >= 0 ? src[i] : 0) * sg.width + b * 64 + (tid & 7) * 8,
                         src[i] >= 0);
          }
          cp_async_commit();
          r.next(nst);
        }
        if (!ok) break;
#pragma unroll 1
        for (int b = 0; b < nb; b++) {
          if (b + 1 < nb) cp_async_wait<1>();
          else cp_async_wait<0>();
          umma::fence_async_smem();
          umma::bar_sync(3, kGather);
          if (tid == 0) umma::mbar_arrive(&full[w.st]);
          w.next(nst);
        }
      }
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&runfree[t & 1]);
    }
    cp_async_wait<0>();
    if (!ok) s_abort = 1;
  }
  umma::fence_before_sync();
  __syncthreads();
  if (s_abort && threadIdx.x == 0) set_err(p.err, 1);
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, 512);
  }
}

// ---- backward: data gradients -------------------------------------------------------

// Shared memory: W1 (128 x k_in), W2 (n_out x 128), dy as bf16 (128 x n_out), one or two
// hidden tiles (a1 in, dz1 out), two output pieces (128 rows x 32 fp32), barriers.
__host__ __device__ constexpr size_t data_fixed_bytes(int k_in, int n_out) {
  return 1024 + static_cast<size_t>(kHid) * k_in * 2 + static_cast<size_t>(n_out) * kHid * 2 +
         static_cast<size_t>(kRows) * n_out * 2 + 2 * kBlk + 256;
}
__host__ __device__ constexpr int data_buffers(int k_in, int n_out) {
  return data_fixed_bytes(k_in, n_out) + 4 * kBlk + 64 <= kSmemMax ? 2 : 1;
}
__host__ __device__ constexpr size_t bwd_data_smem_bytes(int k_in, int n_out) {
  return data_fixed_bytes(k_in, n_out) + static_cast<size_t>(data_buffers(k_in, n_out)) * 2 * kBlk;
}
static_assert(bwd_data_smem_bytes(384, 128) + 64 <= kSmemMax && data_buffers(256, 128) == 2, "shared memory");

struct DataMaps {  // boxes of 64 bf16 or 32 fp32 columns x 128 rows (w2: n_out rows)
  CUtensorMap w1, w2, a1, dz, out[kMaxSeg], add[kMaxSeg];
};

// Warp roles (640 threads), each a tile or more ahead of the next:
//   warp 0       the weights by TMA;
//   warp 1       one thread issues the MMAs: da1 = dy W2, then dA = dz1 W1 in chunks of
//                128 columns, a chunk as soon as the tile before has left its TMEM;
//   warps 4-7    a1 tile in by TMA, dz1 = da1 where a1 > 0 in its place, out by TMA;
//   warps 8-15   two warpgroups, each with pieces of 32 columns of a chunk: the addend in
//                by TMA, the sum in its place, out by TMA (a row to a thread, the direct
//                loads and stores took the L1 32 lines an instruction);
//   warps 16-19  dy rows in order, rounded to bf16.
// da1 takes 128 and dA k_in of the 512 TMEM columns, so neither is doubled.
// What bounds it: the fp32 rows (edge update: 512 B of dy, 256 of a1 and dz1 each, 1536 of
// gradients and 512 of addend from L2 a row).  Measured (us; before, one role a phase):
// edge update 174 (334) at 300,000 rows, 51 (95) at 75,000, 15 (29) at 9,000; node update
// 60 (112) at 100,000 rows, encoder 58 (125) at 300,000, decoder 27 (62) at 100,000.
constexpr int kDataThreads = 640;
__global__ void __launch_bounds__(kDataThreads, 1) k_mlp_bwd_data(const __grid_constant__ MlpBwdData p,
                                                                    const __grid_constant__ DataMaps maps) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = align1024(smem_raw);
  const int ndz = data_buffers(p.k_in, p.n_out);
  uint8_t* w1s = base;                             // [128 hid][k_in] blocks of 64 cols (16 KB)
  uint8_t* w2s = w1s + kHid * p.k_in * 2;          // [n_out][128]   blocks of 64 cols
  uint8_t* dys = w2s + p.n_out * kHid * 2;         // [128][n_out]
  uint8_t* dzs = dys + kRows * p.n_out * 2;        // [ndz][128][128]
  uint8_t* piece = dzs + ndz * 2 * kBlk;           // [2][128][32] fp32
  uint64_t* bars = reinterpret_cast<uint64_t*>(piece + 2 * kBlk);
  uint64_t* wfull = bars;          // weights loaded
  uint64_t* dyfull = bars + 1;     // dy tile written
  uint64_t* d1full = bars + 2;     // da1 complete, dy tile read (commit)
  uint64_t* d1free = bars + 3;     // da1 read
  uint64_t* a1full = bars + 4;     // [2] a1 tile loaded
  uint64_t* dzfull = bars + 6;     // dz1 tile written
  uint64_t* d2full = bars + 7;     // [3] chunk of dA complete (commit)
  uint64_t* d2free = bars + 10;    // [3] chunk of dA read
  uint64_t* addfull = bars + 13;   // [2] addend piece loaded
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool need_da = false;
  for (int s = 0; s < p.nseg; s++) need_da |= (p.dseg[s].out != nullptr);
  if (threadIdx.x == 0) {
    umma::mbar_init(wfull, 1);
    umma::mbar_init(dyfull, kRows);
    umma::mbar_init(d1full, 1);
    umma::mbar_init(d1free, kRows);
    umma::mbar_init(dzfull, kRows);
    for (int i = 0; i < 2; i++) {
      umma::mbar_init(&a1full[i], 1);
      umma::mbar_init(&addfull[i], 1);
    }
    for (int i = 0; i < 3; i++) {
      umma::mbar_init(&d2full[i], 1);
      umma::mbar_init(&d2free[i], 2 * kRows);
    }
    umma::mbar_fence_init();
    umma::fence_async_smem();
    s_abort = 0;
  }
  if (warp == 1) umma::tmem_alloc(tmem_slot, 512);
  umma::grid_wait();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t dda1 = tmem, dda = tmem + 128;
  const int ntiles = p.rows / kRows;
  const int mine = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int nch = (p.k_in + 127) >> 7;
  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const int r = (warp & 3) * 32 + lane;  // row of the tile = TMEM lane

  if (warp == 0) {
    // ---- weights
    if (lane == 0) {
      umma::mbar_expect(wfull, static_cast<uint32_t>((need_da ? kHid * p.k_in * 2 : 0) + p.n_out * kHid * 2));
      for (int x = 0; x < kHid; x += 64) umma::tma_load(w2s + (x >> 6) * (p.n_out * 128), &maps.w2, x, 0, wfull);
      if (need_da)
        for (int x = 0; x < p.k_in; x += 64) umma::tma_load(w1s + (x >> 6) * (kHid * 128), &maps.w1, x, 0, wfull);
    }
    umma::warp_wait(wfull, 0);  // landed before the block's shared memory is given up
  } else if (warp == 1) {
    // ---- MMA issuer
    if (umma::elect_one()) {
      const uint32_t w1a = umma::smem_addr(w1s), w2a = umma::smem_addr(w2s);
      const uint64_t dyd = umma::desc_kmajor(umma::smem_addr(dys)), w2d = umma::desc_mnmajor(w2a, p.n_out * 128);
      // da1 = dy W2 : A = dy [128 x n_out] K-major, B = W2 viewed [N=128 hid x K=n_out] MN-major
      const uint32_t idesc_a1 = umma::idesc_bf16(kRows, kHid, false, true);
      bool ok = umma::mbar_wait(wfull, 0);
      for (int t = 0; t < mine && ok; t++) {
        ok = umma::mbar_wait(dyfull, t & 1) && (t == 0 || umma::mbar_wait(d1free, (t - 1) & 1));
        if (!ok) break;
        umma::fence_after_sync();
        // K = n_out rows of W2; K-step 16 advances dy by 32 bytes (inside a 64-col block)
        // and the MN-major W2 view by 16 rows (2 KB); descriptors count 16 bytes.
#pragma unroll
        for (int k = 0; k < 128; k += 16)
          if (k < p.n_out)
            umma::mma_bf16(dda1, dyd + (k >> 6) * (kBlk / 16) + (k & 63) / 8, w2d + k * 8, idesc_a1, k > 0 ? 1u : 0u);
        umma::commit(d1full);
        if (!need_da) continue;
        // dA = dz1 W1 : A = dz1 [128 x 128] K-major, B = W1 viewed [N=k_in x K=128] MN-major
        ok = umma::mbar_wait(dzfull, t & 1);
        const uint64_t dzd = umma::desc_kmajor(umma::smem_addr(dzs + (t % ndz) * 2 * kBlk));
        for (int c = 0; c < nch && ok; c++) {
          if (t > 0) ok = umma::mbar_wait(&d2free[c], (t - 1) & 1);
          if (!ok) break;
          umma::fence_after_sync();
          const uint32_t idesc = umma::idesc_bf16(kRows, p.k_in - c * 128 >= 128 ? 128 : 64, false, true);
          // W1 rows k.. (K index = hid), columns 128 c.. (two blocks of 16 KB)
          const uint64_t w1d = umma::desc_mnmajor(w1a + c * 2 * (kHid * 128), kHid * 128);
#pragma unroll
          for (int k = 0; k < kHid; k += 16)
            umma::mma_bf16(dda + c * 128, dzd + (k >> 6) * (kBlk / 16) + (k & 63) / 8, w1d + k * 8, idesc, k > 0 ? 1u : 0u);
          umma::commit(&d2full[c]);
        }
      }
      // the last commits, before shared memory and TMEM are given up
      if (ok && mine > 0) {
        ok = umma::mbar_wait(d1full, (mine - 1) & 1);
        if (need_da) ok = umma::mbar_wait(&d2full[nch - 1], (mine - 1) & 1) && ok;
      }
      if (!ok) s_abort = 1;
    }
  } else if (warp >= 4 && warp < 8) {
    // ---- dz1 = da1 * (a1 > 0)
    const bool leader = warp == 4 && lane == 0;
    int issued = 0, t = 0;
    // a1 of the CTA's tile n, once dz1 of the tile before in its buffer has been read
    auto load_a1 = [&](int n) {
      uint8_t* dst = dzs + (n % ndz) * 2 * kBlk;
      if (need_da && n >= ndz && !umma::mbar_wait(&d2full[nch - 1], (n - ndz) & 1)) {
        s_abort = 1;
        return;
      }
      umma::tma_store_wait_read();
      umma::mbar_expect(&a1full[n % ndz], 2 * kBlk);
      umma::tma_load(dst, &maps.a1, 0, (blockIdx.x + n * gridDim.x) * kRows, &a1full[n % ndz]);
      umma::tma_load(dst + kBlk, &maps.a1, 64, (blockIdx.x + n * gridDim.x) * kRows, &a1full[n % ndz]);
      issued = n + 1;
    };
    if (leader && mine > 0) load_a1(0);
    for (; t < mine; t++) {
      uint8_t* dz = dzs + (t % ndz) * 2 * kBlk;
      if (ndz == 2 && leader && t + 1 < mine) load_a1(t + 1);
      const bool ok = umma::warp_wait(&a1full[t % ndz], (t / ndz) & 1) && umma::warp_wait(d1full, t & 1) && !aborted(&s_abort);
      if (!umma::bar_all(1, kRows, ok)) {  // the four warps go on, or stop, together
        s_abort = 1;
        break;
      }
      umma::fence_after_sync();
#pragma unroll
      for (int col0 = 0; col0 < kHid; col0 += 32) {
        float v[32];
        umma::tmem_ld32(dda1 + lane_off + col0, v);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int c = col0 + j * 8;
          uint4* q = reinterpret_cast<uint4*>(dz + (c >> 6) * kBlk + umma::sw128_offset(r, c & 63));
          const uint4 w = *q;
          const uint32_t x[4] = {w.x, w.y, w.z, w.w};
          uint32_t o[4];
#pragma unroll
          for (int u = 0; u < 4; u++)
            o[u] = pack_bf16(__uint_as_float(x[u] << 16) > 0.f ? v[8 * j + 2 * u] : 0.f,
                             __uint_as_float(x[u] & 0xffff0000u) > 0.f ? v[8 * j + 2 * u + 1] : 0.f);
          *q = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      umma::fence_async_smem();
      umma::fence_before_sync();
      umma::mbar_arrive(d1free);
      if (need_da) umma::mbar_arrive(dzfull);
      umma::bar_sync(1, kRows);
      if (leader) {
        if (p.dz1_save) {
          const int row0 = (blockIdx.x + t * gridDim.x) * kRows;
          umma::tma_store(&maps.dz, 0, row0, dz);
          umma::tma_store(&maps.dz, 64, row0, dz + kBlk);
        }
        if (ndz == 1 && t + 1 < mine) load_a1(t + 1);
      }
    }
    if (leader) {
      for (int n = t; n < issued; n++) umma::mbar_wait(&a1full[n % ndz], (n / ndz) & 1);  // (stopped early)
      umma::tma_store_wait();
    }
  } else if (warp >= 8 && warp < 16) {
    // ---- segment gradients (fp32), plus the residual-path addend
    const int wg = (warp >> 2) - 2;
    const bool leader = (warp & 3) == 0 && lane == 0;
    uint8_t* buf = piece + wg * kBlk;
    uint32_t nadd = 0;
    bool ok = true;
    for (int t = 0; t < mine && ok && need_da; t++) {
      const int row0 = (blockIdx.x + t * gridDim.x) * kRows;
      for (int c = 0; c < nch && ok; c++) {
        const int np = p.k_in - c * 128 >= 128 ? 2 : 1;  // the warpgroup's pieces of the chunk
        for (int q = 0; q < np; q++) {
          const int col = c * 128 + (wg * np + q) * 32;
          int s = 0, first = 0;
          while (first + p.seg_width[s] <= col) first += p.seg_width[s++];
          float* out = p.dseg[s].out;
          const bool add = out && p.dseg[s].add;
          if (leader && out) {
            umma::tma_store_wait_read();  // the piece before has been read
            if (add) {
              umma::mbar_expect(&addfull[wg], kBlk);
              umma::tma_load(buf, &maps.add[s], col - first, row0, &addfull[wg]);
            }
          }
          if (q == 0) ok = umma::warp_wait(&d2full[c], t & 1);
          if (add) ok = umma::warp_wait(&addfull[wg], nadd++ & 1) && ok;
          ok = umma::bar_all(2 + wg, kRows, ok && !aborted(&s_abort));
          if (!ok) break;
          if (!out) continue;
          umma::fence_after_sync();
          float v[32];
          umma::tmem_ld32(dda + lane_off + col, v);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            float4* o = reinterpret_cast<float4*>(buf + umma::sw128_offset(r, j * 8));
            float4 a = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            if (add) {
              const float4 b = *o;
              a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
            }
            *o = a;
          }
          umma::fence_async_smem();
          umma::bar_sync(2 + wg, kRows);
          if (leader) umma::tma_store(&maps.out[s], col - first, row0, buf);
        }
        umma::fence_before_sync();
        umma::mbar_arrive(&d2free[c]);
      }
    }
    if (!ok) s_abort = 1;
    if (leader) umma::tma_store_wait();
  } else if (warp >= 16) {
    // ---- dy, rounded to bf16: a float4 a thread, rows in order
    const int tid = threadIdx.x - 512;
    const int sh = p.n_out == 128 ? 5 : 4;  // log2 of the float4s of a row
    const int rounds = p.n_out == 128 ? 2 : 1;
    constexpr int kIn = 16;                 // loads in flight
    bool ok = true;
    for (int t = 0; t < mine && ok; t++) {
      const float4* src = reinterpret_cast<const float4*>(p.dy + static_cast<size_t>(blockIdx.x + t * gridDim.x) * kRows * p.n_out);
      for (int h = 0; h < rounds; h++) {
        float4 v[kIn];
#pragma unroll
        for (int i = 0; i < kIn; i++) v[i] = src[(h * kIn + i) * kRows + tid];
        if (h == 0 && t > 0) ok = umma::warp_wait(d1full, (t - 1) & 1);
        ok = __all_sync(0xffffffffu, ok && !aborted(&s_abort));
        if (!ok) break;
#pragma unroll
        for (int i = 0; i < kIn; i++) {
          const int q = (h * kIn + i) * kRows + tid;
          const int row = q >> sh, c = (q & ((1 << sh) - 1)) * 4;
          *reinterpret_cast<uint2*>(dys + (c >> 6) * kBlk + umma::sw128_offset(row, c & 56) + (c & 4) * 2) =
              make_uint2(pack_bf16(v[i].x, v[i].y), pack_bf16(v[i].z, v[i].w));
        }
      }
      if (!ok) break;
      umma::fence_async_smem();
      umma::mbar_arrive(dyfull);
    }
    if (!ok) s_abort = 1;
  }
  umma::fence_before_sync();
  __syncthreads();
  if (s_abort && threadIdx.x == 0) set_err(p.err, 2);
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, 512);
  }
}

// ---- backward: weight gradients -------------------------------------------------------

// A stage holds 64 rows: A (k_in columns), dz1, a1, dy as bf16, in blocks of 64 columns.
constexpr int kSlab = 64;
constexpr int kSlabBlk = kSlab * 128;  // bytes of a block
__host__ __device__ constexpr int weight_stage_bytes(int k_in, int n_out) {
  return ((k_in + n_out) / 64 + 4) * kSlabBlk;
}
__host__ __device__ constexpr int weight_stages(int k_in, int n_out) {
  const int n = static_cast<int>((kSmemMax - 1024 - 4096) / weight_stage_bytes(k_in, n_out));
  return n < 4 ? n : 4;
}
__host__ __device__ constexpr size_t bwd_weight_smem_bytes(int k_in, int n_out) {
  return 1024 + static_cast<size_t>(weight_stages(k_in, n_out)) * weight_stage_bytes(k_in, n_out) + 256;
}
static_assert(weight_stages(384, 128) == 2, "the widest input leaves two stages");

__host__ __device__ constexpr int part_stride(int k_in, int n_out) {
  return kHid * k_in + kHid + n_out * kHid + n_out;
}

struct WeightMaps {  // boxes of 64 columns x 64 rows
  CUtensorMap seg[kMaxSeg], a1, dz;
};

// Warp roles (384 threads) around a ring of 64-row stages:
//   warp 0      TMA: dz1, a1 and the segments whose rows follow one another;
//   warp 1      one thread issues the MMAs (K = rows), both gradients staying in TMEM;
//   warps 2-3   column sums of dz1 (db1), from the stage;
//   warps 4-7   mapped rows by cp.async, the aggregation's sums of three edge rows;
//   warps 8-11  dy rounded to bf16, with its column sums (db2, of the fp32 values).
// Every role takes part in every stage's use, so none can come two uses early.  At the end
// warps 4-11 write the CTA's partial sums (summed over CTAs, in order, by k_reduce_parts).
// What bounds it: the rows from HBM (edge update: 256 B each of e, dz1 and a1 and 512 of dy
// a row, 3.4k cycles a stage), and for few rows the partial sums (262 KB a CTA, 39 MB in
// all, through L2).  With the reduction, measured (us; before, one stage of 128 rows and
// db1, db2 summed from global memory): edge update 91 (282) at 300,000 rows, 39 (91) at
// 75,000, 19 (35) at 9,000; node update 70 (147) at 100,000 rows, encoder 68 (166) at
// 300,000, decoder 33 (66) at 100,000.
constexpr int kWeightThreads = 384;
__global__ void __launch_bounds__(kWeightThreads, 1) k_mlp_bwd_weight(const __grid_constant__ MlpBwdWeight p,
                                                                        const __grid_constant__ WeightMaps maps) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = align1024(smem_raw);
  const int nst = weight_stages(p.k_in, p.n_out);
  const int stage_bytes = weight_stage_bytes(p.k_in, p.n_out);
  const int dz_off = (p.k_in >> 6) * kSlabBlk, a1_off = dz_off + 2 * kSlabBlk, dy_off = a1_off + 2 * kSlabBlk;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + nst * stage_bytes);
  uint64_t* full = bars;        // [4] stage filled: TMA, 128 gathering and 128 converting threads
  uint64_t* empty = bars + 4;   // [4] stage read: MMAs (commit) and 64 summing threads
  uint64_t* done = bars + 8;    // all MMAs complete (commit)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < nst; i++) {
      umma::mbar_init(&full[i], 1 + 256);
      umma::mbar_init(&empty[i], 1 + 64);
    }
    umma::mbar_init(done, 1);
    umma::mbar_fence_init();
    umma::fence_async_smem();
    s_abort = 0;
  }
  if (warp == 1) umma::tmem_alloc(tmem_slot, 512);
  umma::grid_wait();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t dw1 = tmem, dw2 = tmem + p.k_in;  // dW1 [128 hid][k_in], dW2^T [128 hid][n_out]
  const int nslabs = p.rows / kSlab;
  const int mine = (nslabs - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1;  // (grid <= nslabs / 2)
  auto row_of = [&](int g) { return static_cast<int>(blockIdx.x + g * gridDim.x) * kSlab; };

  float sum[4] = {0.f, 0.f, 0.f, 0.f};  // warps 2-3: two columns of dz1; 8-11: four of dy
  bool ok = true;
  if (warp == 0) {
    // ---- TMA
    int2 ent[kMaxSeg];
#pragma unroll
    for (int s = 0; s < kMaxSeg; s++)
      if (s < p.nseg && p.seg[s].idx) ent[s] = slab_entries(p.seg[s].idx + row_of(0), lane);
    int g = 0;
    for (; g < mine; g++) {
      const int st = g % nst, row0 = row_of(g), next = row_of(g + 1 < mine ? g + 1 : g);
      int run[kMaxSeg];  // first row of a segment whose 64 rows are consecutive, else -1
      uint32_t bytes = 4 * kSlabBlk;
#pragma unroll
      for (int s = 0; s < kMaxSeg; s++) {
        run[s] = -1;
        if (s >= p.nseg || p.seg[s].agg) continue;
        run[s] = row0;
        if (p.seg[s].idx) {
          run[s] = consecutive(ent[s], lane);
          ent[s] = slab_entries(p.seg[s].idx + next, lane);
        }
        if (run[s] >= 0) bytes += (p.seg[s].width >> 6) * kSlabBlk;
      }
      if (g >= nst) ok = umma::warp_wait(&empty[st], (g / nst - 1) & 1);
      ok = __all_sync(0xffffffffu, ok && !aborted(&s_abort));
      if (!ok) break;
      if (lane == 0) {
        uint8_t* dst = ring + st * stage_bytes;
        umma::mbar_expect(&full[st], bytes);
#pragma unroll
        for (int s = 0; s < kMaxSeg; s++) {
          if (s >= p.nseg) break;
          for (int x = 0; x < p.seg[s].width; x += 64, dst += kSlabBlk)
            if (run[s] >= 0) umma::tma_load(dst, &maps.seg[s], x, run[s], &full[st]);
        }
        for (int x = 0; x < kHid; x += 64) {
          umma::tma_load(dst + (x >> 6) * kSlabBlk, &maps.dz, x, row0, &full[st]);
          umma::tma_load(dst + (2 + (x >> 6)) * kSlabBlk, &maps.a1, x, row0, &full[st]);
        }
      }
      __syncwarp();
    }
    // the copies still in flight land before the block's shared memory is given up
    for (int k = g > nst ? g - nst : 0; k < g; k++) umma::warp_wait(&full[k % nst], (k / nst) & 1);
  } else if (warp == 1) {
    // ---- MMA issuer
    if (umma::elect_one()) {
      // dW1 = dz1^T A : A-operand dz1^T [M=128 hid, K=rows] MN-major; B = A^T [N=k_in chunk, K=rows] MN-major
      // dW2^T = a1^T dy : A-operand a1^T [M=128, K=rows] MN-major; B = dy^T [N=n_out, K=rows] MN-major
      const uint32_t idesc_w2 = umma::idesc_bf16(kHid, p.n_out, true, true);
      for (int g = 0; g < mine; g++) {
        const int st = g % nst;
        if (!umma::mbar_wait(&full[st], (g / nst) & 1)) {
          ok = false;
          break;
        }
        umma::fence_after_sync();
        const uint32_t a = umma::smem_addr(ring + st * stage_bytes);
        const uint64_t dzd = umma::desc_mnmajor(a + dz_off, kSlabBlk), a1d = umma::desc_mnmajor(a + a1_off, kSlabBlk);
        const uint64_t dyd = umma::desc_mnmajor(a + dy_off, kSlabBlk), ind = umma::desc_mnmajor(a, kSlabBlk);
#pragma unroll
        for (int k = 0; k < kSlab; k += 16) {  // 16 rows = 2 KB; descriptors count 16 bytes
          const uint32_t acc = (g > 0 || k > 0) ? 1u : 0u;
#pragma unroll
          for (int n0 = 0; n0 < 384; n0 += 128)
            if (n0 < p.k_in)
              umma::mma_bf16(dw1 + n0, dzd + k * 8, ind + (n0 >> 6) * (kSlabBlk / 16) + k * 8,
                             umma::idesc_bf16(kHid, p.k_in - n0 >= 128 ? 128 : 64, true, true), acc);
          umma::mma_bf16(dw2, a1d + k * 8, dyd + k * 8, idesc_w2, acc);
        }
        umma::commit(&empty[st]);
      }
      umma::commit(done);
    }
  } else if (warp < 4) {
    // ---- db1: column sums of dz1, rows in order
    const int c = (threadIdx.x - 64) * 2;
    for (int g = 0; g < mine; g++) {
      const int st = g % nst;
      ok = umma::warp_wait(&full[st], (g / nst) & 1);
      if (!ok) break;
      const uint8_t* src = ring + st * stage_bytes + dz_off + (c >> 6) * kSlabBlk;
#pragma unroll 16
      for (int r = 0; r < kSlab; r++) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(src + umma::sw128_offset(r, c & 63));
        sum[0] += __uint_as_float(w << 16);
        sum[1] += __uint_as_float(w & 0xffff0000u);
      }
      umma::mbar_arrive(&empty[st]);
    }
  } else if (warp < 8) {
    // ---- mapped rows and aggregation
    const int tid = threadIdx.x - 128;
    int2 ent[kMaxSeg];
#pragma unroll
    for (int s = 0; s < kMaxSeg; s++)
      if (s < p.nseg && p.seg[s].idx) ent[s] = slab_entries(p.seg[s].idx + row_of(0), lane);
    for (int g = 0; g < mine; g++) {
      const int st = g % nst, row0 = row_of(g), next = row_of(g + 1 < mine ? g + 1 : g);
      if (g >= nst) ok = umma::warp_wait(&empty[st], (g / nst - 1) & 1);
      ok = __all_sync(0xffffffffu, ok && !aborted(&s_abort));
      if (!ok) break;
      uint8_t* dst = ring + st * stage_bytes;
#pragma unroll
      for (int s = 0; s < kMaxSeg; s++) {
        if (s >= p.nseg) break;
        const Seg& sg = p.seg[s];
        const int nb = sg.width >> 6;
        if (sg.agg) {
          const uint32_t mask = agg_mask<128>(sg, row0, tid);
#pragma unroll 1
          for (int b = 0; b < nb; b++) stage_agg_block<128>(sg, mask, row0, b * 64, dst + b * kSlabBlk, tid);
        } else if (sg.idx) {
          const bool mapped = consecutive(ent[s], lane) < 0;
          ent[s] = slab_entries(sg.idx + next, lane);
          if (mapped) {
            int src[4];
#pragma unroll
            for (int i = 0; i < 4; i++) src[i] = sg.idx[row0 + (tid >> 3) + i * 16];
            for (int b = 0; b < nb; b++)
#pragma unroll
              for (int i = 0; i < 4; i++)
                cp_async16(dst + b * kSlabBlk + umma::sw128_offset((tid >> 3) + i * 16, (tid & 7) * 8),
                           sg.src + static_cast<size_t>(src[i] >= 0 ? src[i] : 0) * sg.width + b * 64 + (tid & 7) * 8,
                           src[i] >= 0);
          }
        }
        dst += nb * kSlabBlk;
      }
      cp_async_commit();
      cp_async_wait<0>();
      umma::fence_async_smem();
      umma::mbar_arrive(&full[st]);
    }
  } else {
    // ---- dy: rounded to bf16, and its column sums
    const int tid = threadIdx.x - 256;
    const int sh = p.n_out == 128 ? 5 : 4;  // log2 of the float4s of a row
    const int n4 = p.n_out == 128 ? 16 : 8; // float4s of a slab and thread, all of one column group
    float4 v[16];
    auto load = [&](int g) {
      const float4* src = reinterpret_cast<const float4*>(p.dy + static_cast<size_t>(row_of(g)) * p.n_out);
#pragma unroll
      for (int i = 0; i < 16; i++)
        if (i < n4) v[i] = src[i * 128 + tid];
    };
    load(0);
    for (int g = 0; g < mine; g++) {
      const int st = g % nst;
      if (g >= nst) ok = umma::warp_wait(&empty[st], (g / nst - 1) & 1);
      ok = __all_sync(0xffffffffu, ok && !aborted(&s_abort));
      if (!ok) break;
      uint8_t* dst = ring + st * stage_bytes + dy_off;
      const int c = (tid & ((1 << sh) - 1)) * 4;
#pragma unroll
      for (int i = 0; i < 16; i++) {
        if (i >= n4) break;
        const int row = (i * 128 + tid) >> sh;
        *reinterpret_cast<uint2*>(dst + (c >> 6) * kSlabBlk + umma::sw128_offset(row, c & 56) + (c & 4) * 2) =
            make_uint2(pack_bf16(v[i].x, v[i].y), pack_bf16(v[i].z, v[i].w));
        sum[0] += v[i].x;
        sum[1] += v[i].y;
        sum[2] += v[i].z;
        sum[3] += v[i].w;
      }
      umma::fence_async_smem();
      umma::mbar_arrive(&full[st]);
      if (g + 1 < mine) load(g + 1);
    }
  }
  if (!ok) s_abort = 1;
  __syncthreads();
  if (!umma::warp_wait(done, 0)) s_abort = 1;
  __syncthreads();
  float* part = p.part + static_cast<size_t>(blockIdx.x) * part_stride(p.k_in, p.n_out);
  float* pw2 = part + kHid * p.k_in + kHid;  // dW2 [n_out][hid]
  float* s_db2 = reinterpret_cast<float*>(ring + 8 * 4096);  // [rows in flight][n_out]
  if (warp >= 8) *reinterpret_cast<float4*>(s_db2 + (threadIdx.x - 256) * 4) = make_float4(sum[0], sum[1], sum[2], sum[3]);
  __syncthreads();
  if (!s_abort) {
    umma::fence_after_sync();
    if (warp >= 2 && warp < 4) {
      *reinterpret_cast<float2*>(part + kHid * p.k_in + (threadIdx.x - 64) * 2) = make_float2(sum[0], sum[1]);
      for (int c = threadIdx.x - 64; c < p.n_out; c += 64) {
        float s = 0.f;
        for (int q = c; q < 512; q += p.n_out) s += s_db2[q];
        pw2[p.n_out * kHid + c] = s;
      }
    } else if (warp >= 4) {
      const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
      const int hid0 = (warp & 3) * 32, half = (warp >> 2) - 1;
      uint8_t* tr = ring + (warp - 4) * 4096;
      // dW1 [hid][k_in]: pieces of 32 x 32, turned in shared memory so that eight lanes
      // write 128 bytes of a row
      for (int col0 = half * 32; col0 < p.k_in; col0 += 64) {
        float v[32];
        umma::tmem_ld32(dw1 + lane_off + col0, v);
#pragma unroll
        for (int j = 0; j < 8; j++)
          *reinterpret_cast<float4*>(tr + umma::sw128_offset(lane, j * 8)) =
              make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int r = j * 4 + (lane >> 3);
          *reinterpret_cast<float4*>(part + static_cast<size_t>(hid0 + r) * p.k_in + col0 + (lane & 7) * 4) =
              *reinterpret_cast<const float4*>(tr + umma::sw128_offset(r, (lane & 7) * 8));
        }
        __syncwarp();
      }
      for (int col0 = half * 32; col0 < p.n_out; col0 += 64) {
        float v[32];
        umma::tmem_ld32(dw2 + lane_off + col0, v);
#pragma unroll
        for (int j = 0; j < 32; j++) pw2[static_cast<size_t>(col0 + j) * kHid + hid0 + lane] = v[j];
      }
    }
  } else if (threadIdx.x == 0) {
    set_err(p.err, 3);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, 512);
  }
}

// ---- small kernels -------------------------------------------------------------------

// grad[i] = sum over CTAs b (in order) of part[b][i]
__global__ void k_reduce_parts(const float* __restrict__ part, int nparts, int n, float* __restrict__ grad) {
  umma::grid_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
  int b = 0;
  for (; b + 16 <= nparts; b += 16) {  // loads ahead of the adds, which keep their order
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = part[static_cast<size_t>(b + j) * n + i];
#pragma unroll
    for (int j = 0; j < 16; j++) s += v[j];
  }
  for (; b < nparts; b++) s += part[static_cast<size_t>(b) * n + i];
  grad[i] = s;
}

// de_tot[k][c] = de[k][c] + (nbr[k][c] >= 0 ? dagg[c] : 0)     (aggregation backward)
// A thread takes four columns of a cell and its three edge rows, all loads in flight together.
// Per layer of 25,000 cells: 22 us with a grid-stride loop over single rows, 14 us now (90 MB).
__global__ void __launch_bounds__(256) k_agg_backward(const float* __restrict__ de, const float* __restrict__ dagg,
                                                      const int32_t* __restrict__ nbr, int Tp, float* __restrict__ out) {
  umma::grid_wait();
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), col = threadIdx.x & 31;  // (Tp is a multiple of 128)
  const size_t row4 = kHid / 4, q = c * row4 + col, kstep = Tp * row4;
  const float4 g = reinterpret_cast<const float4*>(dagg)[q];
  float4 a[3];
  bool edge[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    edge[k] = nbr[static_cast<size_t>(k) * Tp + c] >= 0;
    a[k] = de ? reinterpret_cast<const float4*>(de)[k * kstep + q] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (edge[k]) {
      a[k].x += g.x; a[k].y += g.y; a[k].z += g.z; a[k].w += g.w;
    }
    reinterpret_cast<float4*>(out)[k * kstep + q] = a[k];
  }
}

// dh[c] = dh_in[c] + sum_k ddst[k][c] + sum_k dsrc[rev[k][c]]   (gather backward)
// A thread takes four columns of a cell, its seven rows in flight together:
// 20 us with a grid-stride loop, 19 us now for 25,000 cells (103 MB).
__global__ void __launch_bounds__(256) k_node_backward(const float* __restrict__ dh_in, const float* __restrict__ ddst,
                                                       const float* __restrict__ dsrc, const int32_t* __restrict__ rev,
                                                       int Tp, float* __restrict__ out) {
  umma::grid_wait();
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), col = threadIdx.x & 31;
  const size_t row4 = kHid / 4, q = c * row4 + col, kstep = Tp * row4;
  int e[3];
  float4 d[3], r[3];
#pragma unroll
  for (int k = 0; k < 3; k++) e[k] = rev[static_cast<size_t>(k) * Tp + c];
  float4 a = reinterpret_cast<const float4*>(dh_in)[q];
#pragma unroll
  for (int k = 0; k < 3; k++) d[k] = reinterpret_cast<const float4*>(ddst)[k * kstep + q];
#pragma unroll
  for (int k = 0; k < 3; k++)
    r[k] = e[k] >= 0 ? reinterpret_cast<const float4*>(dsrc)[e[k] * row4 + col] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    a.x += d[k].x; a.y += d[k].y; a.z += d[k].z; a.w += d[k].w;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (e[k] < 0) continue;
    a.x += r[k].x; a.y += r[k].y; a.z += r[k].z; a.w += r[k].w;
  }
  reinterpret_cast<float4*>(out)[q] = a;
}

// Masked mean-squared error over the first `nout` columns of y (row stride ld):
// per-block partial loss and dy = 2 (y - t) w / norm.  A thread sums the loss of its rows, then
// the warps write dy of the block's 256 rows, 128 bytes in a row (a row to a thread took 15 us
// for 25,000 rows).
constexpr int kMseThreads = 256;
__global__ void __launch_bounds__(kMseThreads) k_mse(const float* __restrict__ y, int ld, const float* __restrict__ target,
                                                     const float* __restrict__ wmask, int Tp, int nout, float norm,
                                                     float* __restrict__ dy, float* __restrict__ loss_part) {
  __shared__ float red[kMseThreads];
  umma::grid_wait();
  float acc = 0.f;
  for (int r0 = blockIdx.x * kMseThreads; r0 < Tp; r0 += gridDim.x * kMseThreads) {
    const int i = r0 + threadIdx.x;
    if (i < Tp) {
      const float w = wmask[i];
      for (int j = 0; j < nout; j++) {
        const float d = y[static_cast<size_t>(i) * ld + j] - target[static_cast<size_t>(i) * nout + j];
        acc += w * d * d;
      }
    }
    for (int r = r0 + (threadIdx.x >> 5); r < min(Tp, r0 + kMseThreads); r += kMseThreads / 32) {
      const float w = wmask[r];
      for (int j = threadIdx.x & 31; j < ld; j += 32) {
        float g = 0.f;
        if (j < nout) {
          const float d = y[static_cast<size_t>(r) * ld + j] - target[static_cast<size_t>(r) * nout + j];
          g = 2.f * w * d / norm;
        }
        dy[static_cast<size_t>(r) * ld + j] = g;
      }
    }
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kMseThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) loss_part[blockIdx.x] = red[0] / norm;
}

// Adam on fp32 master weights; writes the bf16 copy the kernels read.
__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, bf16* __restrict__ wb, int n, float lr, float b1,
                       float b2, float eps, float bc1, float bc2, float wd, float clip_scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i] * clip_scale;
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  float wi = w[i];
  wi -= lr * ((mi / bc1) / (sqrtf(vi / bc2) + eps) + wd * wi);
  w[i] = wi;
  if (wb) wb[i] = __float2bfloat16(wi);
}

__global__ void k_sumsq(const float* __restrict__ g, int n, float* __restrict__ out_part) {
  __shared__ float red[256];
  float acc = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += g[i] * g[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) out_part[blockIdx.x] = red[0];
}

}  // namespace gnn
}  // namespace storm

// ---- C-ABI launchers (include/storm_gnn.h) ------------------------------------------

#include <atomic>
#include <string>

#include "../../include/storm_gnn.h"

namespace storm {
int set_error(int code, const std::string& msg);
void clear_error();
}  // namespace storm

namespace {

using namespace storm::gnn;

std::atomic<int64_t> g_launches{0};
constexpr int kMinBwdSmem = 120 * 1024;  // one CTA per SM: the backward kernels take all of TMEM

int cuda_check(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return storm::set_error(STORM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return STORM_OK;
}

int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

bool valid_width(int w) { return w == 64 || w == 128; }

int check_shape(int rows, int nseg, int k_in, int n_out, const int* widths) {
  if (rows <= 0 || rows % kRows) return storm::set_error(STORM_ERR_ARG, "rows must be a positive multiple of 128");
  if (nseg < 1 || nseg > kMaxSeg) return storm::set_error(STORM_ERR_ARG, "1 to 3 input segments");
  int k = 0;
  for (int s = 0; s < nseg; s++) {
    if (!valid_width(widths[s])) return storm::set_error(STORM_ERR_ARG, "segment width must be 64 or 128");
    k += widths[s];
  }
  if (k != k_in || k_in > 384) return storm::set_error(STORM_ERR_ARG, "k_in must equal the segment widths (<= 384)");
  if (n_out != 64 && n_out != 128) return storm::set_error(STORM_ERR_ARG, "n_out must be 64 or 128");
  return STORM_OK;
}

Seg to_seg(const StormGnnSeg& s) {
  Seg o;
  o.src = static_cast<const bf16*>(s.src);
  o.idx = s.agg ? nullptr : s.idx;  // an aggregated segment has no row map: the kernels ask for its entries early
  o.width = s.width;
  o.agg = s.agg;
  o.agg_stride = s.agg_stride;
  o.nbr = s.nbr;
  return o;
}

int check_segs(const StormGnnSeg* seg, int nseg, int rows) {
  for (int s = 0; s < nseg; s++) {
    if (!seg[s].src) return storm::set_error(STORM_ERR_ARG, "segment source is NULL");
    if (seg[s].agg && (!seg[s].nbr || seg[s].agg_stride < rows))
      return storm::set_error(STORM_ERR_ARG, "aggregation segment needs nbr and agg_stride >= rows");
  }
  return STORM_OK;
}

// Launches a kernel that waits for the ones before it by itself (umma::grid_wait), so that
// its blocks are placed, and set up their barriers and TMEM, while those end.  Only the forward
// kernel lets the next one's blocks in before its own have all ended: it is one block to an SM,
// and the next forward needs the room it leaves.  With the others letting them in too, blocks
// of the small kernels waited on SMs where the large ones ran (training step of 25,000 cells
// 1997 us; 1716 so, 1896 with the attribute on the forward kernel alone, 1925 without).
template <class... P, class... A>
int launch(const char* what, void (*kernel)(P...), int grid, int block, size_t smem, void* stream, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  g_launches++;
  return cuda_check(what);
}

int grid_for(int rows) {
  const int tiles = rows / kRows;
  return tiles < num_sms() ? tiles : num_sms();
}

// Row-major [rows][cols] (cols a multiple of 64) in boxes of 64 bf16 or 32 fp32 columns x
// box_rows, 128-byte swizzle.  cuTensorMapEncodeTiled comes from the runtime's driver entry point,
// so the library needs no link to libcuda.
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int tensor_map(CUtensorMap* m, const void* ptr, int rows, int cols, int box_rows, bool f32 = false) {
  static const EncodeFn encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<EncodeFn>(fn);
  }();
  if (!encode) return storm::set_error(STORM_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * (f32 ? 4 : 2)};
  const cuuint32_t box[2] = {f32 ? 32u : 64u, static_cast<cuuint32_t>(box_rows)}, es[2] = {1, 1};
  const CUresult r = encode(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return storm::set_error(STORM_ERR_ARG, "matrix rows must start on 16-byte boundaries (tensor map error " +
                                               std::to_string(static_cast<int>(r)) + ")");
  return STORM_OK;
}

}  // namespace

extern "C" {

int32_t storm_gnn_grad_size(int32_t k_in, int32_t n_out) { return part_stride(k_in, n_out); }

size_t storm_gnn_weight_scratch_bytes(int32_t k_in, int32_t n_out) {
  return static_cast<size_t>(num_sms()) * part_stride(k_in, n_out) * sizeof(float);
}

int storm_gnn_mlp_forward(const StormGnnMlpFwd* a, int32_t* dev_err, void* stream) {
  storm::clear_error();
  if (!a) return storm::set_error(STORM_ERR_ARG, "NULL arguments");
  int widths[kMaxSeg] = {0, 0, 0};
  for (int s = 0; s < a->nseg && s < kMaxSeg; s++) widths[s] = a->seg[s].width;
  int rc = check_shape(a->rows, a->nseg, a->k_in, a->n_out, widths);
  if (rc) return rc;
  if ((rc = check_segs(a->seg, a->nseg, a->rows))) return rc;
  if (!a->w1 || !a->b1 || !a->w2 || !a->b2 || !a->out) return storm::set_error(STORM_ERR_ARG, "NULL weight or output");
  MlpFwd p{};
  p.rows = a->rows; p.nseg = a->nseg; p.k_in = a->k_in; p.n_out = a->n_out;
  for (int s = 0; s < a->nseg; s++) p.seg[s] = to_seg(a->seg[s]);
  p.w1 = static_cast<const bf16*>(a->w1); p.b1 = a->b1;
  p.w2 = static_cast<const bf16*>(a->w2); p.b2 = a->b2;
  p.res = static_cast<const bf16*>(a->res); p.out = static_cast<bf16*>(a->out);
  p.out_f32 = a->out_f32; p.a1_save = static_cast<bf16*>(a->a1_save); p.err = dev_err;
  FwdMaps maps{};
  for (int i = 0; i < a->nseg; i++) {
    const Seg& g = p.seg[i];
    if (g.agg) continue;
    if ((rc = tensor_map(&maps.seg[i], g.src, g.idx ? kAnyRows : a->rows, g.width, kRows))) return rc;
  }
  if ((rc = tensor_map(&maps.w1, p.w1, kHid, a->k_in, kHid)) || (rc = tensor_map(&maps.w2, p.w2, a->n_out, kHid, a->n_out)) ||
      (rc = tensor_map(&maps.out, p.out, a->rows, a->n_out, kRows)))
    return rc;
  if (p.a1_save && (rc = tensor_map(&maps.a1, p.a1_save, a->rows, kHid, kRows))) return rc;
  if (p.res && (rc = tensor_map(&maps.res, p.res, a->rows, a->n_out, kRows))) return rc;
  const size_t smem = fwd_smem_bytes(a->k_in, a->n_out, p.a1_save != nullptr);
  bool agg = false;
  for (int i = 0; i < a->nseg; i++) agg |= p.seg[i].agg != 0;
  auto kernel = agg ? k_mlp_fwd<true> : k_mlp_fwd<false>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  return launch("k_mlp_fwd", kernel, grid_for(a->rows), fwd_threads(agg), smem, stream, p, maps);
}

int storm_gnn_mlp_backward_data(const StormGnnMlpBwdData* a, int32_t* dev_err, void* stream) {
  storm::clear_error();
  if (!a) return storm::set_error(STORM_ERR_ARG, "NULL arguments");
  int rc = check_shape(a->rows, a->nseg, a->k_in, a->n_out, a->seg_width);
  if (rc) return rc;
  if (!a->dy || !a->a1 || !a->w1 || !a->w2) return storm::set_error(STORM_ERR_ARG, "NULL input");
  MlpBwdData p{};
  p.rows = a->rows; p.nseg = a->nseg; p.k_in = a->k_in; p.n_out = a->n_out;
  for (int s = 0; s < a->nseg; s++) {
    p.seg_width[s] = a->seg_width[s];
    p.dseg[s].out = a->dseg[s];
    p.dseg[s].add = a->dseg_add[s];
  }
  p.dy = a->dy; p.a1 = static_cast<const bf16*>(a->a1);
  p.w1 = static_cast<const bf16*>(a->w1); p.w2 = static_cast<const bf16*>(a->w2);
  p.dz1_save = static_cast<bf16*>(a->dz1_save); p.err = dev_err;
  DataMaps maps{};
  if ((rc = tensor_map(&maps.w1, p.w1, kHid, a->k_in, kHid)) || (rc = tensor_map(&maps.w2, p.w2, a->n_out, kHid, a->n_out)) ||
      (rc = tensor_map(&maps.a1, p.a1, a->rows, kHid, kRows)))
    return rc;
  if (p.dz1_save && (rc = tensor_map(&maps.dz, p.dz1_save, a->rows, kHid, kRows))) return rc;
  for (int s = 0; s < a->nseg; s++) {
    if (!p.dseg[s].out) continue;
    if ((rc = tensor_map(&maps.out[s], p.dseg[s].out, a->rows, p.seg_width[s], kRows, true))) return rc;
    if (p.dseg[s].add && (rc = tensor_map(&maps.add[s], p.dseg[s].add, a->rows, p.seg_width[s], kRows, true))) return rc;
  }
  size_t smem = bwd_data_smem_bytes(a->k_in, a->n_out);
  if (smem < static_cast<size_t>(kMinBwdSmem)) smem = kMinBwdSmem;
  cudaFuncSetAttribute(k_mlp_bwd_data, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  return launch("k_mlp_bwd_data", k_mlp_bwd_data, grid_for(a->rows), kDataThreads, smem, stream, p, maps);
}

int storm_gnn_mlp_backward_weight(const StormGnnMlpBwdWeight* a, float* grad, void* scratch, size_t scratch_bytes,
                                  int32_t* dev_err, void* stream) {
  storm::clear_error();
  if (!a || !grad || !scratch) return storm::set_error(STORM_ERR_ARG, "NULL arguments");
  int widths[kMaxSeg] = {0, 0, 0};
  for (int s = 0; s < a->nseg && s < kMaxSeg; s++) widths[s] = a->seg[s].width;
  int rc = check_shape(a->rows, a->nseg, a->k_in, a->n_out, widths);
  if (rc) return rc;
  if ((rc = check_segs(a->seg, a->nseg, a->rows))) return rc;
  if (!a->dy || !a->a1 || !a->dz1) return storm::set_error(STORM_ERR_ARG, "NULL input");
  const int grid = grid_for(a->rows);
  const int n = part_stride(a->k_in, a->n_out);
  if (scratch_bytes < static_cast<size_t>(grid) * n * sizeof(float))
    return storm::set_error(STORM_ERR_ARG, "weight-gradient scratch too small");
  MlpBwdWeight p{};
  p.rows = a->rows; p.nseg = a->nseg; p.k_in = a->k_in; p.n_out = a->n_out;
  for (int s = 0; s < a->nseg; s++) p.seg[s] = to_seg(a->seg[s]);
  p.dy = a->dy; p.a1 = static_cast<const bf16*>(a->a1); p.dz1 = static_cast<const bf16*>(a->dz1);
  p.part = static_cast<float*>(scratch); p.err = dev_err;
  WeightMaps maps{};
  for (int i = 0; i < a->nseg; i++) {
    const Seg& g = p.seg[i];
    if (g.agg) continue;
    if ((rc = tensor_map(&maps.seg[i], g.src, g.idx ? kAnyRows : a->rows, g.width, kSlab))) return rc;
  }
  if ((rc = tensor_map(&maps.a1, p.a1, a->rows, kHid, kSlab)) || (rc = tensor_map(&maps.dz, p.dz1, a->rows, kHid, kSlab)))
    return rc;
  size_t smem = bwd_weight_smem_bytes(a->k_in, a->n_out);
  if (smem < static_cast<size_t>(kMinBwdSmem)) smem = kMinBwdSmem;
  cudaFuncSetAttribute(k_mlp_bwd_weight, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if ((rc = launch("k_mlp_bwd_weight", k_mlp_bwd_weight, grid, kWeightThreads, smem, stream, p, maps))) return rc;
  return launch("k_mlp_bwd_weight", k_reduce_parts, (n + 255) / 256, 256, 0, stream, p.part, grid, n, grad);
}

int storm_gnn_agg_backward(const float* de, const float* dagg, const int32_t* nbr, int32_t Tp, float* out,
                           void* stream) {
  storm::clear_error();
  if (!dagg || !nbr || !out || Tp <= 0 || Tp % kRows) return storm::set_error(STORM_ERR_ARG, "bad arguments");
  return launch("k_agg_backward", k_agg_backward, Tp / 8, 256, 0, stream, de, dagg, nbr, Tp, out);
}

int storm_gnn_node_backward(const float* dh, const float* ddst, const float* dsrc, const int32_t* rev, int32_t Tp,
                            float* out, void* stream) {
  storm::clear_error();
  if (!dh || !ddst || !dsrc || !rev || !out || Tp <= 0 || Tp % kRows)
    return storm::set_error(STORM_ERR_ARG, "bad arguments");
  return launch("k_node_backward", k_node_backward, Tp / 8, 256, 0, stream, dh, ddst, dsrc, rev, Tp, out);
}

int storm_gnn_mse(const float* y, int32_t ld, const float* target, const float* w, int32_t Tp, int32_t nout,
                  float norm, float* dy, float* loss_part, void* stream) {
  storm::clear_error();
  if (!y || !target || !w || !dy || !loss_part || Tp <= 0 || nout <= 0 || nout > ld || !(norm > 0.f))
    return storm::set_error(STORM_ERR_ARG, "bad arguments");
  return launch("k_mse", k_mse, 148, kMseThreads, 0, stream, y, ld, target, w, Tp, nout, norm, dy, loss_part);
}

int storm_gnn_adam(float* w, float* m, float* v, const float* g, void* w_bf16, int32_t n, float lr, float beta1,
                   float beta2, float eps, int32_t step, float weight_decay, float grad_scale, void* stream) {
  storm::clear_error();
  if (!w || !m || !v || !g || n <= 0 || step < 1) return storm::set_error(STORM_ERR_ARG, "bad arguments");
  const float bc1 = 1.f - powf(beta1, static_cast<float>(step));
  const float bc2 = 1.f - powf(beta2, static_cast<float>(step));
  k_adam<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, m, v, g, static_cast<bf16*>(w_bf16), n, lr, beta1, beta2, eps, bc1, bc2, weight_decay, grad_scale);
  g_launches++;
  return cuda_check("k_adam");
}

int storm_gnn_sumsq(const float* g, int32_t n, float* out_part, void* stream) {
  storm::clear_error();
  if (!g || !out_part || n <= 0) return storm::set_error(STORM_ERR_ARG, "bad arguments");
  k_sumsq<<<148, 256, 0, static_cast<cudaStream_t>(stream)>>>(g, n, out_part);
  g_launches++;
  return cuda_check("k_sumsq");
}

int64_t storm_gnn_kernel_launches(void) { return g_launches.load(); }

}  // extern "C"
