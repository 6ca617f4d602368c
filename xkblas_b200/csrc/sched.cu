// sched.cu -- the tile-task executor: one persistent launch runs a whole
// batch of level-3 calls as a DAG of tile tasks.
//
// Replaces the reference's XKaapi machinery for this path: per-tile tasks
// (blas/ztask_gemm.c:107-158, ztask_trsm.c), their data-flow dependencies
// (kaapi/kaapi_task.c:1277-1327) and the device threads that pop ready tasks
// and launch one cuBLAS call each (kaapi/kaapi_offload_device.c:463-683,
// 852-1210).  The host builds the task graph once; persistent CTAs (as many
// as fit, three per SM) take dependency-free tasks from a bulk list and the
// others from a device-side ready queue that completing tasks append their
// successors to.  A batch of small, uneven calls thus costs one launch
// instead of one launch (or thousands of tile tasks with host round trips)
// per call.
//
// Task bodies (four MMA warps and a copy warp, three CTAs per SM):
//   gemm     C[<=BM x <=BN] = alpha op(A) op(B) + beta C over the full K, with
//            the operand tiles, fragments and epilogue of the whole-matrix GEMM
//            (dmma_tile.cuh, gemm_dmma.cuh); the copy warp fills its 4-stage
//            ring by cp.async (16-byte copies, 8-byte ones for an operand not
//            16-byte aligned; zero fill at ragged edges), since a batch has no
//            tensor maps; BM x BN = 64 x 64 (real), 32 x 32 (complex).  Before
//            (eight warps that copied and multiplied, a CTA barrier per stage,
//            128 x 64 tiles, two CTAs per SM): 22 TFLOP/s on mixed DGEMM calls;
//   trsm     one 64-row block X_i of a left triangular solve against up to
//            64 right-hand sides, left-looking: X_i = alpha B_i - sum_k
//            op(A)[i,k] X_k over the blocks already solved (one gemm tile
//            with the whole k range), then the diagonal solve with op(A)[i,i]
//            in the same CTA.  The reference runs the same block algorithm
//            right-looking (blas/ztrsm.c:241-372: diagonal trsm tasks, then
//            gemm updates of the trailing blocks); here each right-hand-side
//            block is one chain of mt tasks, and the sums are formed in
//            registers once instead of read-modified-written per step.
// Ordering rules: a producer stores, then __syncthreads, then thread 0
// issues __threadfence and decrements its successors' dependency counts;
// the consumer's thread 0 takes the queued task, issues __threadfence (a
// gpu-scope acquire, which also leaves no stale L1 line), and after the CTA's
// barrier every warp reads what the producers wrote -- no async-proxy reads.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "gemm_dmma.cuh"
#include "trsm_leaf.cuh"
#include "xkb_dev.cuh"

namespace xkb {
namespace sched {

enum : int { kTaskGemm = 0, kTaskTrsm = 1 };
// kFlagNarrowA / B: that operand's base or leading dimension is not 16-byte
// aligned, so the gemm tile stages it with 8-byte copies
enum : int {
  kFlagSwap = 1, kFlagConj = 2, kFlagLower = 4, kFlagUnit = 8, kFlagNarrowA = 16,
  kFlagNarrowB = 32
};

// One task.  succ0 / nsucc: its successors in the batch's successor array
// (tasks whose dependency count it decrements when it completes).
//   gemm:  C = (ar,ai) op(A) op(B) + (br,bi) C, C is M x N, inner K: a whole
//          call, whose tiles are the bulk entries from tile0 on (tile index =
//          entry - tile0, column by column); a CTA cuts its tile out of it.
//   trsm:  C = X_i (M rows, N right-hand sides); A, B = the op(A) panel and
//          the solved X rows it multiplies (K = their inner length, 0 for
//          the first block); D = the diagonal block; (ar,ai) = alpha.
struct alignas(16) Task {
  int kind, dtype, opA, opB;
  int M, N, K, call;
  const void* A;
  const void* B;
  void* C;
  const void* D;
  long lda, ldb, ldc;
  double ar, ai, br, bi;
  int succ0, nsucc, flags, tile0;
};
static_assert(sizeof(Task) == 144, "task record");

// Device-side queues of one batch (ints in global memory):
//   bulk[nbulk]   the gemm calls' tiles (entry: the call's task), in call
//                 order; claimed with an atomic head;
//   urq[nurg]     the solve tasks: a ready queue.  The first block of every
//                 chain is queued at launch; a task is appended (atomic
//                 tail, then the slot is written) when its last dependency
//                 completes; slots not yet written hold -1.  A CTA takes a
//                 ticket (atomic head) only while the queue shows a task it
//                 could get, then waits for its slot: one atomic per claim,
//                 no retry storms, and no deadlock (slots fill in order and
//                 every queued task's producers were queued before it).
struct Ctl {
  int head_bulk, head_urg, tail_urg, pad;
};

template <class T>
using TileCfg = Cfg<T, St<T>::CPLX ? 32 : 64, St<T>::CPLX ? 32 : 64, 2, 2, 3, 4>;
constexpr int kMma = TileCfg<double>::THREADS;  // MMA threads
constexpr int kThreads = kMma + 32;             // and the copy warp
constexpr int kStages = 4;
constexpr int kLeafS = kLeafRows;  // trsm block (trsm_leaf.cuh)
static_assert(TileCfg<double2>::THREADS == kMma, "one CTA shape");

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)),
               "l"(gmem), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(smem)), "l"(gmem),
               "r"(src_bytes)
               : "memory");
}
// The barrier's pending count (32: one per lane) drops once this thread's
// copies so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }

// Claim the next task for this CTA (thread 0 only): from the ready queue of
// the solves or from the bulk list, in the order `urgent_first` asks.  Spins
// (bounded) while every remaining task still waits for a dependency.
// Returns the task id (entry: its bulk index, -1 for a solve), -1 when every
// task has been claimed, -2 on timeout or when another CTA recorded an error.
__device__ __forceinline__ int claim_task(Ctl* ctl, const int* bulk, int nbulk, const int* urq,
                                          int nurg, bool urgent_first, uint64_t wait_ns,
                                          int& entry) {
  entry = -1;
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    for (int pass = 0; pass < 2; ++pass) {
      if ((pass == 0) == urgent_first) {
        const int h = ld_volatile(&ctl->head_urg);
        if (h < nurg && ld_volatile(&ctl->tail_urg) > h) {
          const int tk = atomicAdd(&ctl->head_urg, 1);
          if (tk < nurg) {  // the slot fills once its task is queued
            uint64_t w0 = 0;
            for (uint32_t k = 0;; ++k) {
              const int t = ld_volatile(urq + tk);
              if (t >= 0) return t;
              __nanosleep(64);
              if ((k & 63u) == 0) {
                if (dev_error_set()) return -2;
                const uint64_t now = globaltimer();
                if (w0 == 0) w0 = now;
                else if (now - w0 > wait_ns) {
                  dev_error(kErrFullWait);
                  return -2;
                }
              }
            }
          }
        }
      } else if (ld_volatile(&ctl->head_bulk) < nbulk) {
        const int b = atomicAdd(&ctl->head_bulk, 1);
        if (b < nbulk) {
          entry = b;
          return bulk[b];
        }
      }
    }
    if (ld_volatile(&ctl->head_bulk) >= nbulk && ld_volatile(&ctl->head_urg) >= nurg) return -1;
    __nanosleep(256);
    if ((spin & 31u) == 0) {
      if (dev_error_set()) return -2;
      const uint64_t now = globaltimer();
      if (t0 == 0) t0 = now;
      else if (now - t0 > wait_ns) {
        dev_error(kErrFullWait);
        return -2;
      }
    }
  }
}

// ---- gemm tile ---------------------------------------------------------------
// One operand's ROWS lines of 128 bytes (OpTile's layout) for k [k0, k0 + BK):
// g = its element (row 0, k 0) in op(A) / op(B)^T; rows past `rows` and k past
// K are zero.  All lanes of the copy warp; consecutive lanes, consecutive
// bytes.  16-byte copies (L2 only), or, narrow, 8-byte ones (through L1, which
// the claim's fence left without lines that other CTAs wrote before it).
template <class T, bool KC, int ROWS>
__device__ __forceinline__ void copy_lines(uint8_t* dst, const char* g, long ld, int rows, int k0,
                                           int K, bool narrow) {
  constexpr int ES = (int)sizeof(T), BK = 128 / ES;
  const int lane = threadIdx.x & 31;
  const size_t ldb = (size_t)ld * ES;
  if (!narrow) {
    constexpr int EPC = 16 / ES;  // elements per chunk
    const int c = lane & 7, l0 = lane >> 3;
    if (rows >= ROWS && k0 + BK <= K) {
      const char* src = KC ? g + (size_t)k0 * ES + c * 16 + l0 * ldb
                           : g + c * 16 + (size_t)(k0 + l0) * ldb;
#pragma unroll
      for (int q = 0; q < ROWS / 4; ++q) {
        const int L = l0 + 4 * q;
        // KC: line = row; else panel L / BK, k = L % BK
        const char* x = KC ? src + (size_t)(4 * q) * ldb
                           : src + (4 * q / BK) * 128 + (size_t)(4 * q % BK) * ldb;
        cp_async16(dst + L * 128 + ((c ^ (L & 7)) << 4), x, 16);
      }
      return;
    }
#pragma unroll 4
    for (int q = 0; q < ROWS / 4; ++q) {
      const int L = l0 + 4 * q;
      int valid;
      const char* x;
      if (KC) {
        valid = L < rows ? max(0, min(EPC, K - k0 - c * EPC)) : 0;
        x = g + (size_t)k0 * ES + c * 16 + (size_t)L * ldb;
      } else {
        const int kk = k0 + L % BK, m = L / BK * BK + c * EPC;
        valid = kk < K ? max(0, min(EPC, rows - m)) : 0;
        x = g + (size_t)(L / BK) * 128 + c * 16 + (size_t)kk * ldb;
      }
      cp_async16(dst + L * 128 + ((c ^ (L & 7)) << 4), valid ? x : g, valid * ES);
    }
    return;
  }
  // 8-byte words: 16 per line
  const int w = lane & 15, l0 = lane >> 4;
  auto at = [&](int L, const char*& x) {
    if (KC) {
      x = g + (size_t)k0 * ES + w * 8 + (size_t)L * ldb;
      return L < rows && k0 + w * 8 / ES < K;
    }
    const int kk = k0 + L % BK, m = L / BK * BK + w * 8 / ES;
    x = g + (size_t)(L / BK) * 128 + w * 8 + (size_t)kk * ldb;
    return kk < K && m < rows;
  };
  auto to = [&](int L) { return dst + L * 128 + (((w >> 1) ^ (L & 7)) << 4) + (w & 1) * 8; };
#pragma unroll 8
  for (int q = 0; q < ROWS / 2; ++q) {
    const int L = l0 + 2 * q;
    const char* x;
    const bool v = at(L, x);
    cp_async8(to(L), v ? x : g, v ? 8 : 0);
  }
}

// The copy warp's part of a tile: stages [pos, pos + KT) of the ring.  False
// if a bounded wait gave up.
template <class T, bool A_KC, bool B_KC>
__device__ __noinline__ bool copy_tile(const Task& t, uint8_t* ring, uint64_t* full,
                                       uint64_t* empty, int pos, bool narrowA, bool narrowB) {
  using C_ = TileCfg<T>;
  const int KT = (t.K + C_::BK - 1) / C_::BK;
  for (int j = pos; j < pos + KT; ++j) {
    const int s = j % kStages;
    if (j >= kStages) {
      const bool free_ = mbar_wait(&empty[s], (j / kStages - 1) & 1, kErrEmptyWait);
      if (!__all_sync(0xffffffffu, free_)) return false;
    }
    uint8_t* sa = ring + s * C_::STAGE_BYTES;
    const int k0 = (j - pos) * C_::BK;
    copy_lines<T, A_KC, C_::BM>(sa, static_cast<const char*>(t.A), t.lda, t.M, k0, t.K, narrowA);
    copy_lines<T, B_KC, C_::BN>(sa + C_::A_BYTES, static_cast<const char*>(t.B), t.ldb, t.N, k0,
                                t.K, narrowB);
    cp_async_arrive(&full[s]);
  }
  return true;
}

// The MMA warps' part: accumulate the stages, then alpha / beta and the store.
// Not inlined: each instantiation keeps its own register allocation.
template <class T, bool A_KC, bool B_KC>
__device__ __noinline__ bool mma_tile(const Task& t, uint8_t* ring, uint64_t* full,
                                      uint64_t* empty, int pos) {
  using C_ = TileCfg<T>;
  const int KT = (t.K + C_::BK - 1) / C_::BK;
  const int warp = threadIdx.x >> 5;
  double acc[C_::MF][C_::NF][C_::NACC];
#pragma unroll
  for (int i = 0; i < C_::MF; ++i)
#pragma unroll
    for (int j = 0; j < C_::NF; ++j)
#pragma unroll
      for (int v = 0; v < C_::NACC; ++v) acc[i][j][v] = 0.0;
  const unsigned fA = t.opA == XKB_OP_C ? 0x80000000u : 0u,
                 fB = t.opB == XKB_OP_C ? 0x80000000u : 0u;
  if (!dmma_mainloop<C_, A_KC, B_KC>(ring, full, empty, pos, KT, acc, (warp / C_::WN) * C_::WTM,
                                     (warp % C_::WN) * C_::WTN, fA, fB))
    return false;
  GemmParams p;
  p.M = t.M;
  p.N = t.N;
  p.C = t.C;
  p.ldc = t.ldc;
  p.ar = t.ar;
  p.ai = t.ai;
  p.br = t.br;
  p.bi = t.bi;
  p.uplo = XKB_FULL;
  p.herm_diag = 0;
  p.diag = 0;
  p.vec = reinterpret_cast<uintptr_t>(t.C) % 16 == 0 && ((size_t)t.ldc * sizeof(T)) % 16 == 0;
  dmma_epilogue<C_, A_KC, B_KC>(p, 0, 0, &acc[0][0][0]);
  return true;
}

// One tile by the whole CTA.  Returns the ring positions used.
template <class T>
__device__ __forceinline__ int run_tile(const Task& t, uint8_t* ring, uint64_t* full,
                                        uint64_t* empty, int pos, int* fail) {
  const bool akc = t.opA != XKB_OP_N, bkc = t.opB == XKB_OP_N;
  bool ok;
  if (threadIdx.x >= kMma) {
    const bool ma = t.flags & kFlagNarrowA, mb = t.flags & kFlagNarrowB;
    if (akc && bkc) ok = copy_tile<T, true, true>(t, ring, full, empty, pos, ma, mb);
    else if (akc) ok = copy_tile<T, true, false>(t, ring, full, empty, pos, ma, mb);
    else if (bkc) ok = copy_tile<T, false, true>(t, ring, full, empty, pos, ma, mb);
    else ok = copy_tile<T, false, false>(t, ring, full, empty, pos, ma, mb);
  } else {
    if (akc && bkc) ok = mma_tile<T, true, true>(t, ring, full, empty, pos);
    else if (akc) ok = mma_tile<T, true, false>(t, ring, full, empty, pos);
    else if (bkc) ok = mma_tile<T, false, true>(t, ring, full, empty, pos);
    else ok = mma_tile<T, false, false>(t, ring, full, empty, pos);
  }
  if (!ok) *reinterpret_cast<volatile int*>(fail) = 1;
  return (t.K + TileCfg<T>::BK - 1) / TileCfg<T>::BK;
}

// Rows [r0, ..) x columns [c0, ..) of a product, at most BM x BN of them.
template <class T>
__device__ __forceinline__ void cut_tile(Task& t, int r0, int c0) {
  using C_ = TileCfg<T>;
  constexpr size_t ES = sizeof(T);
  t.A = static_cast<const char*>(t.A) + (size_t)r0 * (t.opA == XKB_OP_N ? 1 : t.lda) * ES;
  t.B = static_cast<const char*>(t.B) + (size_t)c0 * (t.opB == XKB_OP_N ? t.ldb : 1) * ES;
  t.C = static_cast<char*>(t.C) + ((size_t)r0 + (size_t)c0 * t.ldc) * ES;
  t.M = min(C_::BM, t.M - r0);
  t.N = min(C_::BN, t.N - c0);
}

// ---- trsm diagonal block ------------------------------------------------------
// One 64-row diagonal block against up to 64 right-hand sides
// (trsm_leaf.cuh).  Not inlined: its register allocation stays apart from the
// gemm tile's.
template <class T>
__device__ __noinline__ void trsm_tile(const Task& t, uint8_t* smem, double ar, double ai) {
  using S = typename St<T>::S;
  double* sm = reinterpret_cast<double*>(smem);
  const bool swap = t.flags & kFlagSwap, conj = t.flags & kFlagConj;
  const bool lower = t.flags & kFlagLower, unit = t.flags & kFlagUnit;
  const S* D = static_cast<const S*>(t.D);
  S* X = static_cast<S*>(t.C);
  if (lower) leaf_solve<T, true>(D, t.lda, t.M, swap, conj, unit, X, t.ldc, t.N, ar, ai, sm);
  else leaf_solve<T, false>(D, t.lda, t.M, swap, conj, unit, X, t.ldc, t.N, ar, ai, sm);
}

// dynamic shared memory: the ring, or the solve's staging in its place; a
// batch with a complex solve needs more and runs two CTAs per SM
constexpr size_t kRingBytes = kStages * (size_t)TileCfg<double>::STAGE_BYTES;
static_assert(TileCfg<double2>::STAGE_BYTES <= TileCfg<double>::STAGE_BYTES, "one ring");
constexpr size_t sched_smem(bool ztrsm) {
  const size_t s = ztrsm ? LeafShape<double2>::SMEM : LeafShape<double>::SMEM;
  return (s > kRingBytes ? s : kRingBytes) + 128;
}

__global__ void __launch_bounds__(kThreads, 3)
    k_sched(const Task* __restrict__ tasks, int* ndep, const int* __restrict__ succ,
            const int* __restrict__ bulk, int nbulk, int* urq, int nurg, Ctl* ctl,
            int urgent_first, int* call_left, unsigned long long* call_end,
            unsigned long long* t_start, unsigned long long wait_ns) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  __shared__ int s_idx, s_fail;
  __shared__ Task s_task;  // the claimed task (a gemm call: its tile), read by every thread
  __shared__ Task s_sub;   // a gemm step of a solve task
  __shared__ uint64_t s_full[kStages], s_empty[kStages];
  if (threadIdx.x == 0) {
    for (int q = 0; q < kStages; ++q) {
      mbar_init(&s_full[q], 32);
      mbar_init(&s_empty[q], kMma / 32);
    }
    fence_barrier_init();
    s_fail = 0;
    atomicMin(t_start, (unsigned long long)globaltimer());
  }
  int pos = 0;  // ring position, the same in every thread
  for (;;) {
    if (threadIdx.x == 0) {
      int entry;
      const int i =
          claim_task(ctl, bulk, nbulk, urq, nurg, urgent_first != 0, wait_ns, entry);
      if (i >= 0) {
        __threadfence();  // acquire: the producers' outputs before the reads
        Task t = tasks[i];
        if (t.kind == kTaskGemm) {
          const int b = t.dtype == XKB_Z ? TileCfg<double2>::BM : TileCfg<double>::BM;
          const int tm = (t.M + b - 1) / b, tile = entry - t.tile0;
          if (t.dtype == XKB_Z) cut_tile<double2>(t, tile % tm * b, tile / tm * b);
          else cut_tile<double>(t, tile % tm * b, tile / tm * b);
        }
        s_task = t;
      }
      s_idx = i;
    }
    __syncthreads();
    if (s_idx < 0 || *reinterpret_cast<volatile int*>(&s_fail)) break;
    // only thread 0 rewrites s_task, after every thread is past the barrier
    // that ends this task
    const Task& t = s_task;
    if (t.kind == kTaskGemm) {  // a gemm call's tile: operands read-only here
      if (t.dtype == XKB_Z) pos += run_tile<double2>(t, smem, s_full, s_empty, pos, &s_fail);
      else pos += run_tile<double>(t, smem, s_full, s_empty, pos, &s_fail);
    } else {
      // X_i = alpha B_i - op(A)[i, solved] X_solved in gemm tiles, then the
      // diagonal solve of X_i (same CTA: the tiles' stores are ordered before
      // its loads by the barrier, both go through L2)
      const bool cplx = t.dtype == XKB_Z;
      double sar = t.ar, sai = t.ai;
      if (t.K > 0) {
        const int b = cplx ? TileCfg<double2>::BM : TileCfg<double>::BM;
        for (int c0 = 0; c0 < t.N; c0 += b)
          for (int r0 = 0; r0 < t.M; r0 += b) {
            if (threadIdx.x == 0) {
              s_sub = t;
              if (cplx) cut_tile<double2>(s_sub, r0, c0);
              else cut_tile<double>(s_sub, r0, c0);
              s_sub.ar = -1.0;
              s_sub.ai = 0.0;
              s_sub.br = t.ar;
              s_sub.bi = t.ai;
            }
            __syncthreads();
            if (cplx) pos += run_tile<double2>(s_sub, smem, s_full, s_empty, pos, &s_fail);
            else pos += run_tile<double>(s_sub, smem, s_full, s_empty, pos, &s_fail);
            __syncthreads();  // s_sub is rewritten by the next part
          }
        sar = 1.0;
        sai = 0.0;
      }
      if (threadIdx.x < kMma) {
        if (!cplx) trsm_tile<double>(t, smem, sar, sai);
        else trsm_tile<double2>(t, smem, sar, sai);
      }
    }
    __syncthreads();  // every output of the task is stored
    if (*reinterpret_cast<volatile int*>(&s_fail)) break;  // a bounded wait gave up
    if (threadIdx.x == 0) {
      __threadfence();  // release the outputs before any successor is queued
      for (int k = 0; k < t.nsucc; ++k) {
        const int sidx = succ[t.succ0 + k];
        if (atomicSub(ndep + sidx, 1) == 1) {
          const int q = atomicAdd(&ctl->tail_urg, 1);
          atomicExch(urq + q, sidx);
        }
      }
      if (atomicSub(call_left + t.call, 1) == 1) call_end[t.call] = globaltimer();
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");  // copies in flight after an error
}

// ---------------------------------------------------------------------------
// host: task graph construction
struct Built {
  std::vector<Task> tasks;                 // indexed by task id
  std::vector<int> ndep;                   // initial dependency count
  std::vector<std::pair<int, int>> edges;  // (producer, consumer)
  std::vector<int> bulk;                   // dependency-free gemm tiles
  std::vector<int> urg_ready;              // solve tasks ready at launch
  int nurg = 0;                            // solve tasks in total
  std::vector<int> call_tasks;
  int add(const Task& t, int ndep0) {
    tasks.push_back(t);
    ndep.push_back(ndep0);
    return (int)tasks.size() - 1;
  }
};

static int esz(int dt) { return dt == XKB_Z ? 16 : 8; }

static bool aligned_ok(const void* p, long ld, int es) {
  return (reinterpret_cast<uintptr_t>(p) % 16 == 0) && ((ld * es) % 16 == 0);
}

static bool ptr8(const void* p) { return reinterpret_cast<uintptr_t>(p) % 8 == 0; }

static Task gemm_task(int dtype, int opA, int opB, int M, int N, int K, int call, const void* A,
                      long lda, const void* B, long ldb, void* C, long ldc, double ar, double ai,
                      double br, double bi, int flags) {
  Task t;
  std::memset(&t, 0, sizeof(t));
  t.kind = kTaskGemm;
  t.dtype = dtype;
  t.opA = opA;
  t.opB = opB;
  t.M = M;
  t.N = N;
  t.K = K;
  t.call = call;
  t.A = A;
  t.lda = lda;
  t.B = B;
  t.ldb = ldb;
  t.C = C;
  t.ldc = ldc;
  t.ar = ar;
  t.ai = ai;
  t.br = br;
  t.bi = bi;
  t.flags = flags;
  return t;
}

// C tiles of a gemm call.
static size_t gemm_tiles(const xkb_batch_op& o) {
  const size_t b = o.dtype == XKB_Z ? TileCfg<double2>::BM : TileCfg<double>::BM;
  return ((size_t)o.M + b - 1) / b * (((size_t)o.N + b - 1) / b);
}

// A gemm call: one task record, and a bulk entry per C tile (the reference's
// tile loop, blas/zgemm.c:279-367, with the whole K range in one tile).
static int add_gemm(Built& b, const xkb_batch_op& o, int call) {
  const int es = esz(o.dtype);
  if (!ptr8(o.A) || !ptr8(o.B) || !ptr8(o.C)) return XKB_EINVAL;
  const int flags = (aligned_ok(o.A, o.lda, es) ? 0 : kFlagNarrowA) |
                    (aligned_ok(o.B, o.ldb, es) ? 0 : kFlagNarrowB);
  const size_t n = gemm_tiles(o);
  Task t = gemm_task(o.dtype, o.opA, o.opB, o.M, o.N, o.K, call, o.A, o.lda, o.B, o.ldb, o.C,
                     o.ldc, o.alpha[0], o.alpha[1], o.beta[0], o.beta[1], flags);
  t.tile0 = (int)b.bulk.size();
  b.bulk.insert(b.bulk.end(), n, b.add(t, 0));
  return (int)n;
}

// Left triangular solve: the reference's block algorithm (blas/ztrsm.c:
// 241-372; alpha applied once, its lalpha), left-looking.  Blocks are taken
// in solve order s = 0 .. mt-1 (bk = order(s): forward for an effectively
// lower op(A), backward otherwise); task (s, j) forms
//   X_bk,j = alpha B_bk,j - op(A)[bk, done] X_done,j,   done = order(0..s-1)
// and solves with op(A)[bk,bk].  The blocks already solved are contiguous
// (rows [0, bk*64) forward, [(bk+1)*64, M) backward), so the sum is one gemm
// with K = 64 s (64 (mt-1-s) backward, the last block possibly shorter).
// Task (s, j) depends on task (s-1, j) only: one chain per j.
static int add_trsm(Built& b, const xkb_batch_op& o, int call) {
  const int es = esz(o.dtype);
  if (o.side != 0) return XKB_EINVAL;  // right side: not a batch task
  if (!ptr8(o.A) || !ptr8(o.C)) return XKB_EINVAL;
  const int narrow = (aligned_ok(o.A, o.lda, es) ? 0 : kFlagNarrowA) |
                     (aligned_ok(o.C, o.ldc, es) ? 0 : kFlagNarrowB);
  const bool cplx = o.dtype == XKB_Z;
  const int trans = (!cplx && o.trans == XKB_OP_C) ? XKB_OP_T : o.trans;
  const bool fwd = (o.uplo == XKB_LOWER) ^ (trans != XKB_OP_N);
  const int mt = (o.M + kLeafS - 1) / kLeafS, nt = (o.N + kLeafS - 1) / kLeafS;
  const char* A = static_cast<const char*>(o.A);
  char* X = static_cast<char*>(o.C);
  const int dflags = (trans != XKB_OP_N ? kFlagSwap : 0) | (trans == XKB_OP_C ? kFlagConj : 0) |
                     (fwd ? kFlagLower : 0) | (o.diag ? kFlagUnit : 0);
  // element (r, c) of op(A) lives at A[r + c lda] (trans N) or A[c + r lda]
  auto opA_at = [&](size_t r, size_t c) {
    return trans == XKB_OP_N ? A + (r + c * o.lda) * es : A + (c + r * o.lda) * es;
  };
  int n = 0;
  for (int j = 0; j < nt; ++j) {
    const size_t c0 = (size_t)j * kLeafS;
    int prev = -1;
    for (int s = 0; s < mt; ++s) {
      const int bk = fwd ? s : mt - 1 - s;
      const size_t r0 = (size_t)bk * kLeafS;
      const int rows = std::min(kLeafS, o.M - bk * kLeafS);
      const size_t k0 = fwd ? 0 : r0 + rows;             // first solved row
      const int K = fwd ? (int)r0 : o.M - (int)(r0 + rows);  // solved rows
      Task t;
      std::memset(&t, 0, sizeof(t));
      t.kind = kTaskTrsm;
      t.dtype = o.dtype;
      t.opA = trans;
      t.opB = XKB_OP_N;
      t.M = rows;
      t.N = std::min(kLeafS, o.N - j * kLeafS);
      t.K = K;
      t.call = call;
      t.A = K > 0 ? opA_at(r0, k0) : A;
      t.lda = o.lda;
      t.B = X + (k0 + c0 * o.ldc) * es;
      t.ldb = o.ldc;
      t.C = X + (r0 + c0 * o.ldc) * es;
      t.ldc = o.ldc;
      t.D = A + (r0 + r0 * o.lda) * es;
      t.ar = o.alpha[0];
      t.ai = cplx ? o.alpha[1] : 0.0;
      t.flags = dflags | narrow;
      const int id = b.add(t, prev >= 0 ? 1 : 0);
      ++b.nurg;
      ++n;
      if (prev >= 0) b.edges.emplace_back(prev, id);
      else b.urg_ready.push_back(id);
      prev = id;
    }
  }
  return n;
}

// Device image of one batch: tasks | ndep | succ | bulk | urq | call_left |
// ctl.  tasks, succ and bulk are read-only during a launch; ndep, urq,
// call_left and ctl are consumed by it.
struct Layout {
  int ntasks = 0, nops = 0;
  bool ztrsm = false;  // holds a complex solve (larger shared memory)
  size_t nbulk = 0, nurg = 0, nsucc = 0;
  size_t o_ndep = 0, o_succ = 0, o_bulk = 0, o_urq = 0, o_left = 0, o_ctl = 0, bytes = 0;
  void set(int nt, size_t ns, size_t nb, size_t nu, int no) {
    ntasks = nt;
    nsucc = ns;
    nbulk = nb;
    nurg = nu;
    nops = no;
    o_ndep = (size_t)nt * sizeof(Task);
    o_succ = o_ndep + (size_t)nt * 4;
    o_bulk = o_succ + ns * 4;
    o_urq = o_bulk + nb * 4;
    o_left = o_urq + nu * 4;
    o_ctl = (o_left + (size_t)no * 4 + 15) & ~size_t(15);
    bytes = o_ctl + sizeof(Ctl);
  }
};

// A batch seen before, kept as a CUDA graph: reset the consumed state from
// the pristine image (two device-to-device copies), clear the timestamps,
// run k_sched.  Replaying skips the host-side task construction and the
// upload of the task list.
struct GraphEntry {
  uint64_t key = 0;
  int schedule = 0;
  std::vector<xkb_batch_op> ops;  // the op list, compared on lookup
  Layout L;
  uint8_t* d_img = nullptr;       // pristine image
  uint8_t* d_run = nullptr;       // image the launch consumes
  unsigned long long* d_times = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<int> call_tasks;
  uint64_t last_use = 0;
  cudaEvent_t done = nullptr;     // its last launch, on whatever stream
  size_t bytes() const { return 2 * L.bytes + ((size_t)L.nops + 1) * 8; }
};

struct Batch {
  uint8_t* h_stage = nullptr;  // pinned: the image of the batch being launched
  size_t h_cap = 0;
  uint8_t* d_buf = nullptr;    // device image of uncached batches
  size_t d_cap = 0;
  unsigned long long* d_times = nullptr;  // call_end[ncalls], t_start
  size_t d_cap_times = 0;
  // the staging and device images are shared by the calls of all streams: the
  // last upload out of h_stage, and the last launch that reads d_buf / d_times
  cudaEvent_t staged = nullptr, done = nullptr;
  // the last launch (read by xkb_cuda_batch_latency)
  int ncalls = 0;
  std::vector<int> call_tasks;
  unsigned long long* cur_times = nullptr;
  // graph cache (XKBLAS_BATCH_GRAPHS=0 disables)
  std::vector<GraphEntry*> graphs;
  std::vector<uint64_t> seen;  // keys of recent uncached batches
  uint64_t tick = 0;
  size_t graph_bytes = 0;
};

constexpr size_t kGraphMaxEntries = 8;
constexpr size_t kGraphMaxBytes = size_t(2) << 30;

static bool make_event(cudaEvent_t* e) {
  if (*e || cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess) return true;
  cudaGetLastError();
  *e = nullptr;
  return false;
}

static bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &s) == cudaSuccess && s != cudaStreamCaptureStatusNone;
}

static void free_entry(GraphEntry* e, cudaStream_t st) {
  if (e->done) {
    cudaEventSynchronize(e->done);  // it may be running on another stream
    cudaEventDestroy(e->done);
  }
  if (e->exec) cudaGraphExecDestroy(e->exec);
  if (e->graph) cudaGraphDestroy(e->graph);
  if (e->d_img) cudaFreeAsync(e->d_img, st);
  if (e->d_run) cudaFreeAsync(e->d_run, st);
  if (e->d_times) cudaFreeAsync(e->d_times, st);
  delete e;
}

// field-wise (the struct has padding bytes, which callers need not clear)
static bool same_op(const xkb_batch_op& a, const xkb_batch_op& b) {
  return a.kind == b.kind && a.dtype == b.dtype && a.opA == b.opA && a.opB == b.opB &&
         a.side == b.side && a.uplo == b.uplo && a.trans == b.trans && a.diag == b.diag &&
         a.M == b.M && a.N == b.N && a.K == b.K && a.A == b.A && a.lda == b.lda && a.B == b.B &&
         a.ldb == b.ldb && a.C == b.C && a.ldc == b.ldc && a.alpha[0] == b.alpha[0] &&
         a.alpha[1] == b.alpha[1] && a.beta[0] == b.beta[0] && a.beta[1] == b.beta[1];
}

static uint64_t op_key(const xkb_batch_op* ops, int nops, int schedule) {
  uint64_t h = 1469598103934665603ull ^ (uint64_t)(unsigned)schedule;
  auto mix = [&](uint64_t v) {
    for (int i = 0; i < 8; ++i) h = (h ^ ((v >> (8 * i)) & 0xffu)) * 1099511628211ull;
  };
  auto bits = [](double d) {
    uint64_t u;
    std::memcpy(&u, &d, 8);
    return u;
  };
  for (int c = 0; c < nops; ++c) {
    const xkb_batch_op& o = ops[c];
    mix(((uint64_t)(unsigned)o.kind << 32) ^ (uint64_t)(unsigned)o.dtype);
    mix(((uint64_t)(unsigned)o.opA << 48) ^ ((uint64_t)(unsigned)o.opB << 32) ^
        ((uint64_t)(unsigned)o.side << 16) ^ (uint64_t)(unsigned)o.uplo);
    mix(((uint64_t)(unsigned)o.trans << 32) ^ (uint64_t)(unsigned)o.diag);
    mix(((uint64_t)(unsigned)o.M << 32) ^ (uint64_t)(unsigned)o.N);
    mix((uint64_t)(unsigned)o.K);
    mix(reinterpret_cast<uintptr_t>(o.A));
    mix((uint64_t)o.lda);
    mix(reinterpret_cast<uintptr_t>(o.B));
    mix((uint64_t)o.ldb);
    mix(reinterpret_cast<uintptr_t>(o.C));
    mix((uint64_t)o.ldc);
    mix(bits(o.alpha[0]));
    mix(bits(o.alpha[1]));
    mix(bits(o.beta[0]));
    mix(bits(o.beta[1]));
  }
  return h ^ (uint64_t)nops;
}

// kernel arguments of one launch on image d
// How long a CTA of the executor waits for a task whose dependencies are
// not yet resolved before it records kErrFullWait and the launch ends: the
// tuning key sched_wait_ms (default 4000 ms), a kernel parameter.
static unsigned long long wait_limit_ns() {
  const double ms = tune("sched_wait_ms", (double)(kWaitLimitNs / 1000000ull));
  return (unsigned long long)(std::max(1.0, ms) * 1e6);
}

struct KArgs {
  const Task* tasks;
  int* ndep;
  const int* succ;
  const int* bulk;
  int nbulk;
  int* urq;
  int nurg;
  Ctl* ctl;
  int urgent_first;
  int* left;
  unsigned long long* call_end;
  unsigned long long* t_start;
  unsigned long long wait_ns;
  KArgs(uint8_t* d, const Layout& L, int schedule, unsigned long long* times)
      : tasks(reinterpret_cast<const Task*>(d)),
        ndep(reinterpret_cast<int*>(d + L.o_ndep)),
        succ(reinterpret_cast<const int*>(d + L.o_succ)),
        bulk(reinterpret_cast<const int*>(d + L.o_bulk)),
        nbulk((int)L.nbulk),
        urq(reinterpret_cast<int*>(d + L.o_urq)),
        nurg((int)L.nurg),
        ctl(reinterpret_cast<Ctl*>(d + L.o_ctl)),
        urgent_first(schedule == 0 ? 1 : 0),
        left(reinterpret_cast<int*>(d + L.o_left)),
        call_end(times),
        t_start(times + L.nops),
        wait_ns(wait_limit_ns()) {}
  void* params[13] = {&tasks, &ndep, &succ,         &bulk, &nbulk,    &urq,    &nurg,
                      &ctl,   &urgent_first, &left, &call_end, &t_start, &wait_ns};
};

static Batch& batch() {
  static Batch b;
  return b;
}
static std::mutex g_batch_mu;

// CTAs of a launch: as many as fit, at most one per tile and solve task.
static int grid_size(const Layout& L) {
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sched, kThreads, sched_smem(L.ztrsm));
  if (per <= 0) per = 1;
  return (int)std::min<size_t>((size_t)per * sm_count(), std::max<size_t>(1, L.nbulk + L.nurg));
}

static int set_smem_attr() {
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(k_sched, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sched_smem(true)) != cudaSuccess)
      return XKB_ECUDA;
    attr = true;
  }
  return XKB_OK;
}

// Per-call rows of an executor launch in the event trace (recording on).
static void trace_calls(long long tv, cudaStream_t st, const unsigned long long* d_times,
                        const xkb_batch_op* ops, int n) {
  if (tv < 0) return;
  static const char* const kNames[2][2] = {{"dgemm", "zgemm"}, {"dtrsm", "ztrsm"}};
  std::vector<const char*> names((size_t)n);
  for (int i = 0; i < n; ++i)
    names[i] = kNames[ops[i].kind == XKB_BATCH_TRSM][ops[i].dtype == XKB_Z];
  evlog_kern_calls(tv, st, d_times, n, names.data());
}

static int launch_entry(Batch& B, GraphEntry* e, cudaStream_t st) {
  e->last_use = ++B.tick;
  B.ncalls = e->L.nops;
  B.call_tasks = e->call_tasks;
  B.cur_times = e->d_times;
  const long long tv = evlog_kern_begin(st, "k_sched(graph)");
  const cudaError_t le = cudaGraphLaunch(e->exec, st);
  evlog_kern_end(tv, st);
  if (le != cudaSuccess) return XKB_ECUDA;
  trace_calls(tv, st, e->d_times, e->ops.data(), e->L.nops);
  if (!capturing(st) && cudaEventRecord(e->done, st) != cudaSuccess) return XKB_ECUDA;
  count_launch();
  return XKB_OK;
}

// Build the graph of a cached batch whose image is in e->d_img.
static int build_graph(GraphEntry* e) {
  const Layout& L = e->L;
  if (cudaGraphCreate(&e->graph, 0) != cudaSuccess) return XKB_ECUDA;
  cudaGraphNode_t cp, m0, m1, kn;
  if (cudaGraphAddMemcpyNode1D(&cp, e->graph, nullptr, 0, e->d_run, e->d_img, L.bytes,
                               cudaMemcpyDeviceToDevice) != cudaSuccess)
    return XKB_ECUDA;
  cudaMemsetParams ms{};
  ms.dst = e->d_times;
  ms.value = 0;
  ms.elementSize = 1;
  ms.width = (size_t)L.nops * 8;
  ms.height = 1;
  ms.pitch = ms.width;
  if (cudaGraphAddMemsetNode(&m0, e->graph, nullptr, 0, &ms) != cudaSuccess) return XKB_ECUDA;
  ms.dst = e->d_times + L.nops;
  ms.value = 0xff;
  ms.width = 8;
  ms.pitch = 8;
  if (cudaGraphAddMemsetNode(&m1, e->graph, nullptr, 0, &ms) != cudaSuccess) return XKB_ECUDA;
  KArgs a(e->d_run, L, e->schedule, e->d_times);
  cudaKernelNodeParams kp{};
  kp.func = reinterpret_cast<void*>(k_sched);
  kp.gridDim = dim3((unsigned)grid_size(L));
  kp.blockDim = dim3(kThreads);
  kp.sharedMemBytes = (unsigned)sched_smem(L.ztrsm);
  kp.kernelParams = a.params;
  const cudaGraphNode_t deps[3] = {cp, m0, m1};
  if (cudaGraphAddKernelNode(&kn, e->graph, deps, 3, &kp) != cudaSuccess) return XKB_ECUDA;
  if (cudaGraphInstantiate(&e->exec, e->graph, 0) != cudaSuccess) return XKB_ECUDA;
  return XKB_OK;
}

}  // namespace sched
}  // namespace xkb

using namespace xkb;
using namespace xkb::sched;

extern "C" int xkb_cuda_batch(const xkb_batch_op* ops, int nops, int schedule, void* stream) {
  if (!ops || nops < 0) return XKB_EINVAL;
  if (nops == 0) return XKB_OK;
  std::lock_guard<std::mutex> g(g_batch_mu);
  cudaStream_t st = resolve_stream(stream);
  Batch& B = batch();
  if (int e = set_smem_attr()) return e;
  static const bool use_graphs = [] {
    const char* v = getenv("XKBLAS_BATCH_GRAPHS");
    return !(v && v[0] == '0');
  }();
  const uint64_t key = use_graphs ? op_key(ops, nops, schedule) : 0;
  if (use_graphs) {
    for (GraphEntry* e : B.graphs) {
      if (e->key != key || e->schedule != schedule || (int)e->ops.size() != nops) continue;
      bool same = true;
      for (int c = 0; c < nops && same; ++c) same = same_op(e->ops[(size_t)c], ops[c]);
      if (same) return launch_entry(B, e, st);
    }
  }
  Built b;
  b.call_tasks.assign(nops, 0);
  {  // size every list once: the task build is a hot host path for big batches
    size_t nt = 0, ne = 0, nb = 0;
    for (int c = 0; c < nops; ++c) {
      const xkb_batch_op& o = ops[c];
      if (o.M <= 0 || o.N <= 0) continue;
      if (o.kind == XKB_BATCH_GEMM) {
        nt += 1;
        nb += gemm_tiles(o);
      } else {
        const size_t t = ((size_t)o.M + kLeafS - 1) / kLeafS * (((size_t)o.N + kLeafS - 1) / kLeafS);
        nt += t;
        ne += t;
      }
    }
    b.tasks.reserve(nt);
    b.ndep.reserve(nt);
    b.bulk.reserve(nb);
    b.edges.reserve(ne);
  }
  for (int c = 0; c < nops; ++c) {
    const xkb_batch_op& o = ops[c];
    if ((o.dtype != XKB_D && o.dtype != XKB_Z) || o.M < 0 || o.N < 0 || o.K < 0) return XKB_EINVAL;
    if (o.M == 0 || o.N == 0) continue;
    int n;
    if (o.kind == XKB_BATCH_GEMM) {
      if (o.K == 0) return XKB_EINVAL;  // beta-only calls are not batch tasks
      n = add_gemm(b, o, c);
    } else if (o.kind == XKB_BATCH_TRSM) {
      n = add_trsm(b, o, c);
    } else {
      return XKB_EINVAL;
    }
    if (n < 0) return n;
    b.call_tasks[c] = n;
  }
  const int ntasks = (int)b.tasks.size();
  B.ncalls = nops;
  B.call_tasks = b.call_tasks;
  if (ntasks == 0) return XKB_OK;
  // successor lists (CSR over producers)
  std::vector<int> succ0((size_t)ntasks + 1, 0);
  for (auto& e : b.edges) ++succ0[(size_t)e.first + 1];
  for (int i = 0; i < ntasks; ++i) succ0[(size_t)i + 1] += succ0[(size_t)i];
  std::vector<int> succ(b.edges.size());
  {
    std::vector<int> fill(succ0.begin(), succ0.end() - 1);
    for (auto& e : b.edges) succ[(size_t)fill[(size_t)e.first]++] = e.second;
  }
  for (int i = 0; i < ntasks; ++i) {
    b.tasks[(size_t)i].succ0 = succ0[(size_t)i];
    b.tasks[(size_t)i].nsucc = succ0[(size_t)i + 1] - succ0[(size_t)i];
  }
  Layout L;
  L.set(ntasks, succ.size(), b.bulk.size(), (size_t)b.nurg, nops);
  for (int c = 0; c < nops; ++c)
    L.ztrsm = L.ztrsm || (ops[c].kind == XKB_BATCH_TRSM && ops[c].dtype == XKB_Z);
  // the shared images cannot belong to a captured graph
  if (capturing(st) || !make_event(&B.staged) || !make_event(&B.done)) return XKB_ECUDA;
  // the previous batch's upload may still read the pinned staging buffer
  if (cudaEventSynchronize(B.staged) != cudaSuccess) return XKB_ECUDA;
  if (L.bytes > B.h_cap) {
    if (B.h_stage) cudaFreeHost(B.h_stage);
    B.h_cap = L.bytes * 2;
    if (cudaHostAlloc(&B.h_stage, B.h_cap, cudaHostAllocDefault) != cudaSuccess) {
      B.h_stage = nullptr;
      B.h_cap = 0;
      return XKB_ENOMEM;
    }
  }
  uint8_t* h = B.h_stage;
  std::memcpy(h, b.tasks.data(), L.o_ndep);
  std::memcpy(h + L.o_ndep, b.ndep.data(), (size_t)ntasks * 4);
  if (!succ.empty()) std::memcpy(h + L.o_succ, succ.data(), succ.size() * 4);
  if (L.nbulk) std::memcpy(h + L.o_bulk, b.bulk.data(), L.nbulk * 4);
  int* urq = reinterpret_cast<int*>(h + L.o_urq);
  for (size_t i = 0; i < L.nurg; ++i) urq[i] = i < b.urg_ready.size() ? b.urg_ready[i] : -1;
  std::memcpy(h + L.o_left, b.call_tasks.data(), (size_t)nops * 4);
  Ctl ctl{0, 0, (int)b.urg_ready.size(), 0};
  std::memcpy(h + L.o_ctl, &ctl, sizeof(ctl));

  // a batch seen before (recently, uncached) becomes a cached graph
  bool cache = false;
  if (use_graphs) {
    auto it = std::find(B.seen.begin(), B.seen.end(), key);
    if (it != B.seen.end()) {
      B.seen.erase(it);
      cache = 2 * L.bytes <= kGraphMaxBytes;
    } else {
      B.seen.push_back(key);
      if (B.seen.size() > 32) B.seen.erase(B.seen.begin());
    }
  }
  if (cache) {
    GraphEntry* e = new GraphEntry;
    e->key = key;
    e->schedule = schedule;
    e->ops.assign(ops, ops + nops);
    e->L = L;
    e->call_tasks = b.call_tasks;
    if (!scratch_alloc(reinterpret_cast<void**>(&e->d_img), L.bytes, st) ||
        !scratch_alloc(reinterpret_cast<void**>(&e->d_run), L.bytes, st) ||
        !scratch_alloc(reinterpret_cast<void**>(&e->d_times), ((size_t)nops + 1) * 8, st)) {
      free_entry(e, st);
      return XKB_ENOMEM;
    }
    cudaMemcpyAsync(e->d_img, h, L.bytes, cudaMemcpyHostToDevice, st);
    cudaEventRecord(B.staged, st);
    if (int r = make_event(&e->done) ? build_graph(e) : XKB_ECUDA) {
      free_entry(e, st);
      return r;
    }
    // evict least recently used entries beyond the limits
    while (!B.graphs.empty() && (B.graphs.size() >= kGraphMaxEntries ||
                                 B.graph_bytes + e->bytes() > kGraphMaxBytes)) {
      auto lru = std::min_element(B.graphs.begin(), B.graphs.end(),
                                  [](GraphEntry* x, GraphEntry* y) { return x->last_use < y->last_use; });
      B.graph_bytes -= (*lru)->bytes();
      free_entry(*lru, st);
      B.graphs.erase(lru);
    }
    B.graphs.push_back(e);
    B.graph_bytes += e->bytes();
    return launch_entry(B, e, st);
  }

  // the previous launch, perhaps on another stream, reads what is freed or
  // overwritten below
  if (cudaStreamWaitEvent(st, B.done, 0) != cudaSuccess) return XKB_ECUDA;
  if (L.bytes > B.d_cap) {
    if (B.d_buf) cudaFreeAsync(B.d_buf, st);
    B.d_cap = L.bytes * 2;
    if (!scratch_alloc(reinterpret_cast<void**>(&B.d_buf), B.d_cap, st)) {
      B.d_cap = 0;
      return XKB_ENOMEM;
    }
  }
  if ((size_t)nops + 1 > B.d_cap_times) {
    if (B.d_times) cudaFreeAsync(B.d_times, st);
    B.d_cap_times = ((size_t)nops + 1) * 2;
    if (!scratch_alloc(reinterpret_cast<void**>(&B.d_times),
                       B.d_cap_times * sizeof(unsigned long long), st)) {
      B.d_cap_times = 0;
      return XKB_ENOMEM;
    }
  }
  uint8_t* d = B.d_buf;
  cudaMemcpyAsync(d, h, L.bytes, cudaMemcpyHostToDevice, st);
  cudaEventRecord(B.staged, st);
  cudaMemsetAsync(B.d_times, 0, (size_t)nops * sizeof(unsigned long long), st);
  cudaMemsetAsync(B.d_times + nops, 0xff, sizeof(unsigned long long), st);
  B.cur_times = B.d_times;
  KArgs a(d, L, schedule, B.d_times);
  const long long tv = evlog_kern_begin(st, "k_sched");
  k_sched<<<grid_size(L), kThreads, sched_smem(L.ztrsm), st>>>(
      a.tasks, a.ndep, a.succ, a.bulk, a.nbulk, a.urq, a.nurg, a.ctl, a.urgent_first, a.left,
      a.call_end, a.t_start, a.wait_ns);
  evlog_kern_end(tv, st);
  trace_calls(tv, st, B.d_times, ops, nops);
  cudaEventRecord(B.done, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

extern "C" int xkb_cuda_batch_latency(double* ms, int n) {
  Batch& B = batch();
  std::lock_guard<std::mutex> g(g_batch_mu);
  if (!ms || n < 0 || n > B.ncalls || !B.cur_times) return XKB_EINVAL;
  if (cudaDeviceSynchronize() != cudaSuccess) return XKB_ECUDA;
  std::vector<unsigned long long> t((size_t)B.ncalls + 1);
  if (cudaMemcpy(t.data(), B.cur_times, t.size() * sizeof(unsigned long long),
                 cudaMemcpyDeviceToHost) != cudaSuccess)
    return XKB_ECUDA;
  const unsigned long long t0 = t[B.ncalls];
  for (int i = 0; i < n; ++i)
    ms[i] = (B.call_tasks[i] && t[i] >= t0) ? (double)(t[i] - t0) * 1e-6 : 0.0;
  return XKB_OK;
}

extern "C" int xkb_cuda_batch_release(void) {
  Batch& B = batch();
  std::lock_guard<std::mutex> g(g_batch_mu);
  if (cudaDeviceSynchronize() != cudaSuccess) return XKB_ECUDA;
  for (GraphEntry* e : B.graphs) free_entry(e, nullptr);
  B.graphs.clear();
  B.seen.clear();
  B.graph_bytes = 0;
  if (B.cur_times && B.cur_times != B.d_times) B.cur_times = nullptr;
  return XKB_OK;
}

extern "C" int xkb_cuda_batch_cached(void) {
  Batch& B = batch();
  std::lock_guard<std::mutex> g(g_batch_mu);
  return (int)B.graphs.size();
}

// Exercises the bounded wait on the device: one CTA of the executor is
// launched on a ready queue whose only slot claims a task (the queue's tail
// was advanced) that no producer ever writes -- as if the task's last
// dependency never resolved.  The CTA waits wait_ms, records kErrFullWait
// and ends; the launch returns normally and the context stays usable.  The
// caller reads the outcome with xkb_cuda_take_device_error (or xkblas_sync).
extern "C" int xkb_cuda_sched_wait_test(int wait_ms, void* stream) {
  if (wait_ms < 1 || wait_ms > 10000) return XKB_EINVAL;
  cudaStream_t st = resolve_stream(stream);
  if (int e = set_smem_attr()) return e;
  // layout: ctl | urq[1] | ndep[1] | left[1] | times[2] | task[1]
  const size_t o_urq = 16, o_ndep = 32, o_left = 48, o_times = 64, o_task = 128;
  const size_t bytes = o_task + sizeof(Task);
  uint8_t* d = nullptr;
  if (!scratch_alloc(reinterpret_cast<void**>(&d), bytes, st)) return XKB_ENOMEM;
  uint8_t h[o_task + sizeof(Task)];
  std::memset(h, 0, sizeof h);
  const Ctl ctl{0, 0, 1, 0};  // no bulk work; one queued ticket ...
  std::memcpy(h, &ctl, sizeof ctl);
  const int unset = -1;       // ... whose slot is never written
  std::memcpy(h + o_urq, &unset, sizeof unset);
  const int one = 1;
  std::memcpy(h + o_ndep, &one, sizeof one);
  std::memcpy(h + o_left, &one, sizeof one);
  cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st);
  auto* times = reinterpret_cast<unsigned long long*>(d + o_times);
  cudaMemsetAsync(times + 1, 0xff, sizeof(unsigned long long), st);
  const long long tv = evlog_kern_begin(st, "k_sched");
  k_sched<<<1, kThreads, sched_smem(false), st>>>(
      reinterpret_cast<const Task*>(d + o_task), reinterpret_cast<int*>(d + o_ndep), nullptr,
      nullptr, 0, reinterpret_cast<int*>(d + o_urq), 1, reinterpret_cast<Ctl*>(d), 1,
      reinterpret_cast<int*>(d + o_left), times, times + 1, (unsigned long long)wait_ms * 1000000ull);
  evlog_kern_end(tv, st);
  count_launch();
  cudaFreeAsync(d, st);
  // the staging array h is copied by the time the host can return: pageable
  // memory makes cudaMemcpyAsync stage it synchronously
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}
