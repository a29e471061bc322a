// Persistent CG on the CSR values in place: the iterations of one solve as one
// cooperative launch, the engine behind HOEFEM_CG_ENGINE_CHUNKED (cg.cu keeps
// the graphs of kernel chunks for what this kernel does not take).
//
// Reference: ConjugateGradient::solve_with_guess_ (fenris/src/cg.rs:376-482);
// same recurrence, tests and order of updates as cg.cu.
//
// What bounds it: a large solve streams the matrix (and the inverted Schwarz
// blocks) from HBM once per iteration; a small one waits for its grid-wide
// steps.  An L2 load takes about 1,000 cycles here and a warp's tile needs two
// in a row (neighbours, then p), so without care it is the latency per warp
// that bounds both.  Hence
//  * one warp per CTA fills a ring of shared-memory stages with bulk copies
//    (values, neighbour lists, row offsets of a tile of whole node rows, or
//    some rows of a Schwarz block), one lane per stage, each independent of
//    the others.  The matrix does not change during the solve, so the ring
//    runs ahead across the grid barriers.  If a CTA's tiles all fit, each is
//    copied once.
//  * up to 15 warps take the tiles in turn, one stage each at a time, so that
//    their latencies overlap; more stages than warps are in flight.  (A ring
//    of its own for every warp left room for 4 to 9 warps and was 1.5 to 2
//    times slower.)
//  * a warp multiplies four node rows at once, one 3 x 3 block per lane, the
//    gathers of p of all four in flight together, and sums their row sums in
//    one exchange tree (13 shuffles).  (Eight at once spilled and gained
//    nothing.)
//  * the values are read where the caller has them (scalar CSR order); the
//    rows of a node are contiguous there.  Nothing is packed per solve.
//  * few grid barriers, each one counter with one polling thread per CTA; sums
//    are published before it and added by every CTA after it in the same
//    order, so all take the same decisions.
//
// An iteration with the Schwarz preconditioner (three barriers):
//  1. A p of the CTA's tiles; p.Ap
//  2. y_s = B_s r'_s with r' = r - alpha A p, by rows; r'.r' and, as
//     z.r' = sum_s y_s.r'_s, z.r'
//  3. x, r and p = z + beta p of the CTA's nodes
// With the diagonal or no preconditioner (two barriers): phase 1 also sums
// r.r, r.Ap, Ap.Ap and the same with D, from which r'.r' and z'.r' of the
// updated residual follow without a second pass, to 1e-14; where they drop by more
// than 10 in one step (cancellation, cg_next_sum), the sums are formed from the
// updated residual instead, with a barrier of their own.  r itself is updated as
// ever and its sums are formed anew in every iteration, so nothing accumulates.
// Deterministic: the tile split, the order inside a warp, over warps and over
// CTAs are all fixed.
//
// Measured per iteration (whole solve, the graphs before -> this kernel):
// embedded Hex27 cylinder 24^3, Schwarz, 132,888 DOFs: FP64 91 -> 69 us (272 MB
// of values, of which A p 32 us at 5.8 TB/s), mixed 64 (streamed engine) -> 47
// us; Tet10 box 31 x 29 x 17, diagonal, 390,285 DOFs: FP64 89 -> 68 us, mixed
// 79 -> 60 us; Tet10 box 8^3: 32 -> 15 us.
// FP32 values of the box stay at 4 TB/s: 28 scattered 16-byte gathers a node
// fill the L1 tag stage before the values fill the memory pipe.
//
// Waits are bounded (2 s); one that runs out raises a flag that all CTAs see,
// the copies in flight land before a CTA leaves, and the host gets
// HOEFEM_ERR_DEVICE_TIMEOUT.
#include <cuda_runtime.h>

#include <algorithm>

#include "cg_limit.h"
#include "internal.h"
#include "pcg_layout.h"
#include "solver.h"
#include "stream_pipe.cuh"

namespace hoefem {

namespace {

constexpr int NWARP = 15;              // consumer warps (with the producer 512 threads: 128 registers each)
constexpr int WORKERS = 32 * NWARP;
constexpr int THREADS = WORKERS + 32;  // and the producer warp
constexpr int MAX_STAGES = 32;         // one producer lane each
// Row offsets of a tile or node list of a subdomain (its slots go where a tile's
// neighbours do), from up to three ints ahead: 16-byte granules.
constexpr int IDX_BYTES = 160;
static_assert(IDX_BYTES % 16 == 0 && IDX_BYTES >= (4 * (3 + PCG_MAX_TILE_NODES + 1) + 15) / 16 * 16 &&
                  IDX_BYTES >= (4 * (3 + PCG_MAX_SUB_NODES) + 15) / 16 * 16,
              "the lists fit their part of a stage");
static_assert(3 * PCG_MAX_SUB_NODES <= 96, "a block's columns in three per lane");
constexpr int TILE_COST = 4096;  // bytes a tile's latency is worth in the CTA split
constexpr int MAX_G = 256;      // CTAs the barrier's readers cover (8 entries a lane)
constexpr size_t SMEM_BUDGET = 192 * 1024;  // the rest stays L1 for the gathers of p

struct Args {
  // operator
  const void* vals;
  long long val_limit;  // whole 16-byte granules of the value array, bytes
  const int* adj;
  const int* adj_off;
  const PcgTile* tiles;
  const int* cta_tile;
  // Schwarz blocks
  const void* blocks;
  const int* sub_nodes;
  const int* slot;
  const PcgSwTile* sw_tiles;
  const int* cta_sw;
  const int* pair_off;
  const unsigned char* diag_only;
  const long long* pbase;
  const double* pvals;
  double* y;
  const double* dinv;
  // vectors
  double *x, *r, *z, *p, *Ap;
  void* px;  // padded copy of p: 4 doubles or 4 floats per node
  int nv;
  CgState* st;
  unsigned* counter;  // grid barrier
  double* part;       // partial sums, 2 x MAX_SUMS x G
  int* err;
  int reliable, chunk;  // residual replacements, at multiples of `chunk` iterations
  // shared memory
  int nw, stages, val_bytes, adj_bytes;  // warps that take tiles, ring stages and their parts
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Loads of vectors that this kernel writes: ordinary (not read-only-cache)
// loads, kept in program order with the barriers.
__device__ __forceinline__ double ld_vec(const double* a) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(a) : "memory");
  return v;
}
constexpr int MAX_SUMS = 7;

__device__ __forceinline__ void worker_sync() { pipe::named_sync(1, WORKERS); }

// Grid barrier: every worker thread of every CTA calls it.  With K > 0, the threads'
// shares v[0 .. K) are summed over the grid and the totals replace them
// (partial sums double-buffered by the barrier's parity: a CTA overwrites its
// entries two barriers later, after all CTAs have passed the one between).
// False once a wait ran out anywhere (fail: in this warp).
// 148 CTAs of 512 threads, idle memory: 1.35 us, and 0.5 us for the sums; all
// CTAs reading tagged entries of all others instead of one counter took 2.4 us.
__device__ __noinline__ bool grid_exchange(unsigned* counter, double* part, int* err, unsigned epoch, int K, double* v,
                                           bool fail, int* s_abort) {
  __shared__ double s_red[MAX_SUMS][NWARP];
  __shared__ double s_in[MAX_SUMS];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, G = gridDim.x;
  double* slots = part + (size_t)(epoch & 1) * MAX_SUMS * G;
  for (int k = 0; k < K; ++k) {
    const double t = warp_sum(v[k]);
    if (lane == 0) s_red[k][w] = t;
  }
  if (fail && lane == 0) *(volatile int*)s_abort = 1;
  worker_sync();
  if (w == 0) {
    for (int k = 0; k < K; ++k) {
      double t = lane < NWARP ? s_red[k][lane] : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) slots[(size_t)k * G + blockIdx.x] = t;
    }
    if (lane == 0) {
      if (*(volatile int*)s_abort) atomicExch(err, 1);
      // the CTA's writes (ordered before this thread by the CTA barrier) become visible first
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
      const unsigned target = epoch * (unsigned)G;
      uint64_t start = 0;
      for (unsigned polls = 1;; ++polls) {
        unsigned c;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(counter) : "memory");
        if ((int)(c - target) >= 0) break;
        if (polls & 63) continue;
        if (start == 0) start = pipe::clock_ns();
        if (*(volatile int*)err != 0 || pipe::clock_ns() - start > pipe::HOEFEM_WAIT_NS) {
          atomicExch(err, 1);
          *(volatile int*)s_abort = 1;
          break;
        }
      }
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
    }
  }
  worker_sync();
  if (K > 0) {
    if (w < K) {
      double e[MAX_G / 32];
#pragma unroll
      for (int k = 0; k < MAX_G / 32; ++k) {
        const int i = lane + 32 * k;
        e[k] = 0.0;
        if (i < G) asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(e[k]) : "l"(slots + (size_t)w * G + i) : "memory");
      }
      double t = 0.0;
#pragma unroll
      for (int k = 0; k < MAX_G / 32; ++k) t += e[k];
      t = warp_sum(t);
      if (lane == 0) s_in[w] = t;
    }
    worker_sync();
    for (int k = 0; k < K; ++k) v[k] = s_in[k];
  }
  return *(volatile int*)s_abort == 0;
}

__device__ __forceinline__ void ld_node(const double* a, double* o) {
  double w;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(w) : "l"(a)
               : "memory");
}
__device__ __forceinline__ void ld_node(const float* a, float* o) {
  float w;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(w) : "l"(a)
               : "memory");
}

// Number of the item a stage was last filled for (last word of its header).
__device__ __forceinline__ volatile int& stage_item(unsigned char* stage) {
  return *reinterpret_cast<volatile int*>(stage + 28);
}

// Bounded wait until a stage carries item `n`.
__device__ __forceinline__ bool wait_item(const volatile int* at, int n, const int* abort) {
  if (*at == n) return true;
  const uint64_t t0 = pipe::clock_ns();
  for (;;) {
    if (*at == n) return true;
    if (*(const volatile int*)abort || pipe::clock_ns() - t0 > pipe::HOEFEM_WAIT_NS) return false;
  }
}

// True if the phase with the given parity has completed; does not wait.
__device__ __forceinline__ bool mbar_ready(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(pipe::smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

template <class VA, class VB, int PK>
__global__ void __launch_bounds__(THREADS, 1) k_pcg(const Args A) {
  using X = VA;  // p is gathered in the values' precision
  constexpr int NG = 4;  // node rows multiplied at once
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_full[MAX_STAGES], s_empty[MAX_STAGES];
  __shared__ int s_abort;
  __shared__ volatile int s_stop;
  if (A.st->done) return;  // a replacement before this launch found the solve finished
  const int G = gridDim.x, c = blockIdx.x;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int NS = A.stages, NW = A.nw;
  const int stage_bytes = 32 + IDX_BYTES + A.adj_bytes + A.val_bytes;
  // the CTA's items: operator tiles, then Schwarz tiles, cyclically; item n
  // (counted over the whole launch) goes to stage n % NS
  const int t0 = A.cta_tile[c], nop = A.cta_tile[c + 1] - t0;
  const int u0 = PK == 2 ? A.cta_sw[c] : 0, nsw = PK == 2 ? A.cta_sw[c + 1] - u0 : 0;
  const int per = nop + nsw;
  const bool resident = per <= NS;  // every item keeps a stage of its own
  if (threadIdx.x == 0) {
    s_abort = 0;
    s_stop = 0;
    for (int i = 0; i < NS; ++i) stage_item(smem + (size_t)i * stage_bytes) = -1;
    for (int i = 0; i < MAX_STAGES; ++i) {
      pipe::mbar_init(&s_full[i], 1);
      pipe::mbar_init(&s_empty[i], 1);
    }
    pipe::mbar_fence_init();
  }
  __syncthreads();

  if (w == NWARP) {
    // ---- producer: lane l fills stage l with the items l, l + NS, ... ----
    if (lane >= NS || lane >= per) return;
    const uint64_t policy = pipe::policy_evict_first();
    unsigned char* st = smem + (size_t)lane * stage_bytes;
    unsigned char* s_idx = st + 32;
    unsigned char* s_adj = s_idx + IDX_BYTES;
    unsigned char* s_val = s_adj + A.adj_bytes;
    int k = lane;        // item within the cycle
    unsigned item = lane;  // and counted over the launch (wraps)
    unsigned fills = 0;  // of this stage
    int4 h0, h1 = make_int4(0, 0, 0, 0);
    auto load = [&]() {  // the descriptor of item k, ahead of its use
      if (k < nop) {
        h0 = __ldg(reinterpret_cast<const int4*>(A.tiles) + t0 + k);
      } else {
        h0 = __ldg(reinterpret_cast<const int4*>(A.sw_tiles) + 2 * (u0 + k - nop));
        h1 = __ldg(reinterpret_cast<const int4*>(A.sw_tiles) + 2 * (u0 + k - nop) + 1);
      }
    };
    load();
    uint64_t idle = 0;
    unsigned polls = 0;
    while (!s_stop) {
      if (fills > 0 && !mbar_ready(&s_empty[lane], (fills - 1) & 1)) {
        // nothing to do until the stage is released; bounded by the launch's own waits
        if ((++polls & 255) == 0) {
          const uint64_t now = pipe::clock_ns();
          if (idle == 0) idle = now;
          if (now - idle > 2 * pipe::HOEFEM_WAIT_NS) break;
        }
        continue;
      }
      idle = 0;
      uint64_t* bar = &s_full[lane];
      if (k < nop) {
        const PcgTile T{h0.x, h0.y, h0.z, h0.w};
        const PcgSpan o = pcg_span(4LL * T.n0, 4LL * (T.n0 + T.nn + 1), 1LL << 62);
        const PcgSpan j = pcg_span(4LL * T.o0, 4LL * T.o0 + 4LL * T.nblk, 1LL << 62);
        const long long vb = 9LL * (int)sizeof(VA) * T.o0;
        const PcgSpan v = pcg_span(vb, vb + 9LL * (int)sizeof(VA) * T.nblk, A.val_limit);
        const int jb = T.nblk ? j.bytes : 0, vbytes = T.nblk ? v.bytes : 0;
        *reinterpret_cast<int4*>(st) = h0;
        stage_item(st) = (int)item;
        pipe::mbar_arrive_expect_tx(bar, (unsigned)(o.bytes + jb + vbytes));
        if (vbytes) pipe::bulk_g2s_hint(s_val, (const char*)A.vals + v.from, (unsigned)vbytes, bar, policy);
        if (jb) pipe::bulk_g2s_hint(s_adj, (const char*)A.adj + j.from, (unsigned)jb, bar, policy);
        pipe::bulk_g2s(s_idx, (const char*)A.adj_off + o.from, (unsigned)o.bytes, bar);
      } else {
        const long long src = (long long)(((unsigned long long)(unsigned)h0.y << 32) | (unsigned)h0.x);
        const int o0 = h0.z, dim = h0.w, rows = h1.y;
        const PcgSpan o = pcg_span(4LL * o0, 4LL * (o0 + dim / 3), 1LL << 62);
        const PcgSpan v = pcg_span(src * (int)sizeof(VB), (src + (long long)rows * dim) * (int)sizeof(VB), 1LL << 62);
        reinterpret_cast<int4*>(st)[0] = h0;
        *reinterpret_cast<int2*>(st + 16) = make_int2(h1.x, h1.y);
        stage_item(st) = (int)item;
        pipe::mbar_arrive_expect_tx(bar, (unsigned)(v.bytes + 2 * o.bytes));
        pipe::bulk_g2s_hint(s_val, (const char*)A.blocks + v.from, (unsigned)v.bytes, bar, policy);
        pipe::bulk_g2s(s_idx, (const char*)A.sub_nodes + o.from, (unsigned)o.bytes, bar);
        pipe::bulk_g2s(s_adj, (const char*)A.slot + o.from, (unsigned)o.bytes, bar);
      }
      ++fills;
      if (resident) break;
      item += (unsigned)NS;
      k += NS;
      while (k >= per) k -= per;
      load();
    }
    // the copy in flight lands before the CTA leaves
    if (fills > 0) pipe::mbar_wait(&s_full[lane], (fills - 1) & 1);
    return;
  }

  bool bad = false;     // a wait of this warp ran out
  unsigned item0 = 0;   // items of the phases before this one (wraps), the stage of
  int stage0 = 0;       // the next one and the parity of its turn
  unsigned turn0 = 0;
  // The warp's share (w, w + NW, ...) of the cycle's next n items.
  auto run_items = [&](int n, auto&& compute) {
    const int ring = resident ? max(per, 1) : NS;
    if (w < NW && !bad) {
      for (int i = w; i < n; i += NW) {
        const int q = stage0 + i, turn = q / ring, s = q - turn * ring;
        // The stage's previous item may belong to another warp and not even
        // have landed: its phase's parity would pass for this one's.  Once the
        // header carries this item's number the previous one has been consumed.
        bool got = true;
        if (!resident) got = wait_item(&stage_item(smem + (size_t)s * stage_bytes), (int)(item0 + (unsigned)i), &s_abort);
        got = got && pipe::mbar_wait(&s_full[s], resident ? 0u : (turn0 + turn) & 1u, (const volatile int*)&s_abort);
        if (!__all_sync(0xffffffffu, got)) {
          bad = true;
          break;
        }
        compute(smem + (size_t)s * stage_bytes);
        __syncwarp();
        if (!resident && lane == 0) pipe::mbar_arrive(&s_empty[s]);
      }
    }
    item0 += (unsigned)n;
    turn0 += (unsigned)((stage0 + n) / ring);
    stage0 = (stage0 + n) % ring;
  };

  unsigned epoch = 0;
  double sum[MAX_SUMS];
  auto grid_sum = [&](int K) -> bool {
    ++epoch;
    return grid_exchange(A.counter, A.part, A.err, epoch, K, sum, bad, &s_abort);
  };

  const CgState* st0 = A.st;
  double zTr = st0->zTr, beta = st0->beta, alpha = st0->alpha, pAp = st0->pAp, rr = st0->rr;
  const double bnorm = st0->bnorm, tol = st0->tol, rr_ref = st0->rr_ref, delta2 = st0->delta2;
  long long iters = st0->iters;
  const long long limit = st0->max_iter;  // never negative (cg_limit.h)
  int status = HOEFEM_OK, done = 0, replace = 0;
  const int na = (int)((long long)A.nv * c / G), nb = (int)((long long)A.nv * (c + 1) / G);
  X* px = reinterpret_cast<X*>(A.px);

  auto store_p = [&](int a, const double (&q)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) A.p[3 * a + i] = q[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) px[4LL * a + i] = (X)q[i];
  };

  // first direction: p = z + beta p, z from the preconditioner kernel
  for (int a = na + (int)threadIdx.x; a < nb; a += WORKERS) {
    double q[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      q[i] = ld_vec(A.z + 3 * a + i);
      if (beta != 0.0) q[i] += beta * ld_vec(A.p + 3 * a + i);
    }
    store_p(a, q);
  }
  bool ok = grid_sum(0);
  while (ok) {
    // ---- phase 1: A p ----
    double acc[MAX_SUMS];
#pragma unroll
    for (int k = 0; k < MAX_SUMS; ++k) acc[k] = 0.0;
    // node and component this lane's exchange ends with (the others double one)
    const int on = lane / (32 / NG), oc = lane & (16 / NG) ? 2 : (lane & (8 / NG) ? 1 : 0);
    const bool owner = !(lane & 1) && (lane & 6) != 6;
    run_items(nop, [&](unsigned char* stg) {
      const PcgTile T = *reinterpret_cast<const PcgTile*>(stg);
      const int* off = reinterpret_cast<const int*>(stg + 32) + (T.n0 & 3);
      const int* adj = reinterpret_cast<const int*>(stg + 32 + IDX_BYTES) + (T.o0 & 3) + lane;
      const long long vb = 9LL * T.o0 * (int)sizeof(VA);
      VA* vt = reinterpret_cast<VA*>(stg + 32 + IDX_BYTES + A.adj_bytes + (vb & 15));
      if (vb + 9LL * T.nblk * (int)sizeof(VA) > A.val_limit) {
        // the array's last partial granule is not copied in bulk
        const int n0 = (int)((A.val_limit - vb) / (int)sizeof(VA)), n1 = 9 * T.nblk;
        if (n0 + lane < n1) vt[n0 + lane] = reinterpret_cast<const VA*>(A.vals)[9LL * T.o0 + n0 + lane];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the stage's next bulk copy
        __syncwarp();
      }
      for (int j0 = 0; j0 < T.nn; j0 += NG) {
        int oj[NG], d[NG], dmax = 0;
#pragma unroll
        for (int j = 0; j < NG; ++j) {
          const bool has = j0 + j < T.nn;
          oj[j] = has ? off[j0 + j] - T.o0 : 0;
          d[j] = has ? off[j0 + j + 1] - T.o0 - oj[j] : 0;
          dmax = max(dmax, d[j]);
        }
        X v[NG][3];
#pragma unroll
        for (int j = 0; j < NG; ++j) v[j][0] = v[j][1] = v[j][2] = 0;
        const bool mine = owner && j0 + on < T.nn;
        const long long dof = 3LL * (T.n0 + j0 + on) + oc;
        double po = 0.0, ro = 0.0, di = 0.0;
        if (mine) {
          po = ld_vec(A.p + dof);
          if (PK != 2) ro = ld_vec(A.r + dof);
          if (PK == 1) di = __ldg(A.dinv + dof);
        }
        for (int c0 = 0; c0 < dmax; c0 += 32) {
          X g[NG][3];
#pragma unroll
          for (int j = 0; j < NG; ++j)
            if (c0 + lane < d[j]) ld_node(px + 4LL * adj[oj[j] + c0], g[j]);
#pragma unroll
          for (int j = 0; j < NG; ++j)
            if (c0 + lane < d[j]) {
              const VA* q0 = vt + 9 * oj[j] + 3 * (c0 + lane);
              const VA* q1 = q0 + 3 * d[j];
              const VA* q2 = q1 + 3 * d[j];
              v[j][0] += q0[0] * g[j][0] + q0[1] * g[j][1] + q0[2] * g[j][2];
              v[j][1] += q1[0] * g[j][0] + q1[1] * g[j][1] + q1[2] * g[j][2];
              v[j][2] += q2[0] * g[j][0] + q2[1] * g[j][1] + q2[2] * g[j][2];
            }
        }
        // 3 NG sums over 32 lanes: halve the nodes until a lane carries part
        // of one node's three components, then the components
        int o = 16;
#pragma unroll
        for (int h = NG / 2; h > 0; h >>= 1, o >>= 1) {
          const bool u = lane & o;
#pragma unroll
          for (int j = 0; j < h; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              const X send = u ? v[j][i] : v[j + h][i];
              v[j][i] = (u ? v[j + h][i] : v[j][i]) + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        constexpr int B2 = 16 / NG, B1 = B2 / 2;  // lane bits of component 2, and of 1 against 0
        const bool u2 = lane & B2, u1 = lane & B1;
        X s0 = (u2 ? v[0][2] : v[0][0]) + __shfl_xor_sync(0xffffffffu, u2 ? v[0][0] : v[0][2], B2);
        const X s1 = v[0][1] + __shfl_xor_sync(0xffffffffu, v[0][1], B2);
        s0 = (!u2 && u1 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, u2 || u1 ? s0 : s1, B1);
        s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
        if (mine) {
          const double t = (double)s0;
          A.Ap[dof] = t;
          acc[0] += po * t;
          if (PK != 2) {
            acc[1] += ro * ro;
            acc[2] += ro * t;
            acc[3] += t * t;
          }
          if (PK == 1) {
            acc[4] += di * ro * ro;
            acc[5] += di * ro * t;
            acc[6] += di * t * t;
          }
        }
      }
    });
#pragma unroll
    for (int k = 0; k < MAX_SUMS; ++k) sum[k] = acc[k];
    ok = grid_sum(PK == 2 ? 1 : (PK == 1 ? 7 : 4));
    if (!ok) break;
    pAp = sum[0];
    if (PK == 1) zTr = sum[4];
    if (PK == 0) zTr = sum[1];
    if (!cg_step_begin(pAp, zTr, limit, iters, status)) {
      done = 1;
      break;
    }
    alpha = zTr / pAp;
    double zr;
    bool stepped = false;  // x and r already updated
    if (PK == 2) {
      // ---- phase 2: Schwarz block rows with r' = r - alpha A p ----
      double racc = 0.0, zacc = 0.0;
      run_items(nsw, [&](unsigned char* stg) {
        const PcgSwTile T = *reinterpret_cast<const PcgSwTile*>(stg);
        const int* nodes = reinterpret_cast<const int*>(stg + 32) + (T.o & 3);
        const int* slot = reinterpret_cast<const int*>(stg + 32 + IDX_BYTES) + (T.o & 3);
        const VB* B = reinterpret_cast<const VB*>(stg + 32 + IDX_BYTES + A.adj_bytes + ((T.src * (int)sizeof(VB)) & 15));
        int col[3];
        double rv[3], ap[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          col[i] = min(lane + 32 * i, T.dim - 1);
          const long long t = 3LL * nodes[col[i] / 3] + col[i] % 3;
          rv[i] = ld_vec(A.r + t);
          ap[i] = ld_vec(A.Ap + t);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) rv[i] = lane + 32 * i < T.dim ? rv[i] - alpha * ap[i] : 0.0;
        for (int r0 = 0; r0 < T.rows; r0 += PCG_SW_ROWS) {
          double v[PCG_SW_ROWS];
#pragma unroll
          for (int i = 0; i < PCG_SW_ROWS; ++i) {
            const VB* row = B + min(r0 + i, T.rows - 1) * T.dim;
            v[i] = (double)row[col[0]] * rv[0] + (double)row[col[1]] * rv[1] + (double)row[col[2]] * rv[2];
          }
          // 8 sums over 32 lanes: lane l ends with row r0 + (l >> 2)
#pragma unroll
          for (int h = PCG_SW_ROWS / 2, o = 16; h > 0; h >>= 1, o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < h; ++i) {
              const double send = up ? v[i] : v[i + h];
              const double keep = up ? v[i + h] : v[i];
              v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          }
          double t = v[0];
          t += __shfl_xor_sync(0xffffffffu, t, 2);
          t += __shfl_xor_sync(0xffffffffu, t, 1);
          // the row's own residual entry, held by lane d % 32
          const int r = r0 + (lane >> 2), d = T.row0 + min(r, T.rows - 1);
          const double q0 = __shfl_sync(0xffffffffu, rv[0], d & 31), q1 = __shfl_sync(0xffffffffu, rv[1], d & 31),
                       q2 = __shfl_sync(0xffffffffu, rv[2], d & 31);
          if ((lane & 3) == 0 && r < T.rows) {
            A.y[3LL * slot[d / 3] + d % 3] = t;
            zacc += t * (d < 32 ? q0 : (d < 64 ? q1 : q2));
          }
        }
      });
      for (int a = na + (int)threadIdx.x; a < nb; a += WORKERS) {
        double rn[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) rn[i] = ld_vec(A.r + 3 * a + i);
#pragma unroll
        for (int i = 0; i < 3; ++i) rn[i] -= alpha * ld_vec(A.Ap + 3 * a + i);
        const bool diag = __ldg(A.diag_only + a);
        const long long pb = diag ? __ldg(A.pbase + a) : 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          racc += rn[i] * rn[i];
          if (diag) zacc += __ldg(A.pvals + pb + i) * rn[i] * rn[i];
        }
      }
      sum[0] = racc;
      sum[1] = zacc;
      ok = grid_sum(2);
      if (!ok) break;
      rr = sum[0];
      zr = sum[1];
    } else {
      bool formed = cg_next_sum(alpha, sum[1], sum[2], sum[3], rr);
      zr = rr;
      if (PK == 1) formed = cg_next_sum(alpha, sum[4], sum[5], sum[6], zr) && formed;
      if (!formed) {
        double racc = 0.0, zacc = 0.0;
        for (int a = na + (int)threadIdx.x; a < nb; a += WORKERS)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int t = 3 * a + i;
            const double rn = ld_vec(A.r + t) - alpha * ld_vec(A.Ap + t);
            A.x[t] = ld_vec(A.x + t) + alpha * ld_vec(A.p + t);
            A.r[t] = rn;
            racc += rn * rn;
            zacc += (PK == 1 ? __ldg(A.dinv + t) * rn : rn) * rn;
          }
        sum[0] = racc;
        sum[1] = zacc;
        ok = grid_sum(2);
        if (!ok) break;
        rr = sum[0];
        zr = sum[1];
        stepped = true;
      }
    }
    if (cg_iteration_end(rr, tol, bnorm, limit, iters, status)) {
      done = 1;
    } else {
      beta = zr / zTr;
      zTr = zr;
      // at the ends of chunks, as the graphs
      if (A.reliable && iters % A.chunk == 0 && rr <= delta2 * rr_ref) replace = 1;
    }
    const bool last = done || replace;
    // ---- phase 3: x, r, p of the CTA's nodes ----
    for (int a = na + (int)threadIdx.x; a < nb; a += WORKERS) {
      double pv[3], xv[3], rn[3], ap[3], zv[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        pv[i] = ld_vec(A.p + 3 * a + i);
        rn[i] = ld_vec(A.r + 3 * a + i);
        if (!stepped) {
          xv[i] = ld_vec(A.x + 3 * a + i);
          ap[i] = ld_vec(A.Ap + 3 * a + i);
        }
      }
      if (PK == 2 && !last) {
        zv[0] = zv[1] = zv[2] = 0.0;
        // the node's subdomains in ascending order (zero if it has none)
        const int q1 = __ldg(A.pair_off + a + 1);
        for (int q = __ldg(A.pair_off + a); q < q1; q += 4) {
          double yv[4][3];
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) yv[k][i] = q + k < q1 ? ld_vec(A.y + 3LL * (q + k) + i) : 0.0;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (q + k < q1)
#pragma unroll
              for (int i = 0; i < 3; ++i) zv[i] += yv[k][i];
        }
      }
      if (!stepped) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          A.x[3 * a + i] = xv[i] + alpha * pv[i];
          rn[i] -= alpha * ap[i];
          A.r[3 * a + i] = rn[i];
        }
      }
      if (!last) {
        if (PK == 2) {
          if (__ldg(A.diag_only + a)) {
            const long long pb = __ldg(A.pbase + a);
#pragma unroll
            for (int i = 0; i < 3; ++i) zv[i] = __ldg(A.pvals + pb + i) * rn[i];
          }
        } else {
#pragma unroll
          for (int i = 0; i < 3; ++i) zv[i] = PK == 1 ? __ldg(A.dinv + 3 * a + i) * rn[i] : rn[i];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) zv[i] += beta * pv[i];
        store_p(a, zv);
      }
    }
    if (last) break;
    ok = grid_sum(0);
  }
  if (c == 0 && threadIdx.x == 0) {
    CgState* st = A.st;
    if (ok) {
      st->zTr = zTr;
      st->beta = beta;
      st->alpha = alpha;
      st->pAp = pAp;
      st->rr = rr;
      st->iters = iters;
      st->done = done;
      st->status = status;
      st->replace = replace;
    } else {
      st->done = 1;
      st->status = HOEFEM_ERR_DEVICE_TIMEOUT;
      st->replace = 0;
    }
  }
  worker_sync();
  if (threadIdx.x == 0) s_stop = 1;
}

template <class VA, class VB, int PK>
void launch(const Args& args, int G, size_t smem, cudaStream_t s) {
  auto fn = k_pcg<VA, VB, PK>;
  allow_shared(fn, SMEM_BUDGET);
  Args a = args;
  void* kargs[] = {&a};
  note_launch();
  HOEFEM_CUDA(cudaLaunchCooperativeKernel((const void*)fn, G, THREADS, kargs, smem, s));
}

int align16(long long b) { return (int)((b + 15) & ~15LL); }

}  // namespace

// Whether the persistent kernel takes this solve, with its layouts built on
// first use.  It does not take: Schwarz preconditioners applied as an SpMV or
// without blocks, SpMV variants or a Schwarz apply pinned by the caller (the
// graphs, where the two applies differ in nothing else), solves that report every
// chunk of iterations, rows too long for a stage, values not aligned to 16
// bytes (bulk copies), devices without cooperative launch.
bool cg_persist_usable(CgWork& w, const void* vals, bool f32, const Precond* P, bool p32, cudaStream_t s) {
  Model& m = *w.m;
  if (w.on_chunk || m.spmv_pinned || m.nv == 0 || ((uintptr_t)vals & 15)) return false;
  const bool sw = P && P->kind == PREC_SCHWARZ;
  if (sw && (!P->block_apply || P->apply_pinned || P->nsub == 0 || P->max_nodes > PCG_MAX_SUB_NODES)) return false;
  int dev = 0, coop = 0;
  HOEFEM_CUDA(cudaGetDevice(&dev));
  HOEFEM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  const int G = device_sms();
  if (!coop || G > MAX_G) return false;
  PcgOpLayout& L = m.pcg[f32 ? 1 : 0];
  if (L.state == 0) {
    // stages of 8 KB of values or the longest node rows;
    // smaller ones when the matrix has too few tiles for every warp
    const int vsize = f32 ? 4 : 8;
    long long maxrow = 0;
    for (i64 a = 0; a < m.nv; ++a) maxrow = std::max<long long>(maxrow, 9LL * vsize * (m.adj_off[a + 1] - m.adj_off[a]));
    long long cap = std::min<long long>(8192, 9LL * vsize * m.adj_off[m.nv] / ((long long)G * 12));
    cap = std::max<long long>(std::max<long long>(cap, maxrow), 768);
    std::vector<PcgTile> tiles;
    L.state = -1;
    if (cap > 24 * 1024 || !pcg_op_tiles(m.adj_off, m.nv, vsize, cap, 4, tiles, L.max_blk)) return false;
    std::vector<long long> wt(tiles.size());
    for (size_t k = 0; k < tiles.size(); ++k) wt[k] = (9LL * vsize + 4) * tiles[k].nblk + TILE_COST;
    const std::vector<int> off = pcg_ranges(wt, G);
    L.tiles.upload(tiles, s);
    L.cta.upload(off, s);
    HOEFEM_CUDA(cudaStreamSynchronize(s));
    L.cap = cap;
    L.grid = G;
    L.state = 1;
  }
  if (L.state < 0 || L.grid != G) return false;
  if (sw) {
    PcgSwLayout& W = const_cast<Precond*>(P)->pcg[p32 ? 1 : 0];
    if (W.cap != L.cap || W.grid != G) {
      std::vector<PcgSwTile> tiles;
      if (!pcg_sw_tiles(P->sub_off, p32 ? 4 : 8, L.cap, tiles)) return false;
      std::vector<long long> wt(tiles.size());
      for (size_t k = 0; k < tiles.size(); ++k) wt[k] = (long long)(p32 ? 4 : 8) * tiles[k].rows * tiles[k].dim + TILE_COST;
      const std::vector<int> off = pcg_ranges(wt, G);
      W.tiles.upload(tiles, s);
      W.cta.upload(off, s);
      HOEFEM_CUDA(cudaStreamSynchronize(s));
      W.cap = L.cap;
      W.grid = G;
    }
  }
  return true;
}

void cg_persist_iterate(CgWork& w, const void* vals, bool f32, const Precond* P, bool p32, bool reliable,
                        cudaStream_t s) {
  Model& m = *w.m;
  const PcgOpLayout& L = m.pcg[f32 ? 1 : 0];
  const int G = L.grid;
  const int pk = !P ? 0 : (P->kind == PREC_DIAGONAL ? 1 : 2);
  const int vsize = f32 ? 4 : 8;
  Args a{};
  a.vals = vals;
  a.val_limit = (9LL * m.adj_off[m.nv] * vsize) & ~15LL;
  a.adj = m.d_adj.p;
  a.adj_off = m.d_adj_off.p;
  a.tiles = L.tiles.p;
  a.cta_tile = L.cta.p;
  if (pk == 2) {
    const PcgSwLayout& W = P->pcg[p32 ? 1 : 0];
    a.blocks = p32 ? (const void*)P->bsym32.p : (const void*)P->bsym.p;
    a.sub_nodes = P->d_sub_nodes.p;
    a.slot = P->d_npair.p;
    a.sw_tiles = W.tiles.p;
    a.cta_sw = W.cta.p;
    a.pair_off = P->d_npair_off.p;
    a.diag_only = P->d_diag_only.p;
    a.pbase = P->d_base.p;
    a.pvals = P->vals.p;
    a.y = P->ysub.p;
  }
  if (pk == 1) a.dinv = P->diag.p;
  a.x = w.x.p;
  a.r = w.r.p;
  a.z = w.z.p;
  a.p = w.p.p;
  a.Ap = w.Ap.p;
  if (!f32 && w.p64.n < (size_t)(4 * m.nv)) w.p64.alloc(4 * m.nv);
  a.px = f32 ? (void*)w.p32.p : (void*)w.p64.p;
  a.nv = (int)m.nv;
  a.st = w.st.p;
  if (!w.pbar.p) w.pbar.alloc(1);
  if (w.ppart.n < (size_t)(2 * MAX_SUMS * G)) w.ppart.alloc(2 * MAX_SUMS * G);
  if (!w.serr.p) w.serr.alloc(2);
  a.counter = w.pbar.p;
  a.part = w.ppart.p;
  a.err = w.serr.p;
  a.reliable = reliable ? 1 : 0;
  a.chunk = w.chunk;
  a.val_bytes = align16(L.cap + 32);
  a.adj_bytes = std::max(align16(4LL * L.max_blk + 16), IDX_BYTES);
  // as many stages as fit; three quarters of them at work, the rest in flight
  const size_t stage = 32 + IDX_BYTES + a.adj_bytes + a.val_bytes;
  a.stages = (int)std::min<size_t>(MAX_STAGES, SMEM_BUDGET / stage);
  HOEFEM_REQUIRE(a.stages >= 2, HOEFEM_ERR_INVALID_ARGUMENT, "persistent CG: a stage does not fit");
  a.nw = std::min(NWARP, std::max(1, a.stages * 3 / 4));
  const size_t smem = a.stages * stage;
  HOEFEM_CUDA(cudaMemsetAsync(w.pbar.p, 0, sizeof(unsigned), s));
  HOEFEM_CUDA(cudaMemsetAsync(w.serr.p, 0, 2 * sizeof(int), s));
  if (pk == 2) {
    if (!f32) launch<double, double, 2>(a, G, smem, s);
    else if (p32) launch<float, float, 2>(a, G, smem, s);
    else launch<float, double, 2>(a, G, smem, s);
  } else if (pk == 1) {
    if (f32) launch<float, float, 1>(a, G, smem, s);
    else launch<double, double, 1>(a, G, smem, s);
  } else {
    if (f32) launch<float, float, 0>(a, G, smem, s);
    else launch<double, double, 0>(a, G, smem, s);
  }
  HOEFEM_CUDA(cudaGetLastError());
  int herr[2] = {0, 0};
  HOEFEM_CUDA(cudaMemcpyAsync(w.h_st, w.st.p, sizeof(CgState), cudaMemcpyDeviceToHost, s));
  HOEFEM_CUDA(cudaMemcpyAsync(herr, w.serr.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
  HOEFEM_CUDA(cudaStreamSynchronize(s));
  if (herr[0]) throw Error(HOEFEM_ERR_DEVICE_TIMEOUT, "persistent CG: device wait ran out");
}

}  // namespace hoefem
