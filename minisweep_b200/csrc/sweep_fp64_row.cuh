// sweep_fp64_row.cuh -- the FP64 sweep kernel as rows of independent warps.
//
// A task (octant, block of group pairs, xy tile, z extent of its region) is
// swept by the 8 compute warps of a CTA, each the owner of one tile row: 4
// cells along x, one group pair, every plane.  A warp walks its row cell by
// cell, plane by plane.  The x face stays in its registers, the z faces of
// its cells in its own shared-memory slots, and the y face goes to the warp
// of the next row through a small ring.  So a warp waits only for its own
// inputs and for the row before it: there is no barrier over the CTA, the
// warps drift apart, and while one waits or solves the other warps keep the
// FP64 pipe busy.
//
// rw = 8, 4 or 2 rows form one pipeline (a tile of 4 x rw cells; 2 or 1 cells
// wide where a region is so narrow that one tile would be all of its row); a
// CTA then holds 1, 2 or 4 pipelines, each on a group pair of its own.
//
// What bounds it: per cell, group pair and octant a warp issues 32 FP64
// tensor-core products (m8n8k4, 16 cycles of the scheduler's FP64 pipe each)
// and 56 FP64 instructions of the solve (2 cycles each): 624 cycles at 16
// moments and 32 angles, 1250 for the two warps of a scheduler; and 3 KB of
// state and 4 KB (1/4 + 1/rw) of faces cross L2.  Measured, 64^3 cells x 64
// groups, ms per sweep on the built-in inputs: 57.6 (rw 8; 2040 cycles per two
// cells, DRAM at 4.9 TB/s), 63.0 (rw 2), the staged kernel 120.2; on random
// inputs 63 to 68 from one card to another.  What got it there from 92:
// the vi / vo copies issued by the compute warps themselves (one warp feeding
// all eight by bulk copies was the bound: 92 -> 81), then a cell body without
// branches, in which the next cell's first product, the solve and the second
// product can be interleaved (81 -> 57; one warp alone 1820 -> 1430 cycles a
// cell).  m16n8k8 products are split into m8n8k4 by the compiler and gain
// nothing.
//
// Roles of the producer warpgroup:
//   tasker    grabs tasks in table order, waits for the tasks they depend on
//             as a whole, lays the octant's matrices out in fragment order
//             and posts the task to the other warps.
//   fetcher   brings the faces entering the tile once the upwind tile's
//             progress covers their plane, one 1-D bulk copy each: lane w the
//             x faces of row w, lane 8 + w the y faces of row w where it is a
//             pipeline's first.
//   publisher follows the rows' plane counts and publishes the task's
//             progress (planes every row has finished) to global memory.
//
// The arithmetic of a cell is that of sweep_fp64_ws.cuh (same lane layout,
// same products in the same order, the same exact 7-operation solve), so the
// two kernels agree bit for bit.  Angles: NT tiles of 8 per pass, so that a
// pass over few angles does not pay for 32.
//
// Every wait is bounded by the launch's time budget: the warp that gives up
// records the error and raises the CTA's quit flag, which ends every other
// wait of the CTA; the fetcher lets its copies land before it leaves.
#pragma once

#include "sweep_fp64_ws.cuh"

namespace msb {

// 8-byte asynchronous copy global -> shared, or zeros when !in
__device__ __forceinline__ void cp_async8_zfill(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 8 : 0)
               : "memory");
}

template <int NM_, int NT>
struct RowCfg {
  static constexpr int W = 4, R = 8;          // cells per row, compute warps
  static constexpr int KS = NM_ / 4;          // k-steps of the first product
  static constexpr int MT = (NM_ + 7) / 8;    // m-tiles of the second product
  static constexpr int NTH = (R + 4) * 32;    // threads
  static constexpr int E = NT * 64;           // doubles per face entry (8 columns x 8 NT angles)
  static constexpr int VSZ = 2 * NM_ * NU;    // doubles of vi (or vo) per cell and group pair
  // input ring of a warp, in cells: 4 x 2 KB at 16 moments; a cell of 8 or 4
  // moments takes less time and less room
  static constexpr int D = NM_ == 16 ? 4 : NM_ == 8 ? 6 : 8;
  // y faces between two rows: up to 6, as far as they fit beside the rest,
  // since the rows do not run evenly (37 x 29 x 41, ne 23, na 45, nm 8: 6.53
  // ms with 3, 6.23 so)
  static constexpr int DY = NT <= 2 ? 6 : NT == 3 ? 5 : NM_ == 16 ? 3 : NM_ == 8 ? 4 : 5;
  static constexpr int NREC = 4;              // task records
  static constexpr int MAT = (KS + MT * 2) * NT * 32;
  static constexpr int SM_ZC = 0;                       // [R][W][E]
  static constexpr int SM_Y = SM_ZC + R * W * E;        // [R][DY][E] ring into row b
  static constexpr int SM_X = SM_Y + R * DY * E;        // [R][E] entering x face
  static constexpr int SM_BND = SM_X + R * E;           // [R][E] boundary flux, without its space factor
  static constexpr int SM_RING = SM_BND + R * E;        // [R][D][vi, vo]
  static constexpr int SM_MAT = SM_RING + R * D * 2 * VSZ;  // [2][MAT]
  static constexpr int SM_BAR = SM_MAT + 2 * MAT;       // xfull[R], xempty[R], yfull[R][DY], yempty[R][DY]
  static constexpr int NBAR = 2 * R + 2 * R * DY;
  static constexpr int SM_REC = SM_BAR + NBAR;          // [NREC] RowRec
  static constexpr int SM_CNT = SM_REC + NREC * 24;     // counters (ints)
  static constexpr int SM_END = SM_CNT + 16;
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)SM_END; }

  // The octant's matrices in fragment order, zero beyond the last angle, by
  // the 8-byte asynchronous copies of one warp.
  static __device__ __forceinline__ void load_matrices(double* mat, const Fp64Prob& Q, int oct, int lane) {
    const size_t as = Q.a_stride ? (size_t)Q.a_stride : (size_t)Q.na;
#pragma unroll 4
    for (int e = lane; e < KS * NT * 32; e += 32) {
      const int tt = (e >> 5) % NT, ks = (e >> 5) / NT;
      const int ia = 8 * tt + (lane >> 2), im = KS * (lane & 3) + ks;
      const bool in = ia < Q.na;
      cp_async8_zfill(&mat[e], &Q.afm[in ? ia + as * (im + (size_t)NM_ * oct) : 0], in);
    }
#pragma unroll 4
    for (int e = lane; e < MT * NT * 2 * 32; e += 32) {
      const int i = (e >> 5) & 1, tt = (e >> 6) % NT, mt = (e >> 6) / NT;
      const int ia = 8 * tt + 2 * (lane & 3) + i, im = 8 * mt + (lane >> 2);
      const bool in = ia < Q.na && im < NM_;
      cp_async8_zfill(&mat[KS * NT * 32 + e], &Q.mfa[in ? im + (size_t)NM_ * (ia + as * oct) : 0], in);
    }
  }
};

// A posted task: the table's record, where it starts in the CTA's count of
// planes, and its problem.
struct RowRec {
  int oct, gp, x0, x1, y0, y1, z0, z1, flags, depx, depy, task, stop, plane0, prob, rw;
  Fp64Prob q;
};
static_assert(sizeof(RowRec) <= 24 * sizeof(double), "task record size");

// Counters in shared memory (ints at SM_CNT).
enum RowCounter {
  RC_PLANES = 0,  // [8] planes warp w has finished, over all tasks
  RC_POSTED = 8,  // tasks posted
  RC_PUBLISHED,   // tasks published complete
  RC_FETCHED,     // tasks the fetcher is done with
  RC_QUIT
};

__device__ __forceinline__ int ld_acquire_cta(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_volatile(const int* p) { return *reinterpret_cast<const volatile int*>(p); }
// Predicated forms: the cell loop stays one basic block, so that the
// tensor-core products can be scheduled among everything else.
__device__ __forceinline__ void cp_async16_p(uint32_t dst, const void* src, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %2, 0;\n @p cp.async.cg.shared.global [%0], [%1], 16;\n}" ::"r"(dst),
               "l"(src), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void sts2_p(uint32_t p, double a, double b, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n @p st.shared.v2.f64 [%0], {%1,%2};\n}" ::"r"(p), "d"(a), "d"(b),
               "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void lds2_p(double& a, double& b, uint32_t p, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n @p ld.shared.v2.f64 {%0,%1}, [%2];\n}"
               : "+d"(a), "+d"(b)
               : "r"(p), "r"((int)on));
}
__device__ __forceinline__ void bar_arrive_p(uint32_t b, bool on) {
  asm volatile(
      "{\n .reg .b64 st;\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n @p mbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n}" ::"r"(b),
      "r"((int)on)
      : "memory");
}
// both phases complete (those asked for)
__device__ __forceinline__ bool bar_test2(uint32_t b0, uint32_t p0, bool on0, uint32_t b1, uint32_t p1, bool on1) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p, q, a, b;\n setp.ne.b32 a, %3, 0;\n setp.ne.b32 b, %6, 0;\n setp.eq.b32 p, %3, 0;\n setp.eq.b32 q, %6, 0;\n"
      " @a mbarrier.test_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
      " @b mbarrier.test_wait.parity.acquire.cta.shared::cta.b64 q, [%4], %5;\n and.pred p, p, q;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(b0), "r"(p0), "r"((int)on0), "r"(b1), "r"(p1), "r"((int)on1)
      : "memory");
  return ok != 0;
}
// as dmma(), free to be scheduled among the surrounding arithmetic
__device__ __forceinline__ void dmma_s(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
// the first product of a sum
__device__ __forceinline__ void dmma_0(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};"
      : "=d"(d[0]), "=d"(d[1])
      : "d"(a), "d"(b), "d"(0.0));
}
// shared memory by 32-bit address
__device__ __forceinline__ void lds2(double& a, double& b, uint32_t p) {
  asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(a), "=d"(b) : "r"(p));
}
__device__ __forceinline__ double lds1(uint32_t p) {
  double a;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(a) : "r"(p));
  return a;
}
__device__ __forceinline__ void sts2(uint32_t p, double a, double b) {
  asm volatile("st.shared.v2.f64 [%0], {%1,%2};" ::"r"(p), "d"(a), "d"(b) : "memory");
}
// Bounded wait of a whole warp until the phases of up to two mbarriers
// (address 0: none) are complete, asleep in hardware meanwhile, up to about 2
// us at a time; false once the CTA quits (all lanes agree).
static __device__ __noinline__ bool row_wait(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, int* cnt,
                                             SyncArgs s) {
  long long t0 = 0;
  for (;;) {
    const bool ok = (!b0 || bar_try(b0, p0, 2000)) && (!b1 || bar_try(b1, p1, 2000));
    if (__all_sync(0xffffffffu, ok)) return true;
    bool give_up = ld_volatile(cnt + RC_QUIT) != 0;
    if (!give_up) {
      const long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > s.timeout_ns) {
        raise_error(s.sync, MSB_ERR_TIMEOUT, -1);
        st_release_cta(cnt + RC_QUIT, 1);
        give_up = true;
      }
    }
    if (__any_sync(0xffffffffu, give_up)) return false;
  }
}

// The same on a shared-memory counter: true once *p >= target.
__device__ __forceinline__ bool row_wait_count(const int* p, int target, int* cnt, const SyncArgs& s, int sleep_ns) {
  long long t0 = 0;
  for (;;) {
    if (__all_sync(0xffffffffu, ld_acquire_cta(p) >= target)) return true;
    bool give_up = ld_volatile(cnt + RC_QUIT) != 0;
    if (!give_up) {
      const long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > s.timeout_ns) {
        raise_error(s.sync, MSB_ERR_TIMEOUT, -1);
        st_release_cta(cnt + RC_QUIT, 1);
        give_up = true;
      }
    }
    if (__any_sync(0xffffffffu, give_up)) return false;
    __nanosleep(sleep_ns);
  }
}

template <class C, bool BATCH, class PP>
__device__ __forceinline__ void row_tasker(const PP& P, int cls, double* smem) {
  const int lane = threadIdx.x & 31;
  int* const cnt = reinterpret_cast<int*>(smem + C::SM_CNT);
  int* const sync = P.sy.sync;
  int* const progress = sync + SY_PROGRESS;
  double* const mats = smem + C::SM_MAT;

  auto wait_dep = [&](const int* p, int target, int task) -> bool {
    if (ld_acquire(p) >= target) return true;
    const long long t0 = global_ns();
    for (;;) {
      __nanosleep(64);
      if (ld_acquire(p) >= target) return true;
      if (ld_relaxed(&sync[SY_ABORT]) != 0 || ld_volatile(cnt + RC_QUIT) != 0) return false;
      if (global_ns() - t0 > P.sy.timeout_ns) {
        raise_error(sync, MSB_ERR_TIMEOUT, task);
        return false;
      }
    }
  };
  // every row has finished `planes` planes
  auto rows_past = [&](int planes) -> bool {
    for (int w = 0; w < C::R; ++w)
      if (!row_wait_count(cnt + RC_PLANES + w, planes, cnt, P.sy, 64)) return false;
    return true;
  };

  int plane0 = 0;  // first plane of the task posted last
  int plane_next = 0;
  int preds_done_for = -1;
  for (int k = 0;; ++k) {
    // A task is taken when row 0 enters the last planes of the one before:
    // early enough to wait for its dependencies and lay out its matrices,
    // late enough that a reserved task does not sit behind a whole other one.
    bool ok = k == 0 || row_wait_count(cnt + RC_PLANES, max(plane_next - 4, plane0), cnt, P.sy, 250);
    // the record and the matrix buffer were last used by tasks k - 4 (by the
    // rows, the publisher and the fetcher) and k - 2
    ok = ok && row_wait_count(cnt + RC_PUBLISHED, k - C::NREC + 1, cnt, P.sy, 64) &&
         row_wait_count(cnt + RC_FETCHED, k - C::NREC + 1, cnt, P.sy, 64) && rows_past(plane0);
    int t = -1;
    if (ok && lane == 0 && ld_relaxed(&sync[SY_ABORT]) == 0) {
      if constexpr (BATCH) {
        const long long tt = atomicAdd(&sync[SY_CLASS0 + cls], 1);
        t = tt < P.cls_ntask[cls] ? (int)(P.cls_base[cls] + tt) : -1;
      } else {
        const long long tt = atomicAdd(&sync[SY_COUNTER], 1);
        t = tt < P.ntask ? (int)tt : -1;
      }
    }
    t = __shfl_sync(0xffffffffu, t, 0);
    RowRec* const rec = reinterpret_cast<RowRec*>(smem + C::SM_REC) + (k % C::NREC);
    if (t < 0) {
      if (!ok) {
        if (lane == 0) st_release_cta(cnt + RC_QUIT, 1);
        return;
      }
      if (lane == 0) {
        rec->stop = 1;
        st_release_cta(cnt + RC_POSTED, k + 1);
      }
      return;
    }
    const int rl = lane < MSB_TASK_INTS ? __ldg(&P.tasks[(size_t)t * MSB_TASK_INTS + lane]) : 0;
    int r[MSB_TASK_INTS];
#pragma unroll
    for (int f = 0; f < MSB_TASK_INTS; ++f) r[f] = __shfl_sync(0xffffffffu, rl, f);
    const int mode = r[TK_DEP_MODE], oct = r[TK_OCT];
    Fp64Prob Q;
    int prob = 0;
    if constexpr (BATCH) {
      prob = __ldg(&P.task_prob[t]);
      Q = P.probs[prob];
      if (P.dir) {
        const double* a = Q.vi;
        Q.vi = Q.vo;
        Q.vo = const_cast<double*>(a);
      }
      // the face scratch is free once its previous users completed
      if (prob != preds_done_for) {
        for (int e = __ldg(&P.pred_off[prob]), ee = __ldg(&P.pred_off[prob + 1]); e < ee && ok; ++e) {
          const int q2 = __ldg(&P.pred[e]);
          ok = wait_dep(&P.pdone[q2], __ldg(&P.prob_ntask[q2]), t);
        }
        preds_done_for = prob;
      }
    } else {
      Q = P.pr;
    }
    // the octant's matrices; their copies are in flight while the
    // dependencies are waited for
    C::load_matrices(mats + (k & 1) * C::MAT, Q, oct, lane);
    cp_async_commit();
    const int depx = (mode & DM_X_PLANE) ? r[TK_DEP_X] : -1;
    const int depy = (mode & DM_Y_PLANE) ? r[TK_DEP_Y] : -1;
    // tasks of other phases, complete: one dependency per lane
    int dep = -1;
    if (lane == 0 && depx < 0) dep = r[TK_DEP_X];
    if (lane == 1 && depy < 0) dep = r[TK_DEP_Y];
    if (lane == 2) dep = r[TK_DEP_Z];
    if (lane == 3) dep = r[TK_DEP_VO];
    if (ok && dep >= 0) ok = wait_dep(&progress[dep], kComplete, t);
    __syncwarp();
    cp_async_wait<0>();
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) st_release_cta(cnt + RC_QUIT, 1);
      return;
    }
    plane0 = plane_next;
    plane_next += r[TK_Z1] - r[TK_Z0];
    if (lane == 0) {
      rec->oct = oct; rec->gp = r[TK_GP];
      rec->x0 = r[TK_X0]; rec->x1 = r[TK_X1]; rec->y0 = r[TK_Y0]; rec->y1 = r[TK_Y1];
      rec->z0 = r[TK_Z0]; rec->z1 = r[TK_Z1];
      rec->flags = r[TK_FLAGS]; rec->depx = depx; rec->depy = depy;
      rec->task = t; rec->stop = 0; rec->plane0 = plane0; rec->prob = prob;
      rec->rw = Q.rw;
      rec->q = Q;
    }
    __syncwarp();
    if (lane == 0) st_release_cta(cnt + RC_POSTED, k + 1);
  }
}

template <class C, bool BATCH, class PP>
__device__ __forceinline__ void row_fetcher(const PP& P, double* smem) {
  constexpr int E = C::E, DY = C::DY, R = C::R;
  const int lane = threadIdx.x & 31;
  int* const cnt = reinterpret_cast<int*>(smem + C::SM_CNT);
  int* const sync = P.sy.sync;
  const int* const progress = sync + SY_PROGRESS;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + C::SM_BAR);

  const bool is_x = lane < R, is_y = lane >= R && lane < 2 * R;
  const int wrp = lane % R;  // the compute warp this lane feeds
  const int depth = is_x ? 1 : DY;
  uint64_t* const full = is_x ? bars + wrp : bars + 2 * R + wrp * DY;
  uint64_t* const empty = full + (is_x ? R : R * DY);
  double* const dst = smem + (is_x ? C::SM_X + wrp * E : C::SM_Y + wrp * DY * E);

  bool live = is_x || is_y, have = false;
  int k = 0;           // task
  int a = 0, c = 0;    // next face: position in the row (y), plane
  int w = 0, nzr = 0, dep = -1;
  int F = 0;           // faces the ring has taken
  int own[2] = {0, 0}, prev[2] = {0, 0};  // those this lane copied itself: its last run, the one before
  int seen = 0;        // upwind planes seen complete
  long long t0 = 0;    // start of the present wait for the upwind tile
  bool fail = false, handed = false;  // handed: the row before filled the ring since this lane last did
  int plane0 = 0;
  const char* src = nullptr;
  long long fa = 0, fc = 0;  // byte strides
  bool was_live = live;
  int done_upto = 0, k_seen = 0;  // tasks every lane is past; this lane's task last time
  for (;;) {
    bool moved = false;
    if (live && !have && ld_acquire_cta(cnt + RC_POSTED) > k) {
      const RowRec& rec = reinterpret_cast<const RowRec*>(smem + C::SM_REC)[k % C::NREC];
      moved = true;
      if (rec.stop) {
        live = false;
      } else {
        const Fp64Prob& Q = rec.q;
        const int row = wrp % rec.rw, gp = rec.gp * (R / rec.rw) + wrp / rec.rw;
        const int oct = rec.oct, flags = rec.flags;
        const bool runs = row < rec.y1 - rec.y0 && gp < Q.ngp;  // the warp takes part in the task
        if (!runs || (is_x ? !(flags & TF_X_IN) : row > 0 || !(flags & TF_Y_IN))) {
          // the row before it fills the warp's y ring in this task
          if (runs && is_y && row > 0) {
            F += (rec.x1 - rec.x0) * (rec.z1 - rec.z0);
            handed = true;
          }
          ++k;
        } else {
          have = true;
          const int dx = (oct & 1) ? -1 : 1, dy = (oct & 2) ? -1 : 1, dz = (oct & 4) ? -1 : 1;
          w = is_x ? 1 : rec.x1 - rec.x0;  // faces per plane
          nzr = rec.z1 - rec.z0;
          a = c = 0;
          seen = 0;
          prev[0] = own[0];
          prev[1] = own[1];
          own[0] = F;
          plane0 = rec.plane0;
          const int ix = dx > 0 ? rec.x0 : rec.x1 - 1, iz = dz > 0 ? rec.z0 : rec.z1 - 1;
          const int iy = dy > 0 ? rec.y0 + row : rec.y1 - 1 - row;
          const long long ent = (long long)oct * Q.ngp + gp;
          fence_proxy_async();  // what the tasker's acquires cover, for the copies
          dep = is_x ? rec.depx : rec.depy;
          src = reinterpret_cast<const char*>(is_x ? Q.fyz + ((ent * Q.nz + iz) * Q.ny + iy) * E
                                                   : Q.fxz + ((ent * Q.nz + iz) * Q.nx + ix) * E);
          fa = (long long)dx * E * 8;
          fc = is_x ? (long long)dz * Q.ny * E * 8 : (long long)dz * Q.nx * E * 8 - (w - 1) * fa;
        }
      }
    }
    if (live && have) {
      // A ring that changes its producer may be many phases behind F, where
      // the parity says nothing: first let the warp finish the earlier tasks.
      // Its faces were ordinary stores; the next ones are bulk copies.
      if (handed && ld_acquire_cta(cnt + RC_PLANES + wrp) >= plane0) {
        fence_proxy_async_smem();
        handed = false;
      }
      bool go = !handed && (F < depth || mbar_test_wait(&empty[F % depth], (uint32_t)((F / depth + 1) & 1)));
      if (go && dep >= 0 && seen < c + 1) {
        seen = ld_acquire(progress + dep);
        if (seen < c + 1) {
          go = false;
          const long long t = global_ns();
          if (t0 == 0) t0 = t;
          if (ld_relaxed(&sync[SY_ABORT]) != 0) {
            fail = true;
          } else if (t - t0 > P.sy.timeout_ns) {
            raise_error(sync, MSB_ERR_TIMEOUT, -1);
            fail = true;
          }
        } else {
          fence_proxy_async();
        }
      }
      if (go) {
        moved = true;
        t0 = 0;
        uint64_t* const bar = &full[F % depth];
        mbar_arrive_expect_tx(bar, E * 8);
        bulk_g2s(dst + (F % depth) * E, src, E * 8, bar);
        own[1] = ++F;
        src += fa;
        if (++a == w) {
          a = 0;
          src += fc - fa;  // fc: from a plane's last face to the next plane's first
          if (++c == nzr) {
            have = false;
            ++k;
          }
        }
      }
    }
    // one vote for what the lanes did: the loop's length is the fetcher's
    // latency, which rows of 4 and 8 moments feel (37 x 29 x 41, nm 8: 6.23 ms
    // with three votes and no count of tasks, 6.36 with a count every time)
    const unsigned did = __reduce_or_sync(0xffffffffu, (moved ? 1u : 0u) | (live ? 2u : 0u) | (fail ? 4u : 0u) |
                                                           (k != k_seen || was_live != live ? 8u : 0u));
    k_seen = k;
    was_live = live;
    if (did & 8u) {
      __syncwarp();  // what every lane read of the records it is past, before lane 0 gives them back
      const int past = __reduce_min_sync(0xffffffffu, live ? k : 0x7fffffff);
      if (lane == 0 && past != done_upto) st_release_cta(cnt + RC_FETCHED, past);
      done_upto = past;
    }
    if (did & 4u) {
      if (lane == 0) st_release_cta(cnt + RC_QUIT, 1);
      break;
    }
    if (!(did & 2u)) break;
    if (!(did & 1u)) {
      if (ld_volatile(cnt + RC_QUIT) != 0) break;
      __nanosleep(40);
    }
    __syncwarp();
  }
  __syncwarp();
  // After an early end the compute warps may not have waited for every copy:
  // let them land before the shared memory is reused or released
  // (microseconds; the bound is 1 ms).
  if (ld_volatile(cnt + RC_QUIT) != 0) {
    const long long t1 = global_ns();
    for (int i = 0; i < 2; ++i) {
      const int lo = i ? own[0] : prev[0], hi = i ? own[1] : prev[1];
      for (int n = max(lo, hi - depth); n < hi; ++n)
        while (!mbar_test_wait(&full[n % depth], (uint32_t)((n / depth) & 1)) && global_ns() - t1 < 1000000) {
        }
    }
  }
  __syncwarp();
}

template <class C, bool BATCH, class PP>
__device__ __forceinline__ void row_publisher(const PP& P, double* smem) {
  const int lane = threadIdx.x & 31;
  int* const cnt = reinterpret_cast<int*>(smem + C::SM_CNT);
  int* const progress = P.sy.sync + SY_PROGRESS;
  for (int k = 0;; ++k) {
    if (!row_wait_count(cnt + RC_POSTED, k + 1, cnt, P.sy, 100)) return;
    const RowRec& rec = reinterpret_cast<const RowRec*>(smem + C::SM_REC)[k % C::NREC];
    if (rec.stop) return;
    const int nzr = rec.z1 - rec.z0, plane0 = rec.plane0, task = rec.task;
    // somebody follows this tile plane by plane
    const bool by_plane = (rec.flags & (TF_X_OUT | TF_Y_OUT)) != 0;
    int last = 0;
    long long t0 = 0;
    for (;;) {
      const int mine = lane < C::R ? ld_acquire_cta(cnt + RC_PLANES + lane) : 0x7fffffff;
      const int v = __reduce_min_sync(0xffffffffu, mine) - plane0;
      if (v >= nzr || (by_plane && v > last)) {
        __threadfence();
        __syncwarp();
        if (lane == 0) st_release(&progress[task], v >= nzr ? kComplete : v);
        last = v;
        t0 = 0;
        if (v >= nzr) break;
        continue;
      }
      bool give_up = ld_volatile(cnt + RC_QUIT) != 0;
      if (!give_up) {
        const long long t = global_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > P.sy.timeout_ns) {
          if (lane == 0) raise_error(P.sy.sync, MSB_ERR_TIMEOUT, task);
          st_release_cta(cnt + RC_QUIT, 1);
          give_up = true;
        }
      }
      if (__any_sync(0xffffffffu, give_up)) return;
      __nanosleep(200);
    }
    if constexpr (BATCH) {
      if (lane == 0) {
        const int pr = rec.prob;
        if (atom_add_release(&P.pdone[pr], 1) + 1 == __ldg(&P.prob_ntask[pr])) P.ptime[pr] = global_ns();
      }
    }
    __syncwarp();
    if (lane == 0) st_release_cta(cnt + RC_PUBLISHED, k + 1);
  }
}

// Which of a task's warps a compute warp of the CTA is.  A scheduler holds the
// warps w and w + 4.  Where a pipeline of 4 or 2 rows uses half of them at
// most (SPARE), the rows in use (rows 0, or 0 and 1, of each pipeline) are put
// on different schedulers: 8 x 2 x 96, ne 32, two pipelines of one row, 788 us
// instead of 1014.  With more rows in use the plain order is the better one
// (47 x 6 x 9, ne 77, 3 rows of 4, mixed: 1.04 ms, 1.13 so).  A constant of the
// kernel, and the shuffle last, which tells the compiler that the number is
// the warp's: 64^3 x 64 took 59.7 ms instead of 57.6 with arithmetic behind it.
template <bool SPARE>
__device__ __forceinline__ int row_warp() {
  const int w = threadIdx.x >> 5;
  return __shfl_sync(0xffffffffu, SPARE ? (0x54672310 >> (4 * w)) & 7 : w, 0);
}

// One compute warp: row `warp % rw` of pipeline `warp / rw` of each task.
template <int NM_, int NT, bool BATCH, bool SPARE, class PP>
__device__ __forceinline__ void row_compute(const PP& P, double* smem) {
  using C = RowCfg<NM_, NT>;
  constexpr int E = C::E, VSZ = C::VSZ, W = C::W, D = C::D, DY = C::DY, R = C::R, KS = C::KS, MT = C::MT;
  const int lane = threadIdx.x & 31, warp = row_warp<SPARE>();
  const int q = lane >> 2, r = lane & 3;
  int* const cnt = reinterpret_cast<int*>(smem + C::SM_CNT);
  // shared-memory addresses of this warp's barriers, rings and face slots
  const uint32_t sb = smem_u32(smem);
  const uint32_t xfull = sb + 8 * (C::SM_BAR + warp), xempty = xfull + 8 * R;
  const uint32_t yfull = sb + 8 * (C::SM_BAR + 2 * R + warp * DY), yempty = yfull + 8 * R * DY;
  const uint32_t y_in_ring = sb + 8 * (C::SM_Y + warp * DY * E) + 16 * lane, y_out_ring = y_in_ring + 8 * DY * E;
  const uint32_t zc = sb + 8 * (C::SM_ZC + warp * W * E) + 16 * lane;
  const uint32_t xin = sb + 8 * (C::SM_X + warp * E) + 16 * lane, bnd = sb + 8 * (C::SM_BND + warp * E) + 16 * lane;
  // this lane's column: unknown q & 3 of group q >> 2; its vi fragment
  // (moments KS r + ks) and vo values (moments 8 mt + 2 r + i)
  const uint32_t col = 8 * ((q >> 2) * (VSZ / 2) + NM_ * (q & 3));
  const uint32_t ring = sb + 8 * (C::SM_RING + warp * D * 2 * VSZ);
  double wz[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) wz[i] = 1.0 / 4.0 - 1.0 / (double)(1 << (2 * r + i));

  uint32_t x_ph = 0;                              // phase of the entering x face
  // y rings, this warp's (in) and the next warp's (out): positions and phases
  // (an empty slot's phase lags by one)
  uint32_t yi = 0, yi_ph = 0, yo = 0, yo_ph = 1;
  // A batch changes the pipeline height from task to task, and with it who
  // fills a ring: it counts the faces that passed through each in earlier tasks.
  bool handed = false;  // the fetcher filled the next warp's ring since this warp last did
  uint32_t n_in = 0, n_out = 0;
  int rw = 8, row = 0, pipe = 0;
  if constexpr (!BATCH) {
    rw = P.pr.rw;
    row = warp % rw;
    pipe = warp / rw;
  }
  for (int k = 0;; ++k) {
    if (!row_wait_count(cnt + RC_POSTED, k + 1, cnt, P.sy, 64)) return;
    const RowRec& rec = reinterpret_cast<const RowRec*>(smem + C::SM_REC)[k % C::NREC];
    if (rec.stop) return;
    if constexpr (BATCH) {
      rw = rec.rw;
      row = warp % rw;
      pipe = warp / rw;
    }
    const int oct = rec.oct, flags = rec.flags, gp = rec.gp * (R / rw) + pipe;
    const Fp64Prob& Q = rec.q;
    const int w = rec.x1 - rec.x0, h = rec.y1 - rec.y0, nzr = rec.z1 - rec.z0;
    const bool runs = row < h && gp < Q.ngp;
    if constexpr (BATCH) {
      yi = n_in % DY;
      yi_ph = (n_in / DY) & 1;
      yo = n_out % DY;
      yo_ph = (n_out / DY + 1) & 1;
      const bool passes = runs && row + 1 < h;
      if (runs && (row > 0 || (flags & TF_Y_IN))) n_in += w * nzr;
      // the next warp's ring also takes faces where that warp begins a pipeline
      // and the fetcher feeds it
      const int gp2 = rec.gp * (R / rw) + (warp + 1) / rw;
      const bool fetched = (warp + 1) % rw == 0 && gp2 < Q.ngp && (flags & TF_Y_IN);
      if (passes || fetched) n_out += w * nzr;
      if (passes && handed) {  // as in the fetcher: a ring that changes its producer
        if (!row_wait_count(cnt + RC_PLANES + warp + 1, rec.plane0, cnt, P.sy, 64)) return;
        handed = false;
      }
      if (fetched) handed = true;
    }
    if (!runs) {
      __syncwarp();
      if (lane == 0) st_release_cta(cnt + RC_PLANES + warp, rec.plane0 + nzr);
      continue;
    }
    const bool y_feed = row > 0 || (flags & TF_Y_IN);  // the y face comes through the ring
    const bool y_pass = row + 1 < h;                   // ... and goes on through the next one
    const int dx = (oct & 1) ? -1 : 1, dy = (oct & 2) ? -1 : 1, dz = (oct & 4) ? -1 : 1;
    const bool first = (flags & TF_FIRST) != 0 && !Q.vo_add;
    const int ix0 = dx > 0 ? rec.x0 : rec.x1 - 1, iz0 = dz > 0 ? rec.z0 : rec.z1 - 1;
    const int iy = dy > 0 ? rec.y0 + row : rec.y1 - 1 - row;
    const int g_col = 2 * gp + (q >> 2);  // the lane's group
    const bool gval = g_col < Q.ne;
    const double so = (double)(1 + oct);
    const double so_r = 1.0 / so;  // rounded, as the reference's 1/(1+octant)
    int sp0 = ix0 + 3 * iy + 7 * iz0 + 2 + Q.sp_off;  // log2 s_space of the row's first cell, mod 4
    const bool y_out = !y_pass && (flags & TF_Y_OUT);
    const bool x_in = (flags & TF_X_IN) != 0, z_in = (flags & TF_Z_IN) != 0;
    const bool x_out = (flags & TF_X_OUT) != 0, z_out = (flags & TF_Z_OUT) != 0;
    // Boundary flux (1+ia) 2^(ia&7) s_space s_energy s_unknown (1+oct): exact
    // small integers.  The entry leaves out s_space, whose power of two the
    // solve's coefficient cancels.
    {
      const double face_k =
          gval ? (double)d_scale_energy(Q.ie_base + g_col) * (double)d_scale_unknown(q & 3) * so : 0.0;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        double f[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int ia = 8 * t + 2 * r + i, iag = Q.ia_base + ia;
          f[i] = ia < Q.na ? (double)((1 + iag) << (iag & 7)) * face_k : 0.0;
        }
        sts2(bnd + t * 512, f[0], f[1]);
      }
    }
    // this row's matrices
    double b1r[KS][NT], a2r[MT][NT][2];
    {
      const uint32_t mat = sb + 8 * (C::SM_MAT + (k & 1) * C::MAT + lane);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int t = 0; t < NT; ++t) b1r[ks][t] = lds1(mat + 256 * (ks * NT + t));
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i) a2r[mt][t][i] = lds1(mat + 256 * (KS * NT + (mt * NT + t) * 2 + i));
    }
    const size_t slab = (size_t)NM_ * NU * Q.nx * Q.ny;
    double* vdst = Q.vo + (size_t)NM_ * NU * (ix0 + (size_t)Q.nx * iy) + slab * (size_t)g_col +
                   slab * Q.ne * (size_t)iz0 + NM_ * (q & 3) + 2 * r;
    const long long vda = (long long)dx * NM_ * NU, vdc = (long long)dz * slab * Q.ne - w * vda;
    // This warp's own copies, 16 bytes a lane: vi and the previous vo of cell
    // n + D - 1 are issued at cell n; the entering z faces of the row here.
    constexpr int UNITS = 4 * NM_;  // 16-byte units of a cell's vi: 2 groups
    const int u_g = NM_ == 16 ? 0 : lane / (2 * NM_);
    const bool cp0 = lane < UNITS && 2 * gp + u_g < Q.ne, cp1 = NM_ == 16 && 2 * gp + 1 < Q.ne;
    const char* cpi = reinterpret_cast<const char*>(Q.vi) +
                      ((size_t)NM_ * NU * (ix0 + (size_t)Q.nx * iy) + slab * (2 * (size_t)gp + u_g) +
                       slab * Q.ne * (size_t)iz0) * 8 + 16 * (NM_ == 16 ? lane : lane % (2 * NM_));
    const long long cpo = reinterpret_cast<const char*>(Q.vo) - reinterpret_cast<const char*>(Q.vi);
    const long long cpg = (long long)slab * 8;  // to the second group
    int pa = 0, pleft = nzr * w;                // the next copy's position in the row; copies left
    uint32_t pslot = 0, pdst = ring + 16 * lane;
    auto prefetch = [&]() {
      const bool on = pleft > 0;
      cp_async16_p(pdst, cpi, on && cp0);
      cp_async16_p(pdst + 8 * VSZ, cpi + cpo, on && cp0 && !first);
      if constexpr (NM_ == 16) {
        cp_async16_p(pdst + 4 * VSZ, cpi + cpg, on && cp1);
        cp_async16_p(pdst + 12 * VSZ, cpi + cpo + cpg, on && cp1 && !first);
      }
      cp_async_commit();
      --pleft;
      ++pa;
      cpi += vda * 8 + (pa == w ? vdc * 8 : 0);
      pa = pa == w ? 0 : pa;
      ++pslot;
      pdst += pslot == D ? 16 * VSZ - 16 * VSZ * D : 16 * VSZ;
      pslot = pslot == D ? 0 : pslot;
    };
    const size_t ent = (size_t)oct * Q.ngp + gp;
    if (z_in) {
      const double* f = Q.fxy + ((ent * Q.ny + iy) * Q.nx + ix0) * (size_t)E + 2 * lane;
      for (int a = 0; a < w; ++a, f += dx * E)
#pragma unroll
        for (int t = 0; t < NT; ++t) cp_async16_s(zc + a * (8 * E) + t * 512, f + t * 64);
    }
#pragma unroll
    for (int i = 0; i < D - 1; ++i) prefetch();

    // moments of the cell in ring slot sl (of a group beyond the last one: whatever is there, nobody reads it)
    auto load_vi = [&](double (&vf)[KS], uint32_t sl) {
      const uint32_t in = ring + sl * (16 * VSZ) + col + 8 * KS * r;
      if constexpr (KS == 1) {
        vf[0] = lds1(in);
      } else {
#pragma unroll
        for (int ks = 0; ks < KS; ks += 2) lds2(vf[ks], vf[ks + 1], in + 8 * ks);
      }
    };
    // moments -> angles of the task's first cell; every other cell's runs
    // beside the solve of the one before
    double d1[NT][2];
    {
      cp_async_wait<D - 2>();
      __syncwarp();
      double vf[KS];
      load_vi(vf, 0);
#pragma unroll
      for (int t = 0; t < NT; ++t) dmma_0(d1[t], vf[0], b1r[0][t]);
#pragma unroll
      for (int ks = 1; ks < KS; ++ks)
#pragma unroll
        for (int t = 0; t < NT; ++t) dmma_s(d1[t], vf[ks], b1r[ks][t]);
    }

    uint32_t slot = 0;
    uint32_t zmask = z_in ? 3 : 0;  // 0: the z faces are the boundary flux
    const int ymask = y_feed ? 3 : 0;
    const bool vo_lane = gval && (NM_ >= 8 || r < 2);
    // lane 0 hands on the leaving y face, lane 1 gives the entering one's place back
    const bool arr = (lane == 0 && y_pass) || (lane == 1 && y_feed);
    for (int c = 0; c < nzr; ++c) {
      const bool last = c == nzr - 1;
      int sp = sp0;
      uint32_t xmask = 0, za = zc;
      // ---- the entering x face
      double fx[NT][2];
      if (x_in) {
        xmask = 3;
        if (!__all_sync(0xffffffffu, bar_test(xfull, x_ph)) && !row_wait(xfull, x_ph, 0, 0, cnt, P.sy)) {
          cp_async_wait<0>();
          return;
        }
        x_ph ^= 1;
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) lds2(fx[t][0], fx[t][1], (x_in ? xin : bnd) + t * 512);
      if (x_in) {
        __syncwarp();
        if (lane == 0) bar_arrive(xempty);
      }
      for (int a = 0; a < w; ++a) {
        prefetch();
        cp_async_wait<D - 2>();  // this lane's copies for the next cell
        // ---- wait for the entering y face and for room for the leaving one
        const uint32_t yb = yfull + 8 * yi, eb = yempty + 8 * (DY + yo);
        if (!__all_sync(0xffffffffu, bar_test2(yb, yi_ph, y_feed, eb, yo_ph, y_pass)) &&
            !row_wait(y_feed ? yb : 0, yi_ph, y_pass ? eb : 0, yo_ph, cnt, P.sy)) {
          cp_async_wait<0>();
          return;
        }
        __syncwarp();  // every lane's copies
        // ---- entering faces, the previous vo, the next cell's moments (the
        // task's last cell reads a stale slot, whose product nobody uses)
        double fy[NT][2], fz[NT][2], old[MT][2], vf[KS], dn[NT][2];
        const uint32_t py = y_feed ? y_in_ring + yi * (8 * E) : bnd, pz = zmask ? za : bnd;
        const uint32_t in = ring + slot * (16 * VSZ) + col + 8 * (VSZ + 2 * (NM_ < 8 ? r & 1 : r));
        slot = slot == D - 1 ? 0 : slot + 1;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          lds2(fy[t][0], fy[t][1], py + t * 512);
          lds2(fz[t][0], fz[t][1], pz + t * 512);
        }
        load_vi(vf, slot);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          old[mt][0] = old[mt][1] = -0.0;  // x + -0.0 is x, for the first visitor
          lds2_p(old[mt][0], old[mt][1], in + 64 * mt, !first);
        }
        // ---- Quantities_solve, exact 7-operation form (no contraction)
        {
          const double cxy = d_pow2(-1 - (int)((sp - 7 * dz) & zmask));
          const double cxz = d_pow2(-2 - ((sp - 3 * dy) & ymask));
          const double sx_r = d_pow2(-(int)((sp - dx) & xmask));
          const double cyz[2] = {wz[0] * sx_r, wz[1] * sx_r};
          const double cc = so_r * d_pow2(sp & 3);
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const double bxz = __dmul_rn(fy[t][i], cxz);
              const double sab = __fma_rn(fz[t][i], cxy, bxz);  // fz*cxy is exact
              const double cyzv = __dmul_rn(fx[t][i], cyz[i]);
              const double sm = __dadd_rn(sab, cyzv);
              d1[t][i] = __dadd_rn(d1[t][i], __dmul_rn(sm, cc));  // psi
              fx[t][i] = __dmul_rn(d1[t][i], so);
            }
        }
        // ---- leaving faces
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          sts2_p(y_out_ring + yo * (8 * E) + t * 512, fx[t][0], fx[t][1], y_pass);
          sts2(za + t * 512, fx[t][0], fx[t][1]);
        }
        __syncwarp();
        bar_arrive_p(lane == 0 ? yfull + 8 * (DY + yo) : yempty + 8 * yi, arr);
        // ---- angles -> moments (rows: columns of the state; psi is the A
        // operand as is) and moments -> angles of the next cell
        double d2[MT][2][2];  // two accumulators per m-tile (even / odd t)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              if (t < 2 && i == 0) dmma_0(d2[mt][t], d1[t][i], a2r[mt][t][i]);
              else dmma_s(d2[mt][t & 1], d1[t][i], a2r[mt][t][i]);
            }
#pragma unroll
        for (int t = 0; t < NT; ++t) dmma_0(dn[t], vf[0], b1r[0][t]);
#pragma unroll
        for (int ks = 1; ks < KS; ++ks)
#pragma unroll
          for (int t = 0; t < NT; ++t) dmma_s(dn[t], vf[ks], b1r[ks][t]);
        // ---- accumulate vo in the region's visiting order
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          double2 v;
          v.x = __dadd_rn(old[mt][0], NT > 1 ? __dadd_rn(d2[mt][0][0], d2[mt][1][0]) : d2[mt][0][0]);
          v.y = __dadd_rn(old[mt][1], NT > 1 ? __dadd_rn(d2[mt][0][1], d2[mt][1][1]) : d2[mt][0][1]);
          if (vo_lane) *reinterpret_cast<double2*>(vdst + 8 * mt) = v;
        }
        // ---- faces leaving the tile at its y edge and its last plane
        if (y_out || (last && z_out)) {
          const int ix = ix0 + dx * a;
          double* const fo = Q.fxz + ((ent * Q.nz + (iz0 + dz * c)) * Q.nx + ix) * (size_t)E + 2 * lane;
          double* const fz2 = Q.fxy + ((ent * Q.ny + iy) * Q.nx + ix) * (size_t)E + 2 * lane;
          if (y_out)
#pragma unroll
            for (int t = 0; t < NT; ++t) __stcg(reinterpret_cast<double2*>(fo + t * 64), make_double2(fx[t][0], fx[t][1]));
          if (last && z_out)
#pragma unroll
            for (int t = 0; t < NT; ++t) __stcg(reinterpret_cast<double2*>(fz2 + t * 64), make_double2(fx[t][0], fx[t][1]));
        }
        // ---- next cell
#pragma unroll
        for (int t = 0; t < NT; ++t) d1[t][0] = dn[t][0], d1[t][1] = dn[t][1];
        sp += dx;
        xmask = 3;
        za += 8 * E;
        vdst += vda;
        if (y_feed && ++yi == DY) {
          yi = 0;
          yi_ph ^= 1;
        }
        if (y_pass && ++yo == DY) {
          yo = 0;
          yo_ph ^= 1;
        }
      }
      if (x_out) {
        double* const fo = Q.fyz + ((ent * Q.nz + (iz0 + dz * c)) * Q.ny + iy) * (size_t)E + 2 * lane;
#pragma unroll
        for (int t = 0; t < NT; ++t) __stcg(reinterpret_cast<double2*>(fo + t * 64), make_double2(fx[t][0], fx[t][1]));
      }
      sp0 += 7 * dz;
      zmask = 3;
      vdst += vdc;
      __syncwarp();
      if (lane == 0) st_release_cta(cnt + RC_PLANES + warp, rec.plane0 + c + 1);
    }
  }
}

// Barriers and counters of one body: set up before its first task, and
// invalidated before another body reuses the memory.
template <class C>
__device__ __forceinline__ void row_setup(double* smem, bool init) {
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + C::SM_BAR);
  if (init) {
    for (int i = 0; i < C::NBAR; ++i) mbar_init(&bars[i], 1);
    int* const cnt = reinterpret_cast<int*>(smem + C::SM_CNT);
    for (int i = 0; i < 32; ++i) cnt[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  } else {
    for (int i = 0; i < C::NBAR; ++i) mbar_inval(&bars[i]);
  }
}

// The producer warps of one body.
template <class C, bool BATCH, class PP>
__device__ __forceinline__ void row_producers(const PP& P, int cls, double* smem) {
  const int warp = threadIdx.x >> 5;
  if (warp == C::R) row_tasker<C, BATCH>(P, cls, smem);
  else if (warp == C::R + 1) row_fetcher<C, BATCH>(P, smem);
  else if (warp == C::R + 2) row_publisher<C, BATCH>(P, smem);
}

template <int NM_, int NT, bool SPARE>
__global__ void __launch_bounds__(RowCfg<NM_, NT>::NTH, 1) sweep_fp64_row_kernel(const Fp64Params P) {
  using C = RowCfg<NM_, NT>;
  extern __shared__ __align__(128) double smem[];
  if (threadIdx.x == 0) row_setup<C>(smem, true);
  __syncthreads();
  // 384 threads x 168 registers: 8 warps x 32 x 208 + 4 x 32 x 80
  if ((threadIdx.x >> 5) >= C::R) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(80));
    row_producers<C, false>(P, 0, smem);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(208));
    row_compute<NM_, NT, false, SPARE>(P, smem);
  }
}

}  // namespace msb
