// team.cuh -- many MD steps (or one force evaluation) of small systems in one
// launch.
//
// A system of a few thousand atoms fills a step's kernels for 2-10 us each,
// and the captured step of kernels.cuh is then bound by what lies between
// them: launch latencies, tails and the conditional node of the list rebuild
// (measured on one B200: 31 us per step for 4000 Lennard-Jones atoms in FP64,
// 89 us per step for 64 clusters of 147 atoms).  Here a *team* of CTAs keeps
// one system for a whole chunk of steps: the phases of a step are separated
// by a barrier of the team's CTAs only, the rebuild is a branch, and teams of
// different systems never wait for one another.
//
// Each phase runs the per-atom bodies of kernels.cuh with the same lanes per
// atom, so forces, steps, lists and skin decisions are those of the separate
// kernels.  An atom stays with one thread (lane 0 of its K lanes) from the
// force to both half steps, so only neighbours' data crosses a barrier:
//
//   embedded atom  [rho] | [force, step b, step a] | skin test, rebuild?
//   Tersoff        [bonds] | [gather, step b, step a] | skin test, rebuild?
//   LJ             [force, step b, step a] | skin test, rebuild?
//
// ('|': team barrier.  The LJ step needs one barrier only because the
// records it gathers are double-buffered: a step writes the buffer that no
// CTA reads before the next barrier.)
//
// The half steps cost as much as a short list's forces when one lane of K
// does them (Philox, Box-Muller and FP64 chains), so with four lanes or more
// an atom's three coordinates go to three of its lanes.
//
// Two forms, RES=false and true:
//  * arena: all data stay in the arena; a cooperative launch, so every CTA is
//    resident, and a counter in global memory as the barrier, whose wait is
//    bounded.  For systems of a few thousand atoms: one CTA per BLOCK / K
//    atoms over the whole device.
//  * resident: a team is a thread-block cluster with its hardware barrier,
//    and the steps run in shared memory: every CTA holds all atoms' records
//    (two buffers: a step writes the one that nobody gathers from), its own
//    atoms' lists as 16-bit indices and their integrator state; moved records
//    and densities are written to the cluster's other CTAs through
//    distributed shared memory.  Between rebuilds a step touches no global
//    memory, whose latency (a chain of count, list and record loads, each a
//    miss after a barrier) is most of an arena step of so small a system.
#pragma once
#include <cooperative_groups.h>

#include "kernels.cuh"

namespace gg {

enum TKIND : int { TK_LJ64 = 0, TK_LJ32 = 1, TK_SM64 = 2, TK_SM32 = 3, TK_SM32R = 4, TK_TS64 = 5, TK_TS32 = 6 };
// what a launch does before the steps: build the lists, test the skin
// against the positions given by the host, evaluate (and store) the forces
enum TFLAG : int { TF_REBUILD = 1, TF_SKIN = 2, TF_FORCE = 4 };

struct Team {
  int cta0, ncta;  // its CTAs
  int sys;         // its system (-1: none)
  int pad;
};

struct TeamArgs {
  const Team* team;
  const int* cta_team;  // team of each CTA
  unsigned* bar;        // arena form: per team (TEAM_BAR apart), zero at launch; then the abort flag
  int nteam;
  int nsteps;
  int flags;
  int slots;            // CTAs of the launch: stride of the two sets of skin slots
};

constexpr int TEAM_BAR = 32;               // 128 B between the teams' counters
constexpr int TEAM_TILE = 1024;            // candidates staged per cell in the team's list build
constexpr unsigned TEAM_SPINS = 1u << 23;  // polls before a barrier gives up (seconds)

// warps of a CTA that build lists (rows_fit systems): what 60 KB hold
__host__ __device__ constexpr int team_row_warps(int lcap) {
  const int w = (int)(60 * 1024 / rows_warp_bytes(lcap));
  return w < 1 ? 1 : w > BLOCK / 32 ? BLOCK / 32 : w;
}
// shared memory of the rebuild (and of Tersoff's bonds); rows: rows_fit systems
__host__ __device__ constexpr size_t team_smem(int lcap, int ncell, bool rows, size_t tsf) {
  const size_t scan = (size_t)(ncell + 1) * sizeof(int);
  const size_t list = ncell == 0 ? 0
                      : rows       ? team_row_warps(lcap) * rows_warp_bytes(lcap)
                                   : (size_t)TEAM_TILE * sizeof(float4) +
                                         (size_t)LIST_ATOMS * lcap * (sizeof(int) + sizeof(float));
  const size_t a = scan > list ? scan : list;
  return a > tsf ? a : tsf;
}

// The resident form's shared memory, as byte offsets: n atoms, `own` of them
// this CTA's, lists of up to lcap entries.  The rebuild's scratch shares the
// lists' place (they are loaded again after it).
struct ResLayout {
  int rec, recbuf;  // two record buffers, recbuf bytes each
  int eb, band;     // 1/sqrt(rho) of all atoms, rho of the own ones
  int typ;          // species of all atoms (FP64)
  int pos, vel, acel, pos_old, frc, minv, type;
  int cut, nn, row, stride;  // skip counts, entries, list rows (stride 16-bit ids)
  int total;
};
__host__ __device__ constexpr bool team_mixed(int kind) {
  return kind == TK_LJ32 || kind == TK_SM32 || kind == TK_SM32R || kind == TK_TS32;
}
__host__ __device__ inline ResLayout res_layout(int kind, int n, int own, int lcap, int scratch) {
  ResLayout L{};
  const bool mixed = team_mixed(kind), sm = kind == TK_SM64 || kind == TK_SM32 || kind == TK_SM32R;
  int o = 0;
  auto take = [&](int bytes) {
    const int at = o;
    o += (bytes + 15) / 16 * 16;
    return at;
  };
  L.recbuf = n * (mixed ? 16 : 32);
  L.rec = take(2 * L.recbuf);
  L.eb = sm ? take(n * (mixed ? 4 : 8)) : 0;
  L.band = sm ? take(own * 8) : 0;
  L.typ = mixed ? 0 : take(n);
  L.pos = take(own * 32);
  L.vel = take(own * 32);
  L.acel = take(own * 32);
  L.pos_old = take(own * 32);
  L.frc = take(own * 32);  // force, and the pair sum of the energy
  L.minv = take(own * 16);
  L.type = take(own * 4);
  L.cut = take(own * 16);
  L.nn = take(own * 4);
  L.stride = lcap + 2;  // lcap is a multiple of 8: rows of an odd number of words spread over the banks
  const int rows = own * L.stride * 2;
  L.row = take(rows > scratch ? rows : scratch);
  L.total = o;
  return L;
}

struct TeamCtl {
  int rank, ncta;       // this CTA in its team
  unsigned* bar;
  volatile unsigned* abort;
  int* status;          // the current system's status word
  unsigned goal;        // thread 0: arrivals that complete the next barrier
  int parity;           // which set of skin slots the next skin test uses
  int slot0, slots;     // the team's first skin slot, stride of the sets
};

// Barrier of a team's CTAs, with their writes before it visible after it.
// Resident: the cluster's hardware barrier.  Arena: thread 0 arrives with a
// release and polls with an acquire.  False when that wait ran out or another
// CTA gave up: the caller returns at once.
template <bool RES>
__device__ __forceinline__ bool team_sync(TeamCtl& c) {
  if (c.ncta == 1) {
    __syncthreads();
    return true;
  }
  if constexpr (RES) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  } else {
    __shared__ int ok_sh;
    __syncthreads();
    if (threadIdx.x == 0) {
      int ok = 1;
      c.goal += c.ncta;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c.bar) : "memory");
      unsigned n = 0, v;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c.bar) : "memory");
        if ((int)(v - c.goal) >= 0) break;
        if (++n >= TEAM_SPINS || ((n & 255u) == 0u && *c.abort)) {
          *c.abort = 1u;
          atomicOr(c.status, ST_TIMEOUT);
          ok = 0;
          break;
        }
      }
      ok_sh = ok;
    }
    __syncthreads();
    return ok_sh != 0;
  }
}

// p in the shared memory of the team's CTA r (the cluster's CTAs are one team,
// or each its own)
template <class V>
__device__ __forceinline__ V* team_peer(const TeamCtl& c, V* p, int r) {
  return c.ncta == 1 ? p : cooperative_groups::this_cluster().map_shared_rank(p, r);
}

// test_update over the team (skin_close): every CTA merges all partial
// results itself, so the decision needs no second barrier.  step: the test
// closes a half step, so it also advances the step's counters.
template <bool RES>
__device__ __forceinline__ bool team_skin(const Arena& A, TeamCtl& c, const SysDev& S, SysState& st, double2 t,
                                          bool step, int& rb, int& lk) {
  __shared__ int rb_sh, lk_sh;
  __shared__ double2 top_sh[2];
  t = block_top2(t);
  if (c.ncta > 1) {
    // two sets of slots: a CTA may reach the next test while another still
    // reads this one's
    const int par = c.parity;
    c.parity ^= 1;
    double2* slot = A.blk_top2 + par * c.slots + c.slot0;
    if (threadIdx.x == 0) {
      if (RES) top_sh[par] = t;
      else slot[c.rank] = t;
    }
    if (!team_sync<RES>(c)) return false;
    if (threadIdx.x < 32) {
      t = make_double2(1.e-16, 1.e-16);
      for (int b = threadIdx.x; b < c.ncta; b += 32)
        t = top2_merge(t, RES ? *team_peer(c, &top_sh[par], b) : __ldcg(slot + b));
      for (int o = 16; o; o >>= 1) {
        double2 q;
        q.x = __shfl_xor_sync(0xffffffffu, t.x, o);
        q.y = __shfl_xor_sync(0xffffffffu, t.y, o);
        t = top2_merge(t, q);
      }
    }
  }
  if (threadIdx.x == 0) {
    const double D = __dadd_rn(__dadd_rn(__dsqrt_rn(t.x), __dsqrt_rn(t.y)), 0.0);
    rb_sh = D > S.skin;
    st.dmax = D;
    st.rebuild = rb_sh;
    lk_sh = live_band(S, st);
    if (step && S.integ == IT_ERMAK && !S.use_ext_normals) st.step++;
    if (step && S.integ == IT_FIRE) st.fire_zero = 0;
  }
  __syncthreads();
  rb = rb_sh;
  lk = lk_sh;
  return true;
}

// the list update of one system by its team (the chain of launch_rebuild)
template <bool RES>
__device__ __noinline__ bool team_rebuild(const Arena& A, TeamCtl& c, int s, const SysDev& S, SysState& st,
                                          unsigned char* dyn) {
  __shared__ int wsum[BLOCK / 32];
  __shared__ int nb_start[NSTENCIL], nb_pref[NSTENCIL + 1];
  __shared__ double3 nb_sh[NSTENCIL];
  __shared__ int boff_sh[LIST_ATOMS][16];
  const int warp = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const int beg = S.off, end = S.off + S.n;
  const int t0 = c.rank * BLOCK + threadIdx.x, tn = c.ncta * BLOCK;
  const int w0 = c.rank * (BLOCK / 32) + warp, wn = c.ncta * (BLOCK / 32);
  if (S.use_cells) {
    for (int i = beg + t0; i < end; i += tn) {
      const int cid = atom_cell(A, s, S, A.pos[i]);
      A.cell_of[i] = cid;
      A.slot[i] = atomicAdd(&A.cell_count[cid], 1);
    }
    if (!team_sync<RES>(c)) return false;
    // every CTA scans the counts for itself: no further barrier for the prefix
    int* pre = reinterpret_cast<int*>(dyn);
    const int per = (S.ncell + BLOCK - 1) / BLOCK;
    const int k0 = min((int)threadIdx.x * per, S.ncell), k1 = min(k0 + per, S.ncell);
    int sum = 0;
    for (int k = k0; k < k1; k++) sum += __ldcg(&A.cell_count[S.cell_off + k]);
    int inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(FULL, inc, d);
      if (ln >= d) inc += v;
    }
    if (ln == 31) wsum[warp] = inc;
    __syncthreads();
    int run = inc - sum;
    for (int w = 0; w < warp; w++) run += wsum[w];
    for (int k = k0; k < k1; k++) {
      pre[k] = run;
      run += __ldcg(&A.cell_count[S.cell_off + k]);
    }
    if (k0 < S.ncell && k1 == S.ncell) pre[S.ncell] = run;
    __syncthreads();
    for (int i = beg + t0; i < end; i += tn) A.cell_atoms[beg + pre[A.cell_of[i] - S.cell_off] + A.slot[i]] = i;
    if (!team_sync<RES>(c)) return false;
    for (int k = w0; k < S.ncell; k += wn) {
      const int start = beg + pre[k], n = pre[k + 1] - pre[k];
      if (ln == 0) {
        A.cell_start[S.cell_off + k] = start;
        A.cell_n[S.cell_off + k] = n;
        A.cell_count[S.cell_off + k] = 0;
      }
      sort_cell<2>(A, start, n, ln, rows_fit(S, A.lcap));
    }
    if (!team_sync<RES>(c)) return false;
    if (rows_fit(S, A.lcap)) {
      __shared__ RowsFrame f;
      if (threadIdx.x == 0) f = rows_frame(S);
      __syncthreads();
      const int nw = team_row_warps(A.lcap), sp = rows_split(S.n, c.ncta * nw), per = rows_per_warp(sp);
      int* buf = reinterpret_cast<int*>(dyn + (size_t)warp * rows_warp_bytes(A.lcap));
      if (warp < nw)
        for (int p0 = beg + (c.rank + warp * c.ncta) * per; p0 < end; p0 += c.ncta * nw * per) {
          if (sp == 1) list_rows_warp<1>(A, s, S, f, p0, end, buf, ln);
          else if (sp == 3) list_rows_warp<3>(A, s, S, f, p0, end, buf, ln);
          else list_rows_warp<9>(A, s, S, f, p0, end, buf, ln);
        }
    } else {
      // CTA per cell, or up to four CTAs where the team has more CTAs than cells
      float4* cf = reinterpret_cast<float4*>(dyn);
      int* stage = reinterpret_cast<int*>(cf + TEAM_TILE);
      float* stage_rd = reinterpret_cast<float*>(stage + LIST_ATOMS * A.lcap);
      const int np = max(1, min(LIST_SPLIT, c.ncta / S.ncell));
      for (int q = c.rank; q < S.ncell * np; q += c.ncta) {
        const int k = S.cell_off + q / np;
        if (S.list_img)
          list_cells_item<true, TEAM_TILE>(A, s, S, k, k + 1, q % np, np, cf, stage, stage_rd, nb_start, nb_pref, nb_sh,
                                           boff_sh[warp]);
        else
          list_cells_item<false, TEAM_TILE>(A, s, S, k, k + 1, q % np, np, cf, stage, stage_rd, nb_start, nb_pref,
                                            nb_sh, boff_sh[warp]);
      }
    }
  } else {
    // k_list_n2's lists, a warp per atom: 32 candidates at a time, a ballot
    // keeps the accepted ones in index order
    const unsigned lt = (1u << ln) - 1u;
    for (int i = beg + w0; i < end; i += wn) {
      const double4 xi = A.pos[i];
      int m = 0, mh = 0;
      for (int j0 = beg; j0 < end; j0 += 32) {
        const int j = j0 + ln;
        const bool in = j < end && j != i && !(rd_exact(S, xi, A.pos[min(j, end - 1)]) > S.rlist2);
        const bool hin = in && (!S.half || j > i);
        const unsigned b = __ballot_sync(FULL, in), bh = __ballot_sync(FULL, hin);
        const int e = m + __popc(b & lt), eh = mh + __popc(bh & lt);
        if (in && e < A.lcap) A.flist[(size_t)e * A.cap + i] = j;
        if (hin && eh < A.lcap) A.list[(size_t)eh * A.cap + i] = j;
        m += __popc(b);
        mh += __popc(bh);
      }
      if (ln == 0) list_done(A, s, i, m, mh, true);
    }
  }
  if (!team_sync<RES>(c)) return false;
  if (threadIdx.x == 0) {
    st.nupd++;
    st.dmax = 0.0;
    for (int d = 0; d < 3; d++) st.box_b[d] = S.L[d];
    if (c.rank == 0) A.sys_b[s] = S;
  }
  __syncthreads();
  return true;
}

// step_a of one atom (k_step_a's velocity-Verlet, FIRE and Ermak branches,
// Ermak's with w), q its index in X, i in the arena
template <class State>
__device__ __forceinline__ void team_step_a(const Arena& A, const State& X, int q, const SysDev& S, SysState& st,
                                            int i, const double4& F, BaAtom& b) {
  b.x = X.pos[q];
  b.v = X.vel[q];
  const double2 mi = X.minv[q];
  b.ty = X.type[q];
  b.on = true;
  double4 a;
  if (S.integ == IT_ERMAK) {
    a = X.acel[q];
    double4 vv;
    ermak_a_atom(A, S, st, i, mi, b.v, a, b.x, vv);
    b.v.x = ermak_w(S, b.v.x, a.x, vv.x);
    b.v.y = ermak_w(S, b.v.y, a.y, vv.y);
    b.v.z = ermak_w(S, b.v.z, a.z, vv.z);
  } else {
    const double dt = S.integ == IT_FIRE ? st.fire_dt : S.dt;
    if (S.integ == IT_FIRE && st.fire_zero) b.v = make_double4(0, 0, 0, 0);
    vv_a_atom(dt, mi.x, F, b.x, b.v, a);
  }
  wrap_atom(S, b.x);
  b.d = disp2(S, b.x, X.pos_old[q]);
}

// step_b of one atom (k_step_b's branches of the same integrators); P and
// f2: its terms of FIRE's v.F and |F|^2
template <class State>
__device__ __forceinline__ void team_step_b(const State& X, int q, const SysDev& S, const SysState& st,
                                            const double4& F, double& P, double& f2) {
  double4 v = X.vel[q], a = make_double4(0, 0, 0, 0);
  const double om = X.minv[q].x;
  if (S.integ == IT_ERMAK) {
    v.x = ermak_v(S, om, F.x, v.x);
    v.y = ermak_v(S, om, F.y, v.y);
    v.z = ermak_v(S, om, F.z, v.z);
    a.x = F.x * om; a.y = F.y * om; a.z = F.z * om;
  } else {
    vv_b_atom(S.integ == IT_FIRE ? st.fire_dt : S.dt, om, F, v, a);
    if (S.integ == IT_FIRE) fire_mix(st.fire_alpha, F, v, P, f2);
  }
  X.vel[q] = v;
  X.acel[q] = a;
}

template <int KIND>
struct TeamTab {  // species tables in shared memory
  static constexpr bool LJ64 = KIND == TK_LJ64, LJ32 = KIND == TK_LJ32, SM64 = KIND == TK_SM64, SM32 = KIND == TK_SM32;
  using Lj = typename std::conditional<LJ64, LjF64, LjF32>::type;
  using Sm = typename std::conditional<SM64, SmFP64, SmF32>::type;
  typename std::conditional<LJ64 || LJ32, Lj, Sm>::type t[LJ64 || LJ32 || SM64 || SM32 ? MAXT * MAXT : 1];
};

// The resident form's source of lists and records: atoms are numbered within
// the system, the bodies' atom is the bound one
struct SrcShared {
  unsigned char* sh;
  const ResLayout& L;
  const TeamCtl& c;
  const void* rec;   // the record buffer the gathers read
  int lk, lo;        // live_band; the bound atom's index among the CTA's own
  const unsigned short* row;
  template <class V>
  __device__ __forceinline__ V* at(int off) const { return reinterpret_cast<V*>(sh + off); }
  __device__ __forceinline__ int count(int) const {
    const int nn = at<int>(L.nn)[lo];
    if (lk > 7) return nn;
    const unsigned w = reinterpret_cast<const unsigned*>(at<uint4>(L.cut) + lo)[lk >> 1];
    return min(nn, (int)((lk & 1) ? (w >> 16) : (w & 0xffffu)));
  }
  __device__ __forceinline__ int id(int, int m) const { return row[m]; }
  __device__ __forceinline__ int type(int j) const {
    return L.typ ? (int)at<unsigned char>(L.typ)[j] : static_cast<const int4*>(rec)[j].w;
  }
  __device__ __forceinline__ int4 fx(int j) const { return static_cast<const int4*>(rec)[j]; }
  __device__ __forceinline__ int4 fxe(int j) const {
    int4 r = static_cast<const int4*>(rec)[j];
    r.w = __float_as_int(at<float>(L.eb)[j]);
    return r;
  }
  __device__ __forceinline__ double4 x(int j) const { return static_cast<const double4*>(rec)[j]; }
  __device__ __forceinline__ double4 xe(int j) const {
    double4 r = static_cast<const double4*>(rec)[j];
    r.w = at<double>(L.eb)[j];
    return r;
  }
  __device__ __forceinline__ double band(int) const { return at<double>(L.band)[lo]; }
  __device__ __forceinline__ double eb(int i) const { return at<double>(L.eb)[i]; }
  __device__ __forceinline__ float ebf(int i) const { return at<float>(L.eb)[i]; }
  template <class V>
  __device__ __forceinline__ void publish(V* p, V v) const {  // to every CTA of the team
    for (int r = 0; r < c.ncta; r++) *team_peer(c, p, r) = v;
  }
  __device__ __forceinline__ void put_rho64(int i, double band) const {
    at<double>(L.band)[lo] = band;
    publish(at<double>(L.eb) + i, 1.0 / sqrt(band));
  }
  __device__ __forceinline__ void put_rho32(int i, double band) const {
    at<double>(L.band)[lo] = band;
    publish(at<float>(L.eb) + i, (float)(1.0 / sqrt(band)));
  }
};

// where the half steps find an atom's state
template <bool RES>
__device__ __forceinline__ const auto& team_state(const Arena& A, const StateRef& own) {
  if constexpr (RES) return own;
  else return A;
}

template <int KIND, int K, int MINB, bool RES>
__global__ void __launch_bounds__(BLOCK, MINB) k_team(const __grid_constant__ Arena A,
                                                      const __grid_constant__ TeamArgs T) {
  constexpr int APB = BLOCK / K;  // atoms of a virtual block
  constexpr bool TS = KIND == TK_TS64 || KIND == TK_TS32;
  constexpr bool SM = KIND == TK_SM64 || KIND == TK_SM32 || KIND == TK_SM32R;
  constexpr bool MIXED = team_mixed(KIND);
  using R = typename std::conditional<KIND == TK_TS64, double, float>::type;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ SysDev S;
  __shared__ SysState st;
  __shared__ TeamTab<KIND> tab;
  __shared__ double red_sh[2];
  __shared__ ResLayout L;
  const Team tm = T.team[T.cta_team[blockIdx.x]];
  const int s = tm.sys;
  if (s < 0) return;  // a CTA that fills up a cluster of single-CTA teams
  TeamCtl c;
  c.rank = blockIdx.x - tm.cta0;
  c.ncta = tm.ncta;
  c.bar = T.bar + T.cta_team[blockIdx.x] * TEAM_BAR;
  c.abort = T.bar + T.nteam * TEAM_BAR;
  c.status = &A.st[s].status;
  c.goal = 0;
  c.parity = 0;
  c.slot0 = tm.cta0;
  c.slots = T.slots;
  // the atom of this thread in a virtual block: lane 0 of its lanes (Tersoff's
  // gather: one thread per atom)
  const int la = TS ? (int)threadIdx.x : (int)threadIdx.x / K;
  const int lane = threadIdx.x % K;
  const bool own = TS ? threadIdx.x < APB : lane == 0;
  const BlockMap M0{};
  for (int k = threadIdx.x; k < (int)(sizeof(SysDev) / 4); k += BLOCK)
    reinterpret_cast<int*>(&S)[k] = reinterpret_cast<const int*>(A.sys + s)[k];
  for (int k = threadIdx.x; k < (int)(sizeof(SysState) / 4); k += BLOCK)
    reinterpret_cast<int*>(&st)[k] = reinterpret_cast<const int*>(A.st + s)[k];
  __syncthreads();
  const int off = S.off, n = S.n, end = off + n;
  const int nvb = (n + APB - 1) / APB;
  if (threadIdx.x == 0) {
    st.status = 0;  // this CTA's own bits, merged at the end
    if constexpr (RES) L = res_layout(KIND, n, (nvb + c.ncta - 1) / c.ncta * APB, A.lcap, 0);
  }
  if constexpr (KIND == TK_LJ64) ljd_table(A, S, tab.t);
  if constexpr (KIND == TK_LJ32) ljf_table(A, S, tab.t);
  if constexpr (KIND == TK_SM64) sm_table(A, S, tab.t);
  if constexpr (KIND == TK_SM32) smf_table<false>(A, S, tab.t);
  __syncthreads();
  const bool fire = S.integ == IT_FIRE;
  int lk = live_band(S, st);
  // LJ in the arena form: the buffer the gathers read and the one the next
  // step writes (FIRE moves its atoms between two barriers and needs one
  // only).  Mixed: the first of nsteps moves writes fxp if nsteps is odd, so
  // the last one does.  FP64: copies of pos in pose and pose2.
  const bool two = KIND == TK_LJ32 && !RES && !fire;
  constexpr bool TWO64 = KIND == TK_LJ64 && !RES;
  int4* fx_read = A.fxp;
  int4* fx_write = two && !(T.nsteps & 1) ? A.fxe : A.fxp;
  double4* x_read = TWO64 ? A.pose : A.pos;
  int cur = 0;  // resident form: the record buffer the gathers read
  auto swap = [&]() {
    if (RES) cur ^= 1;
    if (TWO64) x_read = x_read == A.pose ? A.pose2 : A.pose;
    if (!two) return;
    fx_read = fx_write;
    fx_write = fx_read == A.fxp ? A.fxe : A.fxp;
  };
  StateRef own_state{};
  if constexpr (RES) {
    auto at = [&](int o) { return dyn + o; };
    own_state.pos = reinterpret_cast<double4*>(at(L.pos));
    own_state.vel = reinterpret_cast<double4*>(at(L.vel));
    own_state.acel = reinterpret_cast<double4*>(at(L.acel));
    own_state.pos_old = reinterpret_cast<double4*>(at(L.pos_old));
    own_state.minv = reinterpret_cast<double2*>(at(L.minv));
    own_state.type = reinterpret_cast<int*>(at(L.type));
  }
  const auto& X = team_state<RES>(A, own_state);
  // resident form: the CTA's own atoms are numbered through its virtual blocks
  const int ncap = (nvb - c.rank + c.ncta - 1) / c.ncta * APB;
  auto atom_of = [&](int lo) { return off + (c.rank + lo / APB * c.ncta) * APB + lo % APB; };
  double4* frc = reinterpret_cast<double4*>(dyn + L.frc);
  // the resident copies: every atom's record (and species), the own atoms' state
  auto load_state = [&]() {
    for (int j = threadIdx.x; j < n; j += BLOCK) {
      if constexpr (MIXED) {
        const int4 r = A.fxp[off + j];
        reinterpret_cast<int4*>(dyn + L.rec)[j] = r;
        reinterpret_cast<int4*>(dyn + L.rec + L.recbuf)[j].w = r.w;
      } else {
        reinterpret_cast<double4*>(dyn + L.rec)[j] = A.pos[off + j];
        (dyn + L.typ)[j] = (unsigned char)A.type[off + j];
      }
    }
    for (int lo = threadIdx.x; lo < ncap; lo += BLOCK) {
      const int i = atom_of(lo);
      if (i < end) {
        X.pos[lo] = A.pos[i];
        X.vel[lo] = A.vel[i];
        X.acel[lo] = A.acel[i];
        frc[lo] = A.force[i];
        X.pos_old[lo] = A.pos_old[i];
        X.minv[lo] = A.minv[i];
        X.type[lo] = A.type[i];
      }
    }
  };
  auto load_lists = [&]() {  // the own atoms' rows, counts and list positions
    for (int vb = c.rank, q = 0; vb < nvb; vb += c.ncta, q++) {
      const int a = threadIdx.x / K, lo = q * APB + a, i = off + vb * APB + a;
      if (i < end) {
        const int nn = min(A.nn[i], A.lcap);
        unsigned short* row = reinterpret_cast<unsigned short*>(dyn + L.row) + lo * L.stride;
        for (int m = lane; m < nn; m += K) {
          const int j = A.flist[(size_t)m * A.cap + i] - off;
          row[m] = (unsigned short)((unsigned)j < (unsigned)n ? j : 0);
        }
        if (lane == 0) {
          reinterpret_cast<int*>(dyn + L.nn)[lo] = nn;
          reinterpret_cast<uint4*>(dyn + L.cut)[lo] = A.ncut[i];
          X.pos_old[lo] = A.pos_old[i];
        }
      }
    }
    __syncthreads();
  };
  if constexpr (RES) {
    load_state();
    if (!(T.flags & TF_REBUILD)) load_lists();
    team_sync<RES>(c);  // the peers' shared memory is ready
  }
  if constexpr (TWO64) {
    for (int vb = c.rank; vb < nvb; vb += c.ncta) {
      const int i = off + vb * APB + la;
      if (own && i < end) A.pose[i] = A.pos[i];
    }
    if ((T.flags & TF_FORCE) && !team_sync<RES>(c)) return;  // (the first skin test is a barrier too)
  }
  SrcArena<false> srcA{A, lk, fx_read, x_read};
  SrcShared srcS{dyn, L, c, nullptr, lk, 0, nullptr};
  // point the source at this step's buffers and the thread's atom
  auto bind = [&](int q) {
    if constexpr (RES) {
      srcS.lk = lk;
      srcS.rec = dyn + L.rec + cur * L.recbuf;
      srcS.lo = q * APB + (int)threadIdx.x / K;
      srcS.row = reinterpret_cast<const unsigned short*>(dyn + L.row) + srcS.lo * L.stride;
    } else {
      srcA.lk = lk;
      srcA.fxp = fx_read;
      srcA.pos = x_read;
    }
  };
  // a moved atom: its state, and its record where the next step's gathers read it
  auto moved = [&](const BaAtom& b, int i, int q) {
    ba_store(X, q, st, b);
    if constexpr (!RES) {
      ba_fx(S, st, i, b, fx_write);
      if constexpr (TWO64) (x_read == A.pose ? A.pose2 : A.pose)[i] = b.x;
    } else {
      if constexpr (MIXED) {
        int4* buf = reinterpret_cast<int4*>(dyn + L.rec + (cur ^ 1) * L.recbuf);
        int bad = 0;
        const int4 r = fx_record(S, b.x, b.ty, bad);
        if (bad) atomicOr(&st.status, ST_LOST);
        srcS.publish(buf + (i - off), r);
      } else {
        srcS.publish(reinterpret_cast<double4*>(dyn + L.rec + (cur ^ 1) * L.recbuf) + (i - off), b.x);
      }
    }
  };
  double2 t = make_double2(1.e-16, 1.e-16);
  double P = 0.0, f2 = 0.0;
  // step b of atom i (q: its index in X), with FIRE's sums
  auto half_b = [&](int i, int q, const double4& F) {
    double p = 0.0, g = 0.0;
    team_step_b(X, q, S, st, F, p, g);
    P += p;
    f2 = fmax(f2, g);
  };
  // step b and the next step a
  auto half_ba = [&](int i, int q, const double4& F) {
    BaAtom b;
    ba_calc(A, X, q, S, st, i, F, b);
    t = top2_merge(t, make_double2(b.d, 1.e-16));
    moved(b, i, q);
  };
  // the same by coordinate: c of W threads (W divides 32) does coordinate c
  auto half_ba_c = [&](int i, int q, int cc, bool act, const double4& F, int W) {
    double d = 0.0;
    if (act && cc < 3) {
      auto comp = [&](const double4* p) { return const_cast<double*>(reinterpret_cast<const double*>(p + q)) + cc; };
      const double Fc = cc == 0 ? F.x : cc == 1 ? F.y : F.z;
      double x = *comp(X.pos), v = *comp(X.vel), a;
      const double2 mi = X.minv[q];
      const double xo = *comp(X.pos_old);
      if (S.integ == IT_VV) {
        vv_b_c(S.dt, mi.x, Fc, v, a);
        vv_a_c(S.dt, mi.x, Fc, x, v, a);
      } else {
        double vv, r0, r1;
        v = ermak_v(S, mi.x, Fc, v);
        a = Fc * mi.x;
        if (S.use_ext_normals) {
          r0 = A.ext_normals[(size_t)6 * i + 2 * cc];
          r1 = A.ext_normals[(size_t)6 * i + 2 * cc + 1];
        } else {
          normals_c((uint32_t)(i - off), st.step, S.seed, cc, r0, r1);
        }
        ermak_a_c(S, mi, r0, r1, v, a, x, vv);
        v = ermak_w(S, v, a, vv);
      }
      wrap_c(S, cc, x);
      d = disp_c(S, cc, x, xo);
      *comp(X.pos) = x;
      *comp(X.vel) = v;
      if (!(d == d)) atomicOr(&st.status, ST_NAN);
      if constexpr (MIXED) {
        int bad = 0;
        const int xf = fx_coord(S, cc, x, bad);
        if (bad) atomicOr(&st.status, ST_LOST);
        if constexpr (RES) {
          int4* buf = reinterpret_cast<int4*>(dyn + L.rec + (cur ^ 1) * L.recbuf);
          srcS.publish(reinterpret_cast<int*>(buf + (i - off)) + cc, xf);
        } else {
          reinterpret_cast<int*>(fx_write + i)[cc] = xf;
          if (cc == 0) fx_write[i].w = X.type[q];
        }
      } else if constexpr (RES) {
        double4* buf = reinterpret_cast<double4*>(dyn + L.rec + (cur ^ 1) * L.recbuf);
        srcS.publish(reinterpret_cast<double*>(buf + (i - off)) + cc, x);
      } else if constexpr (TWO64) {
        reinterpret_cast<double*>((x_read == A.pose ? A.pose2 : A.pose) + i)[cc] = x;
      }
    }
    const double d0 = __shfl_sync(0xffffffffu, d, 0, W), d1 = __shfl_sync(0xffffffffu, d, 1, W),
                 d2 = __shfl_sync(0xffffffffu, d, 2, W);
    if (act && cc == 0) t = top2_merge(t, make_double2(__dadd_rn(__dadd_rn(d0, d1), d2), 1.e-16));
  };
  int rb = (T.flags & TF_REBUILD) != 0;
  const bool opening = (T.flags & TF_FORCE) != 0;
  const bool steps = T.nsteps > 0 && !(fire && st.fire_done);
  // k = -1: the opening evaluation; k >= 0: step k, whose first half step
  // was made by step k - 1 (not FIRE's, nor step 0's)
  for (int k = opening ? -1 : 0; k < (steps ? T.nsteps : 0); k++) {
    const bool last = k == T.nsteps - 1;
    const bool half_a = k == 0 || (fire && k > 0);
    bool test = k >= 0;
    if (half_a) {
      t = make_double2(1.e-16, 1.e-16);
      auto step_a = [&](int i, int q, const double4& F) {
        BaAtom b;
        team_step_a(A, X, q, S, st, i, F, b);
        t = top2_merge(t, make_double2(b.d, 1.e-16));
        moved(b, i, q);
      };
      if constexpr (RES) {
        for (int lo = threadIdx.x; lo < ncap; lo += BLOCK)
          if (atom_of(lo) < end) step_a(atom_of(lo), lo, frc[lo]);
      } else {
        for (int vb = c.rank; vb < nvb; vb += c.ncta) {
          const int i = off + vb * APB + la;
          if (own && i < end) step_a(i, i, A.force[i]);
        }
      }
      swap();
    } else if (k < 0 && (T.flags & TF_SKIN)) {
      for (int i = off + c.rank * BLOCK + threadIdx.x; i < end; i += c.ncta * BLOCK)
        t = top2_merge(t, make_double2(disp2(S, A.pos[i], A.pos_old[i]), 1.e-16));
      test = true;
    }
    if (test && !team_skin<RES>(A, c, S, st, t, k >= 0, rb, lk)) return;
    if (rb) {
      if constexpr (RES) {
        if (k >= 0) {  // the rebuild reads the arena
          for (int lo = threadIdx.x; lo < ncap; lo += BLOCK)
            if (atom_of(lo) < end) A.pos[atom_of(lo)] = X.pos[lo];
          if (!team_sync<RES>(c)) return;
        }
      }
      if (!team_rebuild<RES>(A, c, s, S, st, dyn + (RES ? L.row : 0))) return;
      if constexpr (RES) load_lists();
      if constexpr (TS) {
        // reverse slots of this CTA's own atoms (k_tsf_rslot)
        for (int vb = c.rank; vb < nvb; vb += c.ncta) {
          const int i = off + vb * APB + (int)threadIdx.x / K;
          if (i < end) tsf_rslot_row(A, i, lane, K);
        }
        __syncthreads();
      }
      lk = live_band(S, st);
    }
    // densities, or Tersoff's bonds, up to the barrier that publishes them
    if constexpr (SM || TS) {
      for (int vb = c.rank, q = 0; vb < nvb; vb += c.ncta, q++) {
        const int first = off + vb * APB;
        if constexpr (TS) {
          __syncthreads();
          tsf_bonds_body<R, K>(A, s, S, lk, first, min(end, first + APB), dyn);
        } else {
          bind(q);
          const int i = first + la;
          auto rho = [&](const auto& src, int e) {
            if constexpr (KIND == TK_SM64) rho_fp64_body<K>(src, S, tab.t, e, lane, i < end);
            else if constexpr (KIND == TK_SM32) rho_mixed_body<K, false>(src, A, S, tab.t, e, lane, i < end);
            else rho_mixed_body<K, true>(src, A, S, nullptr, e, lane, i < end);
          };
          if constexpr (RES) rho(srcS, i - off);
          else rho(srcA, i);
        }
      }
      if (!team_sync<RES>(c)) return;
    }
    const bool store = k < 0 || last || fire;  // nobody sees the forces of the steps between
    t = make_double2(1.e-16, 1.e-16);
    P = f2 = 0.0;
    for (int vb = c.rank, q = 0; vb < nvb; vb += c.ncta, q++) {
      const int i = off + vb * APB + la;
      const bool act = i < end;
      double4 F = make_double4(0, 0, 0, 0);
      bind(q);
      auto force = [&](const auto& src, int e) {
        if constexpr (KIND == TK_LJ64) lj_fp64_body<K, false, false>(src, A, M0, s, S, tab.t, e, lane, act, F);
        if constexpr (KIND == TK_LJ32) lj_mixed_body<K, false, false>(src, A, M0, s, S, tab.t, e, lane, act, F);
        if constexpr (KIND == TK_SM64) force_fp64_body<K, false, false>(src, A, M0, s, S, tab.t, e, lane, act, F);
        if constexpr (KIND == TK_SM32) force_mixed_body<K, false, false, false>(src, A, M0, s, S, tab.t, e, lane, act, F);
        if constexpr (KIND == TK_SM32R) force_mixed_body<K, true, false, false>(src, A, M0, s, S, nullptr, e, lane, act, F);
      };
      if constexpr (RES) {
        force(srcS, i - off);
        if (own && act) frc[q * APB + la] = F;
      } else {
        if constexpr (!TS) force(srcA, i);
        if constexpr (TS)
          if (own && act) F = tsf_gather_body<R>(A, s, i);
        if (own && act && store) {
          A.force[i] = make_double4(F.x, F.y, F.z, 0.0);
          if constexpr (SM) A.epot[i] = sm_energy(F.w, srcA.band(i));
          else if constexpr (!TS) A.epot[i] = lj_energy(F.w);
        }
        if (k < 0) continue;
        F.w = 0.0;
        if (last || fire) {
          if (own && act) half_b(i, i, F);
        } else if constexpr (K >= 4 && !TS) {
          half_ba_c(i, i, lane, act, F, K);
        } else if (own && act) {
          half_ba(i, i, F);
        }
      }
    }
    if constexpr (RES) {
      // the own atoms' half steps, one thread an atom (or four: Ermak's noise)
      __syncthreads();
      if (k >= 0 && !last && !fire && S.integ == IT_ERMAK) {
        for (int e = threadIdx.x; e < (4 * ncap + BLOCK - 1) / BLOCK * BLOCK; e += BLOCK) {
          const int lo = e >> 2;
          const bool act = lo < ncap && atom_of(lo) < end;
          half_ba_c(act ? atom_of(lo) : off, act ? lo : 0, e & 3, act, frc[act ? lo : 0], 4);
        }
      } else if (k >= 0) {
        for (int lo = threadIdx.x; lo < ncap; lo += BLOCK) {
          const int i = atom_of(lo);
          if (i >= end) continue;
          if (last || fire) half_b(i, lo, frc[lo]);
          else half_ba(i, lo, frc[lo]);
        }
      }
    }
    if (k < 0) {
      t = make_double2(1.e-16, 1.e-16);
      if (steps && !team_sync<RES>(c)) return;  // the first half step moves what was gathered
    } else if (fire) {
      // P = sum v.F and max |F|^2 of the system, summed by every CTA in the
      // same order; then the control of dt and alpha
      P = block_sum(P);
      f2 = block_max(f2);
      if (c.ncta > 1) {
        double* red = A.blk_red + 2 * c.slot0;
        if (threadIdx.x == 0) {
          if (RES) red_sh[0] = P, red_sh[1] = f2;
          else red[2 * c.rank] = P, red[2 * c.rank + 1] = f2;
        }
        if (!team_sync<RES>(c)) return;
        if (threadIdx.x < 32) {
          P = f2 = 0.0;
          for (int b = threadIdx.x; b < c.ncta; b += 32) {
            const double* r = RES ? team_peer(c, red_sh, b) : red + 2 * b;
            P += RES ? r[0] : __ldcg(r);
            f2 = fmax(f2, RES ? r[1] : __ldcg(r + 1));
          }
          for (int o = 16; o; o >>= 1) {
            P += __shfl_xor_sync(0xffffffffu, P, o);
            f2 = fmax(f2, __shfl_xor_sync(0xffffffffu, f2, o));
          }
        }
      }
      if (threadIdx.x == 0) fire_control(S, st, P, f2);
      __syncthreads();
      if (st.fire_done) break;
    } else if (!last) {
      swap();
    }
  }
  if constexpr (RES) {
    for (int lo = threadIdx.x; lo < ncap; lo += BLOCK) {  // the own atoms back to the arena
      const int i = atom_of(lo);
      if (i >= end) continue;
      if (opening || steps) {
        const double4 F = frc[lo];
        A.force[i] = make_double4(F.x, F.y, F.z, 0.0);
        A.epot[i] = SM ? sm_energy(F.w, reinterpret_cast<const double*>(dyn + L.band)[lo]) : lj_energy(F.w);
      }
      if (!steps) continue;
      A.pos[i] = X.pos[lo];
      A.vel[i] = X.vel[lo];
      A.acel[i] = X.acel[lo];
      if constexpr (MIXED) A.fxp[i] = reinterpret_cast<const int4*>(dyn + L.rec + cur * L.recbuf)[i - off];
    }
    if (!team_sync<RES>(c)) return;  // no CTA leaves while another may still read its shared memory
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    SysState& g = A.st[s];
    if (st.status) atomicOr(&g.status, st.status);
    if (c.rank == 0) {
      g.rebuild = st.rebuild;
      g.step = st.step;
      g.nupd = st.nupd;
      g.dmax = st.dmax;
      for (int d = 0; d < 3; d++) g.box_b[d] = st.box_b[d];
      g.fire_dt = st.fire_dt;
      g.fire_alpha = st.fire_alpha;
      g.fire_P = st.fire_P;
      g.fire_np = st.fire_np;
      g.fire_done = st.fire_done;
      g.fire_iter = st.fire_iter;
      g.fire_zero = st.fire_zero;
      g.fmax2 = st.fmax2;
    }
  }
}

// the kernel of a kind for K lanes per atom, resident or arena form (team_inst.cu)
const void* team_fn_0(int K, bool res);
const void* team_fn_1(int K, bool res);
const void* team_fn_2(int K, bool res);
const void* team_fn_3(int K, bool res);
const void* team_fn_4(int K, bool res);
const void* team_fn_ts(bool mixed, int K);

}  // namespace gg
