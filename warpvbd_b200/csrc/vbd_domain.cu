// The time step in fp64 by domains: an environment's mesh is divided among the
// blocks that run it -- one block (a light environment of a batch, a small
// mesh), the blocks of a cluster (a heavy environment), or one block on every SM
// (a single mesh in persistent mode).
//
// The mesh is divided into as many domains as it gets blocks (recursive
// bisection of the rest positions, vbd_host.cu).  A block keeps its own
// vertices, and copies of the neighbouring domains' vertices its tets touch
// (the halo), in shared memory for the whole step, beside the records of its
// tets; the slot loop reads nothing but shared memory and its slots.  A vertex
// that other domains read is sent to them when it is updated: its three
// coordinates go to its place in `mail`, each as one 16-byte store of the
// value and a tag (step, sweep).  A block starts colour c once every halo
// vertex of colour c - 1 has arrived: its threads poll the mail of those
// vertices until the tag is the current one, and copy the values to shared
// memory.  The value and its tag are one 128-bit access, so the handoff takes
// one store and one load through L2, with no fence and no flag.
//
// Why the exchange is safe.  Halo membership is symmetric: if block B reads
// vertex v, B owns a vertex w of a tet of v, and v's owner reads w.  v is
// written again in the next sweep only after its owner has received w's
// update that follows B's reading of v, so no value is overwritten unread.
// Every vertex reads the latest values of lower colours and the previous
// sweep's of higher ones, as with a barrier between colours.
//
// End of a sweep: every block posts its max |dx_x + dx_y + dx_z| (and its status
// bits) the same way and reads every other block's post, so all take the same
// decision.  Posts alternate between two places: a block can post exchange k + 2
// only after every block has read exchange k.
//
// Every wait is bounded (polls and wall clock); on expiry the block writes the
// step's number to the abort word, sets the timeout status and returns, and the
// others leave at their next wait.  The host takes a step whose abort word changed as
// timed out, whatever the status words hold.  The blocks of one environment are resident
// together: they form one cluster, or the launch is cooperative.
//
// What bounds it: up to a few thousand vertices the chain of one colour -- one
// vertex's slots, the sums over its lanes, the 3x3 solve -- and the handoff (565
// cycles one way between two blocks; 1,900 through a fence, a release store and
// acquire polling).  From about 300 vertices a domain the fp64 pipe and the
// shared-memory pipe, each about half busy.  B200, fp64, us per sweep, positions
// in global memory and flags between blocks (vbd_persist.cu) -> here: 80x8x8 StVK
// beam 38.1 -> 17.9, 160x16x16 beam 49.1 -> 30.9, 320x32x32 beam 179 -> 121.
// Tried: reading a slot's operands while the previous slot is computed (231
// registers, 8 warps: 35.2 and 137 us on the two larger beams), slots in pairs (no
// change), 16 lanes per vertex on the large ones (42 us at 160x16x16).
#include <cuda_runtime.h>

#include "vbd_device.cuh"
#include "vbd_domain.h"

namespace vbd {

namespace {

__device__ __forceinline__ void st_tagged(ulonglong2* p, unsigned long long v,
                                          unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(
          p),
      "l"(v), "l"(tag)
      : "memory");
}

__device__ __forceinline__ ulonglong2 ld_tagged(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile(
      "{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
      : "=l"(r.x), "=l"(r.y)
      : "l"(p)
      : "memory");
  return r;
}

__device__ __forceinline__ unsigned ld_flag(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Polls `p` until its tag, shifted, is `want`; false when the wait expired here
// or, in this step, elsewhere.
template <int SHIFT>
__device__ __forceinline__ bool wait_tagged(const ulonglong2* p, unsigned long long want,
                                            ulonglong2& got, const DomDev& d,
                                            const PersistLimits& lim) {
  got = ld_tagged(p);
  if ((got.y >> SHIFT) == want) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (long long n = 0;; ++n) {
    const bool expired = n >= lim.max_polls ||
                         ((n & 255) == 255 && globaltimer_ns() - t0 > lim.max_wait_ns);
    if (expired || ((n & 15) == 15 && ld_flag(d.abort) == d.seq)) {
      if (expired) atomicExch(d.abort, d.seq);
      return false;
    }
    got = ld_tagged(p);
    if ((got.y >> SHIFT) == want) return true;
  }
}

// Local state in shared memory; a store also mails a vertex other domains read.
struct MailState {
  double* p;
  double* save;  // where a store first puts the old position, or null
  ulonglong2* mail;  // the vertex's place, or null
  unsigned long long tag;
  __device__ __forceinline__ double4 load(int i) const {
    return make_double4(p[3 * i], p[3 * i + 1], p[3 * i + 2], 0.0);
  }
  __device__ __forceinline__ void store(int i, const double4& v) const {
    if (mail) {
      st_tagged(mail, (unsigned long long)__double_as_longlong(v.x), tag);
      st_tagged(mail + 1, (unsigned long long)__double_as_longlong(v.y), tag);
      st_tagged(mail + 2, (unsigned long long)__double_as_longlong(v.z), tag);
    }
    if (save) {
      save[3 * i] = p[3 * i];
      save[3 * i + 1] = p[3 * i + 1];
      save[3 * i + 2] = p[3 * i + 2];
    }
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
  }
};

// Inertia guess of a vertex (begin_vertex; explicit fused multiply-adds, so that
// every block forms the same bits wherever it forms it).
__device__ __forceinline__ double4 inertia_guess(const DevMesh& m, int gv, const StepConst& sc) {
  const double4 u = reinterpret_cast<const double4*>(m.u)[gv];
  const double4 v = reinterpret_cast<const double4*>(m.vel)[gv];
  return make_double4(fma(sc.g[0], sc.dt2, fma(v.x, sc.dt, u.x)),
                      fma(sc.g[1], sc.dt2, fma(v.y, sc.dt, u.y)),
                      fma(sc.g[2], sc.dt2, fma(v.z, sc.dt, u.z)), 0.0);
}

// What a warp needs of a chunk before any position: loaded before the wait
// for the previous colour.
template <int TPV>
struct ChunkRegs {
  static constexpr int PF = Prefetch<TPV>::steps;
  ushort4 sl[PF];
  const ushort4* slot;
  int steps, lv, k, gv;
  bool valid, mailed;
  double4 tt;   // SPLIT: the vertex's inertia target and mass
  int touched;  // else one word of it, to bring it into L1
};

template <int TPV, bool SPLIT>
__device__ __forceinline__ void load_chunk(ChunkRegs<TPV>& r, const DevMesh& m, const DomDev& d,
                                           const int4* chunk, const int2* local, int q,
                                           int lane) {
  constexpr int CPW = 32 / TPV;
  const int4 c = chunk[q];
  r.steps = c.y;
  r.slot = d.slot + (size_t)c.x * 32 + lane;
#pragma unroll
  for (int s = 0; s < ChunkRegs<TPV>::PF; ++s)
    if (s < c.y) r.sl[s] = __ldg(r.slot + s * 32);
  r.lv = c.z + lane % CPW;
  r.valid = r.lv < c.w;
  r.k = 0;
  r.mailed = false;
  r.gv = 0;
  r.tt = make_double4(0.0, 0.0, 0.0, 0.0);
  r.touched = 0;
  if (r.valid) {
    const int2 o = local[r.lv];
    r.mailed = o.x < 0;
    r.gv = o.x < 0 ? ~o.x : o.x;
    r.k = o.y;
    const double4* tt = reinterpret_cast<const double4*>(m.ut) + r.gv;
    if (lane < CPW) {
      if (SPLIT)
        r.tt = ldcg4(tt);
      else
        r.touched = *reinterpret_cast<const int*>(tt);
    }
  }
}

// One exchange of vertex_sums: the lanes with the bit `off` clear keep the first
// (N + 1) / 2 values, the others the rest, each adding its partner's.
template <int N>
__device__ __forceinline__ void halve(double (&v)[9], int off, int lane) {
  constexpr int K = (N + 1) / 2;
  const bool up = (lane & off) != 0;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const double hi = i + K < N ? v[i + K] : 0.0;
    const double keep = up ? hi : v[i], give = up ? v[i] : hi;
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
  }
}

// Adds the nine sums of a vertex over its TPV lanes (lane, lane ^ CPW, ...); the
// lanes below CPW hold the result.  With 16 or 32 lanes per vertex every exchange
// halves the values a lane carries and the first lane then collects them: 20
// and 21 64-bit shuffles instead of 36 and 45, added in the same order.
template <int TPV>
__device__ __forceinline__ void vertex_sums(double (&g)[3], double (&h)[6], int lane) {
  constexpr int CPW = 32 / TPV;
  if constexpr (TPV < 16) {
#pragma unroll
    for (int off = 16; off >= CPW; off >>= 1) {
#pragma unroll
      for (int i = 0; i < 3; ++i) g[i] += __shfl_xor_sync(0xffffffffu, g[i], off);
#pragma unroll
      for (int i = 0; i < 6; ++i) h[i] += __shfl_xor_sync(0xffffffffu, h[i], off);
    }
  } else {
    double v[9] = {g[0], g[1], g[2], h[0], h[1], h[2], h[3], h[4], h[5]};
    halve<9>(v, 16, lane);  // 5 values a lane
    halve<5>(v, 8, lane);   // 3
    halve<3>(v, 4, lane);   // 2
    halve<2>(v, 2, lane);   // 1
    if constexpr (TPV == 32) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    // value i now sits in the lane whose bits 16, 8, 4, 2 picked it
    const int own = lane & (CPW - 1);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      int j = i, src = 0;
      if (j >= 5) { src |= 16; j -= 5; }
      if (j >= 3) { src |= 8; j -= 3; }
      if (j >= 2) { src |= 4; j -= 2; }
      if (j >= 1) src |= 2;
      const double x = __shfl_sync(0xffffffffu, v[0], src + own);
      if (i < 3)
        g[i] = x;
      else
        h[i - 3] = x;
    }
  }
}

// One warp updates the chunk's vertices; the sums of a vertex are formed as
// process_chunk forms them.
template <int TPV, int MAT, bool SPLIT>
__device__ __forceinline__ void run_chunk(const ChunkRegs<TPV>& r, const DevMesh& m,
                                          const DomDev& d, const DomInfo& di, double* sp, double* save,
                                          const RecTab<double>& tab, int lane,
                                          const StepConst& sc, unsigned long long tag,
                                          unsigned long long& cmax, unsigned& stat,
                                          unsigned long long* dxrec) {
  constexpr int CPW = 32 / TPV;
  const int sub = lane / CPW;
  const MailState st{sp, SPLIT ? save : nullptr, SPLIT && r.mailed ? d.mail + 3 * (size_t)r.gv : nullptr, tag};
  bool valid = r.valid;
#if VBD_CHECK_BOUNDS
  if (valid && ((unsigned)r.lv >= (unsigned)di.nown || (unsigned)r.gv >= (unsigned)m.n_vertices)) {
    stat |= kStatBounds;
    valid = false;
  }
#endif
  double4 uo = make_double4(0.0, 0.0, 0.0, 0.0);
  if (valid) uo = st.load(r.lv);
  double g[3] = {0.0, 0.0, 0.0};
  double h[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  double hI = 0.0;
  const int k = valid ? r.k : 0;
  auto visit = [&](const ushort4& sl) {
    const int4 id = make_int4(sl.x, sl.y, sl.z, sl.w);
#if VBD_CHECK_BOUNDS
    if (id.x >= di.nloc || id.y >= di.nloc || id.z >= di.nloc || slot_record(id.w) >= di.nrec) {
      stat |= kStatBounds;
      return;
    }
#endif
    slot_visit<double, MAT>(st, uo, id, tab, g, h, hI);
  };
#pragma unroll
  for (int s = 0; s < ChunkRegs<TPV>::PF; ++s)
    if (s < r.steps && s * TPV + sub < k) visit(r.sl[s]);
  for (int s = ChunkRegs<TPV>::PF; s < r.steps; ++s)
    if (s * TPV + sub < k) visit(__ldg(r.slot + s * 32));
  add_identity(h, hI);
  vertex_sums<TPV>(g, h, lane);
  if (valid && lane < CPW) {
    double4 tt = r.tt;
    if (!SPLIT) {
      asm volatile("" ::"r"(r.touched));
      tt = reinterpret_cast<const double4*>(m.ut)[r.gv];
    }
    finish_vertex<double, double>(m, r.gv, r.lv, uo, tt, g, h, st, sc, cmax, stat, dxrec);
  }
}

// SPLIT: the launch's environments may be split over several blocks.  Without it
// the handoff leaves the kernel, and with it the registers that made the slot
// loop spill (27K slots on one block: 79 -> 75.5 us per sweep).
template <int TPV, int MAT, bool SPLIT>
__global__ void __launch_bounds__(kDomMaxThreads)
    domain_kernel(DevMesh m, StepParams p, DomDev d, const double* __restrict__ tol_env,
                  PersistLimits lim) {
  extern __shared__ __align__(16) unsigned char dsmem[];
  __shared__ unsigned long long s_post[kDomMaxBlocks];
  __shared__ unsigned long long s_red[2][16];
  __shared__ double s_dsum[16];
  __shared__ unsigned s_stat[2];
  __shared__ DomColor s_color[kDomMaxColors];
  int which = blockIdx.x, launch = 0;
  if (d.work) {
    const int4 w = d.work[blockIdx.x];
    if (w.x < 0) return;  // padding block of a cluster of single-block environments
    which = (w.z > 1 ? d.first_split : d.first_single)[w.x] + w.y;
    launch = w.w;
  }
  const unsigned long long t_start = p.trace ? globaltimer_ns() : 0ull;
  const DomInfo di = d.dom[which];
  const EnvInfo e = m.env[di.env];
  const StepConst sc = make_const(p);
  const double tol = tol_env ? tol_env[di.env] : p.tol;
  const int max_iter = p.max_iter;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
  const int nd = SPLIT ? di.nd : 1, ncolors = di.ncolors;
  double* sp = reinterpret_cast<double*>(dsmem);
  RecTab<double> tab{d.rec + 3 * (size_t)di.rbase, nullptr};
  if (di.flags & kDomRecords) {
    unsigned char* stab = dsmem + dom_smem_records(di.nloc);
    tab = global_table<double>(m.rec_tab, e.rbase);
    const int* id = d.rec_id + di.rbase;
    stage_rows(stab, di.nrec, [&](int rec, int row) {
      return tab.g + 3 * (size_t)__ldg(id + rec) + row;
    });
    tab = staged(tab, stab);
  }
  const int4* chunk = reinterpret_cast<const int4*>(d.chunk) + di.qbase;
  const int2* local = d.local + di.lbase;
  if (di.flags & kDomMeta) {
    int4* s_chunk = reinterpret_cast<int4*>(dsmem + dom_smem_meta(di.nloc, di.nrec, di.flags));
    int2* s_local = reinterpret_cast<int2*>(s_chunk + di.nchunk);
    for (int i = tid; i < di.nchunk; i += nt) s_chunk[i] = __ldg(chunk + i);
    for (int i = tid; i < di.nloc; i += nt) s_local[i] = __ldg(local + i);
    chunk = s_chunk;
    local = s_local;
  }
  for (int i = tid; i < ncolors; i += nt) s_color[i] = d.color[di.cbase + i];
  if (tid < 2) s_stat[tid] = 0u;
  // ORed from here on.  Another block whose wait expires before this store loses its
  // bit; the abort word, which it sets too, tells the host
  if (tid == 0 && di.rank == 0) m.status[di.env] = 0u;
  __syncthreads();
  const unsigned long long seq = (unsigned long long)d.seq << 28;  // tags: step, sweep / exchange
  auto local_gid = [&](int l) {
    const int g = local[l].x;
    return g < 0 ? ~g : g;
  };
  // begin: every local vertex at its inertia guess; the owner writes the
  // step-start state back
  for (int l = tid; l < di.nloc; l += nt) {
    const int gv = local_gid(l);
    double4 un = reinterpret_cast<const double4*>(m.u)[gv];
    if (l < di.nown) reinterpret_cast<double4*>(m.up)[gv] = un;
    if (gv - e.vbase < e.nact) un = inertia_guess(m, gv, sc);
    if (l < di.nown) {
      double4* t = reinterpret_cast<double4*>(m.ut) + gv;
      *t = make_double4(un.x, un.y, un.z, t->w);  // w: the lumped mass
    }
    sp[3 * l] = un.x;
    sp[3 * l + 1] = un.y;
    sp[3 * l + 2] = un.z;
  }
  __syncthreads();

  unsigned stat = 0u;
  unsigned long long ex = 0ull;  // exchanges so far
  auto abort_step = [&]() {
    if (tid == 0) atomicOr(m.status + di.env, kStatTimeout);
  };
  // thread 0 posts this block's value for the next exchange
  auto post = [&](unsigned long long v, unsigned bits) {
    st_tagged(d.post + di.pbase + (int)((ex + 1) & 1) * nd + di.rank, v,
              ((seq | (ex + 1)) << 8) | bits);
  };
  // every block's post of the next exchange into s_post, their status bits into
  // s_stat; false when a wait expired.  Followed by a block barrier.
  // seen: the largest value this thread read, instead
  auto collect = [&](unsigned long long* seen = nullptr) {
    ++ex;
    bool ok = true;
    unsigned bits = 0u;
    for (int b = tid; b < nd; b += nt) {
      ulonglong2 got;
      ok = wait_tagged<8>(d.post + di.pbase + (int)(ex & 1) * nd + b, seq | ex, got, d, lim);
      if (!ok) break;
      if (seen)
        *seen = got.x > *seen ? got.x : *seen;
      else
        s_post[b] = got.x;
      bits |= (unsigned)(got.y & 0xffu);
    }
    bits = __reduce_or_sync(0xffffffffu, bits);
    if (lane == 0 && bits) atomicOr(&s_stat[0], bits);
    return ok;
  };
  // Sum of acc over the environment's blocks, in an order that does not depend on timing
  auto grid_sum = [&](double acc, bool& ok) -> double {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) s_dsum[warp] = acc;
    __syncthreads();
    if (tid == 0) {
      double v = 0.0;
      for (int i = 0; i < nwarps; ++i) v += s_dsum[i];
      if (nd > 1)
        post((unsigned long long)__double_as_longlong(v), 0u);
      else
        s_post[0] = (unsigned long long)__double_as_longlong(v);
    }
    ok = __syncthreads_and(nd > 1 ? collect() : true) != 0;
    double v = 0.0;
    if (ok)
      for (int b = lane; b < nd; b += 32) v += __longlong_as_double((long long)s_post[b]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();  // s_post and s_dsum are reused
    return v;
  };

  if (p.warm && m.ws_pred) {
    // as the block mode's stage: the incremental potential at the inertia guess
    // against inertia guess + alpha x prediction, alpha = 1, 1/2, 1/4
    const MailState st{sp, nullptr, nullptr, 0ull};
    auto pred = [&](int l) { return m.ws_pred[local_gid(l)]; };
    auto moved = [&](double4 v, int l) {
      const float4 c = pred(l);
      if (c.w > 0.f) {
        v.x += double(c.x);
        v.y += double(c.y);
        v.z += double(c.z);
      }
      return v;
    };
    auto energy = [&](bool pair) {
      double a = 0.0, b = 0.0;
      for (int i = tid; i < di.ntets; i += nt) {
        const int4 id = __ldg(d.tet_slot + di.tbase + i);
        const int o = __ldg(d.tet_owner + di.tbase + i);
        const double4 uo = st.load(o), x = st.load(id.x), y = st.load(id.y), z = st.load(id.z);
        a += psi_visit<double, MAT>(uo, x, y, z, id.w, tab);
        if (pair)
          b += psi_visit<double, MAT>(moved(uo, o), moved(x, id.x), moved(y, id.y),
                                      moved(z, id.z), id.w, tab);
      }
      for (int l = tid; l < di.nown; l += nt) {
        const double4 u = pair ? moved(st.load(l), l) : st.load(l);
        const double4 tt = ldcg4(reinterpret_cast<const double4*>(m.ut) + local_gid(l));
        const double dx = u.x - tt.x, dy = u.y - tt.y, dz = u.z - tt.z;
        const double in = 0.5 * tt.w * sc.inv_dt2 * (dx * dx + dy * dy + dz * dz);
        if (pair)
          b += in;  // the inertia guess has none
        else
          a += in;
      }
      return make_double2(a, b);
    };
    // inertia guess + alpha x prediction (alpha = 0: the inertia guess)
    auto place = [&](double alpha) {
      for (int l = tid; l < di.nloc; l += nt) {
        const int gv = local_gid(l);
        if (gv - e.vbase >= e.nsolved) continue;
        double4 v = inertia_guess(m, gv, sc);
        const float4 c = m.ws_pred[gv];
        if (alpha != 0.0 && c.w > 0.f) {
          v.x += alpha * double(c.x);
          v.y += alpha * double(c.y);
          v.z += alpha * double(c.z);
        }
        sp[3 * l] = v.x;
        sp[3 * l + 1] = v.y;
        sp[3 * l + 2] = v.z;
      }
      __syncthreads();
    };
    bool ok = true;
    const double2 el = energy(true);
    const double e0 = grid_sum(el.x, ok);
    const double e1 = ok ? grid_sum(el.y, ok) : 0.0;
    bool used = ok && e1 < e0;  // false on NaN as well
    if (used) place(1.0);
    for (int trial = 1; trial < 3 && ok && !used; ++trial) {
      place(1.0 / double(1 << trial));
      const double et = grid_sum(energy(false).x, ok);
      used = ok && et < e0;
    }
    if (!ok) return abort_step();
    if (used)
      stat |= kStatWarmUsed;
    else
      place(0.0);
  }

  // the previous colour's halo vertices into shared memory
  auto receive = [&](const DomColor& c, unsigned long long tag) {
    const int n = 3 * (c.halo_end - c.halo_begin);
    for (int j = tid; j < n; j += nt) {
      const int l = c.halo_begin + j / 3, x = j % 3;
      ulonglong2 got;
      if (!wait_tagged<0>(d.mail + 3 * (size_t)local_gid(l) + x, tag, got, d, lim)) return false;
      sp[3 * l + x] = __longlong_as_double((long long)got.x);
    }
    return true;
  };
  int it = 0;
  bool conv = false, nan = false;
  ChunkRegs<TPV> r;
  DomColor cc{};
  if (ncolors > 0) cc = s_color[0];
  if (cc.chunk_begin + warp < cc.chunk_end)
    load_chunk<TPV, SPLIT>(r, m, d, chunk, local, cc.chunk_begin + warp, lane);
  if (ncolors == 0) {  // nothing is solved: no update, a largest one of zero
    conv = 0.0 < tol;
    it = conv ? 1 : max_iter;
  }
  // The answer of the convergence test, posted at a sweep's end, takes a trip
  // through L2: the next sweep's first colour is computed meanwhile, its old
  // positions kept in `save` in case the answer is to stop.  Not before the last
  // sweep allowed, whose updates leave a record (dxrec).
  double* save = reinterpret_cast<double*>(
      dsmem + dom_smem_save(di.nloc, di.nrec, di.nchunk, di.flags));
  const bool can_save = SPLIT && (di.flags & kDomSave) && !d.grid_sync;
  bool asked = false;  // posted, answer not read yet
  // every thread votes on the posts it read: all below the tolerance (a NaN, whose
  // bits lie above infinity's, is not), or else something wrong.  False: aborted
  auto answer = [&](bool ok) {
    unsigned long long v = 0ull;
    ok = collect(&v) && ok;
    asked = false;
    conv = __syncthreads_and(ok && __longlong_as_double((long long)v) < tol) != 0;
    if (conv) return true;
    if (__syncthreads_or(!ok)) return false;
    nan = __syncthreads_or(v > 0x7ff0000000000000ull) != 0;
    return true;
  };
  while (ncolors > 0) {
    unsigned long long cmax = 0ull;
    unsigned long long* dxrec = it + 1 == max_iter ? m.dxmax + di.env : nullptr;
    const unsigned long long tag = seq | (unsigned long long)(it + 1);
    bool undo = false;
    for (int c = 0; c < ncolors; ++c) {
      // Warps of one scheduler start a colour 250 cycles apart: together they
      // would all read their first slots and then all wait for the fp64 pipe,
      // step after step (160x16x16 beam 33.2 -> 31.3 us per sweep, 27K slots on
      // one block 75.3 -> 72.8; 150 and 350 cycles within 1 %)
      if (cc.chunk_end - cc.chunk_begin > 4 && warp >= 4) {
        const long long t0 = clock64();
        while (clock64() - t0 < 250 * (warp >> 2 & 3)) {
        }
      }
      for (int q = cc.chunk_begin + warp; q < cc.chunk_end; q += nwarps) {
        // bring the slots of the warp's next chunk of this colour into L1
        int touch = 0;
        if (q + nwarps < cc.chunk_end) {
          const int4 n = chunk[q + nwarps];
          if (lane < 2 * n.y)
            touch = __ldg(reinterpret_cast<const int*>(d.slot + (size_t)n.x * 32 + lane * 16));
        }
        if (q != cc.chunk_begin + warp) load_chunk<TPV, SPLIT>(r, m, d, chunk, local, q, lane);
        run_chunk<TPV, MAT, SPLIT>(r, m, d, di, sp, asked ? save : nullptr, tab, lane, sc, tag,
                                   cmax, stat, dxrec);
        asm volatile("" ::"r"(touch));
      }
      // the next colour's first chunk, then the wait for this one's halo
      const DomColor done = cc;
      cc = s_color[c + 1 < ncolors ? c + 1 : 0];
      if (cc.chunk_begin + warp < cc.chunk_end)
        load_chunk<TPV, SPLIT>(r, m, d, chunk, local, cc.chunk_begin + warp, lane);
      const bool last = c + 1 == ncolors;
      if (asked) {  // c == 0: the previous sweep's answer
        if (!answer(last || receive(done, tag))) return abort_step();
        undo = conv || nan;
        if (undo) break;
        if (!last) continue;
      }
      if (last) {
        // only the lanes below CPW updated vertices
        constexpr int CPW = 32 / TPV;
#pragma unroll
        for (int off = CPW / 2; off > 0; off >>= 1) {
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, cmax, off);
          cmax = o > cmax ? o : cmax;
        }
        const unsigned bits = __reduce_or_sync(0xffffffffu, stat);
        if (lane == 0) {
          s_red[it & 1][warp] = cmax;
          if (bits) atomicOr(&s_stat[1], bits);
        }
      }
      if (nd == 1) {
        __syncthreads();
        continue;
      }
      if (last) {
        __syncthreads();
        if (warp == 0) {
          unsigned long long v = lane < nwarps ? s_red[it & 1][lane] : 0ull;
          v = warp_max_u64(v);
          if (lane == 0) post(v, s_stat[1]);
        }
      }
      bool ok = receive(done, tag);
      if (!last && d.grid_sync) {
        __syncthreads();
        if (tid == 0) post(0ull, 0u);
        ok = collect() && ok;
      }
      if (last && !(can_save && it + 2 < max_iter)) {
        if (!answer(ok)) return abort_step();
      } else {
        if (!__syncthreads_and(ok)) return abort_step();
        asked = last;
      }
    }
    if (undo) {
      // the last finished sweep's positions; `end` below reads each entry with the
      // thread that restores it
      for (int l = tid; l < di.nsave; l += nt)
        for (int x = 0; x < 3; ++x) sp[3 * l + x] = save[3 * l + x];
      break;
    }
    ++it;
    if (nd == 1) {
      const unsigned long long v =
          warp_max_u64(lane < nwarps ? s_red[(it - 1) & 1][lane] : 0ull);
      nan = v > 0x7ff0000000000000ull;
      conv = !nan && __longlong_as_double((long long)v) < tol;
    }
    if (conv || nan || it >= max_iter) break;
  }

  // end: own vertices, then the unsolved ones spread over the blocks
  double4* U = reinterpret_cast<double4*>(m.u);
  for (int l = tid; l < di.nown; l += nt) {
    const int gv = local_gid(l);
    const double4 un = make_double4(sp[3 * l], sp[3 * l + 1], sp[3 * l + 2], 0.0);
    U[gv] = un;
    end_vertex<double>(m, gv, un, sc);
  }
  for (int i = e.nsolved + di.rank * nt + tid; i < e.nv; i += nd * nt) {
    const double4 un = begin_vertex<double>(m, e.vbase + i, i < e.nact, sc, true);
    U[e.vbase + i] = un;
    end_vertex<double>(m, e.vbase + i, un, sc);
  }
  if (m.host_out) {
    // the environment's positions in the caller's order, one double per thread
    // and consecutive threads on consecutive doubles, over the bus while other
    // environments still run: read back from global memory once every block of
    // the environment has written its own
    if (nd > 1) {
      __threadfence();
      __syncthreads();
      if (tid == 0) post(0ull, 0u);
      if (!__syncthreads_and(collect())) return abort_step();
      __threadfence();
    } else {
      __syncthreads();
    }
    double* out = m.host_out + 3 * (size_t)e.vbase;
    const double* rest = m.rest + 3 * (size_t)e.vbase;
    for (int k = di.rank * nt + tid; k < 3 * e.nv; k += nd * nt) {
      const int j = k / 3, c = k - 3 * j;
      out[k] = rest[k] + __ldcg(reinterpret_cast<const double*>(U + m.map[e.vbase + j]) + c);
    }
  }
  if (di.rank == 0 && tid == 0) {
    unsigned st = s_stat[nd == 1 ? 1 : 0];
    if (nan) st |= kStatNonFinite;
    if (!conv) st |= kStatIterCap;
    m.iters[di.env] = it;
    atomicOr(m.status + di.env, st);
  }
  if (p.trace && tid == 0) {
    unsigned long long* t = p.trace + 4 * (size_t)blockIdx.x;
    t[0] = t_start;
    t[1] = globaltimer_ns();
    t[2] = ((unsigned long long)di.env << 32) | ((unsigned long long)di.rank << 16) | sm_id();
    t[3] = ((unsigned long long)it << 8) | (unsigned long long)launch;
  }
}

template <int TPV, typename F>
cudaError_t dom_dispatch(int material, bool split, F& f) {
  if (split)
    return material == kSNH ? f.template run<TPV, kSNH, true>() : f.template run<TPV, kStVK, true>();
  return material == kSNH ? f.template run<TPV, kSNH, false>()
                          : f.template run<TPV, kStVK, false>();
}

template <typename F>
cudaError_t dom_dispatch(int material, int tpv, bool split, F& f) {
  switch (tpv) {
    case 4: return dom_dispatch<4>(material, split, f);
    case 8: return dom_dispatch<8>(material, split, f);
    case 16: return dom_dispatch<16>(material, split, f);
    case 32: return dom_dispatch<32>(material, split, f);
    default: return cudaErrorInvalidValue;
  }
}

template <int TPV, int MAT, bool SPLIT>
cudaError_t dom_configure() {
  // the attributes are per device; each thread sets them for itself
  static thread_local int configured_device = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_device == dev) return cudaSuccess;
  auto* k = domain_kernel<TPV, MAT, SPLIT>;
  cudaError_t e =
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDomMaxSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) configured_device = dev;
  return e;
}

struct DomOccupancy {
  int threads;
  size_t smem;
  int cluster;
  int* out;
  template <int TPV, int MAT, bool SPLIT>
  cudaError_t run() {
    const cudaError_t e = dom_configure<TPV, MAT, SPLIT>();
    if (e != cudaSuccess) return e;
    if (cluster <= 1)
      return cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, domain_kernel<TPV, MAT, SPLIT>, threads,
                                                           smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster * 64);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(out, domain_kernel<TPV, MAT, SPLIT>, &cfg);
  }
};

struct DomLaunch {
  int threads;
  const DevMesh& m;
  const StepParams& p;
  const DomDev& d;
  const double* tol;
  PersistLimits lim;
  int n_blocks, cluster;
  bool cooperative;
  size_t smem;
  cudaStream_t s;
  template <int TPV, int MAT, bool SPLIT>
  cudaError_t run() {
    const cudaError_t e = dom_configure<TPV, MAT, SPLIT>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    if (cooperative) {
      attr[0].id = cudaLaunchAttributeCooperative;
      attr[0].val.cooperative = 1;
      cfg.numAttrs = 1;
    } else if (cluster > 1) {
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = cluster;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, domain_kernel<TPV, MAT, SPLIT>, m, p, d, tol, lim);
  }
};

}  // namespace

cudaError_t dom_occupancy(int material, int tpv, int threads, size_t smem, int cluster,
                          bool split, int* out) {
  if (threads < 32 || threads > kDomMaxThreads || threads % 32) return cudaErrorInvalidValue;
  DomOccupancy f{threads, smem, cluster, out};
  return dom_dispatch(material, tpv, split, f);
}

cudaError_t launch_domain(int material, int tpv, int threads, const DevMesh& m,
                          const StepParams& p, const DomDev& d, const double* tol_env,
                          const PersistLimits& lim, int n_blocks, int cluster, bool cooperative,
                          size_t smem, cudaStream_t s) {
  if (threads < 32 || threads > kDomMaxThreads || threads % 32 || n_blocks < 1 ||
      cluster < 1 || n_blocks % cluster || smem > kDomMaxSmem)
    return cudaErrorInvalidValue;
  DomLaunch f{threads, m, p, d, tol_env, lim, n_blocks, cluster, cooperative, smem, s};
  return dom_dispatch(material, tpv, cluster > 1 || cooperative, f);
}

}  // namespace vbd
