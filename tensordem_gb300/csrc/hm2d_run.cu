// The resident step kernel (see hm2d_run.cuh).
#include "hm2d_run.cuh"

namespace tdem {
namespace hm {

// Reaction of one evaluation from its per-warp partials {warp, fx, fy} (m of
// them, distinct warps), summed in warp order by one warp. Returns the sums in
// lane 0.
__device__ __forceinline__ void sum_indenter(const double* e, unsigned m, double* sorted, double& sx, double& sy) {
  const int lane = threadIdx.x & 31;
  sx = sy = 0.0;
  for (unsigned a = lane; a < m; a += 32) {
    const double k0 = e[3 * a];
    unsigned r = 0;
    for (unsigned u = 0; u < m; ++u) r += (e[3 * u] < k0) ? 1u : 0u;
    sorted[2 * r] = e[3 * a + 1];
    sorted[2 * r + 1] = e[3 * a + 2];
  }
  __syncwarp();
  if (lane == 0) {
    for (unsigned a = 0; a < m; ++a) {
      sx += sorted[2 * a];
      sy += sorted[2 * a + 1];
    }
  }
  __syncwarp();
}

// The indenter's running totals, in lane 0 of the warp that books them.
struct Reaction {
  double work, x, y;
};

// Reaction of evaluation e from its partials (entries[e & 1] of them), by one
// warp, after the evaluation's barrier; the count is cleared for evaluation
// e + 2, whose first partials come after the next barrier.
template <class T>
__device__ __forceinline__ void book_reaction(const Params<T>& P, const Bufs<T>& B, long long e, size_t half,
                                              Reaction& R) {
  const int par = (int)(e & 1);
  const unsigned m = *reinterpret_cast<volatile unsigned*>(&B.ctl->entries[par]);
  double sx, sy;
  sum_indenter(B.ind_part + par * half, m, B.ind_part + 2 * half, sx, sy);
  if ((threadIdx.x & 31) != 0) return;
  R.x = -sx;
  R.y = -sy;
  R.work += (double)P.dt * (sx * P.ind_vx + sy * P.ind_vy);
  if (e < (long long)P.load_cap) {
    B.load[2 * e] = -sx;
    B.load[2 * e + 1] = -sy;
  }
  if (m) *reinterpret_cast<volatile unsigned*>(&B.ctl->entries[par]) = 0u;
}

// One evaluation of a disc from the global arrays (a block whose pairs its
// shared memory does not hold).
template <class T>
__device__ __noinline__ void direct_disc(const Params<T>& P, const Bufs<T>& B, int sp, int lp, int i, int primed,
                                         long long eval, ThreadLedger<T>& L) {
  const PlainFetch<T> fetch{B.pos[sp], B.vel[sp]};
  const V4<T> p = fetch.p(i), v = fetch.v(i);
  const uint4 hd = B.head[lp][i];
  V4<T> q0{}, q1{}, q2{};
  load_head_partners<T>(fetch, hd, q0, q1, q2);
  process_particle_q<T, kBatch, false, PlainFetch<T>>(P, B, fetch, sp, lp, i, p, v, hd, q0, q1, q2, primed, eval, L);
}

// Exclusive prefix of x over the block's threads and the total.
__device__ __forceinline__ unsigned block_prefix(unsigned x, unsigned* s_warp, unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (int)(blockDim.x >> 5);
  unsigned incl = x;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  unsigned before = 0u;
  total = 0u;
  for (int w = 0; w < warps; ++w) {
    if (w < warp) before += s_warp[w];
    total += s_warp[w];
  }
  __syncthreads();
  return before + incl - x;
}

constexpr unsigned kPlaceOwner = 0x8000u;  // this disc is the lower one of the pair
constexpr unsigned kOutside = 0xFFFFu;     // a partner of another block

template <class T, bool LOCAL, bool BIG>
__device__ __forceinline__ void run_pairs(const Params<T>& P, const Bufs<T>& B, unsigned char* run_smem,
                                          cudaGraphConditionalHandle h_rebuild, cudaGraphConditionalHandle h_loop,
                                          int use_cond, int pb, int mc) {
  constexpr int MODE = kBatch;  // the first evaluation of a state primes it
  __shared__ unsigned s_vmax[3], s_out[4], s_warp[32];
  __shared__ int s_bad[3], s_touch[3];
  Ctl* ctl = B.ctl;
  const int t = threadIdx.x, lane = t & 31, nt = (int)blockDim.x;
  const int n = P.n;
  const int i0 = (int)blockIdx.x * pb, mine = min(pb, n - i0);  // this block's discs
  const int i = i0 + t;
  const bool own = t < mine;
  int sp = ctl->sp;
  const int lp = ctl->lp;
  long long eval = ctl->evals;
  const long long target = ctl->target;
  float disp = ctl->disp;
  unsigned epoch = ctl->epoch;
  if (t < 3) {
    s_vmax[t] = 0u;
    s_bad[t] = 0;
    s_touch[t] = 0;
  }
  const PairLayout Y = pair_layout<T>(P.W, pb, mc);
  V4<T>* const spos = reinterpret_cast<V4<T>*>(run_smem + Y.pos);
  V4<T>* const svel = reinterpret_cast<V4<T>*>(run_smem + Y.vel);
  V4<T>* const res = reinterpret_cast<V4<T>*>(run_smem + Y.res);   // force on a, torque per lever, loss
  V2<T>* const hist = reinterpret_cast<V2<T>*>(run_smem + Y.hist);
  uint2* const desc = reinterpret_cast<uint2*>(run_smem + Y.desc);  // {disc | partner's place << 16, partner}
  int* const base = reinterpret_cast<int*>(run_smem + Y.base);     // first pair of each disc
  unsigned short* const place = reinterpret_cast<unsigned short*>(run_smem + Y.place);  // [W][pb]
  unsigned short* const touch = reinterpret_cast<unsigned short*>(run_smem + Y.touch);  // touching pairs
  unsigned char* const on = run_smem + Y.on;  // bit 0: touching, bit 1: stored history, bit 2: eff holds

  // this thread's disc, and its share of the block's pairs: those with discs of
  // other blocks, and of a pair inside the block the lower disc's slot
  V4<T> p{}, v{};
  float2 rem = make_float2(0.0f, 0.0f);
  int cnt = 0;
  unsigned mask0 = 0u;
  const unsigned* nbr = B.nbr[lp];
  auto partner = [&](int s) { return slot_partner(B.head[lp][i], nbr, (size_t)n, i, s); };
  const bool cut = (ctl->status & kStatusCapacity) != 0;  // a list overflowed: disc j may not list this one
  auto lists = [&](int j) {
    const uint4 h = B.head[lp][j];
    const int c = (int)(h.x & 0xFFu);
    for (int s = 0; s < c; ++s)
      if (slot_partner(h, nbr, (size_t)n, j, s) == i) return true;
    return false;
  };
  auto inside = [&](int j) { return (unsigned)(j - i0) < (unsigned)mine; };
  T spin = T(0);      // 1 / moment of inertia, as the torque takes it (FP64)
  unsigned yes = 0u;  // slots this block evaluates under this disc
  if (own) {
    const unsigned word = B.head[lp][i].x;
    cnt = (int)(word & 0xFFu);
    mask0 = word >> 8;
    if (sizeof(T) == 4 && P.prem) rem = B.prem[lp][i];
    p = B.pos[sp][i];
    v = B.vel[sp][i];
    spos[t] = p;
    svel[t] = v;
    if (sizeof(T) == 8) spin = v.w * P.kinv / (p.z * p.z);
    for (int s = 0; s < cnt; ++s) {
      const int j = partner(s);
      if (!inside(j) || i < j || (cut && !lists(j))) yes |= 1u << s;
    }
  }
  unsigned total;
  const unsigned before = block_prefix((unsigned)__popc(yes), s_warp, total);
  const int nc = (int)total;
  const bool direct = nc > mc;  // no room: the discs' threads work on the global arrays
  // FP64, bound by its pipe: a pair's effective radius and mass are constants of
  // the launch, kept from its first contact on (in the room for results that the
  // block's pairs leave, 16 of 32 bytes each), as a disc's torque factor is from
  // the start. The three divisions less take a step of 65,535 touching discs from
  // 66 to 61 us.
  constexpr bool KEEP = sizeof(T) == 8;
  const bool keep = KEEP && 3 * nc <= 2 * mc;
  V2<T>* const eff = reinterpret_cast<V2<T>*>(res + nc);  // {effective radius, mass}
  if (own && !direct) {
    int e = (int)before;
    base[t] = e;
    for (int s = 0; s < cnt; ++s) {
      if (!((yes >> s) & 1u)) continue;
      const int j = partner(s);
      const bool stored = (mask0 >> s) & 1u;
      desc[e] = make_uint2((unsigned)t | (inside(j) ? (unsigned)(j - i0) << 16 : kOutside << 16), (unsigned)j);
      hist[e] = stored ? B.hist[lp][(size_t)s * n + i] : V2<T>{T(0), T(0)};
      on[e] = stored ? 2 : 0;
      place[s * pb + t] = (unsigned short)((unsigned)e | (i < j ? kPlaceOwner : 0u));
      ++e;
    }
    if (t == mine - 1) base[mine] = nc;
  }
  __syncthreads();
  if (own && !direct) {
    for (int s = 0; s < cnt; ++s) {
      if ((yes >> s) & 1u) continue;
      const int o = partner(s) - i0;
      int e = base[o];
      while (e < base[o + 1] - 1 && (int)desc[e].y != i) ++e;
      place[s * pb + t] = (unsigned short)e;
    }
  }
  // ledger partials of this warp's 32 discs (slot i / 32), carried in lane 0
  const size_t gw = (size_t)i >> 5;
  const bool books = lane == 0 && own;
  double acc_diss = books ? B.diss_part[gw] : 0.0;
  int k3 = 0;  // shared-memory reduction slot of the step
  bool late = false;
  unsigned bad = 0u;
  int rebuild = 0;
  __syncthreads();
  while (true) {
    const int primed = eval > 0 ? 1 : 0;
    const int k1 = k3 == 2 ? 0 : k3 + 1;
    if (!direct) {
      const V4<T>* gpos = B.pos[sp];
      const V4<T>* gvel = B.vel[sp];
      auto law = [&](int e, const uint2& d, bool in, const V4<T>& x, const V4<T>& y) {
        const int s = (int)(d.x & 0xFFFFu), o = (int)(d.x >> 16);
        const bool owner = i0 + s < (int)d.y;
        const V4<T> vx = svel[s], vy = in ? svel[o] : gvel[d.y];
        const V4<T>& a = owner ? x : y;
        const V4<T>& b = owner ? y : x;
        const Geo<T> g = pair_geo<T>(P, a, b);
        const unsigned was = on[e];
        const V2<T> xi0 = (was & 2) ? hist[e] : V2<T>{T(0), T(0)};
        PairOut<T> r;
        if (KEEP && vx.w + vy.w > T(0)) {  // pair_force with the constants kept
          V2<T> c;
          if (was & 4) {
            c = eff[e];
          } else {
            pair_effective<T>(x.z, y.z, vx.w, vy.w, c.x, c.y);
            if (keep) eff[e] = c;
          }
          const T d0 = dev_sqrt(g.d2);
          r = contact_law<T>(P, g.rs - d0, g.dx / d0, g.dy / d0, c.x, c.y, a.z, b.z, owner ? vx : vy,
                             owner ? vy : vx, xi0);
        } else {
          r = pair_force<T>(P, g, a, owner ? vx : vy, b, owner ? vy : vx, xi0);
        }
        hist[e] = r.xi;
        on[e] = (unsigned char)(((r.xi.x != T(0)) || (r.xi.y != T(0)) ? 3 : 1) | (KEEP && keep ? 4 : 0));
        res[e] = V4<T>{r.fx, r.fy, r.cr, r.diss};
      };
      // A thread per pair. FP64, whose pipe bounds the law, first lists the pairs
      // that touch and evaluates them on full warps (82 -> 66 us a step at 65,535
      // discs); in FP32 the list costs more than the idle lanes do (5% at 50,071).
      constexpr bool LIST = sizeof(T) == 8;
      for (int e0 = 0; e0 < nc; e0 += nt) {
        const int e = e0 + t;
        bool hit = false;
        if (e < nc) {
          const uint2 d = desc[e];
          const int s = (int)(d.x & 0xFFFFu), o = (int)(d.x >> 16);
          const bool in = LOCAL || o != (int)kOutside;
          const V4<T> x = spos[s], y = in ? spos[o] : gpos[d.y];
          const Geo<T> g = pair_geo<T>(P, x, y);
          hit = g.d2 < g.rs * g.rs;
          if (!hit)
            on[e] = KEEP ? on[e] & 4 : 0;  // contact opened: reset
          else if (!LIST)
            law(e, d, in, x, y);
        }
        if (LIST) {
          const unsigned hits = __ballot_sync(0xffffffffu, hit);
          if (hits) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_touch[k3], __popc(hits));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (hit) touch[at + __popc(hits & ((1u << lane) - 1u))] = (unsigned short)e;
          }
        }
      }
      __syncthreads();
      if (LIST) {
        const int hits = s_touch[k3];
        for (int w = t; w < hits; w += nt) {
          const int e = touch[w];
          const uint2 d = desc[e];
          const int o = (int)(d.x >> 16);
          const bool in = LOCAL || o != (int)kOutside;
          law(e, d, in, spos[d.x & 0xFFFFu], in ? spos[o] : gpos[d.y]);
        }
        if (hits) __syncthreads();
      }
    }
    if (sizeof(T) == 8 && t == 0) s_touch[k1] = 0;  // the next step's count: last read a step ago
    // a disc's sums in slot order, its walls, and its move
    ThreadLedger<T> L;
    if (own) {
      if (direct) {
        ThreadLedger<T> D;  // (its address is taken: L itself stays in registers)
        direct_disc<T>(P, B, sp, lp, i, primed, eval, D);
        L = D;
      } else {
        // (the big build has no registers to keep the state in)
        const V4<T> p0 = BIG ? spos[t] : p, v0 = BIG ? svel[t] : v;
        Acc<T> fx, fy, tq;
        for (int s = 0; s < cnt; ++s) {
          const unsigned at = place[s * pb + t], e = at & ~kPlaceOwner;
          if (!(on[e] & 1)) continue;
          const V4<T> r = res[e];
          if (at & kPlaceOwner) {
            fx.add(r.x);
            fy.add(r.y);
            L.diss += r.w;
          } else {
            fx.add(-r.x);
            fy.add(-r.y);
          }
          tq.add(p0.z * r.z);
        }
        wall_contacts<T, MODE>(P, B.whist[lp], i, p0, v0, fx, fy, tq, L, primed);
        const T Fx = fx.get(), Fy = fy.get(), Tz = tq.get();
        const T inv_m = v0.w;
        const bool free = inv_m > T(0);
        const T ax = free ? Fx * inv_m + P.gx : T(0);
        const T ay = free ? Fy * inv_m + P.gy : T(0);
        T al = Tz;
        if (Tz != T(0)) al = Tz * (KEEP ? spin : inv_m * P.kinv / (p0.z * p0.z));
        const Moved<T> m = move_particle<T, MODE>(P, p0, v0, rem, ax, ay, al, primed, L);
        if (!BIG) {
          p = m.pos;
          v = m.vel;
        }
        rem = m.rem;
        spos[t] = m.pos;
        svel[t] = m.vel;
        if (!LOCAL) {
          B.pos[sp ^ 1][i] = m.pos;
          B.vel[sp ^ 1][i] = m.vel;
        }
      }
    }
    // the warp's ledger partials (most warps have none)
    const unsigned wbits = __reduce_max_sync(0xffffffffu, __float_as_uint(L.vmax2));
    const bool wbad = __any_sync(0xffffffffu, L.bad);
    if (lane == 0) {
      if (wbits) atomicMax(&s_vmax[k3], wbits);
      if (wbad) s_bad[k3] = 1;
    }
    if (__any_sync(0xffffffffu, L.diss != T(0))) {
      T x = L.diss;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
      acc_diss += (double)x;
    }
    unsigned vbits;
    if (t == 0) {  // the next step's slots: last read a step ago
      s_vmax[k1] = 0u;
      s_bad[k1] = 0;
    }
    if (LOCAL) {
      __syncthreads();
      vbits = s_vmax[k3];
      bad = (unsigned)s_bad[k3];
    } else {
      grid_barrier(ctl, gridDim.x, epoch, &s_vmax[k3], &s_bad[k3], P.wait_budget, s_out);
      ++epoch;
      if (s_out[3]) {
        late = true;
        break;
      }
      vbits = s_out[1];
      bad = s_out[2];
    }
    k3 = k1;
    sp ^= 1;
    ++eval;
    disp += sqrtf(__uint_as_float(vbits)) * (float)P.dt;
    rebuild = disp > P.rebuild_disp ? 1 : 0;
    if (rebuild || bad || eval >= target) break;
  }
  if (late) {  // a barrier ran out of time: the state is not usable
    if (t == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  // write back what stayed on the chip
  if (own && !direct) {
    if (LOCAL) {
      B.pos[sp][i] = p;
      B.vel[sp][i] = v;
    }
    if (sizeof(T) == 4 && P.prem) B.prem[lp][i] = rem;
    unsigned mask = 0u;
    for (int s = 0; s < cnt; ++s) {
      const unsigned e = place[s * pb + t] & ~kPlaceOwner;
      const bool stored = (on[e] & 2) != 0;
      if (stored) mask |= 1u << s;
      if (stored || ((mask0 >> s) & 1u))
        B.hist[lp][(size_t)s * n + i] = stored ? hist[e] : V2<T>{T(0), T(0)};
    }
    if (mask != mask0) B.head[lp][i].x = (unsigned)cnt | (mask << 8);
  }
  if (books) B.diss_part[gw] = acc_diss;
  if (blockIdx.x == 0 && t == 0) {
    ctl->sp = sp;
    ctl->evals = eval;
    ctl->disp = disp;
    ctl->epoch = epoch;
    ctl->rebuild_pending = rebuild;
    if (bad) atomicOr(&ctl->status, (int)kStatusNonfinite);
    const int keep_going = eval < target && !bad;
    if (use_cond & 1) cudaGraphSetConditional(h_rebuild, (unsigned)rebuild);
    if (use_cond & 2) cudaGraphSetConditional(h_loop, (unsigned)keep_going);
  }
}

// A thread per disc: it keeps the disc's state in registers and its partner
// indices, contact history and bond slots in shared memory, and evaluates its
// bonds and candidates itself. For engines with bonds or an indenter (dealing
// each bond once to the block's threads was no faster, and a bond's two sides
// round differently in the one-step kernels, so it also changed the results'
// last bits), and for dilute ones.
template <class T, bool FEAT, bool LOCAL, bool BIG>
__device__ __forceinline__ void run_discs(const Params<T>& P, const Bufs<T>& B, unsigned char* run_smem,
                                          cudaGraphConditionalHandle h_rebuild, cudaGraphConditionalHandle h_loop,
                                          int use_cond, int pb) {
  constexpr int MODE = kBatch;  // the first evaluation of a state primes it
  __shared__ unsigned s_vmax[3], s_out[4];
  __shared__ int s_bad[3];
  Ctl* ctl = B.ctl;
  const int t = threadIdx.x, lane = t & 31;
  const int n = P.n;
  const int i = blockIdx.x * pb + t;
  const bool own = t < pb && i < n;
  int sp = ctl->sp;
  const int lp = ctl->lp;
  long long eval = ctl->evals;
  const long long target = ctl->target;
  float disp = ctl->disp;
  unsigned epoch = ctl->epoch;
  if (t < 3) {
    s_vmax[t] = 0u;
    s_bad[t] = 0;
  }
  const RunLayout Y = run_layout<T>(P.W, FEAT ? P.BMAX : 0, pb, LOCAL ? 1 : 0, n);
  V4<T>* const lpos = reinterpret_cast<V4<T>*>(run_smem + Y.pos);
  V4<T>* const lvel = reinterpret_cast<V4<T>*>(run_smem + Y.vel);
  V2<T>* const hist = reinterpret_cast<V2<T>*>(run_smem + Y.hist);
  unsigned* const tail = reinterpret_cast<unsigned*>(run_smem + Y.tail);
  T* const strain = LOCAL ? reinterpret_cast<T*>(run_smem + Y.strain) : B.strain;
  // the bond slots of this block's discs, as do_bond addresses them
  Bufs<T> LB = B;
  if (FEAT) {
    LB.bpart[0] = reinterpret_cast<unsigned*>(run_smem + Y.bpart);
    LB.bref[0] = reinterpret_cast<V2<T>*>(run_smem + Y.bref);
    LB.bus[0] = reinterpret_cast<V2<T>*>(run_smem + Y.bus);
    LB.bstr[0] = reinterpret_cast<T*>(run_smem + Y.bstr);
    LB.bfail[0] = reinterpret_cast<int*>(run_smem + Y.bfail);
  }
  // this thread's disc
  V4<T> p{}, v{}, pi{};
  uint4 hd = make_uint4(0u, 0u, 0u, 0u);
  float2 rem = make_float2(0.0f, 0.0f);
  int bc = 0;
  if (own) {
    p = B.pos[sp][i];
    v = B.vel[sp][i];
    hd = B.head[lp][i];
    if (sizeof(T) == 4 && P.prem) rem = B.prem[lp][i];
    if (LOCAL) {
      lpos[sp * n + i] = p;
      lvel[sp * n + i] = v;
    }
    const int cnt = (int)(hd.x & 0xFFu);
    for (int s = kHeadSlots; s < cnt; ++s) tail[(s - kHeadSlots) * pb + t] = B.nbr[lp][(size_t)(s - kHeadSlots) * n + i];
    for (int s = 0; s < cnt; ++s)
      if ((hd.x >> (8 + s)) & 1u) hist[s * pb + t] = B.hist[lp][(size_t)s * n + i];
    if (FEAT && P.BMAX > 0) {
      bc = B.bcnt[lp][i];
      pi = B.bpinv[lp][i];
      for (int u = 0; u < bc; ++u) {
        const size_t k = (size_t)u * n + i;
        LB.bpart[0][u * pb + t] = B.bpart[lp][k];
        LB.bref[0][u * pb + t] = B.bref[lp][k];
        LB.bus[0][u * pb + t] = B.bus[lp][k];
        LB.bstr[0][u * pb + t] = B.bstr[lp][k];
        LB.bfail[0][u * pb + t] = B.bfail[lp][k];
      }
    }
  }
  const uint4 hd0 = hd;
  // ledger partials of this warp's 32 discs (slot i / 32), carried in lane 0
  const size_t gw = (size_t)i >> 5;
  const bool books = lane == 0 && own;
  double acc_diss = books ? B.diss_part[gw] : 0.0;
  double acc_frac = FEAT && books ? B.frac_part[gw] : 0.0;
  int acc_broke = 0;
  // The helper warp (one more warp than the discs need, engines with an
  // indenter) sums the reaction of the evaluation before, in block 0.
  const bool ind = FEAT && P.irad > T(0);
  const bool helper = ind && blockIdx.x == 0 && t >= pb;
  const size_t half = 3 * (size_t)P.ind_slots;
  Reaction R{0.0, 0.0, 0.0};
  if (helper && lane == 0) R.work = ctl->tool_work;
  const long long first = eval;
  int k3 = 0;  // shared-memory reduction slot of the step
  bool late = false;
  unsigned bad = 0u;
  int rebuild = 0;
  __syncthreads();
  while (true) {
    const int primed = eval > 0 ? 1 : 0;
    const PlainFetch<T> fetch{LOCAL ? lpos + sp * n : B.pos[sp], LOCAL ? lvel + sp * n : B.vel[sp]};
    if (FEAT && P.BMAX > 0) {
      T sv = T(0);
      if (bc > 0) {
        T g00 = 0, g01 = 0, g10 = 0, g11 = 0;
        V4<T> q[kMaxBondSlots];
#pragma unroll
        for (int u = 0; u < kMaxBondSlots; ++u)
          if (u < bc) q[u] = fetch.p((int)(LB.bpart[0][u * pb + t] & kBondIdx));
#pragma unroll
        for (int u = 0; u < kMaxBondSlots; ++u) {
          if (u < bc) {
            const V2<T> r = LB.bref[0][u * pb + t];
            const V2<T> cur = cell_delta<T>(P, p, q[u]);
            const T ux = cur.x - r.x, uy = cur.y - r.y;
            g00 += ux * r.x;
            g01 += ux * r.y;
            g10 += uy * r.x;
            g11 += uy * r.y;
          }
        }
        sv = shear_invariant<T>(g00, g01, g10, g11, pi);
      }
      if (own) strain[i] = sv;
      if (LOCAL) {
        __syncthreads();
      } else {
        grid_barrier(ctl, gridDim.x, epoch, nullptr, nullptr, P.wait_budget, s_out);
        ++epoch;
        if (s_out[3]) {
          late = true;
          break;
        }
      }
    }
    ThreadLedger<T> L;
    if (own) {
      Acc<T> fx, fy, tq;
      if (FEAT && bc > 0) {
        const T si = strain[i];
        constexpr int KB = 2;
#pragma unroll
        for (int s0 = 0; s0 < kMaxBondSlots; s0 += KB) {
          if (s0 >= bc) break;
          BondIn<T> in[KB];
#pragma unroll
          for (int u = 0; u < KB; ++u) {
            if (s0 + u < bc) {
              const int k = (s0 + u) * pb + t;
              in[u].w = LB.bpart[0][k];
              const int j = (int)(in[u].w & kBondIdx);
              in[u].q = fetch.p(j);
              in[u].wv = fetch.v(j);
              in[u].sj = strain[j];
              in[u].rs = LB.bref[0][k];
              in[u].us = LB.bus[0][k];
              in[u].sf = LB.bstr[0][k];
            }
          }
#pragma unroll
          for (int u = 0; u < KB; ++u)
            if (s0 + u < bc)
              do_bond<T, MODE>(P, LB, 0, i, (size_t)((s0 + u) * pb + t), eval, p, v, in[u], si, fx, fy, tq, L, primed);
        }
      }
      const int cnt = (int)(hd.x & 0xFFu);
      const unsigned mask = hd.x >> 8;
      unsigned nmask = 0u;
      // a few candidates at a time: their positions, then the velocities of
      // those that touch, then the laws in slot order
      constexpr int KS = BIG ? 1 : kHeadSlots;
      for (int s0 = 0; s0 < cnt; s0 += KS) {
        int j[KS];
        V4<T> q[KS], w[KS];
        Geo<T> g[KS];
        bool on[KS];
#pragma unroll
        for (int u = 0; u < KS; ++u) {
          on[u] = s0 + u < cnt;
          if (on[u]) {
            const int s = s0 + u;
            j[u] = (int)(s == 0 ? hd.y : s == 1 ? hd.z : s == 2 ? hd.w : tail[(s - kHeadSlots) * pb + t]);
            q[u] = fetch.p(j[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < KS; ++u) {
          if (on[u]) {
            g[u] = pair_geo<T>(P, p, q[u]);
            on[u] = g[u].d2 < g[u].rs * g[u].rs;
            if (on[u]) w[u] = fetch.v(j[u]);
            canonical<T>(g[u], i < j[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < KS; ++u) {
          if (on[u]) {
            const int s = s0 + u;
            const bool stored = (mask >> s) & 1u;
            V2<T>* slot = hist + s * pb + t;
            const V2<T> xi0 = stored ? *slot : V2<T>{T(0), T(0)};
            touching_slot<T, MODE>(P, slot, i, j[u], s, g[u], p, v, q[u], w[u], xi0, stored, nmask, fx, fy, tq, L.diss,
                                   L.un, L.ut, primed);
          }
        }
      }
      hd.x = (hd.x & 0xFFu) | (nmask << 8);
      if (FEAT && P.irad > T(0)) indenter_contact<T>(P, eval, p, v, fx, fy, L);
      wall_contacts<T, MODE>(P, B.whist[lp], i, p, v, fx, fy, tq, L, primed);
      const T Fx = fx.get(), Fy = fy.get(), Tz = tq.get();
      const T inv_m = v.w;
      const bool free = inv_m > T(0);
      const T ax = free ? Fx * inv_m + P.gx : T(0);
      const T ay = free ? Fy * inv_m + P.gy : T(0);
      T al = Tz;
      if (Tz != T(0)) al = Tz * (inv_m * P.kinv / (p.z * p.z));
      const Moved<T> m = move_particle<T, MODE>(P, p, v, rem, ax, ay, al, primed, L);
      p = m.pos;
      v = m.vel;
      rem = m.rem;
      if (LOCAL) {
        lpos[(sp ^ 1) * n + i] = p;
        lvel[(sp ^ 1) * n + i] = v;
      } else {
        B.pos[sp ^ 1][i] = p;
        B.vel[sp ^ 1][i] = v;
      }
    } else if (helper && eval > first) {
      book_reaction(P, B, eval - 1, half, R);
    }
    // the warp's ledger partials (most warps have none)
    const unsigned wbits = __reduce_max_sync(0xffffffffu, __float_as_uint(L.vmax2));
    const bool wbad = __any_sync(0xffffffffu, L.bad);
    if (lane == 0) {
      if (wbits) atomicMax(&s_vmax[k3], wbits);
      if (wbad) s_bad[k3] = 1;
    }
    if (__any_sync(0xffffffffu, L.diss != T(0))) {
      T x = L.diss;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
      acc_diss += (double)x;
    }
    if (FEAT && __any_sync(0xffffffffu, L.frac != T(0) || L.broke != 0 || L.ifx != T(0) || L.ify != T(0))) {
      T wf = L.frac, wx = L.ifx, wy = L.ify;
      int wb = L.broke;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        wf += __shfl_xor_sync(0xffffffffu, wf, off);
        wx += __shfl_xor_sync(0xffffffffu, wx, off);
        wy += __shfl_xor_sync(0xffffffffu, wy, off);
        wb += __shfl_xor_sync(0xffffffffu, wb, off);
      }
      acc_frac += (double)wf;
      acc_broke += wb;
      if (lane == 0 && (wx != T(0) || wy != T(0))) {
        const unsigned e = atomicAdd(&ctl->entries[eval & 1], 1u);
        double* o = B.ind_part + (eval & 1) * half + 3 * (size_t)e;
        o[0] = (double)gw;
        o[1] = (double)wx;
        o[2] = (double)wy;
      }
    }
    const int k1 = k3 == 2 ? 0 : k3 + 1;
    unsigned vbits;
    if (t == 0) {  // the next step's slots: last read a step ago
      s_vmax[k1] = 0u;
      s_bad[k1] = 0;
    }
    if (LOCAL) {
      __syncthreads();
      vbits = s_vmax[k3];
      bad = (unsigned)s_bad[k3];
    } else {
      grid_barrier(ctl, gridDim.x, epoch, &s_vmax[k3], &s_bad[k3], P.wait_budget, s_out);
      ++epoch;
      if (s_out[3]) {
        late = true;
        break;
      }
      vbits = s_out[1];
      bad = s_out[2];
    }
    k3 = k1;
    sp ^= 1;
    ++eval;
    disp += sqrtf(__uint_as_float(vbits)) * (float)P.dt;
    rebuild = disp > P.rebuild_disp ? 1 : 0;
    if (rebuild || bad || eval >= target) break;
  }
  if (late) {  // a barrier ran out of time: the state is not usable
    if (t == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  // write back what stayed on the chip
  if (own) {
    if (LOCAL) {
      B.pos[sp][i] = p;
      B.vel[sp][i] = v;
    }
    if (sizeof(T) == 4 && P.prem) B.prem[lp][i] = rem;
    const int cnt = (int)(hd.x & 0xFFu);
    const unsigned any = (hd.x | hd0.x) >> 8;
    for (int s = 0; s < cnt; ++s)
      if ((any >> s) & 1u) B.hist[lp][(size_t)s * n + i] = ((hd.x >> (8 + s)) & 1u) ? hist[s * pb + t] : V2<T>{T(0), T(0)};
    if (hd.x != hd0.x) B.head[lp][i].x = hd.x;
    if (FEAT) {
      for (int u = 0; u < bc; ++u) {
        const size_t k = (size_t)u * n + i;
        B.bpart[lp][k] = LB.bpart[0][u * pb + t];
        B.bus[lp][k] = LB.bus[0][u * pb + t];
        B.bfail[lp][k] = LB.bfail[0][u * pb + t];
      }
      if (P.BMAX > 0 && LOCAL) B.strain[i] = strain[i];
    }
  }
  if (books) {
    B.diss_part[gw] = acc_diss;
    if (FEAT) {
      B.frac_part[gw] = acc_frac;
      if (acc_broke) atomicAdd(&ctl->broken, acc_broke);
    }
  }
  if (helper) {
    book_reaction(P, B, eval - 1, half, R);
    if (lane == 0) {
      ctl->reaction_x = R.x;
      ctl->reaction_y = R.y;
      ctl->tool_work = R.work;
    }
  }
  if (blockIdx.x == 0 && t == 0) {
    ctl->sp = sp;
    ctl->evals = eval;
    ctl->disp = disp;
    ctl->epoch = epoch;
    ctl->rebuild_pending = rebuild;
    if (bad) atomicOr(&ctl->status, (int)kStatusNonfinite);
    const int keep_going = eval < target && !bad;
    if (use_cond & 1) cudaGraphSetConditional(h_rebuild, (unsigned)rebuild);
    if (use_cond & 2) cudaGraphSetConditional(h_loop, (unsigned)keep_going);
  }
}

template <class T, bool FEAT, bool LOCAL, bool BIG>
__global__ void __launch_bounds__(run_block<T>(FEAT, BIG), 1)
    force_kernel_run(Params<T> P, Bufs<T> B, cudaGraphConditionalHandle h_rebuild, cudaGraphConditionalHandle h_loop,
                     int use_cond, int pb, int mc) {
  extern __shared__ __align__(16) unsigned char run_smem[];
  if (B.ctl->status & (kStatusNonfinite | kStatusTimeout)) {  // nothing to do with such a state
    if (blockIdx.x == 0 && threadIdx.x == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  // from one candidate pair per disc on, pairs pay for their barrier (FP32, us a
  // step, discs / pairs: 50,071 touching discs 8.6 / 7.1, 90,000 dilute ones 4.3 / 5.6)
  if (!FEAT && B.ctl->candidates >= 2ll * P.n)
    run_pairs<T, LOCAL, BIG>(P, B, run_smem, h_rebuild, h_loop, use_cond, pb, mc);
  else
    run_discs<T, FEAT, LOCAL, BIG>(P, B, run_smem, h_rebuild, h_loop, use_cond, pb);
}

// Resident form of the pipelined step (FP32), for engines of many discs per
// thread: the one-step kernel's pass over the discs, with a grid barrier in the
// place of the launch. At 1,048,576 discs the launch, its ramp and its last
// block cost 6 us of a 24 us step. Measured (GB300, steps and a state read):
// 1,048,576 discs x 100 steps 2,894 -> 2,717 us, 4,194,304 discs x 40 steps
// 6,708 -> 4,920 us (the default loop had been the one-thread-per-disc kernel),
// the 1,048,576-disc bonded sheet x 40 steps 6,026 -> 5,605 us; with read_kernel
// and the lean contact test 2,425, 3,747 and 5,435 us.
// CHUNKED: ledger partials per 32 sorted discs, as variant 0 books them; else
// per warp of the grid, as the pipelined variants do.
template <class T, int BLOCK, bool FEAT, bool CHUNKED>
__global__ void __launch_bounds__(BLOCK, 1)
    force_kernel_run_async(Params<T> P, Bufs<T> B, cudaGraphConditionalHandle h_rebuild,
                           cudaGraphConditionalHandle h_loop, int use_cond, int, int) {
  extern __shared__ __align__(16) unsigned char run_smem[];
  __shared__ unsigned s_vmax[3], s_out[4];
  __shared__ int s_bad[3];
  Ctl* ctl = B.ctl;
  const int t = threadIdx.x, lane = t & 31;
  int sp = ctl->sp;
  const int lp = ctl->lp;
  long long eval = ctl->evals;
  const long long target = ctl->target, first = eval;
  float disp = ctl->disp;
  unsigned epoch = ctl->epoch;
  if (ctl->status & (kStatusNonfinite | kStatusTimeout)) {
    if (blockIdx.x == 0 && t == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  if (t < 3) {
    s_vmax[t] = 0u;
    s_bad[t] = 0;
  }
  const size_t warp = (size_t)blockIdx.x * (BLOCK / 32) + (t >> 5);
  double acc_diss = 0.0, acc_frac = 0.0;
  int acc_broke = 0;
  if (!CHUNKED && lane == 0) {
    acc_diss = B.diss_part[warp];
    if (FEAT) acc_frac = B.frac_part[warp];
  }
  const size_t half = 3 * (size_t)P.ind_slots;
  // block 0's first warp sums the reaction of the evaluation before
  const bool books = FEAT && P.irad > T(0) && blockIdx.x == 0 && t < 32;
  Reaction R{books && lane == 0 ? ctl->tool_work : 0.0, 0.0, 0.0};
  int k3 = 0, rebuild = 0;
  unsigned bad = 0u;
  bool late = false;
  __syncthreads();
  while (true) {
    if (FEAT && books && eval > first) book_reaction(P, B, eval - 1, half, R);
    if (FEAT && P.BMAX > 0) {
      strain_pass<T, BLOCK>(P, B, run_smem, sp, lp);
      grid_barrier(ctl, gridDim.x, epoch++, nullptr, nullptr, P.wait_budget, s_out);
      if (s_out[3]) {
        late = true;
        break;
      }
    }
    ThreadLedger<T> L;
    const PlainFetch<T> fetch{B.pos[sp], B.vel[sp]};
    // one ledger slot: the terms of `count` lanes (the last chunk may be short)
    auto book = [&](unsigned m, int count, size_t slot) {
      auto total = [&](auto x) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const auto y = __shfl_xor_sync(m, x, off);
          x += (lane ^ off) < count ? y : decltype(x)(0);
        }
        return x;
      };
      if (__any_sync(m, L.diss != T(0))) {
        const T x = total(L.diss);
        if (CHUNKED) {
          if (lane == 0) atomicAdd(&B.diss_part[slot], (double)x);
        } else {
          acc_diss += (double)x;
        }
      }
      if (FEAT && __any_sync(m, L.frac != T(0) || L.broke != 0 || L.ifx != T(0) || L.ify != T(0))) {
        const T f = total(L.frac), x = total(L.ifx), y = total(L.ify);
        const int broke = total(L.broke);
        if (CHUNKED) {
          if (lane == 0 && f != T(0)) atomicAdd(&B.frac_part[slot], (double)f);
        } else {
          acc_frac += (double)f;
        }
        acc_broke += broke;
        if (lane == 0 && (x != T(0) || y != T(0))) {
          const unsigned e = atomicAdd(&ctl->entries[eval & 1], 1u);
          double* o = B.ind_part + (eval & 1) * half + 3 * (size_t)e;
          o[0] = (double)slot;
          o[1] = (double)x;
          o[2] = (double)y;
        }
      }
    };
    async_pass<T, kBatch, BLOCK, FEAT, true, FEAT>(
        P, B, fetch, reinterpret_cast<uint4*>(run_smem), sp, lp, eval > 0 ? 1 : 0, eval, L, [&](int i) {
          if (CHUNKED) {
            const int count = min(32, P.n - (i - lane));
            book(count == 32 ? 0xffffffffu : (1u << count) - 1u, count, (size_t)i >> 5);
            L.diss = L.frac = L.ifx = L.ify = T(0);
            L.broke = 0;
          }
        });
    __syncwarp();
    if (!CHUNKED) book(0xffffffffu, 32, warp);
    const unsigned wbits = __reduce_max_sync(0xffffffffu, __float_as_uint(L.vmax2));
    const bool wbad = __any_sync(0xffffffffu, L.bad);
    if (lane == 0) {
      if (wbits) atomicMax(&s_vmax[k3], wbits);
      if (wbad) s_bad[k3] = 1;
    }
    const int k1 = k3 == 2 ? 0 : k3 + 1;
    if (t == 0) {
      s_vmax[k1] = 0u;
      s_bad[k1] = 0;
    }
    grid_barrier(ctl, gridDim.x, epoch++, &s_vmax[k3], &s_bad[k3], P.wait_budget, s_out);
    if (s_out[3]) {
      late = true;
      break;
    }
    bad = s_out[2];
    k3 = k1;
    sp ^= 1;
    ++eval;
    disp += sqrtf(__uint_as_float(s_out[1])) * (float)P.dt;
    rebuild = disp > P.rebuild_disp ? 1 : 0;
    if (rebuild || bad || eval >= target) break;
  }
  if (late) {
    if (t == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  if (lane == 0) {
    if (!CHUNKED) {
      B.diss_part[warp] = acc_diss;
      if (FEAT) B.frac_part[warp] = acc_frac;
    }
    if (FEAT && acc_broke) atomicAdd(&ctl->broken, acc_broke);
  }
  if (FEAT && books) {
    book_reaction(P, B, eval - 1, half, R);
    if (lane == 0) {
      ctl->reaction_x = R.x;
      ctl->reaction_y = R.y;
      ctl->tool_work = R.work;
    }
  }
  if (blockIdx.x == 0 && t == 0) {
    ctl->sp = sp;
    ctl->evals = eval;
    ctl->disp = disp;
    ctl->epoch = epoch;
    ctl->rebuild_pending = rebuild;
    if (bad) atomicOr(&ctl->status, (int)kStatusNonfinite);
    if (use_cond & 1) cudaGraphSetConditional(h_rebuild, (unsigned)rebuild);
    if (use_cond & 2) cudaGraphSetConditional(h_loop, (unsigned)(eval < target && !bad ? 1 : 0));
  }
}

template <class T>
RunFn<T> run_fn(bool feat, bool local, bool big) {
  if (local) return feat ? &force_kernel_run<T, true, true, false> : &force_kernel_run<T, false, true, false>;
  if (big) return feat ? &force_kernel_run<T, true, false, true> : &force_kernel_run<T, false, false, true>;
  return feat ? &force_kernel_run<T, true, false, false> : &force_kernel_run<T, false, false, false>;
}
template RunFn<float> run_fn<float>(bool, bool, bool);
template RunFn<double> run_fn<double>(bool, bool, bool);

RunFn<float> run_async_fn(bool feat, bool chunked) {
  constexpr int W = kRunAsync<false>, H = kRunAsync<true>;
  if (feat) return chunked ? &force_kernel_run_async<float, H, true, true> : &force_kernel_run_async<float, H, true, false>;
  return chunked ? &force_kernel_run_async<float, W, false, true> : &force_kernel_run_async<float, W, false, false>;
}

}  // namespace hm
}  // namespace tdem
