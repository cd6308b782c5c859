// Resident step kernel of the batched engine.
//
// A batch step was three launches in a WHILE iteration (strain, granular
// tiles, other tiles), each with its own ramp and tail, and its warps held
// one tile at a time with the next tile's loads in registers. Here one
// 512-thread block per SM stays for the whole step block. Each warp owns a
// contiguous range of the granular tiles and one of the bonded tiles
// (contiguous, so an instance's parameters are copied to shared memory once;
// ranges of equal length, warp-major over the SMs, so the SMs differ by less
// than a tile per warp), and runs the single-solve engine's cp.async pipeline
// over them: the head of tile k+2, the state, bond words and partners of tile
// k+1 land while tile k is computed.
//
// Ledger rows stay per tile, in two column sets by evaluation parity: while
// the next evaluation runs, the warp that an instance falls to sums its rows
// of the last one in tile order. Every value is computed as in the one-step
// kernels, so the results are theirs bit for bit.
//
// Measured (GB300, a block of steps with its ledgers and two states read;
// one-step launches -> this): 32 runs of 100 to 2,000 discs (22,673 discs) x
// 100 steps 10,625 -> 2,209 us (99 -> 19 us a step: 91 chunks of 8 tiles had
// kept 91 of 4,864 warps busy); 256 runs of 100 to 20,000 discs (1.16M) x 40
// steps 12,832 -> 6,696 us (310 -> 124 us a step; L2 prefetches of the next tile's
// bond rows cost 9% of it).
#include "batch_run.cuh"

namespace tdem {
namespace hm {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kRowHalf = kTileVals / 2;  // columns of one parity: 5 sums and a "stepped" mark

template <class T>
__device__ __forceinline__ T lanes_sum(T x) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(kAll, x, off);
  return x;
}

// What a warp keeps across its tiles of one evaluation. No more than this: the
// bonded build is short of registers (an instance's evaluation index, its state
// in two words and the evaluation that these were read in, kept as well, were 7%
// of a step of 256 runs with 1.16M discs).
template <class T>
struct TileRun {
  Params<T>* Q;  // the open instance's parameters (shared memory, per warp)
  int inst;      // the open instance, -1: none
  int go;        // -1: to be read in this evaluation, 0: retired, 1: frozen, 2: stepped
  float vmax;    // max over the thread's discs of (|v| dt / rebuild displacement)^2
};

// Marks instance k non-finite in the batch's evaluation eval: the evaluation
// first, then the bit that says to look for it. (No memory clobber, here and
// below: nothing else needs these orders.)
template <class T>
__device__ __forceinline__ void mark_bad(const Bufs<T>& B, int k, long long eval) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;\n\tred.release.gpu.global.or.b32 [%2], %3;" ::"l"(
                   B.iled + (size_t)k * kInstLedger + kInstBadAt),
               "d"((double)(eval + 1)), "l"(B.istate + k), "r"((int)kStatusNonfinite));
}

// What mark_bad wrote, after its bit was seen: the evaluation after, 0 if the
// bit is not a resident step's.
template <class T>
__device__ __forceinline__ double marked_at(const Bufs<T>& B, int k) {
  double at;
  asm volatile("{\n\t.reg .b32 t;\n\tld.acquire.gpu.global.b32 t, [%1];\n\tld.relaxed.gpu.global.f64 %0, [%2];\n\t}"
               : "=d"(at)
               : "l"(B.istate + k), "l"(B.iled + (size_t)k * kInstLedger + kInstBadAt));
  return at;
}

template <class T>
__device__ __forceinline__ void open_instance(const Bufs<T>& B, TileRun<T>& S, int k, long long eval) {
  if (k == S.inst && S.go >= 0) return;
  const int lane = threadIdx.x & 31;
  const int st = *reinterpret_cast<volatile int*>(&B.istate[k]);
  if (k != S.inst) {
    S.inst = k;
    __syncwarp();
    const unsigned* src = reinterpret_cast<const unsigned*>(B.iparams + k);
    unsigned* dst = reinterpret_cast<unsigned*>(S.Q);
    for (int w = lane; w < (int)(sizeof(Params<T>) / 4); w += 32) dst[w] = src[w];
    __syncwarp();
  }
  // quarantine: see batch_kernel. The evaluation in which an instance goes
  // non-finite is taken by all its tiles, whichever warp opens it after the
  // mark: its rows are then of one evaluation, and are booked.
  int bad = (st | (st >> kInstRebuildShift)) & (kStatusNonfinite | kStatusEscaped | kStatusCapacity);
  if ((st & kStatusNonfinite) && !((st >> kInstRebuildShift) & kStatusNonfinite) &&
      marked_at(B, k) == (double)(eval + 1))
    bad &= ~(int)kStatusNonfinite;
  S.go = !(st & kInstAlive) ? 0 : eval - S.Q->eval0 >= S.Q->stop || bad != 0 ? 1 : 2;
}

// One disc of the tile is done: the tile's ledger row and the speed bound.
template <class T, bool FEAT>
__device__ __forceinline__ void close_tile(const Bufs<T>& B, TileRun<T>& S, int tile, long long eval, bool stepped,
                                           const ThreadLedger<T>& L) {
  const int lane = threadIdx.x & 31;
  double* row = B.tpart + (size_t)tile * kTileVals + (int)(eval & 1) * kRowHalf;
  if (!stepped) {
    if (lane == 0) row[5] = 0.0;
    return;
  }
  const float f = (float)S.Q->dt / S.Q->rebuild_disp;
  S.vmax = fmaxf(S.vmax, L.vmax2 * f * f);
  T wd = T(0), wf = T(0), wix = T(0), wiy = T(0);
  int wb = 0;
  if (__any_sync(kAll, L.diss != T(0))) wd = lanes_sum<T>(L.diss);
  if (FEAT && __any_sync(kAll, L.frac != T(0) || L.ifx != T(0) || L.ify != T(0) || L.broke != 0)) {
    wf = lanes_sum<T>(L.frac);
    wix = lanes_sum<T>(L.ifx);
    wiy = lanes_sum<T>(L.ify);
    wb = lanes_sum<int>(L.broke);
  }
  const bool bad = __any_sync(kAll, L.bad);
  if (lane == 0) {
    row[0] = (double)wd;
    row[1] = (double)wf;
    row[2] = (double)wix;
    row[3] = (double)wiy;
    row[4] = (double)wb;
    row[5] = 1.0;
    if (bad) mark_bad(B, S.inst, eval);
  }
}

// The force pass over tiles [tb, te), FP64: loads one tile ahead in registers.
template <class T, bool FEAT>
__device__ __forceinline__ void force_tiles_plain(const Bufs<T>& B, TileRun<T>& S, int tb, int te, int sp, int lp,
                                                  long long eval) {
  const int lane = threadIdx.x & 31;
  const PlainFetch<T> fetch{B.pos[sp], B.vel[sp]};
  for (int tile = tb; tile < te; ++tile) {
    const int4 d = B.tiles[tile];
    open_instance<T>(B, S, d.x, eval);
    const int i = d.y + lane;
    const bool on = lane < d.z;
    ThreadLedger<T> L;
    if (on && S.go) {
      const V4<T> p = fetch.p(i), v = fetch.v(i);
      if (S.go == 1) {
        B.pos[sp ^ 1][i] = p;
        B.vel[sp ^ 1][i] = v;
      } else {
        const uint4 hd = B.head[lp][i];
        V4<T> q0{}, q1{}, q2{};
        load_head_partners<T>(fetch, hd, q0, q1, q2);
        process_particle_q<T, kBatch, FEAT, PlainFetch<T>>(*S.Q, B, fetch, sp, lp, i, p, v, hd, q0, q1, q2, eval > S.Q->eval0 ? 1 : 0,
                                                           eval - S.Q->eval0, L);
      }
    }
    close_tile<T, FEAT>(B, S, tile, eval, S.go == 2, L);
  }
}

// The force pass over tiles [tb, te), FP32, pipelined as force_kernel_async.
template <class T, bool FEAT>
__device__ __forceinline__ void force_tiles(const Bufs<T>& B, TileRun<T>& S, unsigned char* smem, int n, int BM,
                                            int tb, int te, int sp, int lp, long long eval) {
  if constexpr (sizeof(T) == 8) {
    force_tiles_plain<T, FEAT>(B, S, tb, te, sp, lp, eval);
  } else {
    using bulk::cp16;
    using bulk::cp4;
    using bulk::cp8;
    using bulk::cp_commit;
    using bulk::cp_wait;
    constexpr int BL = kBatchRunBlock<T>;
    const int t = threadIdx.x, lane = t & 31;
    uint4* sh = reinterpret_cast<uint4*>(smem);                 // [3][BL]
    V4<T>* spos = reinterpret_cast<V4<T>*>(sh + 3 * BL);        // [2][BL]
    V4<T>* svel = spos + 2 * BL;                                 // [2][BL]
    V4<T>* sq = svel + 2 * BL;                                   // [2][3][BL]
    float2* srem = reinterpret_cast<float2*>(sq + 6 * BL);       // [2][BL]
    const float2* prem = B.prem[lp];
    const bool pr = prem != nullptr;
    unsigned* sbw = reinterpret_cast<unsigned*>(smem + (size_t)kAsyncRecords * BL * 16 + (pr ? (size_t)2 * BL * 8 : 0));
    int* sbc = reinterpret_cast<int*>(sbw + 2 * BM * BL);
    T* ssi = reinterpret_cast<T*>(sbc + 2 * BL);
    const PlainFetch<T> fetch{B.pos[sp], B.vel[sp]};
    auto desc = [&](int tile) { return tile < te ? B.tiles[tile] : make_int4(-1, 0, 0, 0); };
    auto head = [&](const int4& d, int h) {
      if (lane < d.z) cp16(sh + h * BL + t, B.head[lp] + d.y + lane);
    };
    auto own = [&](const int4& d, int s) {
      if (lane >= d.z) return;
      const int i = d.y + lane;
      cp16(spos + s * BL + t, fetch.pos + i);
      cp16(svel + s * BL + t, fetch.vel + i);
      if (pr) cp8(srem + s * BL + t, prem + i);
      if (FEAT && BM > 0) {
        for (int u = 0; u < BM; ++u) cp4(sbw + (s * BM + u) * BL + t, B.bpart[lp] + (size_t)u * n + i);
        cp4(sbc + s * BL + t, B.bcnt[lp] + i);
        cp4(ssi + s * BL + t, B.strain + i);
      }
    };
    auto gather = [&](const int4& d, int h, int s) {
      if (lane >= d.z) return;
      const uint4 hd = sh[h * BL + t];
      const int cnt = (int)(hd.x & 0xFFu);
      V4<T>* q = sq + (size_t)s * 3 * BL + t;
      if (cnt > 0) cp16(q, fetch.pos + hd.y);
      if (cnt > 1) cp16(q + BL, fetch.pos + hd.z);
      if (cnt > 2) cp16(q + 2 * BL, fetch.pos + hd.w);
    };
    int4 d0 = desc(tb), d1 = desc(tb + 1), d2 = desc(tb + 2);
    head(d0, 0);
    own(d0, 0);
    head(d1, 1);
    cp_commit();
    cp_wait<0>();
    gather(d0, 0, 0);
    cp_commit();
    int h0 = 0, s = 0;
    for (int tile = tb; tile < te; ++tile) {
      const int h1 = h0 == 2 ? 0 : h0 + 1, h2 = h1 == 2 ? 0 : h1 + 1;
      const int4 d3 = desc(tile + 3);
      head(d2, h2);
      own(d1, s ^ 1);
      cp_commit();
      cp_wait<2>();  // the head of the next tile has landed
      gather(d1, h1, s ^ 1);
      cp_commit();
      cp_wait<2>();  // this tile's partners have landed
      open_instance<T>(B, S, d0.x, eval);
      ThreadLedger<T> L;
      if (lane < d0.z && S.go) {
        const int i = d0.y + lane;
        const V4<T> p = spos[s * BL + t], v = svel[s * BL + t];
        if (S.go == 1) {
          B.pos[sp ^ 1][i] = p;
          B.vel[sp ^ 1][i] = v;
        } else {
          const uint4 hd = sh[h0 * BL + t];
          const V4<T>* q = sq + (size_t)s * 3 * BL + t;
          const int cnt = (int)(hd.x & 0xFFu);
          V4<T> q0{}, q1{}, q2{};
          if (cnt > 0) q0 = q[0];
          if (cnt > 1) q1 = q[BL];
          if (cnt > 2) q2 = q[2 * BL];
          const float2 rm = pr ? srem[s * BL + t] : make_float2(0.0f, 0.0f);
          if constexpr (FEAT) {
            process_particle_q<T, kBatch, true, PlainFetch<T>, false, true>(
                *S.Q, B, fetch, sp, lp, i, p, v, hd, q0, q1, q2, eval > S.Q->eval0 ? 1 : 0, eval - S.Q->eval0, L, &rm, sbw + s * BM * BL + t, BL,
                BM > 0 ? sbc[s * BL + t] : 0, BM > 0 ? ssi[s * BL + t] : T(0));
          } else {
            process_particle_q<T, kBatch, false, PlainFetch<T>>(*S.Q, B, fetch, sp, lp, i, p, v, hd, q0, q1, q2,
                                                                eval > S.Q->eval0 ? 1 : 0, eval - S.Q->eval0, L, &rm);
          }
        }
      }
      __syncwarp();
      close_tile<T, FEAT>(B, S, tile, eval, S.go == 2, L);
      d0 = d1;
      d1 = d2;
      d2 = d3;
      h0 = h1;
      s ^= 1;
    }
    cp_wait<0>();
  }
}

// The objective shear of the discs of tiles [tb, te), as strain_kernel (FP32:
// the next tile's first round staged by cp.async).
template <class T>
__device__ __forceinline__ void strain_tiles(const Bufs<T>& B, unsigned char* smem, int n, int BM, int tb, int te,
                                             int sp, int lp) {
  constexpr int BL = kBatchRunBlock<T>, S = kMaxBondSlots;
  const int t = threadIdx.x, lane = t & 31;
  const V4<T>* pos = B.pos[sp];
  auto sum = [&](const Params<T>& Q, int bc, const V4<T>& p, const V4<T>& pi, auto word, auto ref) {
    V4<T> q[S];
#pragma unroll
    for (int u = 0; u < S; ++u)
      if (u < bc) q[u] = pos[(int)(word(u) & kBondIdx)];
    T g00 = 0, g01 = 0, g10 = 0, g11 = 0;
#pragma unroll
    for (int u = 0; u < S; ++u) {
      if (u < bc) {
        const V2<T> r = ref(u);
        const V2<T> cur = cell_delta<T>(Q, p, q[u]);
        const T ux = cur.x - r.x, uy = cur.y - r.y;
        g00 += ux * r.x;
        g01 += ux * r.y;
        g10 += uy * r.x;
        g11 += uy * r.y;
      }
    }
    return bc > 0 ? shear_invariant<T>(g00, g01, g10, g11, pi) : T(0);
  };
  if constexpr (sizeof(T) == 8) {
    for (int tile = tb; tile < te; ++tile) {
      const int4 d = B.tiles[tile];
      if (lane >= d.z) continue;
      const int i = d.y + lane;
      const unsigned* bp = B.bpart[lp] + i;
      const V2<T>* br = B.bref[lp] + i;
      B.strain[i] = sum(B.iparams[d.x], B.bcnt[lp][i], pos[i], B.bpinv[lp][i],
                        [&](int u) { return bp[(size_t)u * n]; }, [&](int u) { return br[(size_t)u * n]; });
    }
  } else {
    using bulk::cp16;
    using bulk::cp4;
    using bulk::cp8;
    V4<T>* spos = reinterpret_cast<V4<T>*>(smem);                   // [2][BL]
    V4<T>* spi = spos + 2 * BL;                                      // [2][BL]
    V2<T>* sref = reinterpret_cast<V2<T>*>(spi + 2 * BL);            // [2][S][BL]
    unsigned* sw = reinterpret_cast<unsigned*>(sref + 2 * S * BL);   // [2][S][BL]
    int* sbc = reinterpret_cast<int*>(sw + 2 * S * BL);              // [2][BL]
    auto desc = [&](int tile) { return tile < te ? B.tiles[tile] : make_int4(-1, 0, 0, 0); };
    auto stage = [&](const int4& d, int st) {
      if (lane >= d.z) return;
      const int i = d.y + lane;
      cp4(sbc + st * BL + t, B.bcnt[lp] + i);
      cp16(spos + st * BL + t, pos + i);
      cp16(spi + st * BL + t, B.bpinv[lp] + i);
#pragma unroll
      for (int u = 0; u < S; ++u) {
        if (u < BM) {
          const size_t k = (size_t)u * n + i;
          cp4(sw + (st * S + u) * BL + t, B.bpart[lp] + k);
          cp8(sref + (st * S + u) * BL + t, B.bref[lp] + k);
        }
      }
    };
    int4 d0 = desc(tb), d1 = desc(tb + 1);
    stage(d0, 0);
    bulk::cp_commit();
    int st = 0;
    for (int tile = tb; tile < te; ++tile, st ^= 1) {
      const int4 d2 = desc(tile + 2);
      stage(d1, st ^ 1);
      bulk::cp_commit();
      bulk::cp_wait<1>();
      if (lane < d0.z)
        B.strain[d0.y + lane] =
            sum(B.iparams[d0.x], sbc[st * BL + t], spos[st * BL + t], spi[st * BL + t],
                [&](int u) { return sw[(st * S + u) * BL + t]; }, [&](int u) { return sref[(st * S + u) * BL + t]; });
      d0 = d1;
      d1 = d2;
    }
    bulk::cp_wait<0>();
  }
}

// Sums of instance k's rows of evaluation `eval` (one warp, tile order by lane).
template <class T>
__device__ __forceinline__ void book_instance(const Bufs<T>& B, int k, long long eval) {
  const int lane = threadIdx.x & 31;
  const int4 r = B.irange[k];
  const double* rows = B.tpart + (size_t)r.z * kTileVals + (eval & 1) * kRowHalf;
  if (__ldcg(rows + 5) == 0.0) return;  // not stepped in that evaluation
  double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int tt = lane; tt < r.w; tt += 32) {
    const double* rr = rows + (size_t)tt * kTileVals;
#pragma unroll
    for (int c = 0; c < 5; ++c) s[c] += __ldcg(rr + c);
  }
#pragma unroll
  for (int c = 0; c < 5; ++c) s[c] = lanes_sum<double>(s[c]);
  if (lane != 0) return;
  const Params<T>& Q = B.iparams[k];
  const long long le = eval - Q.eval0;
  double* led = B.iled + (size_t)k * kInstLedger;
  led[0] += s[0];                                              // dissipated
  led[1] += s[1];                                              // fracture release
  led[2] += (double)Q.dt * (s[2] * Q.ind_vx + s[3] * Q.ind_vy);  // tool work
  led[3] += s[4];                                              // bonds broken
  led[4] = -s[2];                                              // reaction on the indenter
  led[5] = -s[3];
  const double R = sqrt(s[2] * s[2] + s[3] * s[3]);
  if (R > led[6]) {
    led[6] = R;
    led[7] = (double)le;
  }
  led[8] = (double)(le + 1);  // evaluations committed
}

template <class T>
__global__ void __launch_bounds__(kBatchRunBlock<T>, 1)
    batch_run_kernel(Bufs<T> B, cudaGraphConditionalHandle h_rebuild, cudaGraphConditionalHandle h_loop, int use_cond,
                     int rebuild_every, int n, int BM, int slots, long long budget) {
  constexpr int NW = kBatchRunBlock<T> / 32;
  extern __shared__ __align__(16) unsigned char run_smem[];
  __shared__ alignas(16) Params<T> s_par[2 * NW];
  __shared__ unsigned s_vmax[3], s_out[4];
  Ctl* ctl = B.ctl;
  const int t = threadIdx.x, lane = t & 31;
  int sp = ctl->sp;
  const int lp = ctl->lp;
  long long eval = ctl->evals;
  const long long target = ctl->target, first = eval;
  float disp = ctl->disp;
  int since = ctl->since;
  unsigned epoch = ctl->epoch;
  const int nt = ctl->ntiles, ntp = ctl->ntiles_plain;
  if (ctl->status & kStatusTimeout) {
    if (blockIdx.x == 0 && t == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  if (t < 3) s_vmax[t] = 0u;
  const int nw = (int)gridDim.x * NW, gw = (t >> 5) * (int)gridDim.x + (int)blockIdx.x;
  auto part = [&](int count, int w) { return (int)((long long)count * w / nw); };
  const int pb = part(ntp, gw), pe = part(ntp, gw + 1);
  const int fb = ntp + part(nt - ntp, gw), fe = ntp + part(nt - ntp, gw + 1);
  const bool strains = BM > 0 && nt > ntp;
  // the instances this warp books: slots gw, gw + nw, ... that own tiles
  const int per = (slots - gw + nw - 1) / nw;  // slots of this warp (<= 0: none)
  unsigned mine = 0u;
  if (per <= 32) {
    const int k = gw + lane * nw;
    mine = __ballot_sync(kAll, lane < per && B.irange[k].w > 0 && (B.istate[k] & kInstAlive));
  }
  auto book = [&](long long e) {
    if (per <= 32) {
      for (unsigned m = mine; m; m &= m - 1) book_instance<T>(B, gw + (__ffs(m) - 1) * nw, e);
    } else {
      for (int k = gw; k < slots; k += nw)
        if (B.irange[k].w > 0 && (B.istate[k] & kInstAlive)) book_instance<T>(B, k, e);
    }
  };
  // open instances of the bonded and the granular range
  TileRun<T> S{&s_par[t >> 5], -1, -1, 0.0f}, G{&s_par[NW + (t >> 5)], -1, -1, 0.0f};
  int k3 = 0, rebuild = 0;
  bool late = false;
  __syncthreads();
  while (true) {
    if (strains) {
      strain_tiles<T>(B, run_smem, n, BM, fb, fe, sp, lp);
      grid_barrier(ctl, gridDim.x, epoch++, nullptr, nullptr, budget, s_out);
      if (s_out[3]) {
        late = true;
        break;
      }
    }
    S.vmax = G.vmax = 0.0f;
    S.go = G.go = -1;  // state words are read anew
    force_tiles<T, true>(B, S, run_smem, n, BM, fb, fe, sp, lp, eval);
    force_tiles<T, false>(B, G, run_smem, n, BM, pb, pe, sp, lp, eval);
    const unsigned bits = __reduce_max_sync(kAll, __float_as_uint(fmaxf(S.vmax, G.vmax)));
    if (lane == 0 && bits) atomicMax(&s_vmax[k3], bits);
    if (eval > first) book(eval - 1);
    const int k1 = k3 == 2 ? 0 : k3 + 1;
    if (t == 0) s_vmax[k1] = 0u;  // the next evaluation's slot: last read an evaluation ago
    grid_barrier(ctl, gridDim.x, epoch++, &s_vmax[k3], nullptr, budget, s_out);
    if (s_out[3]) {
      late = true;
      break;
    }
    k3 = k1;
    sp ^= 1;
    ++eval;
    ++since;
    disp += sqrtf(__uint_as_float(s_out[1]));  // in units of each instance's allowed displacement
    rebuild = (disp > 1.0f || (rebuild_every > 0 && since >= rebuild_every)) ? 1 : 0;
    if (rebuild || eval >= target) break;
  }
  if (late) {  // a barrier ran out of time: the state is not usable
    if (t == 0 && (use_cond & 2)) cudaGraphSetConditional(h_loop, 0u);
    return;
  }
  book(eval - 1);
  if (blockIdx.x == 0 && t == 0) {
    ctl->sp = sp;
    ctl->evals = eval;
    ctl->disp = disp;
    ctl->since = since;
    ctl->epoch = epoch;
    ctl->rebuild_pending = rebuild;
    if (use_cond & 1) cudaGraphSetConditional(h_rebuild, (unsigned)rebuild);
    if (use_cond & 2) cudaGraphSetConditional(h_loop, (unsigned)(eval < target ? 1 : 0));
  }
}

}  // namespace

template <class T>
BatchRunFn<T> batch_run_fn() {
  return &batch_run_kernel<T>;
}
template BatchRunFn<float> batch_run_fn<float>();
template BatchRunFn<double> batch_run_fn<double>();

}  // namespace hm
}  // namespace tdem
