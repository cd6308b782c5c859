// Resident step kernel of the single-solve engine: one cooperative launch
// advances many steps, with a grid barrier in the place of the kernel boundary.
//
// What bounds a small or middle-sized engine is not bandwidth but the chain of
// one step. In the step graph a WHILE iteration costs 3.9 us with an empty body
// (a step of 3,249 discs took 11 us). Here a block owns a contiguous range of
// sorted discs for the whole launch, and a grid barrier (one arrival per block,
// one 16-byte poll that also returns the speed bound and the error flag) costs
// 1.2 us on 152 blocks; an engine of one block needs none. Only positions and
// velocities that other blocks read go through L2. Two ways through a step:
//
// A thread per disc keeps the disc's state in registers and its partner indices,
// history and bond slots in shared memory, and evaluates its bonds and
// candidates one after another.
//
// A thread per pair (no bonds, a candidate pair per disc or more): each pair of
// the block is evaluated once, also when both discs are the block's, by any of
// its threads; a disc's thread then sums the results in slot order. At this
// occupancy a contact law is a chain of 0.4 us, and a disc of a bed has six
// candidates; in FP64 the pipe (two lanes a clock) bounds the law itself.
//
// Measured (GB300, a pass of upload where it says so, n steps, read-back):
//                                              one-step  per disc  per pair
//   300 touching discs x 100 steps, upload        1,924       950       713 us
//   3,249 dilute discs x 200 steps, upload        2,405       814       852
//     (667 and 801 with the lists of small engines built by one block)
//   50,071 touching discs x 100 steps             1,822       954       835
//   65,535 touching discs x 50 steps, FP64        7,618     6,486     3,938
//     (3,636 with each pair's effective radius and mass kept)
//   2,328-disc bonded sheet x 200 steps, upload   5,083     2,620         -
//
// The launch ends when the list must be rebuilt, the step target is reached or
// the state went non-finite; the step graph loops around it. Every disc is
// evaluated by the same code in the same order as in the one-step kernels, so
// the states are bit-identical to theirs.
#pragma once

#include "hm2d_dev.cuh"

namespace tdem {
namespace hm {

// Grid barrier k = epoch of a cooperative launch of nb blocks, called by every
// thread; vmax2_bits and bad (shared, or null) hold the block's own values. out
// (shared) gets {arrivals, largest vmax2_bits, any bad, 1 if the wait ran out}.
// The words rotate by three: block 0 zeroes the next one before it arrives,
// when the last waiters of its previous use (two barriers ago) have passed.
// Waits at most `budget` clocks.
__device__ __forceinline__ void grid_barrier(Ctl* ctl, unsigned nb, unsigned epoch, const unsigned* block_vmax2,
                                             const int* block_bad, long long budget, unsigned* out) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned vmax2_bits = block_vmax2 ? *block_vmax2 : 0u;
    const int bad = block_bad ? *block_bad : 0;
    GridWord* w = &ctl->word[epoch % 3];
    if (blockIdx.x == 0) *reinterpret_cast<uint4*>(&ctl->word[(epoch + 1) % 3]) = make_uint4(0u, 0u, 0u, 0u);
    if (vmax2_bits) atomicMax(&w->vmax2_bits, vmax2_bits);
    if (bad) atomicOr(&w->bad, 1u);
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&w->count) : "memory");
    const long long start = clock64();
    unsigned long long lo, hi;
    unsigned late = 0;
    while (true) {
      asm volatile(
          "{\n\t.reg .b128 t;\n\t"
          "ld.acquire.gpu.global.b128 t, [%2];\n\t"
          "mov.b128 {%0, %1}, t;\n\t}"
          : "=l"(lo), "=l"(hi)
          : "l"(w)
          : "memory");
      if ((unsigned)lo >= nb) break;
      if (clock64() - start > budget || budget <= 0) {
        late = 1;
        atomicOr(&ctl->status, (int)kStatusTimeout);
        break;
      }
    }
    out[0] = (unsigned)lo;
    out[1] = (unsigned)(lo >> 32);
    out[2] = (unsigned)hi;
    out[3] = late;
  }
  __syncthreads();
}

// Partner state through plain (coherent) loads: the buffers change under a
// resident launch, so nothing may promise that they are read-only.
template <class T>
struct PlainFetch {
  const V4<T>* pos;
  const V4<T>* vel;
  __device__ __forceinline__ V4<T> p(int j) const { return pos[j]; }
  __device__ __forceinline__ V4<T> v(int j) const { return vel[j]; }
};

// Threads per block, in two builds: `big` halves the registers of a thread for
// engines that need every thread of the chip. Without spills bonds and FP64
// take up to 255 registers, FP32 contacts 128.
template <class T>
constexpr int run_block(bool feat, bool big) {
  return (sizeof(T) == 4 && !feat ? 512 : 256) * (big ? 2 : 1);
}

// Discs of a block: at least kRunDiscs in a grid; up to kRunLocal (with bonds
// kRunLocalBonds) stay in one block. Measured (GB300, us a step):
//   blocks of 32 / 64 / 128 / 256 discs: 3,249 touching discs 4.9 / 5.0 / 5.0 / 5.8,
//     dilute 2.5 / 2.4 / 2.5 / 2.6, 2,328 bonded 10.4 / 10.0 / 10.0 / 10.3, 182
//     bonded 10.5 / 9.6 / 9.5 / 9.5; in FP64 3,249 touching discs 16.1 / 17.2 / 25.0 /
//     39.1 (smaller blocks would pay there), 16,384 24.9 / 24.9 / 24.9 / 38.7;
//   one block / a grid: 256 touching discs 3.9 / 4.6, 400 4.7 / 4.9, 506 4.8 / 4.6;
//     256 dilute 1.1 / 2.3, 484 1.3 / 2.5; 128 bonded 7.6 / 10.0 (182 would still gain,
//     7.6 / 9.5); FP64, 256 touching discs 29.9 / 20.4 (a grid would pay from there).
constexpr int kRunDiscs = 128;
constexpr int kRunLocal = 512;
constexpr int kRunLocalBonds = 128;

// Shared memory of a block without bonds that owns `pb` discs and has room for
// mc pairs: byte offsets. kRunPairs: pairs per disc it must have room for (a
// hexagonal bed evaluates 3.4 per disc of a 128-disc block, 3.2 of a 352-disc
// one); a block with more works on the global arrays.
constexpr int kRunPairs = 4;

struct PairLayout {
  size_t pos, vel, res, hist, desc, base, place, touch, on, total;
};

template <class T>
__host__ __device__ inline PairLayout pair_layout(int W, int pb, int mc) {
  PairLayout L;
  size_t o = 0;
  const size_t b = (size_t)pb, c = (size_t)mc;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 15) & ~size_t(15);
    return at;
  };
  L.pos = take(b * sizeof(V4<T>));
  L.vel = take(b * sizeof(V4<T>));
  L.res = take(c * sizeof(V4<T>));
  L.hist = take(c * sizeof(V2<T>));
  L.desc = take(c * 8);
  L.base = take((b + 1) * 4);
  L.place = take((size_t)W * b * 2);
  L.touch = take(c * 2);
  L.on = take(c);
  L.total = o;
  return L;
}

// Shared memory of a block with bonds that owns `pb` discs: byte offsets.
struct RunLayout {
  size_t pos, vel, strain, hist, bref, bus, bstr, tail, bpart, bfail, total;
};

// local: the whole engine (n discs) in one block, positions in shared memory.
template <class T>
__host__ __device__ inline RunLayout run_layout(int W, int BM, int pb, int local, int n) {
  RunLayout L;
  size_t o = 0;
  const size_t m = local ? (size_t)n : 0, b = (size_t)pb;
  L.pos = o;
  o += 2 * m * sizeof(V4<T>);
  L.vel = o;
  o += 2 * m * sizeof(V4<T>);
  L.hist = o;
  o += (size_t)W * b * sizeof(V2<T>);
  L.bref = o;
  o += (size_t)BM * b * sizeof(V2<T>);
  L.bus = o;
  o += (size_t)BM * b * sizeof(V2<T>);
  L.strain = o;
  o += (BM > 0 ? m : 0) * sizeof(T);
  L.bstr = o;
  o += (size_t)BM * b * sizeof(T);
  o = (o + 7) & ~size_t(7);
  L.tail = o;
  o += (size_t)(W > kHeadSlots ? W - kHeadSlots : 0) * b * 4;
  L.bpart = o;
  o += (size_t)BM * b * 4;
  L.bfail = o;
  o += (size_t)BM * b * 4;
  L.total = o;
  return L;
}

// The kernel for an engine with (feat) or without bonds or an indenter, in one
// block with its positions in shared memory (local) or over a cooperative grid
// (of big blocks).
template <class T>
using RunFn = void (*)(Params<T>, Bufs<T>, cudaGraphConditionalHandle, cudaGraphConditionalHandle, int, int, int);
template <class T>
RunFn<T> run_fn(bool feat, bool local, bool big);

// The pipelined form for FP32 engines of many discs per thread, in the block
// shapes of variants 10 (without bonds or indenter) and 11 (with).
template <bool FEAT>
constexpr int kRunAsync = FEAT ? 512 : 1024;
RunFn<float> run_async_fn(bool feat, bool chunked);

}  // namespace hm
}  // namespace tdem
