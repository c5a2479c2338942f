// Kernels of one stream whose launches overlap.
//
// The passes of a step follow one another on a stream, and a small grid's pass
// takes about as long as its launch.  They are launched with programmatic stream
// serialisation: a pass's CTAs start, load the twiddle tables (which nothing writes
// after a context's creation) and set up their barriers before the pass in front has
// been retired, then wait here for its completion and its memory.  Every CTA
// waits, so that a pass's completion implies the completion of all before it.
// Nothing that another kernel or a copy writes is read before the wait, and none of
// it through the non-coherent path: __restrict__ stands on twiddle tables alone, in
// the kernels and in the helpers inlined into them (it measured the same).  The
// Stockham passes wait before they load their twiddles, which the allocation-free
// Poisson solve fills on the same stream;
// the adjoint at 128^3, 40 steps, went from 8.5 to 7.3 ms.
//
// When the next pass may start:
// - As a rule once every CTA of this one has exited (no trigger).  A trigger at the
//   start would let the next CTAs in beside the running ones, and they pile up on the
//   SMs that have room instead of spreading: 384^3 1277 -> 1384 us a step, 256^3
//   373 -> 422 (without overlap at all 1302 and 391).
// - At the start in grids of at most CHAIN_SMALL threads, which leave most SMs empty
//   in any case: 64^3 23.3 -> 21.1 us a step (without overlap 31.9), 48^3 23.3 -> 20.7.
//   The line, against a quarter and four times of it (8192 / 32768 / 131072), us a
//   step: 32^3 15.4 / 14.4 / 14.4, 64^3 23.1 / 20.8 / 20.8, two of 64^3 24.2 / 24.2 /
//   24.7, 96^3 38.8 / 38.5 / 44.1, 64 x 96 x 64 26.3 / 26.0 / 25.4.
//   Row passes, whose CTAs stay longest, at most CHAIN_SMALL_ROWS: replayed 192 x 32 x
//   32 (8192 threads) 36.2 -> 29.1, 192 x 48 x 8 28.6 -> 27.2, 256 x 8 x 48 33.9 ->
//   27.8; but 128 x 256 x 16 (16384) 34.8 -> 37.6, 192 x 96 x 48 (18432) 42.6 -> 49.5.
#pragma once

namespace wdm {

constexpr unsigned CHAIN_SMALL = 32768;
constexpr unsigned CHAIN_SMALL_ROWS = 8192;

// MOST: the most threads of a grid that lets the next pass start (0: none does).
template <unsigned MOST>
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  if (MOST && gridDim.x * gridDim.y * blockDim.x <= MOST)
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

}  // namespace wdm
