// Exact replay of a left-to-right IEEE-754 double summation, in parallel.
//
// The reference computes every reduction on the dense path as a sequential
// loop `c += term(s)` (totalProbability, dense_state_backend.cpp:161-171;
// sampleMeasurement, :173-188; logicalAmplitudeSum,
// quantum_register.cpp:176-190).  A tree reduction rounds differently, so
// its total -- and the index at which a cumulative sum first reaches a
// random draw -- can differ from the reference's.  This header holds the
// math that lets a GPU reproduce the sequential rounding exactly:
//
//  * While the running sum C stays inside one binade [2^e, 2^(e+1)) (or its
//    negative mirror), every rounded add lands on the fixed grid
//    u = 2^(e-52).  So C_j = C_{j-1} + u * inc_j, where inc_j is the term
//    rounded to the grid -- exactly, except that a term lying half-way
//    between two grid points rounds to the even result, which depends on
//    the parity of C/u.
//  * Each term is therefore a function {parity -> integer increment}; such
//    functions compose associatively (tq_compose), so a tile of terms
//    reduces to one pair (inc if C/u is even, inc if odd).  A run's pair comes
//    from two chains of real additions, from an even and an odd start.
//  * A tile's pair for a binade applies when the exact C at its start lies in
//    that binade and every prefix stays in it: for non-negative terms when the
//    end does, for signed terms by the extremes of the tile's prefix sums.
//    Where it does not apply the terms are replayed, with one real double
//    add wherever the binade changes.
//
// The functions are host+device so that the CPU model in the tests and the
// CUDA kernels share one implementation.
#ifndef TMFQS_B200_SEQSUM_CORE_H
#define TMFQS_B200_SEQSUM_CORE_H

#include <stdint.h>

#ifdef __CUDACC__
#define TQ_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define TQ_HD inline
#endif

namespace tq {

// Integer increment (in grid units) of a run of terms, for an even (i0) and
// an odd (i1) value of C/u at the start of the run.
struct Inc {
	int64_t i0;
	int64_t i1;
};

TQ_HD Inc inc_identity() { return Inc{0, 0}; }

// Run L followed by run R.
TQ_HD Inc compose(Inc L, Inc R) {
	const int64_t par0 = L.i0 & 1;        // parity after L when starting even
	const int64_t par1 = (L.i1 + 1) & 1;  // parity after L when starting odd
	Inc o;
	o.i0 = L.i0 + (par0 ? R.i1 : R.i0);
	o.i1 = L.i1 + (par1 ? R.i1 : R.i0);
	return o;
}

TQ_HD int64_t apply(Inc g, int64_t c) { return (c & 1) ? g.i1 : g.i0; }

#ifdef __CUDACC__
// Binade of a normal positive x (|x| in [2^e, 2^(e+1))), and 2^e for |e| < 1023.
__device__ __forceinline__ int binade(double x) { return ((__double2hiint(x) >> 20) & 0x7ff) - 1023; }
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// Grid scale 2^(52-e) for binade e (C/u = C * scale is an integer).
__device__ __forceinline__ double grid_scale(int e) { return pow2(52 - e); }
#endif

constexpr int kDirty = -100000;
constexpr int kIdentity = 100000;  // all terms zero: C unchanged, any binade

}  // namespace tq

#endif
