// General fused passes as register stages: any mix of Hadamards, X, CNOTs,
// swaps, dense one- and two-qubit gates, controlled phases and basis-state flips
// on a tile's local bits.
//
// A pass's moving operations (H, X, CNOT, dense gates) are cut, in circuit order, into stages
// of up to four (complex64: five) distinct targets.  In a stage every thread
// holds the 16 (32) amplitudes of the tile that differ in the stage's register
// bits and applies the stage's operations to them in registers; diagonal operations run
// in whatever stage they fall into, under per-thread and per-register
// conditions.  The first stage reads the tile from HBM, the last writes it back,
// those between pass it on through shared memory with one barrier each.  A swap
// of two local bits moves nothing: it relabels them, and the last stage stores
// every amplitude at its final place.
//
// Exact form: the IEEE operations of the per-gate path in circuit order for each
// amplitude (dense_state_backend.cpp:255-319), zero pairs and zero amplitudes
// skipped as there, so the result is bit-identical.  Fast forms: butterflies
// without their 1/sqrt(2), which is applied once as a power at the end; on the way
// the powers of two in it after every kMaxDeferred butterflies, exactly.
//
// Bound: HBM (one read and one write per pass) and, behind it, instruction issue:
// about 60 instructions per operation and 16 amplitudes, at half the issue rate
// (16 warps per SM, one code path after another through the instruction caches).
// A pass of 11-35 mixed operations on 23 qubits complex128 (41 us at the copy rate)
// takes 77-167 us, and one of 10-21 on 26 qubits complex64 (164 us) 276-483 us; op
// by op through shared memory with a barrier each (k_fused) 205-471 and 900-1850 us.
// 32 complex64 amplitudes per thread against 16: 12% less; zero tests on the high
// words first: 3%; dense gates in a kernel of their own: 9%.
// Dense two-qubit gates are arithmetic: 30 us of FP64 each on 24 qubits exact (four
// in a pass 230 us, alone 104 us each), 75 us each on 27 qubits complex64 (four in
// a pass 660 us; as tensor-core blocks of two 515 us per block).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

namespace tqb {

namespace {

constexpr unsigned kMaxRB = 5;
constexpr unsigned kMaxK = 13;
constexpr unsigned kMaxStages = 64;
constexpr unsigned kMaxOps = 240;
// Fast forms: the Hadamards whose 1/sqrt(2) is outstanding at one time: values stay
// within 2^6 of their true size.  (240 of them would be 2^120: a complex64 register
// that is not normalised overflowed from values of 10^3 on.)
constexpr unsigned kMaxDeferred = 12;

// Tiles of 64 KiB.
template <typename R>
constexpr unsigned tile_bits() {
	return sizeof(R) == 8 ? 12u : 13u;
}
// Register bits per stage: 16 complex128 or 32 complex64 amplitudes per thread
// (64 registers), 256 threads.  Passes of no more tiles than SMs leave most of the
// chip idle and wait on each thread's chain of operations: half the amplitudes per
// thread there (QFT-12 complex128, 84 operations: 38 -> 31 us; circuit of 60 on 14
// qubits 86 -> 73 us in all).
template <typename R>
constexpr unsigned reg_bits() {
	return sizeof(R) == 8 ? 4u : 5u;
}
template <typename R>
constexpr unsigned small_bits() {
	return reg_bits<R>() - 1u;
}
constexpr unsigned kThreadBits = 8, kThreads = 1u << kThreadBits;  // of the large form
constexpr unsigned kMaxTB = 9;
// Index bits of a 128-byte line: lanes in stages that touch HBM, and the shared-memory slot bits that pick a bank group.
template <typename R>
constexpr unsigned line_bits() {
	return sizeof(R) == 8 ? 3u : 4u;
}

// Operation codes: kCodeH + register bit; kCodeX + 5 * target + control register
// bit (the target itself: none); kCodeCP + mask of register bits that must be
// set; kCodeFlip; kCodeU1 + register bit; kCodeU2 + 5 * first + second register
// bit (the first is the more significant one of the gate's block index; in the
// fast forms always the higher one).
// kCodeDiag: a merged run of controlled phases, tmask the register bits with a
// factor, rval its number, omask the thread bits with a factor per tile.
// kCodeScale (a phase on three register bits, which there is not): all
// amplitudes times cr.
constexpr unsigned kCodeH = 0, kCodeX = 5, kCodeCP = 30, kCodeScale = kCodeCP + 7, kCodeFlip = 62, kCodeU1 = 63, kCodeU2 = 68, kCodeDiag = 100;

// Merged runs of controlled phases (fast complex128 form).  In a run the phases commute, so
// those without two register bits collect into one factor per thread and one
// per register bit: a part that depends on the thread index only, formed once
// per launch (entry 0: all amplitudes, 1 + i: those with register bit i), and
// one that depends on the tile, formed once per tile (the same entries, then
// 6 + k: for threads with thread bit k).  Both are products in FP64, rounded once.
// Against the radix stages, 24 qubits: 4, 6 and 12 phases behind four Hadamards 128,
// 129 and 131 us, there 178, 180 and 184 (2 and 3 phases 164 and 175 in both); a ring of
// 24 phases with 8, 16 and 24 more on register bits 169, 200 and 232 us, there 211, 215
// and 218 (14 qubits: 38, 42 and 46; 45, 49 and 52).
constexpr unsigned kMaxLoose = 8;
constexpr unsigned kMaxDiag = 2, kDiagMin = 6, kDiagThread = 6, kDiagTile = 6 + 8;

struct GateOp {
	uint32_t code;
	uint16_t tmask, rval;  // thread index bits that must be set; flips: the thread index and the register of the state
	uint64_t omask;        // outer index bits that must be set; flips: the state's outer bits; dense gates: the matrix
	double cr, ci;
};

// A stage as the kernel uses it, in shared memory: the slot of thread index t
// (three nibbles, XORed) and of each register bit, and its operations.
struct StageSlots {
	uint16_t reg[8];
	uint16_t first, end, pad[6];
	uint16_t nib[3][16];
};

// An operation in the kernel's precision, in shared memory.
template <typename R>
struct alignas(16) OpS {
	uint32_t code;
	uint16_t tmask, rval;
	uint64_t omask;
	R cr, ci;
};

struct GateGeom {
	unsigned n, nstages, nops, nmat;  // nmat: complex matrix elements of the dense gates
	unsigned ndiag, nterms;           // merged phase runs, and the phases in them (after the operations)
	uint16_t term[kMaxDiag][kDiagThread + kDiagTile + 1];  // first phase of each entry: the thread's, then the tile's
	uint64_t o_begin, ntiles;  // the launch runs tiles [o_begin, ntiles)
	double inv, scale;  // 1/sqrt(2); fast forms: the pass's power of it
	uint64_t outer;     // mask of the index bits outside the tile
	uint8_t lpos[kMaxK], opos[kMaxK];  // index bit of a tile bit when loaded and when stored
	uint16_t first[kMaxStages], count[kMaxStages];
	uint8_t rbit[kMaxStages][kMaxRB];        // tile bit of register bit i
	uint8_t tbit[kMaxStages][kMaxTB];  // tile bit of thread index bit k
};

// Non-sign bits of an amplitude: zero exactly for +-0 +- 0i (integer units, not the FP64 pipe).
__device__ __forceinline__ unsigned nonzero_bits(double2 x) {
	return ((unsigned)(__double2hiint(x.x) | __double2hiint(x.y)) << 1) | (unsigned)__double2loint(x.x) |
	       (unsigned)__double2loint(x.y);
}

// A thread's amplitudes of a stage.
template <typename R, unsigned RB>
struct Amps {
	static constexpr unsigned kRegs = 1u << RB;
	typename Vec2<R>::type v[kRegs];
	__device__ __forceinline__ typename Vec2<R>::type &operator[](unsigned r) { return v[r]; }
};

// x + y and x - y, one packed instruction each for complex64.
__device__ __forceinline__ float2 cadd(float2 x, float2 y) { return __fadd2_rn(x, y); }
__device__ __forceinline__ float2 csub(float2 x, float2 y) { return __ffma2_rn(y, make_float2(-1.0f, -1.0f), x); }
__device__ __forceinline__ double2 cadd(double2 x, double2 y) { return make_double2(radd(x.x, y.x), radd(x.y, y.y)); }
__device__ __forceinline__ double2 csub(double2 x, double2 y) { return make_double2(rsub(x.x, y.x), rsub(x.y, y.y)); }

// Zero for an amplitude that may be zero: its exponents' words are (then
// nonzero_bits decides; sums of normal numbers never get here otherwise).
__device__ __forceinline__ unsigned maybe_zero(double2 x) {
	return (unsigned)(__double2hiint(x.x) | __double2hiint(x.y)) & 0x7fffffffu;
}

template <typename R, unsigned RB, bool EXACT, unsigned I>
__device__ __forceinline__ void op_h(Amps<R, RB> &v, R inv) {
	typedef typename Vec2<R>::type V;
	auto bfly = [&](V &x, V &y) {
		V o0 = cadd(x, y), o1 = csub(x, y);
		if(EXACT) {
			o0.x = rmul(o0.x, inv);
			o0.y = rmul(o0.y, inv);
			o1.x = rmul(o1.x, inv);
			o1.y = rmul(o1.y, inv);
		}
		x = o0;
		y = o1;
	};
	constexpr unsigned kRegs = Amps<R, RB>::kRegs;
	if constexpr(EXACT) {
		// An all-zero pair is left as it is (dense_state_backend.cpp:265).
		unsigned least = ~0u;
#pragma unroll
		for(unsigned r = 0; r < kRegs; ++r)
			if(!((r >> I) & 1u)) least = min(least, maybe_zero(v[r]) | maybe_zero(v[r | (1u << I)]));
		if(least == 0u) {
#pragma unroll
			for(unsigned r = 0; r < kRegs; ++r)
				if(!((r >> I) & 1u) && (nonzero_bits(v[r]) | nonzero_bits(v[r | (1u << I)])) != 0u) bfly(v[r], v[r | (1u << I)]);
			return;
		}
	}
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r)
		if(!((r >> I) & 1u)) bfly(v[r], v[r | (1u << I)]);
}

// X on register bit I of the pairs whose register bit C is set (C == I: all).
template <typename R, unsigned RB, bool EXACT, unsigned I, unsigned C>
__device__ __forceinline__ void op_x(Amps<R, RB> &v, bool on) {
	constexpr unsigned kRegs = Amps<R, RB>::kRegs;
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r) {
		if(((r >> I) & 1u) || (C != I && !((r >> C) & 1u))) continue;
		const auto x = v[r], y = v[r | (1u << I)];
		// Equal pairs (zeros of either sign) are left as they are (dense_state_backend.cpp:283,315).
		const bool move = on && !(EXACT && x.x == y.x && x.y == y.y);
		v[r].x = move ? y.x : x.x;
		v[r].y = move ? y.y : x.y;
		v[r | (1u << I)].x = move ? x.x : y.x;
		v[r | (1u << I)].y = move ? x.y : y.y;
	}
}

// One phase product of the fast forms.  complex64: each component updated in its
// own register; from the plain expressions the new values went to registers of
// their own and were moved back where the operations' paths meet (random circuits
// of 26 qubits 3.30 ms, now 3.2; complex128 was 8% slower this way, by spills).
__device__ __forceinline__ void phase_fast(float pr, float pi, float2 &x) {
	asm volatile(
		"{\n\t.reg .f32 b, d;\n\t"
		"mul.rn.f32 b, %3, %1;\n\t"
		"mul.rn.f32 d, %3, %0;\n\t"
		"neg.f32 b, b;\n\t"
		"fma.rn.f32 %0, %2, %0, b;\n\t"
		"fma.rn.f32 %1, %2, %1, d;\n\t}"
		: "+f"(x.x), "+f"(x.y)
		: "f"(pr), "f"(pi));
}
__device__ __forceinline__ void phase_fast(double pr, double pi, double2 &x) {
	const double re = x.x, im = x.y;
	x.x = fma(pr, re, -(pi * im));
	x.y = fma(pr, im, pi * re);
}

// Phase on the registers that have all bits of M.
template <typename R, unsigned RB, bool EXACT, unsigned M>
__device__ __forceinline__ void op_cp(Amps<R, RB> &v, R pr, R pi) {
	constexpr unsigned kRegs = Amps<R, RB>::kRegs;
	unsigned least = ~0u;
	if constexpr(EXACT) {
#pragma unroll
		for(unsigned r = 0; r < kRegs; ++r)
			if((r & M) == M) least = min(least, maybe_zero(v[r]));
	}
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r) {
		if((r & M) != M) continue;
		if constexpr(EXACT) {
			// Zero amplitudes are skipped (dense_state_backend.cpp:299).
			R re = v[r].x, im = v[r].y;
			cmul_ref(pr, pi, re, im);
			if(least != 0u || nonzero_bits(v[r]) != 0u) {
				v[r].x = re;
				v[r].y = im;
			}
		} else {
			phase_fast(pr, pi, v[r]);
		}
	}
}

// A matrix element g in shared memory: complex128 as it is; complex64 as the two
// operand pairs of a packed complex product, (re, re) and (-im, im).
template <typename R>
struct MatElem;
template <>
struct MatElem<double> {
	typedef double2 type;
	static __device__ __forceinline__ double2 make(double2 g) { return g; }
};
template <>
struct MatElem<float> {
	typedef float4 type;
	static __device__ __forceinline__ float4 make(double2 g) { return make_float4((float)g.x, (float)g.x, -(float)g.y, (float)g.y); }
};

// Loaded where it is used: a broadcast, and cheaper than the spills of keeping
// the whole matrix in registers.
__device__ __forceinline__ double2 mat_at(const double2 *m) {
	double2 x;
	asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x.x), "=d"(x.y) : "r"((unsigned)__cvta_generic_to_shared(m)));
	return x;
}
__device__ __forceinline__ float4 mat_at(const float4 *m) {
	float4 x;
	asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
	             : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"((unsigned)__cvta_generic_to_shared(m)));
	return x;
}

// o += g * x in the fast forms; xs is x with its components exchanged.
__device__ __forceinline__ void cfma(float4 g, float2 x, float2 xs, float2 &o) {
	o = __ffma2_rn(make_float2(g.x, g.y), x, o);
	o = __ffma2_rn(make_float2(g.z, g.w), xs, o);
}
__device__ __forceinline__ void cfma(double2 g, double2 x, double2, double2 &o) {
	o.x = fma(-g.y, x.y, fma(g.x, x.x, o.x));
	o.y = fma(g.y, x.x, fma(g.x, x.y, o.y));
}

// Dense gate on register bit I: the unrolled formula of gate_block_apply.h:117-140.
template <typename R, unsigned RB, bool EXACT, unsigned I>
__device__ __forceinline__ void op_u1(Amps<R, RB> &v, const typename MatElem<R>::type *m) {
	typedef typename Vec2<R>::type V;
	const auto g00 = m[0], g01 = m[1], g10 = m[2], g11 = m[3];
#pragma unroll
	for(unsigned r = 0; r < Amps<R, RB>::kRegs; ++r) {
		if((r >> I) & 1u) continue;
		const V x = v[r], y = v[r | (1u << I)];
		if constexpr(EXACT) {
			if((nonzero_bits(x) | nonzero_bits(y)) == 0u) continue;
			v[r].x = rsub(radd(rsub(rmul(g00.x, x.x), rmul(g00.y, x.y)), rmul(g01.x, y.x)), rmul(g01.y, y.y));
			v[r].y = radd(radd(radd(rmul(g00.x, x.y), rmul(g00.y, x.x)), rmul(g01.x, y.y)), rmul(g01.y, y.x));
			v[r | (1u << I)].x = rsub(radd(rsub(rmul(g10.x, x.x), rmul(g10.y, x.y)), rmul(g11.x, y.x)), rmul(g11.y, y.y));
			v[r | (1u << I)].y = radd(radd(radd(rmul(g10.x, x.y), rmul(g10.y, x.x)), rmul(g11.x, y.y)), rmul(g11.y, y.x));
		} else {
			V xs, ys, o0, o1;
			xs.x = x.y, xs.y = x.x, ys.x = y.y, ys.y = y.x;
			o0.x = o0.y = o1.x = o1.y = R(0);
			cfma(g00, x, xs, o0);
			cfma(g10, x, xs, o1);
			cfma(g01, y, ys, o0);
			cfma(g11, y, ys, o1);
			v[r] = o0;
			v[r | (1u << I)] = o1;
		}
	}
}

// Dense gate on register bits A (more significant) and B: row sums term by term
// (gate_block_apply.h:165-176); all-zero blocks are left alone.  Fast forms: two
// blocks per matrix element loaded.
template <typename R, unsigned RB, bool EXACT, unsigned A, unsigned B>
__device__ __forceinline__ void op_u2(Amps<R, RB> &v, const typename MatElem<R>::type *m) {
	typedef typename Vec2<R>::type V;
	constexpr unsigned mask = (1u << A) | (1u << B);
	// Register of index c of block b.
	auto at = [](unsigned b, unsigned c) {
		unsigned r = 0, k = 0;
		for(unsigned i = 0; i < RB; ++i)
			if(!((mask >> i) & 1u)) r |= ((b >> k++) & 1u) << i;
		return r | ((c >> 1) << A) | ((c & 1u) << B);
	};
	if constexpr(EXACT) {
#pragma unroll
		for(unsigned b = 0; b < Amps<R, RB>::kRegs / 4; ++b) {
			V o[4];
			if((nonzero_bits(v[at(b, 0)]) | nonzero_bits(v[at(b, 1)]) | nonzero_bits(v[at(b, 2)]) | nonzero_bits(v[at(b, 3)])) == 0u) continue;
#pragma unroll
			for(unsigned row = 0; row < 4; ++row) {
				V n;
				n.x = n.y = R(0);
#pragma unroll
				for(unsigned c = 0; c < 4; ++c) {
					const auto g = mat_at(m + 4 * row + c);
					const V x = v[at(b, c)];
					n.x = radd(n.x, rsub(rmul(g.x, x.x), rmul(g.y, x.y)));
					n.y = radd(n.y, radd(rmul(g.x, x.y), rmul(g.y, x.x)));
				}
				o[row] = n;
			}
#pragma unroll
			for(unsigned c = 0; c < 4; ++c) v[at(b, c)] = o[c];
		}
	} else {
#pragma unroll
		for(unsigned b = 0; b < Amps<R, RB>::kRegs / 4; b += 2) {
			V o[2][4];
#pragma unroll
			for(unsigned k = 0; k < 2; ++k)
#pragma unroll
				for(unsigned c = 0; c < 4; ++c) o[k][c].x = o[k][c].y = R(0);
#pragma unroll
			for(unsigned c = 0; c < 4; ++c) {
				V xs[2];
#pragma unroll
				for(unsigned k = 0; k < 2; ++k) {
					xs[k].x = v[at(b + k, c)].y;
					xs[k].y = v[at(b + k, c)].x;
				}
#pragma unroll
				for(unsigned row = 0; row < 4; ++row) {
					const auto g = mat_at(m + 4 * row + c);
#pragma unroll
					for(unsigned k = 0; k < 2; ++k) cfma(g, v[at(b + k, c)], xs[k], o[k][row]);
				}
			}
#pragma unroll
			for(unsigned k = 0; k < 2; ++k)
#pragma unroll
				for(unsigned c = 0; c < 4; ++c) v[at(b + k, c)] = o[k][c];
		}
	}
}

template <typename V>
__device__ __forceinline__ V cprod(V a, V b) {
	V o;
	o.x = fma(a.x, b.x, -(a.y * b.y));
	o.y = fma(a.x, b.y, a.y * b.x);
	return o;
}

// A merged run: dth this run's thread entries (per thread), dti its tile entries.
template <typename R, unsigned RB>
__device__ __forceinline__ void op_diag(const OpS<R> &op, Amps<R, RB> &v, const typename Vec2<R>::type *dth, const typename Vec2<R>::type *dti,
                                        unsigned t) {
	typedef typename Vec2<R>::type V;
	constexpr unsigned kRegs = Amps<R, RB>::kRegs;
	V p = cprod(dth[t], dti[0]);
	for(unsigned m = (unsigned)op.omask; m; m &= m - 1u) {
		const unsigned k = __ffs(m) - 1;
		if((t >> k) & 1u) p = cprod(p, dti[6 + k]);
	}
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r) v[r] = cprod(p, v[r]);
#pragma unroll
	for(unsigned i = 0; i < RB; ++i) {
		if(!((op.tmask >> i) & 1u)) continue;
		const V f = cprod(dth[(1 + i) * kThreads + t], dti[1 + i]);
#pragma unroll
		for(unsigned r = 0; r < kRegs; ++r)
			if((r >> i) & 1u) v[r] = cprod(f, v[r]);
	}
}

template <typename R, unsigned RB, bool EXACT, bool DENSE, bool MERGED>
__device__ __forceinline__ void run_op(const OpS<R> &op, Amps<R, RB> &v, const GateGeom &g, const typename MatElem<R>::type *mats,
                                       const typename Vec2<R>::type *dth, const typename Vec2<R>::type *dti, uint64_t base, unsigned t) {
	if(MERGED && op.code == kCodeDiag) {
		op_diag<R, RB>(op, v, dth + op.rval * kDiagThread * kThreads, dti + op.rval * kDiagTile, t);
		return;
	}
	if(DENSE && op.code >= kCodeU1) {
		const typename MatElem<R>::type *m = mats + op.omask;
		switch(op.code) {
#define TQB_U1(I)                                                         \
	case kCodeU1 + I:                                                     \
		if constexpr(DENSE && I < RB) op_u1<R, RB, EXACT, I < RB ? I : 0u>(v, m);      \
		return;
#define TQB_U2(A, B)                                                                                    \
	case kCodeU2 + 5 * A + B:                                                                           \
		if constexpr(DENSE && A < RB && B < RB && (EXACT || A > B)) op_u2<R, RB, EXACT, A < RB ? A : 0u, B < RB ? B : 0u>(v, m); \
		return;
			TQB_U1(0) TQB_U1(1) TQB_U1(2) TQB_U1(3) TQB_U1(4)
			TQB_U2(0, 1) TQB_U2(0, 2) TQB_U2(0, 3) TQB_U2(1, 0) TQB_U2(1, 2) TQB_U2(1, 3)
			TQB_U2(2, 0) TQB_U2(2, 1) TQB_U2(2, 3) TQB_U2(3, 0) TQB_U2(3, 1) TQB_U2(3, 2)
			TQB_U2(4, 0) TQB_U2(4, 1) TQB_U2(4, 2) TQB_U2(4, 3)
#undef TQB_U1
#undef TQB_U2
			default: return;
		}
	}
	if(op.code == kCodeFlip) {
		const unsigned at = (base & g.outer) == op.omask && t == op.tmask ? op.rval : Amps<R, RB>::kRegs;
#pragma unroll
		for(unsigned r = 0; r < Amps<R, RB>::kRegs; ++r) {
			v[r].x = r == at ? -v[r].x : v[r].x;
			v[r].y = r == at ? -v[r].y : v[r].y;
		}
		return;
	}
	if((base & op.omask) != op.omask) return;
	const bool on = (t & op.tmask) == op.tmask;
	const R inv = (R)g.inv, pr = op.cr, pi = op.ci;
	switch(op.code) {
#define TQB_H(I)                                                          \
	case kCodeH + I:                                                      \
		if constexpr(I < RB) op_h<R, RB, EXACT, I < RB ? I : 0u>(v, inv);     \
		return;
#define TQB_XC(I, C)                                                                                       \
	case kCodeX + 5 * I + C:                                                                               \
		if constexpr(I < RB && C < RB) op_x<R, RB, EXACT, I < RB ? I : 0u, C < RB ? C : 0u>(v, on);            \
		return;
#define TQB_X(I) TQB_XC(I, 0) TQB_XC(I, 1) TQB_XC(I, 2) TQB_XC(I, 3) TQB_XC(I, 4)
		TQB_H(0) TQB_H(1) TQB_H(2) TQB_H(3) TQB_H(4)
		TQB_X(0) TQB_X(1) TQB_X(2) TQB_X(3) TQB_X(4)
#define TQB_CP(M)                                                                                    \
	case kCodeCP + M:                                                                                \
		if constexpr(M < (1u << RB))                                                                 \
			if(on) op_cp<R, RB, EXACT, M < (1u << RB) ? M : 0u>(v, pr, pi);                          \
		return;
		TQB_CP(0) TQB_CP(1) TQB_CP(2) TQB_CP(3) TQB_CP(4) TQB_CP(5) TQB_CP(6) TQB_CP(8) TQB_CP(9) TQB_CP(10) TQB_CP(12)
		TQB_CP(16) TQB_CP(17) TQB_CP(18) TQB_CP(20) TQB_CP(24)
	case kCodeScale:
		if constexpr(!EXACT) {
#pragma unroll
			for(unsigned r = 0; r < Amps<R, RB>::kRegs; ++r) {
				v[r].x *= pr;
				v[r].y *= pr;
			}
		}
		return;
		default: return;
#undef TQB_H
#undef TQB_X
#undef TQB_XC
#undef TQB_CP
	}
}

// Shared-memory slot of tile bit b: a bit above the bank-group bits also flips
// one of them, so that lanes on bits of different residues spread over the banks.
template <typename R>
__device__ __forceinline__ unsigned slot_of(unsigned b) {
	constexpr unsigned s = line_bits<R>();
	return (1u << b) | (b >= s ? 1u << (b % s) : 0u);
}

// What a pass holds beside the plain operations: each costs the others registers.
enum Extra { kPlain, kDense, kMerged };

// Shared memory: tile, operations, phases of merged runs, stages, matrices,
// entries of the merged runs.  mirror: a second place for
// the result of a pass with merged runs (or null).
template <typename R, unsigned RB, bool EXACT, Extra EXTRA>
__global__ void __launch_bounds__(1u << (tile_bits<R>() - RB), RB == small_bits<R>() ? 1 : 2) k_gate_pass(typename Vec2<R>::type *a, typename Vec2<R>::type *mirror,
                                                           const __grid_constant__ GateGeom g, const GateOp *gops, const double2 *gmats) {
	typedef typename Vec2<R>::type V;
	constexpr unsigned K = tile_bits<R>(), TB = K - RB, kThreads = 1u << TB, kRegs = 1u << RB;
	constexpr bool MERGED = EXTRA == kMerged;
	static_assert(!MERGED || TB == kThreadBits, "entries of merged runs are per thread of the large form");
	extern __shared__ __align__(16) unsigned char smem_raw[];
	V *s = reinterpret_cast<V *>(smem_raw);
	OpS<R> *ops = reinterpret_cast<OpS<R> *>(smem_raw + (sizeof(V) << K));
	GateOp *terms = reinterpret_cast<GateOp *>(ops + g.nops);
	StageSlots *stages = reinterpret_cast<StageSlots *>(terms + g.nterms);
	typedef typename MatElem<R>::type ME;
	ME *mats = reinterpret_cast<ME *>(stages + g.nstages);
	V *dth = reinterpret_cast<V *>(mats + g.nmat), *dti = dth + g.ndiag * kDiagThread * kThreads;
	const unsigned t = threadIdx.x;
	for(unsigned e = t; e < g.nops; e += blockDim.x) {
		const GateOp q = gops[e];
		ops[e] = OpS<R>{q.code, q.tmask, q.rval, q.omask, (R)q.cr, (R)q.ci};
	}
	for(unsigned e = t; e < g.nterms; e += blockDim.x) terms[e] = gops[g.nops + e];
	for(unsigned e = t; e < g.nmat; e += blockDim.x) mats[e] = MatElem<R>::make(gmats[e]);
	for(unsigned e = t; e < g.nstages * 64u; e += blockDim.x) {
		const unsigned st = e >> 6, i = e & 63u;
		if(i < 48u) {
			unsigned x = 0;
			for(unsigned k = 0; k < 4; ++k)
				if(4 * (i >> 4) + k < TB && ((i >> k) & 1u)) x ^= slot_of<R>(g.tbit[st][4 * (i >> 4) + k]);
			stages[st].nib[i >> 4][i & 15u] = (uint16_t)x;
		} else if(i < 48u + RB) {
			stages[st].reg[i - 48u] = (uint16_t)slot_of<R>(g.rbit[st][i - 48u]);
		} else if(i == 60u) {
			stages[st].first = g.first[st];
			stages[st].end = (uint16_t)(g.first[st] + g.count[st]);
		}
	}
	// And in HBM, when the tile is loaded and stored.
	V *pin = a, *pout = a;
	{
		const unsigned e = g.nstages - 1u;
		uint64_t x = 0, y = 0;
#pragma unroll
		for(unsigned k = 0; k < TB; ++k) {
			x |= (uint64_t)((t >> k) & 1u) << g.lpos[g.tbit[0][k]];
			y |= (uint64_t)((t >> k) & 1u) << g.opos[g.tbit[e][k]];
		}
		pin += x;
		pout += y;
	}
	const ptrdiff_t other = MERGED && mirror ? mirror - a : 0;
	__syncthreads();
	// Product of the phases of entry e of run d (thread entries, then tile
	// entries) whose conditions hold.
	auto entry = [&](unsigned d, unsigned e, uint64_t base) {
		double re = 1.0, im = 0.0;
		for(unsigned k = g.term[d][e]; k < g.term[d][e + 1]; ++k) {
			const GateOp &q = terms[k];
			if((base & q.omask) != q.omask || (t & q.tmask) != q.tmask) continue;
			const double x = fma(re, q.cr, -(im * q.ci));
			im = fma(re, q.ci, im * q.cr);
			re = x;
		}
		V f;
		f.x = (R)re;
		f.y = (R)im;
		return f;
	};
	auto tile_base = [&](uint64_t o) {
#pragma unroll
		for(unsigned i = 0; i < K; ++i) o = insert0(o, g.lpos[i]);
		return o;
	};
	// The next tile's entries come from one warp while its loads of the current
	// tile are in flight.
	const unsigned ntile = MERGED ? g.ndiag * kDiagTile : 0u;
	auto prepare = [&](uint64_t o, unsigned buf) {
		if(t < ntile && o < g.ntiles) dti[buf * ntile + t] = entry(t / kDiagTile, kDiagThread + t % kDiagTile, tile_base(o));
	};
	if(MERGED) {
		for(unsigned d = 0; d < g.ndiag; ++d)
			for(unsigned e = 0; e < kDiagThread; ++e) dth[(d * kDiagThread + e) * kThreads + t] = entry(d, e, 0);
		prepare(g.o_begin + blockIdx.x, 0);
		__syncthreads();
	}
	unsigned buf = 0;
	for(uint64_t o = g.o_begin + blockIdx.x; o < g.ntiles; o += gridDim.x, buf ^= 1u) {
		const uint64_t base = tile_base(o);
		for(unsigned st = 0; st < g.nstages; ++st) {
			const bool last = st + 1 == g.nstages;
			Amps<R, RB> v;
			// Where this thread's amplitudes sit in shared memory.
			const StageSlots &sl = stages[st];
			const unsigned slot = (unsigned)sl.nib[0][t & 15u] ^ sl.nib[1][(t >> 4) & 15u] ^ (TB > 8 ? sl.nib[2][t >> 8] : 0u);
			unsigned ro[RB];
#pragma unroll
			for(unsigned i = 0; i < RB; ++i) ro[i] = sl.reg[i];
			auto at = [&](unsigned r) {
				unsigned x = 0;
#pragma unroll
				for(unsigned i = 0; i < RB; ++i)
					if((r >> i) & 1u) x ^= ro[i];
				return slot ^ x;
			};
			// Offset of register r from the thread's place in HBM (uniform).
			auto global = [&](const uint8_t *pos, unsigned r) {
				uint64_t x = base;
#pragma unroll
				for(unsigned i = 0; i < RB; ++i)
					if((r >> i) & 1u) x |= 1ull << pos[g.rbit[st][i]];
				return x;
			};
			if(st == 0) {
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) v[r] = pin[global(g.lpos, r)];
				if(MERGED) prepare(o + gridDim.x, buf ^ 1u);
			} else {
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) v[r] = s[at(r)];
			}
			const unsigned k1 = sl.end;
			for(unsigned k = sl.first; k < k1; ++k) run_op<R, RB, EXACT, EXTRA == kDense, MERGED>(ops[k], v, g, mats, dth, dti + buf * ntile, base, t);
			if(last) {
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) {
					if(!EXACT) {
						v[r].x *= (R)g.scale;
						v[r].y *= (R)g.scale;
					}
					V *q = pout + global(g.opos, r);
					*q = v[r];
					if(MERGED && mirror) q[other] = v[r];
				}
			} else {
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) s[at(r)] = v[r];
			}
			// Between stages, and before the next tile's first stage writes what the last one read.
			if(g.nstages > 1 || MERGED) __syncthreads();
		}
	}
}

// One operation of the pass on tile bits: `pm` the tile bits and `om` the outer
// index bits that must be set.
struct PlanOp {
	enum Kind { kH, kX, kCP, kFlip, kU1, kU2 } kind;
	unsigned p, p2;  // the moving tile bit(s)
	unsigned mat;    // dense gates: first element of the matrix
	uint32_t pm;
	uint64_t om;
	double cr, ci;
};

// The stage plan of a pass; false: it does not fit (another kernel runs it).
// `merge`: merge runs of controlled phases; `loose` is the number of them that were not.
bool plan_gates(const FusedPass &pass, unsigned K, unsigned RB, unsigned line, bool exact, bool merge, GateGeom &g, std::vector<GateOp> &out,
                std::vector<GateOp> &terms, std::vector<double> &mats, unsigned &loose) {
	if(pass.K != K || pass.ops.empty() || pass.n < K) return false;
	g = GateGeom{};
	g.n = pass.n;
	g.o_begin = 0;
	g.ntiles = 1ull << (pass.n - K);
	if(pass.tile_end) {
		if(pass.tile_begin >= pass.tile_end || pass.tile_end > g.ntiles) fail(TMFQS_ERR_LOGIC, "gate pass: bad tile range");
		g.o_begin = pass.tile_begin;
		g.ntiles = pass.tile_end;
	}
	g.inv = 1.0 / std::sqrt(2.0);
	unsigned m = 0;  // contiguous low bits in the tile
	while(m < K && pass.lpos[m] == m) ++m;
	const unsigned low = std::min(m, line);
	std::vector<int> local(pass.n, -1);
	uint64_t tile_mask = 0;
	for(unsigned i = 0; i < K; ++i) {
		g.lpos[i] = (uint8_t)pass.lpos[i];
		local[pass.lpos[i]] = (int)i;
		tile_mask |= 1ull << pass.lpos[i];
	}
	g.outer = (pass.n < 64 ? (1ull << pass.n) - 1ull : ~0ull) & ~tile_mask;
	// Swaps relabel: where[l] is the tile bit that holds logical local bit l.
	std::vector<unsigned> where(K);
	for(unsigned i = 0; i < K; ++i) where[i] = i;
	std::vector<PlanOp> ops;
	unsigned nh = 0;
	auto require = [&](PlanOp &q, uint64_t mask) {
		q.om |= mask & ~tile_mask;
		for(uint64_t x = mask & tile_mask; x; x &= x - 1) q.pm |= 1u << where[local[__builtin_ctzll(x)]];
	};
	for(const FusedOp &op : pass.ops) {
		PlanOp q{};
		switch(op.kind) {
			case kFH:
			case kFHChain:
			case kFHTwiddle:
				q.kind = PlanOp::kH;
				q.p = where[op.lt];
				ops.push_back(q);
				++nh;
				for(unsigned e = 0; op.kind != kFH && e < op.lc; ++e) {
					const ChainEntry &ce = pass.chain[op.tab + e];
					PlanOp c{};
					c.kind = PlanOp::kCP;
					c.cr = ce.cr;
					c.ci = ce.ci;
					require(c, (1ull << ce.bit) | (1ull << pass.lpos[op.lt]));
					ops.push_back(c);
				}
				break;
			case kFX:
			case kFCnot:
				q.kind = PlanOp::kX;
				q.p = where[op.lt];
				require(q, op.mask);
				ops.push_back(q);
				break;
			case kFCP:
				q.kind = PlanOp::kCP;
				q.cr = op.cr;
				q.ci = op.ci;
				require(q, op.mask);
				ops.push_back(q);
				break;
			case kFFlip:
				q.kind = PlanOp::kFlip;
				require(q, op.state);
				ops.push_back(q);
				break;
			case kFDense1:
			case kFDense2:
				q.kind = op.kind == kFDense1 ? PlanOp::kU1 : PlanOp::kU2;
				q.p = where[op.lt];
				if(op.kind == kFDense2) q.p2 = where[op.lc];
				q.mat = op.tab / 2;
				ops.push_back(q);
				break;
			case kFSwap: std::swap(where[op.lt], where[op.lc]); break;
			default: return false;
		}
	}
	if(ops.size() > kMaxOps) return false;
	for(unsigned l = 0; l < K; ++l) g.opos[where[l]] = (uint8_t)pass.lpos[l];
	uint32_t keep_in = 0, keep_out = 0;  // tile bits that stay lanes where the tile is loaded / stored
	for(unsigned b = 0; b < K; ++b) {
		if(g.lpos[b] < low) keep_in |= 1u << b;
		if(g.opos[b] < low) keep_out |= 1u << b;
	}
	// Stages: consecutive operations while their targets fit in the register bits.
	std::vector<uint32_t> regs{0u};
	std::vector<std::vector<unsigned>> of(1);
	for(unsigned k = 0; k < ops.size(); ++k) {
		uint32_t bits = 0;
		if(ops[k].kind != PlanOp::kCP && ops[k].kind != PlanOp::kFlip) bits = 1u << ops[k].p;
		if(ops[k].kind == PlanOp::kU2) bits |= 1u << ops[k].p2;
		if(bits & ~regs.back()) {
			if(__builtin_popcount(regs.back() | bits) > (int)RB || (regs.size() == 1 && (keep_in & bits))) {
				regs.push_back(bits);
				of.push_back({});
			} else {
				regs.back() |= bits;
			}
		}
		of.back().push_back(k);
	}
	// The last stage must leave the line bits to the lanes, and with relabelled
	// bits no thread may store before all have loaded.
	const bool moved = !std::equal(g.lpos, g.lpos + K, g.opos);
	if((regs.back() & keep_out) || (moved && regs.size() == 1)) {
		regs.push_back(0);
		of.push_back({});
	}
	g.nstages = (unsigned)regs.size();
	if(g.nstages > kMaxStages) return false;
	out.clear();
	terms.clear();
	loose = 0;
	mats = pass.mats;
	unsigned deferred = 0, halvings = 0;  // Hadamards since the last kCodeScale, and the powers of two applied by those
	for(unsigned st = 0; st < g.nstages; ++st) {
		const bool in = st == 0, outs = st + 1 == g.nstages;
		const uint32_t fixed = (in ? keep_in : 0u) | (outs ? keep_out : 0u);
		// How many of the stage's conditions each tile bit is in: the most frequent
		// fill up the register bits (fewer amplitudes to touch, no divergence), the
		// least frequent become lanes.
		unsigned cost[kMaxK] = {};
		for(unsigned k : of[st])
			for(unsigned b = 0; b < K; ++b) cost[b] += ops[k].kind != PlanOp::kFlip && ((ops[k].pm >> b) & 1u);
		uint32_t r = regs[st];
		while(__builtin_popcount(r) < (int)RB) {
			int best = -1;
			for(int b = (int)K - 1; b >= 0; --b)
				if(!((r | fixed) >> b & 1u) && (best < 0 || cost[b] > cost[best])) best = b;
			if(best < 0) return false;
			r |= 1u << best;
		}
		std::vector<unsigned> rb, rest, tb;
		for(unsigned b = 0; b < K; ++b) ((r >> b) & 1u ? rb : rest).push_back(b);
		std::stable_sort(rest.begin(), rest.end(), [&](unsigned x, unsigned y) { return cost[x] < cost[y]; });
		auto take = [&](unsigned b) {
			tb.push_back(b);
			rest.erase(std::find(rest.begin(), rest.end(), b));
		};
		if(in || outs) {
			// Lanes along the line, in the order of the index bits.
			for(unsigned i = 0; i < low; ++i)
				for(unsigned b = 0; b < K; ++b)
					if((in ? g.lpos[b] : g.opos[b]) == i && std::find(rest.begin(), rest.end(), b) != rest.end()) take(b);
		} else {
			// Lanes on different bank groups.
			uint32_t seen = 0;
			for(unsigned want = 0; want < line; ++want)
				for(unsigned b : std::vector<unsigned>(rest))
					if(!((seen >> (b % line)) & 1u)) {
						seen |= 1u << (b % line);
						take(b);
						break;
					}
		}
		while(!rest.empty()) take(rest.front());
		for(unsigned i = 0; i < RB; ++i) g.rbit[st][i] = (uint8_t)rb[i];
		for(unsigned k = 0; k < tb.size(); ++k) g.tbit[st][k] = (uint8_t)tb[k];
		g.first[st] = (uint16_t)out.size();
		for(unsigned pos = 0; pos < of[st].size(); ++pos) {
			const unsigned k = of[st][pos];
			const PlanOp &q = ops[k];
			GateOp o{};
			uint32_t rm = 0, tm = 0;
			// A run of controlled phases from here on.
			unsigned end = pos, few = 0;
			while(merge && end < of[st].size() && ops[of[st][end]].kind == PlanOp::kCP) few += __builtin_popcount(ops[of[st][end++]].pm & r) < 2;
			if(g.ndiag < kMaxDiag && few >= kDiagMin) {
				o.code = kCodeDiag;
				o.rval = (uint16_t)g.ndiag;
				for(unsigned e = pos; e < end; ++e) {
					const PlanOp &c = ops[of[st][e]];
					GateOp x{};
					x.cr = c.cr;
					x.ci = c.ci;
					x.rval = o.rval;
					uint32_t crm = 0, ctm = 0;
					for(unsigned i = 0; i < RB; ++i) crm |= ((c.pm >> rb[i]) & 1u) << i;
					for(unsigned i = 0; i < tb.size(); ++i) ctm |= ((c.pm >> tb[i]) & 1u) << i;
					if(__builtin_popcount(crm) == 2) {
						x.code = kCodeCP + crm;
						x.rval = 0;
						out.push_back(x);
						++loose;
						continue;
					}
					x.code = (c.om ? kDiagThread : 0u) + (crm ? 1u + (unsigned)__builtin_ctz(crm) : 0u);
					if(crm) o.tmask |= (uint16_t)crm;
					x.tmask = (uint16_t)ctm;
					x.omask = c.om;
					if(c.om && ctm) {
						x.code = kDiagThread + 6u + (unsigned)__builtin_ctz(ctm);
						x.tmask = 0;
						o.omask |= ctm;
					}
					terms.push_back(x);
				}
				out.push_back(o);
				const auto from = terms.begin() + (g.ndiag ? g.term[g.ndiag - 1][kDiagThread + kDiagTile] : 0);
				std::stable_sort(from, terms.end(), [](const GateOp &x, const GateOp &y) { return x.code < y.code; });
				unsigned at = (unsigned)(from - terms.begin());
				for(unsigned e = 0; e <= kDiagThread + kDiagTile; ++e) {
					while(at < terms.size() && terms[at].code < e) ++at;
					g.term[g.ndiag][e] = (uint16_t)at;
				}
				++g.ndiag;
				pos = end - 1;
				continue;
			}
			loose += q.kind == PlanOp::kCP;
			for(unsigned i = 0; i < RB; ++i) rm |= ((q.pm >> rb[i]) & 1u) << i;
			for(unsigned i = 0; i < tb.size(); ++i) tm |= ((q.pm >> tb[i]) & 1u) << i;
			unsigned target = 0, second = 0;
			for(unsigned i = 0; i < RB; ++i) {
				if(rb[i] == q.p) target = i;
				if(rb[i] == q.p2) second = i;
			}
			o.tmask = (uint16_t)tm;
			o.omask = q.om;
			o.cr = q.cr;
			o.ci = q.ci;
			switch(q.kind) {
				case PlanOp::kH: o.code = kCodeH + target; break;
				case PlanOp::kX: o.code = kCodeX + 5 * target + (rm ? (unsigned)__builtin_ctz(rm) : target); break;
				case PlanOp::kCP: o.code = kCodeCP + rm; break;
				case PlanOp::kFlip:
					o.code = kCodeFlip;
					o.rval = (uint16_t)rm;
					break;
				case PlanOp::kU1:
				case PlanOp::kU2:
					if(q.kind == PlanOp::kU2 && !exact && target < second) {
						// The block index with its two bits exchanged (exact: the order of
						// the row sums is the gate's own).
						std::swap(target, second);
						double *m = mats.data() + 2 * q.mat;
						const unsigned x[4] = {0, 2, 1, 3};
						double y[32];
						for(unsigned r = 0; r < 4; ++r)
							for(unsigned c = 0; c < 4; ++c)
								for(unsigned k2 = 0; k2 < 2; ++k2) y[2 * (4 * x[r] + x[c]) + k2] = m[2 * (4 * r + c) + k2];
						std::copy(y, y + 32, m);
					}
					o.code = q.kind == PlanOp::kU1 ? kCodeU1 + target : kCodeU2 + 5 * target + second;
					o.omask = q.mat;
					break;
			}
			out.push_back(o);
			if(!exact && q.kind == PlanOp::kH && ++deferred == kMaxDeferred) {
				GateOp x{};
				x.code = kCodeScale;
				x.cr = std::ldexp(1.0, -(int)(kMaxDeferred / 2));
				out.push_back(x);
				deferred = 0;
				halvings += kMaxDeferred / 2;
			}
		}
		g.count[st] = (uint16_t)(out.size() - g.first[st]);
	}
	g.nops = (unsigned)out.size();
	g.nterms = (unsigned)terms.size();
	g.nmat = (unsigned)(pass.mats.size() / 2);
	// The power of the reference's 1/sqrt(2), rounded as it is (the difference adds up).
	g.scale = std::ldexp(std::pow(g.inv, (double)nh), (int)halvings);
	return true;
}

template <typename R, unsigned RB, bool EXACT>
bool run_gate_pass(const LaunchCtx &c, void *a, const FusedPass &pass, void *&dev_prog, size_t &dev_prog_bytes, void *mirror, bool merged) {
	// (the kernel for merged runs has no dense gates: a pass with both takes the one for dense gates)
	if(merged && (EXACT || sizeof(R) != 8 || !pass.mats.empty())) return false;
	constexpr unsigned K = tile_bits<R>();
	GateGeom g;
	std::vector<GateOp> ops;
	std::vector<GateOp> terms;
	std::vector<double> mats;
	unsigned loose = 0;
	if(!plan_gates(pass, K, RB, line_bits<R>(), EXACT, merged, g, ops, terms, mats, loose)) return false;
	if(merged && (g.ndiag == 0 || loose > kMaxLoose)) return false;
	ops.insert(ops.end(), terms.begin(), terms.end());
	const size_t ops_bytes = ops.size() * sizeof(GateOp), mat_bytes = mats.size() * sizeof(double);
	const size_t need = std::max<size_t>(sizeof(GateOp), ops_bytes + mat_bytes);
	if(need > dev_prog_bytes) {
		if(dev_prog) {
			check_cuda(cudaStreamSynchronize(c.stream), "gate pass program sync");
			cudaFree(dev_prog);
		}
		dev_prog = nullptr;
		dev_prog_bytes = 0;
		if(device_alloc(&dev_prog, need * 2) != cudaSuccess) {
			cudaGetLastError();
			fail(TMFQS_ERR_NOMEM, "gate pass program allocation failed");
		}
		dev_prog_bytes = need * 2;
	}
	std::vector<unsigned char> host(need);
	if(ops_bytes) std::memcpy(host.data(), ops.data(), ops_bytes);
	if(mat_bytes) std::memcpy(host.data() + ops_bytes, mats.data(), mat_bytes);
	if(ops_bytes + mat_bytes) upload_async(c, dev_prog, host.data(), ops_bytes + mat_bytes, "gate pass program upload");
	typedef typename Vec2<R>::type V;
	const size_t smem = (sizeof(V) << K) + g.nops * sizeof(OpS<R>) + g.nterms * sizeof(GateOp) + g.nstages * sizeof(StageSlots) +
	                    g.nmat * sizeof(typename MatElem<R>::type) + g.ndiag * (kDiagThread * kThreads + 2 * kDiagTile) * sizeof(V);
	constexpr unsigned threads = 1u << (K - RB);
	auto kern = mats.empty() ? k_gate_pass<R, RB, EXACT, kPlain> : k_gate_pass<R, RB, EXACT, kDense>;
	if constexpr(!EXACT && sizeof(R) == 8 && RB != small_bits<R>())
		if(merged) kern = k_gate_pass<R, RB, EXACT, kMerged>;
	allow_dynamic_smem(kern, "gate pass smem");
	int per_sm = 1;
	check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem), "gate pass occupancy");
	const uint64_t grid = std::min<uint64_t>(g.ntiles - g.o_begin, (uint64_t)c.num_sms * std::max(1, per_sm));
	kern<<<(unsigned)grid, threads, smem, c.stream>>>(static_cast<V *>(a), static_cast<V *>(mirror), g, static_cast<const GateOp *>(dev_prog),
	                                                 reinterpret_cast<const double2 *>(static_cast<unsigned char *>(dev_prog) + ops_bytes));
	check_cuda(cudaGetLastError(), "gate pass");
	if(c.launches) ++*c.launches;
	return true;
}

template <typename R, bool EXACT>
bool pick_gate_pass(const LaunchCtx &c, void *a, const FusedPass &pass, void *&dev_prog, size_t &dev_prog_bytes, void *mirror, bool merged) {
	const uint64_t tiles = pass.n >= tile_bits<R>() ? 1ull << (pass.n - tile_bits<R>()) : 0;
	if(!merged && tiles <= (uint64_t)c.num_sms && run_gate_pass<R, small_bits<R>(), EXACT>(c, a, pass, dev_prog, dev_prog_bytes, mirror, merged))
		return true;
	return run_gate_pass<R, reg_bits<R>(), EXACT>(c, a, pass, dev_prog, dev_prog_bytes, mirror, merged);
}

}  // namespace

bool launch_gate_pass(const LaunchCtx &c, int prec, bool exact, void *a, const FusedPass &pass, void *&dev_prog, size_t &dev_prog_bytes,
                      void *mirror, bool merged) {
	if(prec == TMFQS_FP32) return pick_gate_pass<float, false>(c, a, pass, dev_prog, dev_prog_bytes, mirror, merged);
	return exact ? pick_gate_pass<double, true>(c, a, pass, dev_prog, dev_prog_bytes, mirror, merged)
	             : pick_gate_pass<double, false>(c, a, pass, dev_prog, dev_prog_bytes, mirror, merged);
}

void launch_fused_pass(const LaunchCtx &c, int prec, bool exact, void *a, const FusedPass &pass, void *&dev_prog,
                       size_t &dev_prog_bytes) {
	if(launch_fused_stages(c, prec, a, pass, dev_prog, dev_prog_bytes)) return;
	if(launch_gate_pass(c, prec, exact, a, pass, dev_prog, dev_prog_bytes)) return;
	launch_fused_ops(c, prec, a, pass, dev_prog, dev_prog_bytes);
}

}  // namespace tqb
