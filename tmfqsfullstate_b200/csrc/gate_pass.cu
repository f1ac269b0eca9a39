// General fused passes as register stages: any mix of Hadamards, X, CNOTs,
// swaps, dense one- and two-qubit gates, controlled phases and basis-state flips
// on a tile's local bits.
//
// A pass's moving operations (H, X, CNOT, dense gates) are cut, in circuit order, into stages
// of up to four distinct targets.  In a stage every thread holds the 16
// amplitudes of the tile that differ in the stage's four register bits and
// applies the stage's operations to them in registers; diagonal operations run
// in whatever stage they fall into, under per-thread and per-register
// conditions.  The first stage reads the tile from HBM, the last writes it back,
// those between pass it on through shared memory with one barrier each.  A swap
// of two local bits moves nothing: it relabels them, and the last stage stores
// every amplitude at its final place.
//
// Exact form: the IEEE operations of the per-gate path in circuit order for each
// amplitude (dense_state_backend.cpp:255-319), zero pairs and zero amplitudes
// skipped as there, so the result is bit-identical.  Fast forms: butterflies
// without their 1/sqrt(2), which is applied once as a power at the end.
//
// Bound: HBM (one read and one write per pass) and, behind it, instruction issue:
// about 100 instructions per operation and 16 amplitudes.  A pass of 12-35 mixed
// operations on 23 qubits complex128 (41 us at the copy rate) takes 81-181 us, and
// one of 10-21 on 26 qubits complex64 (164 us) 345-612 us; op by op through shared
// memory with a barrier each (k_fused) they took 205-471 us and 900-1850 us.
// Dense two-qubit gates are arithmetic: 30 us of FP64 each on 24 qubits exact (four
// in a pass 235 us, alone 104 us each), 107 us each on 27 qubits complex64 (four in
// a pass 750 us; as tensor-core blocks of two 515 us per block).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

namespace tqb {

namespace {

constexpr unsigned kRB = 4;            // register bits per stage
constexpr unsigned kRegs = 1u << kRB;  // amplitudes per thread
constexpr unsigned kMaxK = 13;
constexpr unsigned kMaxStages = 64;
constexpr unsigned kMaxOps = 240;

// Tiles of 64 KiB.
template <typename R>
constexpr unsigned tile_bits() {
	return sizeof(R) == 8 ? 12u : 13u;
}
// Index bits of a 128-byte line: lanes in stages that touch HBM, and the shared-memory slot bits that pick a bank group.
template <typename R>
constexpr unsigned line_bits() {
	return sizeof(R) == 8 ? 3u : 4u;
}

// Operation codes: kCodeH + register bit; kCodeX + 4 * target + control register
// bit (the target itself: none); kCodeCP + mask of register bits that must be
// set; kCodeFlip; kCodeU1 + register bit; kCodeU2 + 4 * first + second register
// bit (the first is the more significant one of the gate's block index).
constexpr unsigned kCodeH = 0, kCodeX = 4, kCodeCP = 20, kCodeFlip = 36, kCodeU1 = 37, kCodeU2 = 41;

struct GateOp {
	uint32_t code;
	uint16_t tmask, rval;  // thread index bits that must be set; flips: the thread index and the register of the state
	uint64_t omask;        // outer index bits that must be set; flips: the state's outer bits; dense gates: the matrix
	double cr, ci;
};

struct GateGeom {
	unsigned n, nstages, nops, nmat;  // nmat: complex matrix elements of the dense gates
	uint64_t o_begin, ntiles;  // the launch runs tiles [o_begin, ntiles)
	double inv, scale;  // 1/sqrt(2); fast forms: the pass's power of it
	uint64_t outer;     // mask of the index bits outside the tile
	uint8_t lpos[kMaxK], opos[kMaxK];  // index bit of a tile bit when loaded and when stored
	uint8_t first[kMaxStages], count[kMaxStages];
	uint8_t rbit[kMaxStages][kRB];          // tile bit of register bit i
	uint8_t tbit[kMaxStages][kMaxK - kRB];  // tile bit of thread index bit k
};

// Non-sign bits of an amplitude: zero exactly for +-0 +- 0i (integer units, not the FP64 pipe).
__device__ __forceinline__ unsigned nonzero_bits(double2 x) {
	return ((unsigned)(__double2hiint(x.x) | __double2hiint(x.y)) << 1) | (unsigned)__double2loint(x.x) |
	       (unsigned)__double2loint(x.y);
}

template <typename R, bool EXACT, unsigned I>
__device__ __forceinline__ void op_h(typename Vec2<R>::type (&v)[kRegs], R inv) {
	typedef typename Vec2<R>::type V;
	auto bfly = [&](V &x, V &y) {
		V o0, o1;
		o0.x = radd(x.x, y.x);
		o0.y = radd(x.y, y.y);
		o1.x = rsub(x.x, y.x);
		o1.y = rsub(x.y, y.y);
		if(EXACT) {
			o0.x = rmul(o0.x, inv);
			o0.y = rmul(o0.y, inv);
			o1.x = rmul(o1.x, inv);
			o1.y = rmul(o1.y, inv);
		}
		x = o0;
		y = o1;
	};
	if constexpr(EXACT) {
		// An all-zero pair is left as it is (dense_state_backend.cpp:265).
		bool zero = false;
#pragma unroll
		for(unsigned r = 0; r < kRegs; ++r)
			if(!((r >> I) & 1u)) zero = zero || (nonzero_bits(v[r]) | nonzero_bits(v[r | (1u << I)])) == 0u;
		if(__any_sync(0xffffffffu, zero)) {
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
template <typename R, bool EXACT, unsigned I, unsigned C>
__device__ __forceinline__ void op_x(typename Vec2<R>::type (&v)[kRegs], bool on) {
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

// Phase on the registers that have all bits of M.
template <typename R, bool EXACT, unsigned M>
__device__ __forceinline__ void op_cp(typename Vec2<R>::type (&v)[kRegs], R pr, R pi) {
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r) {
		if((r & M) != M) continue;
		R re = v[r].x, im = v[r].y;
		if constexpr(EXACT) {
			// Zero amplitudes are skipped (dense_state_backend.cpp:299).
			const bool nz = nonzero_bits(v[r]) != 0u;
			cmul_ref(pr, pi, re, im);
			v[r].x = nz ? re : v[r].x;
			v[r].y = nz ? im : v[r].y;
		} else {
			v[r].x = fma(pr, re, -(pi * im));
			v[r].y = fma(pr, im, pi * re);
		}
	}
}

// Dense gate on register bit I: the unrolled formula of gate_block_apply.h:117-140.
template <typename R, bool EXACT, unsigned I>
__device__ __forceinline__ void op_u1(typename Vec2<R>::type (&v)[kRegs], const typename Vec2<R>::type *m) {
	const auto g00 = m[0], g01 = m[1], g10 = m[2], g11 = m[3];
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r) {
		if((r >> I) & 1u) continue;
		const auto x = v[r], y = v[r | (1u << I)];
		if constexpr(EXACT) {
			if((nonzero_bits(x) | nonzero_bits(y)) == 0u) continue;
			v[r].x = rsub(radd(rsub(rmul(g00.x, x.x), rmul(g00.y, x.y)), rmul(g01.x, y.x)), rmul(g01.y, y.y));
			v[r].y = radd(radd(radd(rmul(g00.x, x.y), rmul(g00.y, x.x)), rmul(g01.x, y.y)), rmul(g01.y, y.x));
			v[r | (1u << I)].x = rsub(radd(rsub(rmul(g10.x, x.x), rmul(g10.y, x.y)), rmul(g11.x, y.x)), rmul(g11.y, y.y));
			v[r | (1u << I)].y = radd(radd(radd(rmul(g10.x, x.y), rmul(g10.y, x.x)), rmul(g11.x, y.y)), rmul(g11.y, y.x));
		} else {
			v[r].x = fma(-g01.y, y.y, fma(g01.x, y.x, fma(-g00.y, x.y, g00.x * x.x)));
			v[r].y = fma(g01.y, y.x, fma(g01.x, y.y, fma(g00.y, x.x, g00.x * x.y)));
			v[r | (1u << I)].x = fma(-g11.y, y.y, fma(g11.x, y.x, fma(-g10.y, x.y, g10.x * x.x)));
			v[r | (1u << I)].y = fma(g11.y, y.x, fma(g11.x, y.y, fma(g10.y, x.x, g10.x * x.y)));
		}
	}
}

// A matrix element from shared memory, loaded where it is used: a broadcast,
// and cheaper than the spills of keeping the whole matrix in registers.
__device__ __forceinline__ double2 mat_at(const double2 *m) {
	double2 x;
	asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x.x), "=d"(x.y) : "r"((unsigned)__cvta_generic_to_shared(m)));
	return x;
}
__device__ __forceinline__ float2 mat_at(const float2 *m) {
	float2 x;
	asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x.x), "=f"(x.y) : "r"((unsigned)__cvta_generic_to_shared(m)));
	return x;
}

// Dense gate on register bits A (more significant) and B: row sums term by term
// (gate_block_apply.h:165-176); all-zero blocks are left alone.
template <typename R, bool EXACT, unsigned A, unsigned B>
__device__ __forceinline__ void op_u2(typename Vec2<R>::type (&v)[kRegs], const typename Vec2<R>::type *m) {
#pragma unroll
	for(unsigned r = 0; r < kRegs; ++r) {
		if(((r >> A) & 1u) || ((r >> B) & 1u)) continue;
		const unsigned at[4] = {r, r | (1u << B), r | (1u << A), r | (1u << A) | (1u << B)};
		typename Vec2<R>::type o[4];
		if constexpr(EXACT)
			if((nonzero_bits(v[at[0]]) | nonzero_bits(v[at[1]]) | nonzero_bits(v[at[2]]) | nonzero_bits(v[at[3]])) == 0u) continue;
#pragma unroll
		for(unsigned row = 0; row < 4; ++row) {
			R nr = R(0), ni = R(0);
#pragma unroll
			for(unsigned c = 0; c < 4; ++c) {
				const auto g = mat_at(m + 4 * row + c), x = v[at[c]];
				if constexpr(EXACT) {
					nr = radd(nr, rsub(rmul(g.x, x.x), rmul(g.y, x.y)));
					ni = radd(ni, radd(rmul(g.x, x.y), rmul(g.y, x.x)));
				} else {
					nr = fma(-g.y, x.y, fma(g.x, x.x, nr));
					ni = fma(g.y, x.x, fma(g.x, x.y, ni));
				}
			}
			o[row].x = nr;
			o[row].y = ni;
		}
#pragma unroll
		for(unsigned c = 0; c < 4; ++c) v[at[c]] = o[c];
	}
}

template <typename R, bool EXACT>
__device__ __forceinline__ void run_op(const GateOp &op, typename Vec2<R>::type (&v)[kRegs], const GateGeom &g, const typename Vec2<R>::type *mats, uint64_t base, unsigned t) {
	if(op.code == kCodeFlip) {
		const unsigned at = (base & g.outer) == op.omask && t == op.tmask ? op.rval : kRegs;
#pragma unroll
		for(unsigned r = 0; r < kRegs; ++r) {
			v[r].x = r == at ? -v[r].x : v[r].x;
			v[r].y = r == at ? -v[r].y : v[r].y;
		}
		return;
	}
	if(op.code >= kCodeU1) {
		const typename Vec2<R>::type *m = mats + op.omask;
		switch(op.code) {
#define TQB_U1(I) \
	case kCodeU1 + I: op_u1<R, EXACT, I>(v, m); return;
#define TQB_U2(A, B) \
	case kCodeU2 + 4 * A + B: op_u2<R, EXACT, A, B>(v, m); return;
			TQB_U1(0) TQB_U1(1) TQB_U1(2) TQB_U1(3)
			TQB_U2(0, 1) TQB_U2(0, 2) TQB_U2(0, 3) TQB_U2(1, 0) TQB_U2(1, 2) TQB_U2(1, 3)
			TQB_U2(2, 0) TQB_U2(2, 1) TQB_U2(2, 3) TQB_U2(3, 0) TQB_U2(3, 1) TQB_U2(3, 2)
#undef TQB_U1
#undef TQB_U2
			default: return;
		}
	}
	if((base & op.omask) != op.omask) return;
	const bool on = (t & op.tmask) == op.tmask;
	const R inv = (R)g.inv;
	switch(op.code) {
		case kCodeH + 0: op_h<R, EXACT, 0>(v, inv); return;
		case kCodeH + 1: op_h<R, EXACT, 1>(v, inv); return;
		case kCodeH + 2: op_h<R, EXACT, 2>(v, inv); return;
		case kCodeH + 3: op_h<R, EXACT, 3>(v, inv); return;
#define TQB_X(I, C) \
	case kCodeX + 4 * I + C: op_x<R, EXACT, I, C>(v, on); return;
		TQB_X(0, 0) TQB_X(0, 1) TQB_X(0, 2) TQB_X(0, 3)
		TQB_X(1, 0) TQB_X(1, 1) TQB_X(1, 2) TQB_X(1, 3)
		TQB_X(2, 0) TQB_X(2, 1) TQB_X(2, 2) TQB_X(2, 3)
		TQB_X(3, 0) TQB_X(3, 1) TQB_X(3, 2) TQB_X(3, 3)
#undef TQB_X
		default: break;
	}
	if(!on) return;
	const R pr = (R)op.cr, pi = (R)op.ci;
	switch(op.code) {
#define TQB_CP(M) \
	case kCodeCP + M: op_cp<R, EXACT, M>(v, pr, pi); return;
		TQB_CP(0) TQB_CP(1) TQB_CP(2) TQB_CP(3) TQB_CP(4) TQB_CP(5) TQB_CP(6) TQB_CP(8) TQB_CP(9) TQB_CP(10) TQB_CP(12)
#undef TQB_CP
		default: break;
	}
}

// Shared-memory slot of tile bit b: a bit above the bank-group bits also flips
// one of them, so that lanes on bits of different residues spread over the banks.
template <typename R>
__device__ __forceinline__ unsigned slot_of(unsigned b) {
	constexpr unsigned s = line_bits<R>();
	return (1u << b) | (b >= s ? 1u << (b % s) : 0u);
}

template <typename R, bool EXACT>
__global__ void __launch_bounds__(1u << (tile_bits<R>() - kRB), 2) k_gate_pass(typename Vec2<R>::type *a, const __grid_constant__ GateGeom g,
                                                                              const GateOp *gops, const double2 *gmats) {
	typedef typename Vec2<R>::type V;
	constexpr unsigned K = tile_bits<R>(), TB = K - kRB;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	V *s = reinterpret_cast<V *>(smem_raw);
	GateOp *ops = reinterpret_cast<GateOp *>(smem_raw + (sizeof(V) << K));
	V *mats = reinterpret_cast<V *>(ops + g.nops);
	const unsigned t = threadIdx.x;
	for(unsigned e = t; e < g.nops * (sizeof(GateOp) / 16); e += blockDim.x)
		reinterpret_cast<int4 *>(ops)[e] = reinterpret_cast<const int4 *>(gops)[e];
	for(unsigned e = t; e < g.nmat; e += blockDim.x) {
		const double2 x = gmats[e];
		mats[e].x = (R)x.x;
		mats[e].y = (R)x.y;
	}
	__syncthreads();
	for(uint64_t o = g.o_begin + blockIdx.x; o < g.ntiles; o += gridDim.x) {
		uint64_t base = o;
#pragma unroll
		for(unsigned i = 0; i < K; ++i) base = insert0(base, g.lpos[i]);
		for(unsigned st = 0; st < g.nstages; ++st) {
			const bool last = st + 1 == g.nstages;
			V v[kRegs];
			// Where this thread's amplitudes sit in shared memory.
			unsigned slot = 0, ro[kRB];
#pragma unroll
			for(unsigned k = 0; k < TB; ++k) slot ^= (t >> k) & 1u ? slot_of<R>(g.tbit[st][k]) : 0u;
#pragma unroll
			for(unsigned i = 0; i < kRB; ++i) ro[i] = slot_of<R>(g.rbit[st][i]);
			auto at = [&](unsigned r) {
				unsigned x = slot;
#pragma unroll
				for(unsigned i = 0; i < kRB; ++i)
					if((r >> i) & 1u) x ^= ro[i];
				return x;
			};
			// And in HBM.
			auto global = [&](const uint8_t *pos, uint64_t (&go)[kRB]) {
				uint64_t x = base;
#pragma unroll
				for(unsigned k = 0; k < TB; ++k) x |= (uint64_t)((t >> k) & 1u) << pos[g.tbit[st][k]];
#pragma unroll
				for(unsigned i = 0; i < kRB; ++i) go[i] = 1ull << pos[g.rbit[st][i]];
				return x;
			};
			if(st == 0) {
				uint64_t go[kRB];
				const uint64_t gb = global(g.lpos, go);
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) {
					uint64_t x = gb;
#pragma unroll
					for(unsigned i = 0; i < kRB; ++i)
						if((r >> i) & 1u) x |= go[i];
					v[r] = a[x];
				}
			} else {
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) v[r] = s[at(r)];
			}
			const unsigned k1 = (unsigned)g.first[st] + g.count[st];
			for(unsigned k = g.first[st]; k < k1; ++k) run_op<R, EXACT>(ops[k], v, g, mats, base, t);
			if(last) {
				uint64_t go[kRB];
				const uint64_t gb = global(g.opos, go);
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) {
					uint64_t x = gb;
#pragma unroll
					for(unsigned i = 0; i < kRB; ++i)
						if((r >> i) & 1u) x |= go[i];
					if(!EXACT) {
						v[r].x *= (R)g.scale;
						v[r].y *= (R)g.scale;
					}
					a[x] = v[r];
				}
			} else {
#pragma unroll
				for(unsigned r = 0; r < kRegs; ++r) s[at(r)] = v[r];
			}
			// Between stages, and before the next tile's first stage writes what the last one read.
			if(g.nstages > 1) __syncthreads();
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
bool plan_gates(const FusedPass &pass, unsigned K, unsigned line, GateGeom &g, std::vector<GateOp> &out) {
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
	// Stages: consecutive operations while their targets fit in four register bits.
	std::vector<uint32_t> regs{0u};
	std::vector<std::vector<unsigned>> of(1);
	for(unsigned k = 0; k < ops.size(); ++k) {
		uint32_t bits = 0;
		if(ops[k].kind != PlanOp::kCP && ops[k].kind != PlanOp::kFlip) bits = 1u << ops[k].p;
		if(ops[k].kind == PlanOp::kU2) bits |= 1u << ops[k].p2;
		if(bits & ~regs.back()) {
			if(__builtin_popcount(regs.back() | bits) > (int)kRB || (regs.size() == 1 && (keep_in & bits))) {
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
		while(__builtin_popcount(r) < (int)kRB) {
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
		for(unsigned i = 0; i < kRB; ++i) g.rbit[st][i] = (uint8_t)rb[i];
		for(unsigned k = 0; k < tb.size(); ++k) g.tbit[st][k] = (uint8_t)tb[k];
		g.first[st] = (uint8_t)out.size();
		g.count[st] = (uint8_t)of[st].size();
		for(unsigned k : of[st]) {
			const PlanOp &q = ops[k];
			GateOp o{};
			uint32_t rm = 0, tm = 0;
			for(unsigned i = 0; i < kRB; ++i) rm |= ((q.pm >> rb[i]) & 1u) << i;
			for(unsigned i = 0; i < tb.size(); ++i) tm |= ((q.pm >> tb[i]) & 1u) << i;
			unsigned target = 0, second = 0;
			for(unsigned i = 0; i < kRB; ++i) {
				if(rb[i] == q.p) target = i;
				if(rb[i] == q.p2) second = i;
			}
			o.tmask = (uint16_t)tm;
			o.omask = q.om;
			o.cr = q.cr;
			o.ci = q.ci;
			switch(q.kind) {
				case PlanOp::kH: o.code = kCodeH + target; break;
				case PlanOp::kX: o.code = kCodeX + 4 * target + (rm ? (unsigned)__builtin_ctz(rm) : target); break;
				case PlanOp::kCP: o.code = kCodeCP + rm; break;
				case PlanOp::kFlip:
					o.code = kCodeFlip;
					o.rval = (uint16_t)rm;
					break;
				case PlanOp::kU1:
				case PlanOp::kU2:
					o.code = q.kind == PlanOp::kU1 ? kCodeU1 + target : kCodeU2 + 4 * target + second;
					o.omask = q.mat;
					break;
			}
			out.push_back(o);
		}
	}
	g.nops = (unsigned)out.size();
	g.nmat = (unsigned)(pass.mats.size() / 2);
	g.scale = std::pow(2.0, -0.5 * (double)nh);
	return true;
}

template <typename R, bool EXACT>
bool run_gate_pass(const LaunchCtx &c, void *a, const FusedPass &pass, void *&dev_prog, size_t &dev_prog_bytes) {
	constexpr unsigned K = tile_bits<R>();
	GateGeom g;
	std::vector<GateOp> ops;
	if(!plan_gates(pass, K, line_bits<R>(), g, ops)) return false;
	const size_t ops_bytes = ops.size() * sizeof(GateOp), mat_bytes = pass.mats.size() * sizeof(double);
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
	if(mat_bytes) std::memcpy(host.data() + ops_bytes, pass.mats.data(), mat_bytes);
	if(ops_bytes + mat_bytes) upload_async(c, dev_prog, host.data(), ops_bytes + mat_bytes, "gate pass program upload");
	typedef typename Vec2<R>::type V;
	const size_t smem = (sizeof(V) << K) + ops_bytes + g.nmat * sizeof(V);
	auto kern = k_gate_pass<R, EXACT>;
	check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "gate pass smem");
	const unsigned threads = 1u << (K - kRB);
	int per_sm = 1;
	check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem), "gate pass occupancy");
	const uint64_t grid = std::min<uint64_t>(g.ntiles - g.o_begin, (uint64_t)c.num_sms * std::max(1, per_sm));
	kern<<<(unsigned)grid, threads, smem, c.stream>>>(static_cast<V *>(a), g, static_cast<const GateOp *>(dev_prog),
	                                                 reinterpret_cast<const double2 *>(static_cast<unsigned char *>(dev_prog) + ops_bytes));
	check_cuda(cudaGetLastError(), "gate pass");
	if(c.launches) ++*c.launches;
	return true;
}

}  // namespace

bool launch_gate_pass(const LaunchCtx &c, int prec, bool exact, void *a, const FusedPass &pass, void *&dev_prog, size_t &dev_prog_bytes) {
	if(prec == TMFQS_FP32) return run_gate_pass<float, false>(c, a, pass, dev_prog, dev_prog_bytes);
	return exact ? run_gate_pass<double, true>(c, a, pass, dev_prog, dev_prog_bytes)
	             : run_gate_pass<double, false>(c, a, pass, dev_prog, dev_prog_bytes);
}

}  // namespace tqb
