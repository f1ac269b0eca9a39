// Exact replay of the reference's sequential double sums on the GPU.
//
// Reductions replaced (all left-to-right loops in the reference):
//   totalProbability      dense_state_backend.cpp:161-171  (terms |a|^2)
//   sampleMeasurement     dense_state_backend.cpp:173-188  (first s with rnd <= running sum)
//   logicalAmplitudeSum   quantum_register.cpp:176-190     (terms re, im; signed)
//   overlay branches      quantum_register.cpp:269-310     (terms of scale*a+bias)
//
// Tile = 4096 terms, group = 32 tiles; math in seqsum_core.h.  Launches:
//   k_seq_guess  (large sums) estimates the running sum's course from a few
//                samples of each of 1024 strata.
//   k_seq_tiles  reads the state once: each tile's sum and, where the estimate
//                names the binade the running sum should be in (two, near a
//                crossing), the tile's increment on that grid.
//   k_seq_join   worker blocks: the prefixes of the tile sums tell which tiles
//                have the increment they need; the others are read again (all of
//                them where nothing was guessed).  They compose the groups.
//                walk block, one per sum, alongside: carries the exact running
//                sum over the groups as they become ready, then tiles, checking
//                each step against the binade it really is in.  A tile whose
//                increment does not apply (a binade crossing, the first tile, the
//                measured index) is replayed from its terms, 4096 at a time.
// Estimates and prefixes are approximate: a wrong one costs time only, the walk
// decides what applies.  Sums of at most kDirectTiles tiles are replayed by the
// walk block alone.
//
// Bound: HBM, one read of the state, and behind it the walk, a serial chain of
// about 5 us per binade crossing.  Total probability, complex128, n = 28:
// 0.86 ms (4.3 GB; 2.5 ms with two reads, double-double tile sums and 32-term
// replays); n = 20: 0.08 ms (0.38).  A single-read look-back over the tiles
// measured 1.8 ms and more (its waits drain the loads in flight), the walk in
// one warp 1.38 ms (a lone warp's step costs as much as the block's).
#include <algorithm>
#include <cmath>
#include <mutex>

#include "device_common.cuh"
#include "internal.h"
#include "seqsum_core.h"

namespace tqb {

namespace {

constexpr unsigned kThreads = 256;
constexpr unsigned kPer = 16;                // terms per thread
constexpr unsigned kTile = kThreads * kPer;  // terms per tile
constexpr unsigned kGroup = 32;              // tiles per group
constexpr unsigned kWarps = kThreads / 32;
constexpr unsigned kStage = kTile + kThreads;  // staged terms: a thread's run of 16 padded to 17
constexpr unsigned kDirectTiles = 4;
constexpr unsigned kStrata = 1024;            // strata of the estimate, kThreads samples each
constexpr uint64_t kGuessTerms = 1ull << 22;  // sums from this length on are estimated first
constexpr unsigned kMaxSums = 2;
constexpr double kBinade = 4503599627370496.0;  // 2^52, the start of the binade on its own grid
constexpr unsigned FULL = 0xffffffffu;
// Sums outside this range are added term by term (the grid scale and its inverse stay normal inside it).
constexpr double kTiny = 1e-280, kHuge = 1e280;
constexpr unsigned kSpinLimit = 1u << 20;

// Effect of a run of terms on the running sum (tile or group): grid increments
// for binades e and e + 1, and for signed sums the run's sum and the extremes
// of its prefix sums.  (Copied in 16-byte words.)
struct alignas(16) SeqRec {
	int e;        // tq::kIdentity: all terms zero
	unsigned ok;  // kHasE, kHasE1: the increments that are known; kUp, kDown: no term is negative / positive
	long long i0[2], i1[2];
	double s, mn, mx;
};

constexpr unsigned kHasE = 1, kHasE1 = 2, kUp = 4, kDown = 8, kAny = 15;

struct SeqTables {
	SeqRec *tiles, *groups;  // [sum][ntiles], [sum][ngroups]
	double *est;             // [sum][kStrata] estimated sums of the strata
	double *chunk;           // [sum][nchunks] sums of the chunks of tiles that the blocks take
	unsigned *gcount;        // tiles of the group that are final
	unsigned *gready;        // 1: the group's record is written
	unsigned ntiles, ngroups, nchunks;
	bool guess;
	double rel;  // relative distance a sequential sum of this length may be off
};

struct WalkOut {
	unsigned long long index;
	double value;
};

// Terms of one state: kind Prob |a|^2 (one sum), kind Amp the real and
// imaginary parts (two sums).
template <typename R, int KIND>
struct TermF {
	static constexpr int kSums = KIND == kTermProb ? 1 : 2;
	static constexpr bool kSigned = KIND != kTermProb;
	const typename Vec2<R>::type *a;
	int ov;
	double sr, si, br, bi;
	typedef typename Vec2<R>::type Raw;
	__device__ __forceinline__ Raw load(uint64_t j) const { return a[j]; }
	__device__ __forceinline__ void terms(const Raw &v, double (&p)[kSums]) const {
		double re = (double)v.x, im = (double)v.y;
		if(ov) {
			// applyAffineOverlay, quantum_register.cpp:160-165.
			const double mr = rsub(rmul(sr, re), rmul(si, im));
			const double mi = radd(rmul(sr, im), rmul(si, re));
			re = radd(mr, br);
			im = radd(mi, bi);
		}
		if constexpr(KIND == kTermProb) {
			p[0] = radd(rmul(re, re), rmul(im, im));
		} else {
			p[0] = re;
			p[1] = im;
		}
	}
};

// Squared distance of two states at j, as experiment::compareStates forms it
// (comparison.cpp:29-38): the candidate minus the reference, per component,
// in double.
template <typename RA, typename RB>
struct TermDiff {
	static constexpr int kSums = 1;
	static constexpr bool kSigned = false;
	const typename Vec2<RA>::type *ref;
	const typename Vec2<RB>::type *got;
	typedef double Raw;  // formed at the load: two states' amplitudes would not fit the registers
	__device__ __forceinline__ Raw load(uint64_t j) const {
		const auto r = ref[j];
		const auto g = got[j];
		const double dr = rsub((double)g.x, (double)r.x), di = rsub((double)g.y, (double)r.y);
		return radd(rmul(dr, dr), rmul(di, di));
	}
	__device__ __forceinline__ void terms(const Raw &v, double (&p)[1]) const { p[0] = v; }
};

__device__ __forceinline__ tq::Inc shfl_up_inc(tq::Inc v, unsigned d) {
	return tq::Inc{__shfl_up_sync(FULL, v.i0, d), __shfl_up_sync(FULL, v.i1, d)};
}

// Inclusive ordered scan of increments over lanes: a plain sum where no lane
// depends on the parity (nearly always).
__device__ __forceinline__ tq::Inc warp_scan_inc(tq::Inc v) {
	const unsigned lane = threadIdx.x & 31u;
	if(__all_sync(FULL, v.i0 == v.i1)) {
#pragma unroll
		for(unsigned d = 1; d < 32; d <<= 1) {
			const long long o = __shfl_up_sync(FULL, v.i0, d);
			if(lane >= d) v.i0 += o;
		}
		v.i1 = v.i0;
		return v;
	}
	for(unsigned d = 1; d < 32; d <<= 1) {
		const tq::Inc o = shfl_up_inc(v, d);
		if(lane >= d) v = tq::compose(o, v);
	}
	return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
	for(unsigned d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
	return v;
}

__device__ __forceinline__ unsigned stage_slot(unsigned i) { return i + i / kPer; }

__device__ __forceinline__ SeqRec load_rec(const SeqRec *p) {
	static_assert(alignof(SeqRec) >= alignof(int4) && sizeof(SeqRec) % sizeof(int4) == 0, "records are copied as int4");
	SeqRec r;
	const int4 *src = reinterpret_cast<const int4 *>(p);
	int4 *dst = reinterpret_cast<int4 *>(&r);
#pragma unroll
	for(unsigned k = 0; k < sizeof(SeqRec) / 16; ++k) dst[k] = __ldcg(src + k);
	return r;
}
__device__ __forceinline__ SeqRec identity_rec() {
	SeqRec r;
	r.e = tq::kIdentity;
	r.ok = kAny;
	r.i0[0] = r.i0[1] = r.i1[0] = r.i1[1] = 0;
	r.s = r.mn = r.mx = 0.0;
	return r;
}

// Composition of 32 records (one per lane) for binades e0 and e0 + 1, e0 the
// lowest first binade of theirs.  Lane 0 returns the result.
template <bool SIGNED>
__device__ SeqRec compose_group(const SeqRec &r) {
	const unsigned lane = threadIdx.x & 31u;
	const bool id = r.e == tq::kIdentity;
	int e0 = id || !(r.ok & (kHasE | kHasE1)) ? tq::kIdentity : r.e;
#pragma unroll
	for(unsigned d = 16; d > 0; d >>= 1) e0 = min(e0, __shfl_xor_sync(FULL, e0, d));
	SeqRec g;
	g.e = e0;
	g.ok = (__all_sync(FULL, r.ok & kUp) ? kUp : 0u) | (__all_sync(FULL, r.ok & kDown) ? kDown : 0u);
	if(__all_sync(FULL, id)) {
		g.ok = kAny;
	} else if(e0 == tq::kIdentity) {
		g.e = tq::kDirty;
	}
#pragma unroll
	for(unsigned c = 0; c < 2; ++c) {
		const int e = e0 + (int)c;
		tq::Inc v = tq::inc_identity();
		bool has = id;
		if(!id && r.e == e && (r.ok & kHasE)) {
			v = tq::Inc{r.i0[0], r.i1[0]};
			has = true;
		} else if(!id && r.e + 1 == e && (r.ok & kHasE1)) {
			v = tq::Inc{r.i0[1], r.i1[1]};
			has = true;
		}
		if(__all_sync(FULL, has)) g.ok |= kHasE << c;
		v = warp_scan_inc(v);
		g.i0[c] = __shfl_sync(FULL, v.i0, 31);
		g.i1[c] = __shfl_sync(FULL, v.i1, 31);
	}
	g.s = g.mn = g.mx = 0.0;
	if(SIGNED) {
		double s = id ? 0.0 : r.s;
		const double own = s;
		for(unsigned d = 1; d < 32; d <<= 1) {
			const double o = __shfl_up_sync(FULL, s, d);
			if(lane >= d) s += o;
		}
		double mn = id ? 0.0 : s - own + r.mn, mx = id ? 0.0 : s - own + r.mx;
#pragma unroll
		for(unsigned d = 16; d > 0; d >>= 1) {
			mn = fmin(mn, __shfl_xor_sync(FULL, mn, d));
			mx = fmax(mx, __shfl_xor_sync(FULL, mx, d));
		}
		g.s = __shfl_sync(FULL, s, 31);
		g.mn = fmin(mn, 0.0);
		g.mx = fmax(mx, 0.0);
	}
	return g;
}

// Effect of a thread's 16 consecutive terms on a running sum in the binade of
// `scale` that starts at an even and at an odd grid value: two chains of real
// double additions from a representative start of each parity, which round as
// the sequential sum does.  Non-negative terms start at the bottom of the
// binade, signed ones in its middle; the run must not leave it.
template <bool SIGNED>
__device__ __forceinline__ tq::Inc run_increment(const double *p, double scale) {
	const double start = SIGNED ? 1.5 * kBinade : kBinade;
	double c0 = start, c1 = start + 1.0;
#pragma unroll
	for(unsigned k = 0; k < kPer; ++k) {
		const double x = p[k] * scale;
		c0 += x;
		c1 += x;
	}
	return tq::Inc{(long long)(c0 - start), (long long)(c1 - (start + 1.0))};
}

// What a warp's 512 terms of a tile come to (signs: kUp, kDown).
struct WarpPart {
	double s, mag, mn, mx;
	tq::Inc inc[2];
	unsigned wide, signs;
};

// The record of one sum of a tile from its terms in `st` (this thread's run of
// 16 at p), for binades e and, with `two`, e + 1 (kDirty: none): each warp
// leaves its part, and after the block's next barrier parts_join makes the
// record.
template <bool SIGNED>
__device__ __forceinline__ void tile_parts(const double *p, int e, bool two, WarpPart *parts) {
	const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	WarpPart w;
	double s = 0.0, least = 0.0, most = 0.0;
#pragma unroll
	for(unsigned k = 0; k < kPer; ++k) {
		s += p[k];
		if(SIGNED) {
			least = fmin(least, p[k]);
			most = fmax(most, p[k]);
		}
	}
	const double own = s;
	s = warp_sum(s);
	w.s = s;
	w.mag = s;
	w.mn = 0.0;
	w.mx = s;
	w.signs = kUp;
	if(SIGNED) {
		const bool up = __all_sync(FULL, least >= 0.0), down = __all_sync(FULL, most <= 0.0);
		w.signs = (up ? kUp : 0u) | (down ? kDown : 0u);
		w.mag = fabs(s);  // terms of one sign
		if(down) {
			w.mn = s;
			w.mx = 0.0;
		}
		if(!up && !down) {
			// Extremes of the prefix sums.
			double run = 0.0, lo = 0.0, hi = 0.0, mag = fmax(-least, most);
#pragma unroll
			for(unsigned k = 0; k < kPer; ++k) {
				run += p[k];
				lo = fmin(lo, run);
				hi = fmax(hi, run);
			}
			double incl = own;
#pragma unroll
			for(unsigned d = 1; d < 32; d <<= 1) {
				const double o = __shfl_up_sync(FULL, incl, d);
				if(lane >= d) incl += o;
			}
			lo += incl - own;
			hi += incl - own;
#pragma unroll
			for(unsigned d = 16; d > 0; d >>= 1) {
				lo = fmin(lo, __shfl_xor_sync(FULL, lo, d));
				hi = fmax(hi, __shfl_xor_sync(FULL, hi, d));
				mag = fmax(mag, __shfl_xor_sync(FULL, mag, d));
			}
			w.mag = mag * (double)kPer;
			w.mn = lo;
			w.mx = hi;
		}
	}
	w.wide = 0;
	if(e != tq::kDirty) {
#pragma unroll
		for(int k = 0; k < 2; ++k) {
			if(k && !two) break;
			const double scale = tq::grid_scale(e + k);
			tq::Inc v = run_increment<SIGNED>(p, scale);
			// Every run must stay in the binade: it gets at most `mag` away from
			// where it starts, the middle for signed sums and else the bottom.  (`mag` of
			// mixed signs knows nothing of a NaN; the sum does.)
			const bool wide = !(w.mag * (SIGNED ? 2.0 : 1.0) * scale < kBinade) || w.s != w.s;
			if(__all_sync(FULL, v.i0 == v.i1)) {
#pragma unroll
				for(unsigned d = 16; d > 0; d >>= 1) v.i0 += __shfl_xor_sync(FULL, v.i0, d);
				v.i1 = v.i0;
			} else {
				v = warp_scan_inc(v);
				v.i0 = __shfl_sync(FULL, v.i0, 31);
				v.i1 = __shfl_sync(FULL, v.i1, 31);
			}
			w.inc[k] = v;
			w.wide |= (unsigned)wide << k;
		}
	}
	if(lane == 0) parts[warp] = w;
}

template <bool SIGNED>
__device__ __forceinline__ SeqRec parts_join(const WarpPart *parts, int e, bool two) {
	SeqRec r = identity_rec();
	double mag = 0.0;
	unsigned wide = 0, signs = kUp | kDown;
	r.i0[0] = r.i0[1] = r.i1[0] = r.i1[1] = 0;
	tq::Inc v[2] = {tq::inc_identity(), tq::inc_identity()};
	for(unsigned w = 0; w < kWarps; ++w) {
		const WarpPart &q = parts[w];
		if(SIGNED) {
			r.mn = fmin(r.mn, r.s + q.mn);
			r.mx = fmax(r.mx, r.s + q.mx);
		}
		r.s += q.s;
		mag = fmax(mag, q.mag);
		wide |= q.wide;
		signs &= q.signs;
		if(e != tq::kDirty) {
			v[0] = tq::compose(v[0], q.inc[0]);
			if(two) v[1] = tq::compose(v[1], q.inc[1]);
		}
	}
	if(!SIGNED) r.mx = r.s;
	if(mag == 0.0 && r.s == 0.0) return r;  // (fmax passes over a NaN)
	r.e = e;
	r.ok = signs | (e == tq::kDirty ? 0u : (two ? kHasE | kHasE1 : kHasE) & ~wide);
	for(unsigned k = 0; k < 2; ++k) {
		r.i0[k] = v[k].i0;
		r.i1[k] = v[k].i1;
	}
	return r;
}

// Binades a running sum passes while it goes from P to P + [mn, mx], each end
// widened by the relative `slack`: e and, with `two`, e + 1; false: more than
// two, zero in between, or outside the normal range.
__device__ __forceinline__ bool binades(double P, double mn, double mx, double slack, int &e, bool &two) {
	const double lo = P + mn, hi = P + mx;
	const bool neg = hi < 0.0;
	const double nearer = (neg ? -hi : lo) * (1.0 - slack), farther = (neg ? -lo : hi) * (1.0 + slack);
	e = tq::kDirty;
	two = false;
	if(!(nearer >= kTiny && farther <= kHuge)) return false;
	const int a = tq::binade(nearer), b = tq::binade(farther);
	if(b - a > 1) return false;
	e = a;
	two = b != a;
	return true;
}

// Estimated sum of each stratum: one block per stratum, one sample per thread
// at a hashed place of the thread's share.
template <class F>
__global__ void __launch_bounds__(kThreads) k_seq_guess(F term, uint64_t N, double *est) {
	__shared__ double sh[F::kSums][kWarps];
	const uint64_t share = N / ((uint64_t)kStrata * kThreads);
	uint32_t z = (blockIdx.x * kThreads + threadIdx.x) * 0x9e3779b9u + 0x7f4a7c15u;
	z = (z ^ (z >> 16)) * 0x85ebca6bu;
	z = (z ^ (z >> 13)) * 0xc2b2ae35u;
	const uint64_t at = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) * share + (z ^ (z >> 16)) % share;
	double v[F::kSums];
	term.terms(term.load(at), v);
#pragma unroll
	for(int c = 0; c < F::kSums; ++c) {
		const double s = warp_sum(v[c]);
		if((threadIdx.x & 31u) == 0) sh[c][threadIdx.x >> 5] = s;
	}
	__syncthreads();
	if(threadIdx.x < F::kSums) {
		double s = 0.0;
		for(unsigned w = 0; w < kWarps; ++w) s += sh[threadIdx.x][w];
		est[threadIdx.x * kStrata + blockIdx.x] = s * (double)share;
	}
}

template <class F>
__device__ __forceinline__ void load_tile(const F &term, unsigned tile, typename F::Raw (&raw)[kPer]) {
	const uint64_t base = (uint64_t)tile * kTile + threadIdx.x;
#pragma unroll
	for(unsigned q = 0; q < kPer; ++q) raw[q] = term.load(base + q * kThreads);
}
template <class F>
__device__ __forceinline__ void stage_tile(const F &term, const typename F::Raw (&raw)[kPer], double *st) {
#pragma unroll
	for(unsigned q = 0; q < kPer; ++q) {
		double v[F::kSums];
		term.terms(raw[q], v);
#pragma unroll
		for(int c = 0; c < F::kSums; ++c) st[c * kStage + stage_slot(q * kThreads + threadIdx.x)] = v[c];
	}
}

// First tile of chunk b.
__device__ __forceinline__ unsigned chunk_begin(const SeqTables &T, unsigned b) {
	return (unsigned)((uint64_t)b * T.ntiles / T.nchunks);
}

// Bound: HBM, one read of the state.  A block streams a contiguous chunk of
// tiles: the next tile's loads are in flight while the current one, in shared
// memory in the order of its terms, is added up.
template <class F>
__global__ void __launch_bounds__(kThreads, 2) k_seq_tiles(F term, SeqTables T) {
	constexpr int NC = F::kSums;
	extern __shared__ double st[];                     // staged terms, kStage per sum
	__shared__ double pre[F::kSums][kStrata + 1];  // estimated prefixes of the strata
	__shared__ double tot[F::kSums][kWarps];
	__shared__ WarpPart parts[NC][kWarps];
	const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	for(unsigned g = blockIdx.x * kThreads + tid; g < T.ngroups; g += gridDim.x * kThreads) T.gready[g] = T.gcount[g] = 0u;
	if(T.guess) {
		constexpr unsigned kEach = kStrata / kThreads;
		for(int c = 0; c < NC; ++c) {
			double v[kEach], s = 0.0;
#pragma unroll
			for(unsigned k = 0; k < kEach; ++k) {
				v[k] = T.est[c * kStrata + tid * kEach + k];
				s += v[k];
			}
			double incl = s;
			for(unsigned d = 1; d < 32; d <<= 1) {
				const double o = __shfl_up_sync(FULL, incl, d);
				if(lane >= d) incl += o;
			}
			if(lane == 31) tot[c][warp] = incl;
			__syncthreads();
			double run = incl - s;
			for(unsigned w = 0; w < warp; ++w) run += tot[c][w];
#pragma unroll
			for(unsigned k = 0; k < kEach; ++k) {
				pre[c][tid * kEach + k] = run;
				run += v[k];
			}
			if(tid == kThreads - 1) pre[c][kStrata] = run;
		}
		__syncthreads();
	}
	const unsigned t0 = chunk_begin(T, blockIdx.x), t1 = chunk_begin(T, blockIdx.x + 1);
	const unsigned per = T.ntiles / kStrata;  // tiles per stratum (guessing: at least one)
	typename F::Raw raw[kPer];
	double sum = 0.0;
	load_tile(term, t0, raw);
	for(unsigned t = t0; t < t1; ++t) {
		stage_tile(term, raw, st);
		if(t + 1 < t1) load_tile(term, t + 1, raw);
		__syncthreads();
		int e[NC];
		bool two[NC];
#pragma unroll
		for(int c = 0; c < NC; ++c) {
			e[c] = tq::kDirty;
			two[c] = false;
			if(T.guess) {
				const unsigned k = t / per;
				const double step = (pre[c][k + 1] - pre[c][k]) / (double)per;
				const double P = pre[c][k] + step * (double)(t - k * per);
				binades(P, fmin(step, 0.0), fmax(step, 0.0), 0.01, e[c], two[c]);
			}
			tile_parts<F::kSigned>(st + c * kStage + tid * (kPer + 1), e[c], two[c], parts[c]);
		}
		__syncthreads();
		// (the warps take turns)
		if(warp == t % kWarps && lane < NC) {
			const SeqRec r = lane == 0 ? parts_join<F::kSigned>(parts[0], e[0], two[0])
			                           : parts_join<F::kSigned>(parts[NC - 1], e[NC - 1], two[NC - 1]);
			T.tiles[(size_t)lane * T.ntiles + t] = r;
			sum += r.s;
		}
	}
	if(lane < NC) tot[lane][warp] = sum;
	__syncthreads();
	if(tid < NC) {
		double s = 0.0;
		for(unsigned w = 0; w < kWarps; ++w) s += tot[tid][w];
		T.chunk[tid * T.nchunks + blockIdx.x] = s;
	}
}

// ---- walk -------------------------------------------------------------------
// Applies the records of lanes [l, cnt) (r, one per lane, `terms` terms each)
// to the exact running sum C while they provably apply; returns the first that
// does not (or that the draw falls into), or cnt.  One warp.
template <bool SIGNED, bool STOP>
__device__ unsigned walk_records(const SeqRec &r, unsigned l, unsigned cnt, double terms, double rnd, double &C) {
	const unsigned lane = threadIdx.x & 31u;
	const bool id = r.e == tq::kIdentity;
	const double mag = fabs(C);
	const bool normal = mag >= kTiny && mag <= kHuge;
	const int e = normal ? tq::binade(mag) : 0;
	tq::Inc v = tq::inc_identity();
	bool has = id;
	if(!id && normal && r.e == e && (r.ok & kHasE)) {
		v = tq::Inc{r.i0[0], r.i1[0]};
		has = true;
	} else if(!id && normal && r.e + 1 == e && (r.ok & kHasE1)) {
		v = tq::Inc{r.i0[1], r.i1[1]};
		has = true;
	}
	bool bad = !has;
	double Cl = C;
	if(normal) {
		const double inv = tq::pow2(e - 52);
		const long long c0 = (long long)(C * tq::grid_scale(e));  // exact: C is in binade e
		v = warp_scan_inc(lane >= l && lane < cnt ? v : tq::inc_identity());
		const long long cl = c0 + tq::apply(v, c0);
		Cl = (double)cl * inv;
		long long cs = __shfl_up_sync(FULL, cl, 1);
		if(lane <= l) cs = c0;
		if(!id && !SIGNED) bad = bad || cl >= (1ll << 53);
		if(!id && SIGNED && C > 0.0 && (r.ok & kUp)) {
			bad = bad || cl >= (1ll << 53);
		} else if(!id && SIGNED && C < 0.0 && (r.ok & kDown)) {
			bad = bad || cl <= -(1ll << 53);
		} else if(!id && SIGNED) {
			// Every prefix inside the binade, rounding drift included.
			const double lo = (double)cs * inv + r.mn - 2.0 * terms * inv, hi = (double)cs * inv + r.mx + 2.0 * terms * inv;
			const double b0 = tq::pow2(e), b1 = 2.0 * b0;
			bad = bad || !(C > 0.0 ? (lo > b0 && hi < b1) : (hi < -b0 && lo > -b1));
		}
	}
	const bool hit = STOP && rnd <= Cl;
	const unsigned stop = __ballot_sync(FULL, lane >= l && lane < cnt && (bad || hit));
	const unsigned f = stop ? (unsigned)__ffs(stop) - 1u : cnt;
	const double Cf = __shfl_sync(FULL, Cl, f ? f - 1u : 0u);
	if(f > l) C = Cf;
	return f;
}

struct ReplayShared {
	double C;
	unsigned pos, event, step, forgiven;
	unsigned done;
	unsigned long long answer;
	tq::Inc w[kWarps];
	unsigned tile;
};

// Adds staged terms from i on to c one by one, one warp (the same c in every
// lane), and returns the place after the last: `end`, where `most` of them and
// more are added, or where c reaches the draw (hit).  Zeros change no sum and are
// passed over.  Some 11 cycles a term (one thread with its loads in between 27:
// signed sums that hover around zero, 2% of 2^21 amplitudes not zero: 29.9 ms,
// now 8.3).
template <bool STOP>
__device__ __forceinline__ unsigned add_terms(const double *st, unsigned i, unsigned end, int most, double rnd, double &c, bool &hit) {
	const unsigned lane = threadIdx.x & 31u;
	double next = i + lane < end ? st[stage_slot(i + lane)] : 0.0;
	while(i < end && most > 0) {
		const double v = next, c0 = c;
		const unsigned n = min(32u, end - i);
		next = i + 32u + lane < end ? st[stage_slot(i + 32u + lane)] : 0.0;
		const unsigned some = __ballot_sync(FULL, !(v == 0.0));
		if(__popc(some) > 8) {
#pragma unroll 8
			for(unsigned k = 0; k < 32; ++k) c = radd(c, __shfl_sync(FULL, v, k));
		} else {
#pragma unroll 1
			for(unsigned m = some; m; m &= m - 1u) c = radd(c, __shfl_sync(FULL, v, __ffs(m) - 1));
		}
		if(STOP && !(c < rnd)) {  // one of these reaches it, or c is NaN
			c = c0;
#pragma unroll 1
			for(unsigned k = 0; k < n; ++k) {
				c = radd(c, __shfl_sync(FULL, v, k));
				if(rnd <= c) {
					hit = true;
					return i + k + 1u;
				}
			}
		}
		most -= __popc(some);
		i += n;
	}
	return min(i, end);
}

// Adds terms [base, base + cnt) to S.C exactly, the whole block.  Each thread
// has 16 consecutive terms on the grid of the sum's binade; a scan of their
// parity-indexed increments gives every thread its exact start, from which it
// adds its terms as doubles.  The first thread whose sum leaves the binade (or
// reaches the draw) ends the step: it is exact to the end of its run, and the
// next step starts there.  Sums that keep leaving it, and sums outside the normal
// range (zero at the start, infinities), are added one term at a time.
template <class F, bool STOP>
__device__ void replay_tile(const F &term, unsigned sum, uint64_t base, unsigned cnt, double rnd, double *st, ReplayShared &S) {
	constexpr bool SIGNED = F::kSigned;
	const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	// All 16 loads of a thread before the first use: one at a time, each waiting
	// for HBM, they were half of the walk (n = 26: 9 us a tile, now 2).
	typename F::Raw raw[kPer];
#pragma unroll
	for(unsigned q = 0; q < kPer; ++q) raw[q] = term.load(base + min(q * kThreads + tid, cnt - 1u));
#pragma unroll
	for(unsigned q = 0; q < kPer; ++q) {
		const unsigned i = q * kThreads + tid;
		double v[F::kSums];
		term.terms(raw[q], v);
		const double x = F::kSums == 2 && sum == 1 ? v[F::kSums - 1] : v[0];
		st[stage_slot(i)] = i < cnt ? x : 0.0;
	}
	if(tid == 0) {
		S.pos = 0;
		S.step = kTile;
		S.forgiven = 0;
	}
	__syncthreads();
	const double *p = st + tid * (kPer + 1);
	const unsigned i0 = tid * kPer;
	for(;;) {
		const double C = S.C;
		const unsigned pos = S.pos, step = S.step;
		if(pos >= cnt || S.done || C != C) break;
		__syncthreads();
		if(tid == 0) S.event = cnt;
		__syncthreads();
		const double mag = fabs(C);
		const bool normal = mag >= kTiny && mag <= kHuge;
		// (a step takes 1 us, 256 single additions 2)
		if(!normal || step < (SIGNED ? 512u : 48u)) {
			unsigned first = pos;
			if(C == 0.0 && !(STOP && rnd <= 0.0)) {
				// Zeros leave a zero sum as it is: to the first other term.
				first = cnt;
				for(unsigned k = kPer; k-- > 0;) {
					const unsigned i = i0 + k;
					if(i >= pos && i < cnt && !(p[k] == 0.0)) first = i;
				}
				if(first < cnt) atomicMin(&S.event, first);
				__syncthreads();
				first = S.event;
			}
			if(warp == 0) {
				double c = C;
				bool hit = false;
				// A sum that starts leaves zero with its first terms; one whose terms are
				// too large for its binade has nothing to gain from another step.
				const unsigned end = step == 0u ? cnt : min(cnt, first + (SIGNED || C != 0.0 ? 256u : 32u));
				const unsigned to = add_terms<STOP>(st, first, end, 256, rnd, c, hit);
				if(lane == 0) {
					if(hit) {
						S.done = 1;
						S.answer = base + to - 1;
					}
					S.C = c;
					S.pos = to;
					S.step = kTile;
				}
			}
			__syncthreads();
			continue;
		}
		const int e = tq::binade(mag);
		const double scale = tq::grid_scale(e), inv = tq::pow2(e - 52);
		const long long c0 = (long long)(C * scale);
		const unsigned k0 = pos > i0 ? min(pos - i0, kPer) : 0u, k1 = cnt > i0 ? min(cnt - i0, kPer) : 0u;
		double x[kPer];
		const double start = SIGNED ? 1.5 * kBinade : kBinade;
		double a0 = start, a1 = start + 1.0;
		bool wide = false;
#pragma unroll
		for(unsigned k = 0; k < kPer; ++k) {
			x[k] = k >= k0 && k < k1 ? p[k] * scale : 0.0;
			a0 += x[k];
			a1 += x[k];
			// (64 terms' worth of it keep a signed run inside the binade)
			if(SIGNED) wide = wide || !(fabs(x[k]) < kBinade / 64.0);
		}
		if(SIGNED && __syncthreads_or(wide)) {
			if(tid == 0) S.step = 0;  // one term at a time from here
			__syncthreads();
			continue;
		}
		tq::Inc v = warp_scan_inc(tq::Inc{(long long)(a0 - start), (long long)(a1 - (start + 1.0))});
		if(lane == 31) S.w[warp] = v;
		tq::Inc ex = shfl_up_inc(v, 1);
		if(lane == 0) ex = tq::inc_identity();
		__syncthreads();
		tq::Inc before = tq::inc_identity();
#pragma unroll
		for(unsigned w = 0; w + 1 < kWarps; ++w)
			if(w < warp) before = tq::compose(before, S.w[w]);
		ex = tq::compose(before, ex);
		double c = (double)(c0 + tq::apply(ex, c0)), chit = 0.0;
		bool left = false;
		unsigned hit = kPer;
#pragma unroll
		for(unsigned k = 0; k < kPer; ++k) {
			c += x[k];
			left = left || !(SIGNED ? fabs(c) > kBinade && fabs(c) < 2.0 * kBinade : c < 2.0 * kBinade);
			if(STOP && hit == kPer && k >= k0 && k < k1 && rnd <= c * inv) {
				hit = k;
				chit = c * inv;
			}
		}
		const bool mine = k0 < k1 && (left || (STOP && hit < kPer));
		if(mine) atomicMin(&S.event, i0);
		__syncthreads();
		const unsigned at = S.event;
		if(at == cnt) {
			if(tid == kThreads - 1) {
				S.C = c * inv;
				S.pos = cnt;
			}
		} else if(mine && at == i0) {
			const unsigned to = i0 + k1;
			S.C = c * inv;
			S.pos = to;
			// (A tile's first short step is often a sum that was about to leave anyway:
			// 256 single additions after it were half of a signed walk, n = 26.)
			S.step = S.forgiven ? to - pos : kTile;
			S.forgiven = 1;
			if(STOP && hit < kPer) {
				S.C = chit;
				S.done = 1;
				S.answer = base + i0 + hit;
			}
		}
		__syncthreads();
	}
}

// The walk of one sum (see the top of the file), the whole block; warp 0 steps
// over the records, replays take every thread.
template <class F, bool STOP>
__device__ void walk_block(const F &term, unsigned sum, uint64_t N, const SeqTables &T, bool direct, double rnd, double *st,
                           ReplayShared &S, WalkOut *out) {
	const unsigned tid = threadIdx.x, lane = tid & 31u;
	const SeqRec *tiles = T.tiles + (size_t)sum * T.ntiles, *groups = T.groups + (size_t)sum * T.ngroups;
	if(tid == 0) {
		S.C = 0.0;
		S.done = 0;
		S.answer = N;
	}
	__syncthreads();
	// Position of warp 0: record gl of the `ready` groups from g on whose records
	// are in gr, and within that group (in_group) record t of tr.  A group that
	// is not written within the limit is replayed tile by tile.
	unsigned g = 0, gl = 0, ready = 0, t = 0;
	bool in_group = false, blind = false;
	SeqRec gr = identity_rec(), tr = identity_rec();
	for(;;) {
		if(tid < 32) {
			unsigned tile = T.ntiles;
			double C = S.C;
			if(S.done || C != C) {  // (no term changes a NaN, and no draw reaches it)
			} else if(direct) {
				tile = t++;
			} else {
				for(;;) {
					if(in_group) {
						const unsigned t0 = (g + gl) * kGroup, cnt = min(kGroup, T.ntiles - t0);
						const unsigned f = blind ? t : walk_records<F::kSigned, STOP>(tr, t, cnt, (double)kTile, rnd, C);
						if(f < cnt) {
							tile = t0 + f;
							t = f + 1;
							break;
						}
						in_group = blind = false;
						++gl;
					}
					if(gl >= ready) {
						g += gl;
						gl = 0;
						if(g >= T.ngroups) break;
						ready = 0;
						for(unsigned spin = 0; ready == 0 && spin < kSpinLimit; ++spin) {
							unsigned f = 0;
							if(g + lane < T.ngroups)
								asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(T.gready + g + lane) : "memory");
							const unsigned m = __ballot_sync(FULL, f == 1u);
							ready = m == FULL ? 32u : (unsigned)__ffs(~m) - 1u;
							if(ready == 0) __nanosleep(100);
						}
						blind = ready == 0;
						if(blind) {
							ready = 1;
							in_group = true;
							t = 0;
							continue;
						}
						gr = lane < ready ? load_rec(groups + g + lane) : identity_rec();
					}
					gl = walk_records<F::kSigned, STOP>(gr, gl, ready, (double)kTile * kGroup, rnd, C);
					if(gl < ready) {
						const unsigned t0 = (g + gl) * kGroup;
						tr = t0 + lane < T.ntiles ? load_rec(tiles + t0 + lane) : identity_rec();
						in_group = true;
						t = 0;
					}
				}
			}
			__syncwarp();
			if(tid == 0) {
				S.C = C;
				S.tile = tile;
			}
		}
		__syncthreads();
		const unsigned tile = S.tile;
		if(tile >= T.ntiles) break;
		const uint64_t base = (uint64_t)tile * kTile;
		replay_tile<F, STOP>(term, sum, base, (unsigned)min((unsigned long long)kTile, (unsigned long long)(N - base)), rnd, st, S);
		__syncthreads();
	}
	if(tid == 0) out[sum] = WalkOut{S.answer, S.C};
}

// A worker block: chunk b of the tiles, in order, with the approximate prefix
// from the sums of the chunks before it.
template <class F>
__device__ void join_chunk(const F &term, const SeqTables &T, unsigned b, double *st, WarpPart (*parts)[kWarps], double (*sh)[kWarps]) {
	constexpr int NC = F::kSums;
	const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	double P[NC];
	for(int c = 0; c < NC; ++c) {
		double s = 0.0;
		for(unsigned k = tid; k < b; k += kThreads) s += T.chunk[c * T.nchunks + k];
		s = warp_sum(s);
		if(lane == 0) sh[c][warp] = s;
	}
	__syncthreads();
#pragma unroll
	for(int c = 0; c < NC; ++c) {
		P[c] = 0.0;
		for(unsigned w = 0; w < kWarps; ++w) P[c] += sh[c][w];
	}
	const unsigned t0 = chunk_begin(T, b), t1 = chunk_begin(T, b + 1);
	typename F::Raw raw[kPer];
	unsigned loaded = T.ntiles;  // the tile in raw
	for(unsigned f = t0; f < t1;) {
		const unsigned g = f / kGroup, cnt = min((g + 1) * kGroup, t1) - f;  // the chunk's tiles in group g
		// Which binades each of them needs: one lane per tile, the same in every warp.
		int e[NC];
		bool two[NC];
		bool again = false;
#pragma unroll
		for(int c = 0; c < NC; ++c) {
			SeqRec r = identity_rec();
			if(lane < cnt) r = load_rec(T.tiles + (size_t)c * T.ntiles + f + lane);
			double incl = r.s;
			for(unsigned d = 1; d < 32; d <<= 1) {
				const double o = __shfl_up_sync(FULL, incl, d);
				if(lane >= d) incl += o;
			}
			const bool can = binades(P[c] + (incl - r.s), r.mn, r.mx, T.rel, e[c], two[c]);
			if(r.e != tq::kIdentity && can) {
				const bool has = (r.e == e[c] && (r.ok & kHasE) && (!two[c] || (r.ok & kHasE1))) || (r.e + 1 == e[c] && (r.ok & kHasE1) && !two[c]);
				again = again || !has;
			} else {
				e[c] = tq::kDirty;
				two[c] = false;
			}
			P[c] += __shfl_sync(FULL, incl, 31);
		}
		unsigned todo = __ballot_sync(FULL, again);
		while(todo) {
			const unsigned i = __ffs(todo) - 1u;
			todo &= todo - 1u;
			const unsigned t = f + i;
			if(loaded != t) load_tile(term, t, raw);
			stage_tile(term, raw, st);
			if(todo || f + cnt < t1) {
				// The next one in need (without a guess so far, the next group's first).
				loaded = todo ? f + __ffs(todo) - 1u : f + cnt;
				load_tile(term, loaded, raw);
			}
			__syncthreads();
			int ei[NC];
			bool twoi[NC];
#pragma unroll
			for(int c = 0; c < NC; ++c) {
				ei[c] = __shfl_sync(FULL, e[c], i);
				twoi[c] = __shfl_sync(FULL, (int)two[c], i) != 0;
				tile_parts<F::kSigned>(st + c * kStage + tid * (kPer + 1), ei[c], twoi[c], parts[c]);
			}
			__syncthreads();
			if(tid < NC) {
				T.tiles[(size_t)tid * T.ntiles + t] = tid == 0 ? parts_join<F::kSigned>(parts[0], ei[0], twoi[0])
				                                               : parts_join<F::kSigned>(parts[NC - 1], ei[NC - 1], twoi[NC - 1]);
			}
		}
		// The last block to finish tiles of the group composes it.
		if(warp == 0) {
			__threadfence();
			__syncwarp();
			unsigned n = 0;
			if(lane == 0) n = atomicAdd(T.gcount + g, cnt) + cnt;
			if(__shfl_sync(FULL, n, 0) == min(kGroup, T.ntiles - g * kGroup)) {
				__threadfence();
#pragma unroll
				for(int c = 0; c < NC; ++c) {
					SeqRec r = identity_rec();
					if(g * kGroup + lane < T.ntiles) r = load_rec(T.tiles + (size_t)c * T.ntiles + g * kGroup + lane);
					const SeqRec gr = compose_group<F::kSigned>(r);
					if(lane == 0) T.groups[(size_t)c * T.ngroups + g] = gr;
				}
				if(lane == 0) {
					__threadfence();
					asm volatile("st.release.gpu.global.u32 [%0], 1;" ::"l"(T.gready + g) : "memory");
				}
			}
		}
		f += cnt;
	}
}

template <class F, bool STOP>
__global__ void __launch_bounds__(kThreads, 2) k_seq_join(F term, uint64_t N, SeqTables T, bool direct, double rnd, WalkOut *out) {
	extern __shared__ double st[];  // staged terms, kStage per sum
	__shared__ WarpPart parts[F::kSums][kWarps];
	__shared__ double sh[F::kSums][kWarps];
	__shared__ ReplayShared S;
	if(blockIdx.x < F::kSums) walk_block<F, STOP>(term, blockIdx.x, N, T, direct, rnd, st, S, out);
	else join_chunk(term, T, blockIdx.x - F::kSums, st, parts, sh);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Byte layout of the scratch for `sums` sums of N terms.
struct ScratchLayout {
	uint64_t tiles, groups;
	size_t tile_rec, group_rec, est, chunk, count, ready, out, total;
};
constexpr unsigned kMaxChunks = 1024;
ScratchLayout scratch_layout(uint64_t N, unsigned sums) {
	ScratchLayout l{};
	l.tiles = (N + kTile - 1) / kTile;
	l.groups = (l.tiles + kGroup - 1) / kGroup;
	l.group_rec = align256(sums * l.tiles * sizeof(SeqRec));
	l.est = l.group_rec + align256(sums * l.groups * sizeof(SeqRec));
	l.chunk = l.est + align256(sums * kStrata * sizeof(double));
	l.count = l.chunk + align256(sums * kMaxChunks * sizeof(double));
	l.ready = l.count + align256(l.groups * sizeof(unsigned));
	l.out = l.ready + align256(l.groups * sizeof(unsigned));
	l.total = l.out + align256(kMaxSums * sizeof(WalkOut));
	return l;
}

// Runs the engine in `base` (scratch_layout bytes); host_out receives one
// WalkOut per sum.  Synchronises.
template <class F>
void run_engine(const F &term, uint64_t N, bool stop, double rnd, unsigned char *base, WalkOut *host_out, cudaStream_t stream,
                int num_sms, uint64_t *launches) {
	constexpr unsigned NC = F::kSums;
	const ScratchLayout l = scratch_layout(N, NC);
	if(l.tiles > 0xfffffff0ull) fail(TMFQS_ERR_INVALID_ARGUMENT, "exact reduction: state too large");
	SeqTables T{};
	T.ntiles = (unsigned)l.tiles;
	T.ngroups = (unsigned)l.groups;
	T.tiles = reinterpret_cast<SeqRec *>(base + l.tile_rec);
	T.groups = reinterpret_cast<SeqRec *>(base + l.group_rec);
	T.est = reinterpret_cast<double *>(base + l.est);
	T.chunk = reinterpret_cast<double *>(base + l.chunk);
	T.gcount = reinterpret_cast<unsigned *>(base + l.count);
	T.gready = reinterpret_cast<unsigned *>(base + l.ready);
	T.guess = N >= kGuessTerms;
	T.rel = (double)N * 2.3e-16 + 1e-9;
	auto *wo = reinterpret_cast<WalkOut *>(base + l.out);
	const bool direct = l.tiles <= kDirectTiles;
	const size_t smem = NC * kStage * sizeof(double);
	unsigned count = 1;
	// Blocks per SM of a kernel with that much dynamic shared memory.
	auto resident = [&](auto kern) {
		int per_sm = 1;
		check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "reduction smem");
		check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem), "reduction occupancy");
		return (unsigned)num_sms * (unsigned)std::max(1, per_sm);
	};
	auto launch = [&](auto join) {
		const unsigned fit = resident(join);
		if(!direct) {  // N is a power of two: whole tiles
			// Both kernels' blocks take the same chunks; the walk blocks run beside the join's.
			T.nchunks = std::min<unsigned>({T.ntiles, resident(k_seq_tiles<F>), fit > NC ? fit - NC : 1u, kMaxChunks});
			if(T.guess) k_seq_guess<F><<<kStrata, kThreads, 0, stream>>>(term, N, T.est);
			k_seq_tiles<F><<<T.nchunks, kThreads, smem, stream>>>(term, T);
			count += T.guess ? 2 : 1;
		}
		join<<<NC + T.nchunks, kThreads, smem, stream>>>(term, N, T, direct, rnd, wo);
	};
	if constexpr(!F::kSigned) {
		if(stop) launch(k_seq_join<F, true>);
		else launch(k_seq_join<F, false>);
	} else {
		launch(k_seq_join<F, false>);
	}
	check_cuda(cudaGetLastError(), "exact reduction");
	if(launches) *launches += count;
	check_cuda(cudaMemcpyAsync(host_out, wo, NC * sizeof(WalkOut), cudaMemcpyDeviceToHost, stream), "reduction readback");
	check_cuda(cudaStreamSynchronize(stream), "reduction sync");
}

template <typename R, int KIND>
TermF<R, KIND> make_term(const void *amps, const Overlay &ov) {
	return TermF<R, KIND>{static_cast<const typename Vec2<R>::type *>(amps), ov.active ? 1 : 0, ov.sre, ov.sim, ov.bre, ov.bim};
}

void ensure_scratch(SeqScratch &s, uint64_t N) {
	const size_t total = scratch_layout(N, kMaxSums).total;
	if(s.base && s.bytes == total) return;
	seq_scratch_free(s);
	void *base = nullptr;
	if(device_alloc(&base, total) != cudaSuccess) {
		cudaGetLastError();
		fail(TMFQS_ERR_NOMEM, "exact reduction scratch: device allocation of " + std::to_string(total) + " bytes failed");
	}
	void *host = nullptr;
	if(cudaMallocHost(&host, kMaxSums * sizeof(WalkOut)) != cudaSuccess) {
		cudaGetLastError();
		cudaFree(base);
		fail(TMFQS_ERR_NOMEM, "exact reduction scratch: pinned allocation failed");
	}
	s.base = base;
	s.bytes = total;
	s.host_out = host;
}

// ---------------------------------------------------------------------------
// Fixed device scratch for the allocation-free measurement entry point.
//
// Some callers cannot let this library call cudaMalloc: a host application
// whose caching allocator has already reserved nearly all device memory for
// itself (so a fresh allocation fails or fragments its pool), or a loop that
// must not pay the device-wide synchronisation cudaMalloc/cudaFree imply.
// For them tmfqs_sample_static runs the exact measurement replay with its
// per-tile tables in this fixed array, which every GPU that loads the library
// holds until the process exits.  Every region of it is fully written before
// it is read on each call, so no clearing is needed; calls that overlap on
// the GPU share the array and race.
// ---------------------------------------------------------------------------
constexpr unsigned kStaticMaxQubits = 24;
constexpr size_t kStaticScratchBytes = size_t(2) << 20;  // 2 MiB
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

std::mutex g_static_mutex;
void *g_static_addr[64] = {nullptr};  // device address of g_static_scratch, per device ordinal

// Host code cannot use &g_static_scratch as a device address; the runtime
// gives the real address for the current device.  It is looked up again on
// every call made outside stream capture: a context reset (cudaDeviceReset)
// reloads the module, and the array may then sit at another address.  While
// `stream` is capturing, the address of the last call outside capture on this
// device is used (no lookup, which could load the module inside a capture);
// a capturing call on a device that never had one fails.
void *static_scratch_address(cudaStream_t stream) {
	int dev = 0;
	check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
	if(dev < 0 || dev >= 64) fail(TMFQS_ERR_INVALID_ARGUMENT, "device ordinal out of range for the static scratch");
	cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
	check_cuda(cudaStreamIsCapturing(stream, &cap), "cudaStreamIsCapturing");
	std::lock_guard<std::mutex> lock(g_static_mutex);
	if(cap == cudaStreamCaptureStatusNone) {
		void *p = nullptr;
		check_cuda(cudaGetSymbolAddress(&p, g_static_scratch), "cudaGetSymbolAddress(static scratch)");
		g_static_addr[dev] = p;
	} else if(!g_static_addr[dev]) {
		fail(TMFQS_ERR_LOGIC, "tmfqs_sample_static: the first call on a device must come before any stream capture");
	}
	return g_static_addr[dev];
}

}  // namespace

SeqResult seq_sample_static(int precision, const void *amps, unsigned num_qubits, double rnd, cudaStream_t stream) {
	if(num_qubits > kStaticMaxQubits)
		fail(TMFQS_ERR_INVALID_ARGUMENT, "tmfqs_sample_static: at most " + std::to_string(kStaticMaxQubits) +
		                                     " qubits (its fixed " + std::to_string(kStaticScratchBytes >> 20) +
		                                     " MiB device scratch); use tmfqs_gpu_sample for larger states");
	const uint64_t N = 1ull << num_qubits;
	if(scratch_layout(N, 1).total > kStaticScratchBytes)
		fail(TMFQS_ERR_INVALID_ARGUMENT, "state too large for the static scratch");
	int dev = 0, sms = 0;
	check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
	check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
	WalkOut host[kMaxSums] = {};  // pageable: the readback copy is synchronous
	auto *base = static_cast<unsigned char *>(static_scratch_address(stream));
	if(precision == TMFQS_FP64) run_engine(make_term<double, kTermProb>(amps, Overlay{}), N, true, rnd, base, host, stream, sms, nullptr);
	else run_engine(make_term<float, kTermProb>(amps, Overlay{}), N, true, rnd, base, host, stream, sms, nullptr);
	return SeqResult{host[0].index, host[0].value};
}

void seq_scratch_free(SeqScratch &s) {
	if(s.base) cudaFree(s.base);
	if(s.host_out) cudaFreeHost(s.host_out);
	s = SeqScratch{};
}

double seq_diff_norm(int prec_ref, const void *ref, int prec_got, const void *got, uint64_t N, SeqScratch &scratch,
                     cudaStream_t stream, int num_sms, uint64_t *launches) {
	ensure_scratch(scratch, N);
	auto *out = static_cast<WalkOut *>(scratch.host_out);
	auto run = [&](auto term) {
		run_engine(term, N, false, 0.0, static_cast<unsigned char *>(scratch.base), out, stream, num_sms, launches);
		return out[0].value;
	};
	if(prec_ref == TMFQS_FP64 && prec_got == TMFQS_FP64)
		return run(TermDiff<double, double>{static_cast<const double2 *>(ref), static_cast<const double2 *>(got)});
	if(prec_ref == TMFQS_FP64)
		return run(TermDiff<double, float>{static_cast<const double2 *>(ref), static_cast<const float2 *>(got)});
	if(prec_got == TMFQS_FP64)
		return run(TermDiff<float, double>{static_cast<const float2 *>(ref), static_cast<const double2 *>(got)});
	return run(TermDiff<float, float>{static_cast<const float2 *>(ref), static_cast<const float2 *>(got)});
}

SeqResult seq_replay(int precision, const void *amps, uint64_t N, const Overlay &ov, bool stop, double rnd, SeqScratch &scratch,
                     cudaStream_t stream, int num_sms, uint64_t *launches) {
	ensure_scratch(scratch, N);
	auto *base = static_cast<unsigned char *>(scratch.base);
	auto *out = static_cast<WalkOut *>(scratch.host_out);
	if(precision == TMFQS_FP64) run_engine(make_term<double, kTermProb>(amps, ov), N, stop, rnd, base, out, stream, num_sms, launches);
	else run_engine(make_term<float, kTermProb>(amps, ov), N, stop, rnd, base, out, stream, num_sms, launches);
	return SeqResult{out[0].index, out[0].value};
}

void seq_amplitude_sum(int precision, const void *amps, uint64_t N, const Overlay &ov, double &re, double &im,
                       SeqScratch &scratch, cudaStream_t stream, int num_sms, uint64_t *launches) {
	ensure_scratch(scratch, N);
	auto *base = static_cast<unsigned char *>(scratch.base);
	auto *out = static_cast<WalkOut *>(scratch.host_out);
	if(precision == TMFQS_FP64) run_engine(make_term<double, kTermAmp>(amps, ov), N, false, 0.0, base, out, stream, num_sms, launches);
	else run_engine(make_term<float, kTermAmp>(amps, ov), N, false, 0.0, base, out, stream, num_sms, launches);
	re = out[0].value;
	im = out[1].value;
}

}  // namespace tqb
