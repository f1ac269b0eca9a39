// Host-side check that the op-by-op fused pass (launch_fused_ops in
// tmfqsfullstate_b200/csrc/fused.cu) refuses the operations its kernel has no
// code for, for tests/test_fused_kinds.py.  No GPU is touched: the program
// buffer's allocation fails here, so an accepted pass ends there.
#include "../tmfqsfullstate_b200/csrc/fused.cu"

#include <cstdio>

namespace tqb {
[[noreturn]] void fail(int code, const std::string &) { throw code; }
void check_cuda(cudaError_t, const char *) {}
void upload_async(const LaunchCtx &, void *, const void *, size_t, const char *) {}
cudaError_t device_alloc(void **, size_t) { return cudaErrorMemoryAllocation; }
}  // namespace tqb

using namespace tqb;

int main() {
	for(uint32_t kind = 0; kind <= kFDense2; ++kind)
		for(int prec : {TMFQS_FP64, TMFQS_FP32}) {
			FusedPass p;
			p.n = 14;
			p.K = prec == TMFQS_FP64 ? 12 : 13;
			for(unsigned i = 0; i < p.K; ++i) p.lpos[i] = i;
			FusedOp op{};
			op.kind = kind;
			op.lt = 1;
			op.lc = kind == kFHChain || kind == kFHTwiddle ? 0 : 2;
			p.ops = {FusedOp{}, op};
			p.mats.assign(32, 0.0);
			void *prog = nullptr;
			size_t bytes = 0;
			int code = 0;
			try {
				launch_fused_ops(LaunchCtx{}, prec, nullptr, p, prog, bytes);
			} catch(int c) {
				code = c;
			}
			std::printf("kind %u prec %d %s\n", kind, prec,
			            code == TMFQS_ERR_LOGIC ? "refused" : code == TMFQS_ERR_NOMEM ? "accepted" : "?");
		}
}
