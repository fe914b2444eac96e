// Run kernel of sparse single graphs: contraction (contract_device.cuh)
// between the trim and the searches.  In its own translation unit, so that
// the default run kernels keep their code.
#include "run_kernel.cuh"
#include "contract_device.cuh"

namespace gb {
namespace {

struct ContractExtra {
  static constexpr bool kOn = true;
  static __device__ __forceinline__ void run(const Args& A, Smem& sm) { contract_phase(A, sm); }
};

}  // namespace

cudaError_t launch_run_contract(const GraphView& g, const RunParams& p, const Work& w, int grid,
                                cudaStream_t stream) {
  Args a{};
  a.g = g;
  a.p = p;
  a.w = w;
  a.kind = kSCC;
  return coop(k_run<1, false, ContractExtra>, grid, a, stream);
}

int run_contract_blocks_per_sm() { return run_blocks_per_sm(k_run<1, false, ContractExtra>); }

}  // namespace gb
