// engine_eyuk.cu -- fused step kernels of the resident engine for pair evaluator
// ExpandedYukawa (one translation unit per evaluator so the instantiations compile in parallel).
#include "engine_kernels.cuh"

namespace azp
{
int launch_md_eyuk(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s)
{
    return launch_md_pe<ExpandedYukawa>(bond_kind, precision, integ, a, s);
}

int launch_run_eyuk(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s)
{
    return launch_run_pe<ExpandedYukawa>(bond_kind, precision, integ, r, s);
}
}  // namespace azp
