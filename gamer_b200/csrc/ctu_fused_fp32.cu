// Instantiations of the plane-streaming hydro CTU kernel for the P_FP32 policy.
#include "ctu_fused.cuh"
namespace gb {
int ctu_fused_fp32( const gb_fluid_config &cfg, const void *in, void *out, void *flux, int npg, const gb_fluid_params *prm,
                  int *status, cudaStream_t st )
{
   return hctu_fused_pick<float,P_FP32>( cfg, in, out, flux, npg, prm, status, st );
}
} // namespace gb
