// Path-replay adjoint instantiations of the wave kernels (the backward pass
// of ymrt_render_backward / ymrt_render_backward_ex), compiled apart from the
// forward kernels so that the library builds in parallel. Surface adjoint
// shading is instantiated on surface_features() (its closest hits are the
// forward k_extend's); with media, one instantiation with every feature
// serves both free flight and shading.
#include "wave_device.cuh"

namespace ym {

void launch_adjoint_extend_media(const WaveArgs& w, const WaveOptions& opt) {
  // free flight with the density-grid terms (one instantiation, all features)
  const auto k = k_extend<true, kFeatAll, true>;
  k<<<w.trace_blocks, w.trace_block, traversal_shared_bytes(w.trace_block), w.stream>>>(w.A, w.ctl, w.H, w.jobs, w.counters,
                                                                           opt.grid_grads, opt.grid_tex, w.ray_order);
}

uint32_t launch_adjoint_shade(bool volumes, uint32_t features, const WaveArgs& w, const WaveOptions& opt) {
  if (volumes) return launch_shade_phases<true, kFeatAll>(w, opt);
  switch (surface_features(features)) {
    case 0: return launch_shade_phases<false, 0>(w, opt);
    case kFeatSpheres: return launch_shade_phases<false, kFeatSpheres>(w, opt);
    case kFeatTextures: return launch_shade_phases<false, kFeatTextures>(w, opt);
    default: return launch_shade_phases<false, kFeatSpheres | kFeatTextures>(w, opt);
  }
}

void prepare_adjoint_kernels() { allow_trace_shared(k_extend<true, kFeatAll, true>); }

cudaError_t upload_slots_adjoint(const DeviceScene* scenes, const uint32_t* slots, uint32_t n,
                                 cudaStream_t stream) {
  return upload_slots_here(scenes, slots, n, stream);
}

cudaError_t read_bound_adjoint(BoundRecord* out, bool clear, cudaStream_t stream) {
  return read_bound_here(out, clear, stream);
}

}  // namespace ym
