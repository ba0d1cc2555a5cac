// tess_clip_f64.cu -- the FP64 clipping: the cells the FP32 passes could not
// settle, and single-cell geometry; kernel source in tess_clip_impl.cuh.
#include "tess_clip_impl.cuh"

namespace tess {

cudaError_t launch_clip_f64(const ClipParams& p, int slots, int wpb, int blocks, cudaStream_t s) {
    using namespace clipk;
    if (p.geo) return launch_t<8, true>(p, wpb, blocks, s);
    if (slots <= 2) return launch_t<2, false>(p, wpb, blocks, s);
    return slots <= 4 ? launch_t<4, false>(p, wpb, blocks, s)
                      : launch_t<8, false>(p, wpb, blocks, s);
}

int clip_blocks_f64(int slots, int wpb, int device) {
    using namespace clipk;
    if (slots <= 2) return blocks_t<2, false>(wpb, device);
    return slots <= 4 ? blocks_t<4, false>(wpb, device) : blocks_t<8, false>(wpb, device);
}

}  // namespace tess
