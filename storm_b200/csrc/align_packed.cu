// align_packed.cu -- the packed nucleotide form of the alignment at every odd band width up to 41.
#include "align_core.cuh"

namespace sg {

const void* align_packed_kernel(int bw) {
#define SG_ALIGN(BW) case BW: return (const void*)align_kernel<BW, 2>;
  switch (bw) {
    SG_ALIGN(3) SG_ALIGN(5) SG_ALIGN(7) SG_ALIGN(9) SG_ALIGN(11) SG_ALIGN(13) SG_ALIGN(15) SG_ALIGN(17)
    SG_ALIGN(19) SG_ALIGN(21) SG_ALIGN(23) SG_ALIGN(25) SG_ALIGN(27) SG_ALIGN(29) SG_ALIGN(31) SG_ALIGN(33)
    SG_ALIGN(35) SG_ALIGN(37) SG_ALIGN(39) SG_ALIGN(41)
  default: return nullptr;
  }
#undef SG_ALIGN
}

}  // namespace sg
