// align_general.cu -- the general form of the alignment: colour space, and scores the packed form has no room for.
// Widths of -i 3, 5, 7, 15 and 20 with their cells in registers; the others have them in local memory: 3,000
// windows of 101 colours 674 us at -i 10, 535 at -i 15, 292 at -i 7.
#include "align_core.cuh"

namespace sg {

const void* align_general_kernel(int bw, int colour) {
#define SG_ALIGN(BW) \
  case BW: return colour ? (const void*)align_kernel<BW, 1> : (const void*)align_kernel<BW, 0>;
  switch (bw) {
    SG_ALIGN(7)
    SG_ALIGN(11)
    SG_ALIGN(15)
    SG_ALIGN(31)
    SG_ALIGN(41)
  default: return colour ? (const void*)align_kernel<0, 1> : (const void*)align_kernel<0, 0>;
  }
#undef SG_ALIGN
}

}  // namespace sg
