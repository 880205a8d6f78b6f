// align_unit.cu -- the form of the unit entry points: packed in windows without masked codes, general in the others.
// Widths of -i 3, 5, 7, 10, 15 and 20; the others run the general form in local memory (align_general.cu):
// 3,000 windows of 101 codes 412 us at -i 13, 127 at -i 15.
#include "align_core.cuh"

namespace sg {

const void* align_unit_kernel(int bw) {
#define SG_ALIGN(BW) case BW: return (const void*)align_kernel<BW, 3>;
  switch (bw) {
    SG_ALIGN(7) SG_ALIGN(11) SG_ALIGN(15) SG_ALIGN(21) SG_ALIGN(31) SG_ALIGN(41)
  default: return nullptr;
  }
#undef SG_ALIGN
}

}  // namespace sg
