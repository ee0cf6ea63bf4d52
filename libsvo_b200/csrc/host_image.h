// host_image.h -- host images that a kernel can write itself.
#pragma once
#include <cstdint>

namespace svo {

// The device-side address of a host image, `pixels` (at least one) long, every byte
// of which is page-locked and mapped (one allocation or registration, or several
// side by side), at a pixel's alignment; else null.
uint32_t* mapped_image(uint32_t* h, uint64_t pixels);

}  // namespace svo
