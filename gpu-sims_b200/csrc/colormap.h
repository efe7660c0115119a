// The velocity-magnitude colour map (build_colormap_lut of the reference,
// src/main.cpp:529-563): entry i of 256, as bytes.  Evaluated in single precision
// without contraction, at compile time for the raymarch's table.
#pragma once

namespace lbm {

struct ColormapEntry {
  unsigned char rgb[3];
};

constexpr ColormapEntry colormap_entry(int i) {
  const float t = (float)i / 255.0f;
  float c[3] = {};
  if (t < 0.25f) {
    const float f = t / 0.25f;
    c[0] = 0.05f; c[1] = 0.05f + 0.6f * f; c[2] = 0.4f + 0.6f * f;
  } else if (t < 0.5f) {
    const float f = (t - 0.25f) / 0.25f;
    c[0] = 0.05f; c[1] = 0.65f + 0.3f * f; c[2] = 1.0f - 0.7f * f;
  } else if (t < 0.75f) {
    const float f = (t - 0.5f) / 0.25f;
    c[0] = 0.05f + 0.95f * f; c[1] = 0.95f - 0.05f * f; c[2] = 0.3f - 0.25f * f;
  } else {
    const float f = (t - 0.75f) / 0.25f;
    c[0] = 1.0f; c[1] = 0.9f - 0.7f * f; c[2] = 0.05f;
  }
  ColormapEntry e{};
  for (int k = 0; k < 3; ++k) {
    const float v = c[k] < 0.0f ? 0.0f : (c[k] > 1.0f ? 1.0f : c[k]);
    e.rgb[k] = (unsigned char)(v * 255.0f);
  }
  return e;
}

}  // namespace lbm
