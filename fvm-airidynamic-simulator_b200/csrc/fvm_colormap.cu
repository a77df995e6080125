// fvm_colormap.cu -- headless counterpart of the renderer's field pass:
// colour tables and the C ABI entry fvm_colormap_to_device.  The reference
// draws the field with an OpenGL fragment shader (src/renderer.cpp:47-77)
// sampling a 256-entry RGB table built on the CPU (src/renderer.cpp:672-799);
// here the same arithmetic runs as a CUDA kernel (k_colormap, fvm_aux.cu)
// into a caller device buffer, one RGBA pixel per cell, with no graphics API.
#include <algorithm>

#include "fvm_colortable.h"
#include "fvm_handle.h"

extern "C" int fvm_colormap_table(int colormap, float *rgb_out) {
    if (!rgb_out) return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_table: null output");
    if (colormap < FVM_CMAP_JET || colormap > FVM_CMAP_VIRIDIS)
        return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_table: unknown colormap");
    const ColormapLUT L = colormap_lut(colormap);
    std::copy(L.rgb, L.rgb + 256 * 3, rgb_out);
    return FVM_OK;
}

extern "C" int fvm_colormap_to_device(fvm_handle *h, int field_kind, int colormap, float min_val, float max_val,
                                      void *dev_rgba, int format) {
    if (!h) return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_to_device: null handle");
    if (!h->Un) return fvm_internal_set_error(FVM_ERR_STATE, "fvm_colormap_to_device: solver not initialized");
    if (!dev_rgba) return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_to_device: null destination");
    if (field_kind < 0 || field_kind > 4)
        return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_to_device: unknown field kind");
    if (colormap < FVM_CMAP_JET || colormap > FVM_CMAP_VIRIDIS)
        return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_to_device: unknown colormap");
    if (format != FVM_RGBA_F32 && format != FVM_RGBA_U8)
        return fvm_internal_set_error(FVM_ERR_INVALID, "fvm_colormap_to_device: unknown pixel format");
    cudaError_t e =
        launch_colormap(field_kind, h->g, h->Un, h->mask, colormap, min_val, max_val, dev_rgba, format, h->stream);
    if (e != cudaSuccess) return fvm_internal_set_error(FVM_ERR_CUDA, cudaGetErrorString(e));
    h->launches++;
    return FVM_OK;
}
