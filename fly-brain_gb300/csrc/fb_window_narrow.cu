// The windowed kernel (fb_window.cu) with the block width for one brain.
#include "fb_window.cuh"
#define FB_WINDOW_WIDTH kWinNarrow
#define FB_WINDOW_NAME narrow
#define FB_WINDOW_IS_NARROW
#include "fb_window.cu"
