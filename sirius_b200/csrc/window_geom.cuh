// Geometry of shifted-window attention, shared by the window kernels.
//
// Tokens live in the natural [B][Hs][Ws] order. A window of WS x WS tokens of the cyclically shifted map is
// window (wy, wx), token (iy, ix): shifted position (wy*WS+iy, wx*WS+ix), natural position that plus `shift`
// modulo the map size.
#pragma once
#include <stdint.h>

namespace srt {

struct WinGeom {
  int B, Hs, Ws, WS, shift, nWy, nWx;
};
__device__ inline int64_t win_token_to_natural(const WinGeom& g, int64_t win, int tok) {
  const int wx = (int)(win % g.nWx);
  const int wy = (int)((win / g.nWx) % g.nWy);
  const int64_t b = win / ((int64_t)g.nWx * g.nWy);
  const int iy = tok / g.WS, ix = tok - iy * g.WS;
  int h = wy * g.WS + iy + g.shift, w = wx * g.WS + ix + g.shift;
  if (h >= g.Hs) h -= g.Hs;
  if (w >= g.Ws) w -= g.Ws;
  return (b * g.Hs + h) * g.Ws + w;
}
__device__ inline int shift_region(int p, int size, int WS, int shift) {  // region of a shifted coordinate
  return p < size - WS ? 0 : (p < size - shift ? 1 : 2);
}

}  // namespace srt
