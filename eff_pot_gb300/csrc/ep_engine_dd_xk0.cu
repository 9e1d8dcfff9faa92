// ep_engine_dd_xk0.cu - double-float engine: the X-pass kernels of the general
// shared-memory engine (half-lines that ep_xw.cuh has no kernels for).
#define EP_ENGINE_PARTS 16
#include "ep_engine_impl.cuh"
template int Engine<dfloat>::x_launch(int, bool);
template int Engine<dfloat>::x_attrs_general();
