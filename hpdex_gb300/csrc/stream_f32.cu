// stream kernel for float values (see stream_impl.cuh)
#define HPDEX_STREAM_T f32
#define HPDEX_STREAM_V float
#include "stream_impl.cuh"
