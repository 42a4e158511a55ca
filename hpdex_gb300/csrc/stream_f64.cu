// stream kernel for double values (see stream_impl.cuh)
#define HPDEX_STREAM_T f64
#define HPDEX_STREAM_V double
#include "stream_impl.cuh"
