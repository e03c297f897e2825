// host stand-in for <cuda.h> (see cuda_runtime.h beside it)
#pragma once
struct CUtensorMap { unsigned long long opaque[16]; };
