// toed_detect_inst.cuh -- one translation unit per kernel radius keeps the
// heavily unrolled instantiations compiling in parallel.
#pragma once
#include "toed_detect.cuh"
#include "toed_internal.h"

#define TOED_DETECT_INSTANCE(R)                                                    \
    namespace toed {                                                               \
    DetectEntry detect_entry_r##R(bool nmsto)                                      \
    {                                                                              \
        if (nmsto) return {(const void*)toed_detect_kernel<R, true>, Cfg<R, true>::smem}; \
        return {(const void*)toed_detect_kernel<R>, Cfg<R>::smem};                 \
    }                                                                              \
    }
