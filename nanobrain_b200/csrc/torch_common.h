// Shared by the binding's sources.
#pragma once

#include <torch/extension.h>

#include "../../include/nb_attn.h"

namespace nbt {

// The device's status word (one pinned int32 that kernels write to when something went wrong).
volatile int32_t* status_ptr(int64_t device);
// Raises what a finished kernel reported. Never synchronises.
void raise_for_status(volatile int32_t* word);
// NB_ATTN_DEBUG=1: synchronise and look at the status word after every call.
void after_launch(volatile int32_t* word);
void check_rc(int rc, const char* what);

void bind_encoder(pybind11::module_& m);

}  // namespace nbt
