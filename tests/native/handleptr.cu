// The device array of a handle's particle tags, for a test that damages one.
#include "gkm_handle.h"

extern "C" void* hp_tags(void* handle) { return static_cast<gkm_handle*>(handle)->tag; }
