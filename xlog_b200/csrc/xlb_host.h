// Page-locked host memory for results (see xlb_host.cu).
#pragma once
#include <cstdint>

void host_pool_context_opened(int device);
void host_pool_context_closed(int device);
