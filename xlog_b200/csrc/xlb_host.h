// Page-locked host memory for results (see xlb_host.cu).
#pragma once
#include <cstdint>

void host_pool_context_opened(int device);
void host_pool_context_closed(int device);
void host_pool_ranks(unsigned ranks);  // processes that share the machine
uint64_t host_pool_most();             // bytes that may be registered at a time
unsigned host_pool_cores();            // this process's share of the cores it may run on, and of the time it may have on them
unsigned host_cores_quota(const char* groups, const char* mount);
