// Instance of the persistent decode kernel for one GPU and long contexts: CTAs share query heads.
#include "kernel_table.h"
#include "mega_kernel.cuh"

const void* mg::mega_kernel_shared() { return (const void*)mg::mega_decode_kernel<false, true>; }
