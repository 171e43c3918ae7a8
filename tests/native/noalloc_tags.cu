// g4s_run_noalloc with a way to set the tag word of its scratch, which otherwise takes 2^32 steps
// to come near its end.  Linked with the library's other objects.
#include "g4s_noalloc.cu"

extern "C" int set_next_tag(unsigned next) {
  return (int)cudaMemcpyToSymbol(g_noalloc_scratch, &next, sizeof next, kOffCtl + 4 * sizeof(int));
}
