// Batch solution files as text on the GPU (cs_text.cu), called by the runtime.
#pragma once
#include <stddef.h>

struct CsTextArgs {
  const double *t, *y, *z, *p;  // device: t [T], y [T][ny], z at the nodes [T][nz], p [B][np]
  long long T;                  // node slots
  int B, ny, nz, np;
  const int *dN, *doff;         // device: nodes and first slot of every instance
  const int* hN;                // host: nodes
  void* stream;
  struct CsTextScratch* scratch;
};

// Device scratch of the writer (index and offsets, text), grown on demand and
// kept by its owner.
struct CsTextScratch {
  void* p[2] = {nullptr, nullptr};
  size_t bytes[2] = {0, 0};
};
void cs_text_scratch_free(CsTextScratch* s);

// Sizes every file (offsets: B + 1 host entries) and, with out non-null and cap
// large enough, writes the files to out.
int cs_text_files(const CsTextArgs& a, char* out, long long cap, long long* offsets);
