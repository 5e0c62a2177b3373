/* Candidate harvest and collapse on the GPU (cs_collapse.cu), used by the
 * session's collect path in cs_gpu.cu.  Internal to libcsgpu.so. */
#ifndef CS_COLLAPSE_H
#define CS_COLLAPSE_H

#include <cuda_runtime.h>
#include "cs_internal.h"

typedef struct CsCollapse CsCollapse;

CsCollapse *cs_collapse_new(void);
void cs_collapse_free(CsCollapse *w);

/* Enqueue, on `st` and without synchronising, the collapse of the n records
 * at device address recs into the candidate list search_file returns after
 * its post-processing (src/search.c:1467-1478).  0 or -1. */
int cs_collapse_enqueue(CsCollapse *w, const CsRec *recs, unsigned n, const CsChunk *chunks,
                        long long nchunks, const int *slot_k, const int *slot_Hk, int nslot,
                        int nprof, double r_lo, double lodr, double N, double T,
                        double threshold, int remove, double dr_tol, int harm_remove,
                        int numharm, double harm_tol, cudaStream_t st);

/* The same for a search whose record count is still on the device (count, err:
 * the search's counter and error flag; cap: the record buffer's capacity; total:
 * trials), in one launch that only works on up to cs_collapse_small_cap()
 * records.  After a wait on `st`, cs_collapse_small_status gives the count and
 * the error flag, and 1 when the list is ready (cs_collapse_finish hands it
 * over), 0 when the records have to go through cs_collapse_enqueue.  Returns 0, 1
 * when the geometry does not fit (nothing queued), or -1. */
int cs_collapse_small_enqueue(CsCollapse *w, const CsRec *recs, const unsigned *count,
                              const int *err, unsigned cap, const CsChunk *chunks,
                              const int *slot_k, const int *slot_Hk, int nslot, long long total,
                              double r_lo, double lodr, double N, double T, double threshold,
                              int remove, double dr_tol, int harm_remove, int numharm,
                              double harm_tol, cudaStream_t st);
unsigned cs_collapse_small_cap(void);
int cs_collapse_small_status(const CsCollapse *w, unsigned *n, int *err);

/* Wait for the enqueued collapse and copy its list to host memory (out;
 * the caller frees it with candlist_free).  0 or -1. */
int cs_collapse_finish(CsCollapse *w, cudaStream_t st, CandidateList *out);

#endif
