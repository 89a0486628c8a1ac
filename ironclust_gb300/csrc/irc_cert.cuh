// irc_cert.cuh -- entry points of the proven search of the plain forms
// (irc_cert.cu) and the plain kernels it falls back on (internal).
#pragma once
#include "irc_plan.cuh"

// irc_cert_*: the call is not served here; the caller runs the plain kernels.
#define IRC_CERT_PASS 1

int irc_cert_site_knn(irc_plan *pl, const float *F, int nC, int knn, int nThreads, int mode, float *vrKnn, float *rho,
                      int32_t *miKnn, float *d2Knn, cudaStream_t s);
int irc_cert_site_delta_ref(irc_plan *pl, const float *F, int nC, const float *R, int nThreads, float *delta,
                            int32_t *nneigh, cudaStream_t s);
void irc_cert_release(irc_plan *pl);

// The plain kernels over a tile queue (irc_site.cu, irc_exact.cu).
int irc_ref_tiles(irc_plan *pl, const float *F, int nC, int knn, int nThreads, float *vrKnn, float *rho,
                  int32_t *miKnn, const irc::TileQueue &tq, cudaStream_t s);
int irc_exact_tiles(irc_plan *pl, const float *F, int nC, int knn, float *vrKnn, float *rho, int32_t *miKnn,
                    float *d2Knn, const irc::TileQueue &tq, cudaStream_t s);

// Device scratch of the drift-window delta search: unit and list counters,
// per chunk the number of queries to search and (a segment of list) which, the
// queries searched one by one, per-query keys and the units of 16-query tiles,
// up to 8 parts each.
struct irc_delta_scratch {
    int *words, *counts, *list;  // (a chunk's segment of list: from PlanDev::qseg)
    int2 *sparse, *items;
    unsigned long long *keys;
    const int *all;              // if not null and set: search every query
};
inline size_t delta_part(size_t n) { return (n + 255) & ~(size_t)255; }
inline size_t delta_bytes(long long n_out, long long n_qry, long long nChunks)
{
    const size_t n = (size_t)n_qry, c = (size_t)nChunks;
    return delta_part(4 * (4 + c)) + delta_part(4 * n) + delta_part(8 * n) + delta_part(8 * (size_t)n_out) +
           delta_part(8 * 8 * (n / 16 + c + 1));
}
irc_delta_scratch irc_delta_carve(const irc_plan *pl, void *mem, const int *all);
cudaError_t irc_delta_clear(const irc_plan *pl, const irc_delta_scratch &sc, cudaStream_t s);
int irc_delta_window(irc_plan *pl, const float *F, int nC, const float *R, int nT, const irc_delta_scratch &sc,
                     float *delta, int32_t *nneigh, cudaStream_t s);
