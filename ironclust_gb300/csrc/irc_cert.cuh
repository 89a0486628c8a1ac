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
                    float *d2Knn, const irc::TileQueue &tq, int *cnt, int *ovf_list, cudaStream_t s);

// Device scratch of the drift-window delta search: the unit counter, one flag
// and one key per query, the compacted queries [n_out] and their units, up to
// 8 parts of every 16-query tile.
struct irc_delta_scratch {
    int *n_items, *flags, *list;
    int2 *items;                 // [delta_items(...)]
    unsigned long long *keys;    // [n_out]
};
inline size_t delta_items(long long n_out, long long nChunks)
{
    return 8 * ((size_t)n_out / 16 + (size_t)nChunks + 1);
}
int irc_delta_window(irc_plan *pl, const float *F, int nC, const float *R, int nT, const irc_delta_scratch &sc,
                     float *delta, int32_t *nneigh, cudaStream_t s);
