/* The oracle's S-Merge from two sub-graphs that the caller gives (the steps
 * InitSGraph, InitialGraph, nnDescent, merge2one in a fresh process). */
#include "../../oracle/nnm_oracle.c"

int nno_smerge_graphs(const float *x, uint32_t n, uint32_t d, uint32_t k, uint32_t pre, const uint32_t *g1,
                      const uint32_t *g2, uint32_t seed, uint32_t *ids, float *dists, uint8_t *flags) {
    grand_t rnd;
    grand_seed(&rnd, seed);
    graph_t g;
    g_init(&g, x, n, d, k, NNO_L2, &rnd, NULL);
    g.n = n;
    init_sgraph(&g, 0, g1, 0, pre);
    init_sgraph(&g, pre, g2, 1, n - pre);
    mt_t rng;
    mt_seed(&rng, seed);
    const uint32_t cut = k / 2;
    uint32_t seeds[1024];
    int rc = 0;
    for (uint32_t i = 0; i < n && !rc; i++)
        rc = cross_sample_row(&g, i, &rng, cut, 2 * cut, i < pre ? n - pre : pre, i < pre ? pre : 0, i < pre, seeds);
    if (!rc) {
        nndescent(&g, MODE_SMERGE, pre, 0);
        merge2one(&g, n);
        out_pools(&g, ids, dists, flags);
    }
    g_free(&g);
    return rc;
}
