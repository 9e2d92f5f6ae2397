/* partition_plans.c -- the plans of requested partition counts, on the host
 * alone: spike_host.c with stand-ins for the device calls that building a plan
 * makes (other symbols stay unresolved; nothing here reaches them).  Built by
 * tests/test_partition_plans.py; test code only. */
#include "../../hspike_gb300/csrc/spike_host.c"

static size_t cap = (size_t)-1, used;
int spk_malloc_on(void **p, size_t bytes, void *stream)
{
    *p = NULL;
    if (bytes > cap - used) return SPK_EMEM;
    used += bytes;
    size_t *q = malloc(sizeof *q); /* holds its size; nothing is stored through it */
    *q = bytes;
    *p = q;
    return SPK_OK;
}
static void release(void *p)
{
    if (p) used -= *(size_t *)p;
    free(p);
}
int spk_malloc(void **p, size_t bytes) { return spk_malloc_on(p, bytes, NULL); }
void spk_free(void *p) { release(p); }
void spk_free_on(void *p, void *stream) { release(p); }
int spk_memcpy_h2d(void *d, const void *s, size_t b, void *st) { return SPK_OK; }
int spk_stream_sync(void *st) { return SPK_OK; }
int spk_sm_count(void) { return 152; }
size_t spk_factor_smem(int KB, int cplx, int mode) { return 1; }
int spk_twist_supported(int KB, int cplx, int mode) { return 1; }
void spk_phase_destroy(spk_plan *P) {}
void spk_shard_release(spike_context_t c) {}

#define CHECK(c)                                                                                                \
    do {                                                                                                        \
        if (!(c)) {                                                                                             \
            printf("line %d: %s\n", __LINE__, #c);                                                              \
            return 1;                                                                                           \
        }                                                                                                       \
    } while (0)

int main(void)
{
    const int n = 100000, k = 2, p = 4;
    spk_plan *P, *E;
    /* split: pieces inside each of the four, whose boundaries stay */
    CHECK(plan_create(n, 0, k, k, 0, SPK_PLAIN, p, 1, 1, NULL, 0, &P) == SPK_OK);
    const size_t split_bytes = used;
    CHECK(P->p_user == p && P->p > 100 * p && P->p % p == 0);
    for (int i = 0; i <= p; i++) CHECK(P->part_start[i * (P->p / p)] == i * (n / p));
    CHECK(same_partitions(P, p, 1) && !same_partitions(P, p, 0) && !same_partitions(P, p + 1, 1));
    spk_plan_destroy(P);
    CHECK(used == 0);
    /* exactly four */
    CHECK(plan_create(n, 0, k, k, 0, SPK_PLAIN, p, 0, 1, NULL, 0, &E) == SPK_OK);
    CHECK(E->p_user == p && E->p == p && E->n_iface == p - 1 && used < split_bytes);
    for (int i = 0; i <= p; i++) CHECK(E->part_start[i] == i * (n / p));
    CHECK(same_partitions(E, p, 0) && !same_partitions(E, p, 1));
    spk_plan_destroy(E);
    /* memory for four but not for the pieces: four, and the next call takes the plan again */
    cap = split_bytes - 1;
    CHECK(plan_create(n, 0, k, k, 0, SPK_PLAIN, p, 1, 1, NULL, 0, &P) == SPK_OK);
    CHECK(P->p == p && P->p_user == p && same_partitions(P, p, 1));
    spk_plan_destroy(P);
    /* not for four either */
    cap = 1000;
    CHECK(plan_create(n, 0, k, k, 0, SPK_PLAIN, p, 1, 1, NULL, 0, &P) == SPK_EMEM && !P && used == 0);
    cap = (size_t)-1;
    /* what a plan holds is what the admission estimate says, at every tile size;
     * FP64 copies of the reduced system's blocks only where they are read */
    const int ks[] = {1, 3, 8, 16, 17, 40, 64, 100};
    for (int i = 0; i < 8; i++)
        for (int mode = SPK_MIXED; mode <= SPK_PLAIN; mode++)
            for (int parts = 0; parts <= 5; parts += 5) {
                const int nn = 30011, nr = 3;
                CHECK(plan_create(nn, 0, ks[i], ks[i], 0, mode, parts, 1, nr, NULL, 0, &P) == SPK_OK);
                const size_t staging = sizeof(int) * ((size_t)nn + 1) + 8 * (size_t)nn * 3 * nr;
                CHECK(P->bytes == used);
                CHECK(spk_solve_footprint(nn, 0, ks[i], nr, 0, mode, parts) == P->bytes + staging);
                CHECK((P->d_RP != NULL) == (P->KB <= 16) && (P->d_RY != NULL) == (P->KB <= 16));
                spk_plan_destroy(P);
            }
    CHECK(spk_plan_reduced_build(9, 64, 0, SPK_MIXED, 2, &P) == SPK_OK && P->d_RP && P->d_RY);
    spk_plan_destroy(P);
    CHECK(used == 0);
    /* the option itself */
    struct spike_context_s c = {.split = 1};
    double v = 0;
    CHECK(spike_get_option(&c, SPIKE_OPT_SPLIT_PARTITIONS, &v) == SPIKE_SUCCESS && v == 1);
    CHECK(spike_set_option(&c, SPIKE_OPT_SPLIT_PARTITIONS, 0) == SPIKE_SUCCESS && !c.split);
    return 0;
}
