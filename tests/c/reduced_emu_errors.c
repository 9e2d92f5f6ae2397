/* reduced_emu_errors.c -- the reduced factorization of 64-row FP64 tiles when a
 * digit-product launch fails.  Linked with spike_reduced.o alone; the two
 * launchers of spike_emu64.cu are stand-ins here that fail on request, so no
 * GPU is needed.  Built by tests/test_reduced_errors.py; test code only. */
#include <stdio.h>
#include <string.h>

#include "spike_internal.h"

/* the runtime's error state: clean, as after a launcher that checked (and
 * cleared) it itself */
int __wrap_cudaGetLastError(void) { return 0; } /* (linked with --wrap) */

static int odd_rc, even_rc, odd_calls, even_calls;

int spk_emu_cr_odd(const double *P, const double *Q, int first, int stride, int count, double *M, unsigned *err,
                   void *stream)
{
    odd_calls++;
    return odd_rc;
}
int spk_emu_cr_even(const double *P, const double *Q, const double *X, const double *Y, const double *M, int cnt,
                    double *Pn, double *Qn, double *Xn, double *Yn, void *stream)
{
    even_calls++;
    return even_rc;
}

/* a plan of n_iface interfaces whose tiles no kernel here touches */
static int factor(int n_iface, int orc, int erc)
{
    static int count[8];
    static long long off[9], moff[9];
    spk_plan P;
    memset(&P, 0, sizeof P);
    P.KB = 64;
    P.mode = SPK_PLAIN;
    P.n_iface = n_iface;
    P.red_direct = 1;
    int L = 0;
    for (int c = n_iface; c > 1; c = (c + 1) / 2) count[L++] = c;
    count[L] = 1;
    P.cr_levels = L;
    P.cr_count = count;
    P.cr_off = off;
    P.cr_moff = moff;
    odd_rc = orc;
    even_rc = erc;
    odd_calls = even_calls = 0;
    return spk_reduced_factor(&P, NULL);
}

int main(void)
{
    int bad = 0;
    struct {
        int nif, orc, erc, want, odd, even;
    } t[] = {{1, SPK_OK, SPK_OK, SPK_OK, 1, 0},       {5, SPK_OK, SPK_OK, SPK_OK, 4, 3},
             {1, SPK_ECUDA, SPK_OK, SPK_ECUDA, 1, 0}, {5, SPK_ECUDA, SPK_OK, SPK_ECUDA, 1, 0},
             {5, SPK_OK, SPK_ECUDA, SPK_ECUDA, 1, 1}};
    for (unsigned i = 0; i < sizeof t / sizeof t[0]; i++) {
        const int rc = factor(t[i].nif, t[i].orc, t[i].erc);
        if (rc != t[i].want || odd_calls != t[i].odd || even_calls != t[i].even) {
            printf("case %u: rc %d (want %d), odd calls %d (%d), even calls %d (%d)\n", i, rc, t[i].want, odd_calls,
                   t[i].odd, even_calls, t[i].even);
            bad = 1;
        }
    }
    return bad;
}
