/* Two threads share one plan, each with a transform of its own.
 *
 * The plan's launch lists are built beforehand, so both threads only look them
 * up: minfft_b200_launch_count reads the list that a call would launch.  For a
 * real DFT of 1 x 64 points and its inverse the lists differ in length, so a
 * lookup that returns the other thread's list shows.  No kernel is launched.
 * Exits 0, or 1 if a count was off, 2 if the plan could not be made. */
#include <pthread.h>
#include <stdio.h>

#include "minfft.h"
#include "minfft_b200.h"

enum { THREADS = 4, CALLS = 3000000 };

struct arg {
    const minfft_aux *plan;
    int op, want;
    long off;
};

static void *count(void *p) {
    struct arg *a = p;
    for (long i = 0; i < CALLS; ++i) a->off += minfft_b200_launch_count(a->op, a->plan) != a->want;
    return NULL;
}

int main(void) {
    minfft_aux *plan = minfft_mkaux_realdft_2d(1, 64);
    if (!plan) return 2;
    pthread_t t[THREADS];
    struct arg a[THREADS];
    long off = 0;
    for (int i = 0; i < THREADS; ++i) {
        a[i].plan = plan;
        a[i].op = i % 2 ? MINFFT_B200_INVREALDFT : MINFFT_B200_REALDFT;
        a[i].want = minfft_b200_launch_count(a[i].op, plan);
        a[i].off = 0;
    }
    if (a[0].want == a[1].want) return 2;
    for (int i = 0; i < THREADS; ++i) pthread_create(&t[i], NULL, count, &a[i]);
    for (int i = 0; i < THREADS; ++i) {
        pthread_join(t[i], NULL);
        off += a[i].off;
    }
    minfft_free_aux(plan);
    printf("%ld of %ld lookups gave another transform's launches\n", off, (long)THREADS * CALLS);
    return off ? 1 : 0;
}
