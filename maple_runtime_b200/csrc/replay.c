/* replay.c -- the table of captured layer loops, by (tokens, first layer, layers, ...).
 *
 * A host that comes back for every layer asks for 24 keys per batch size, in the same order every time.  With slots reused in turn, one key more than
 * slots means that none is ever found again; and a miss costs more than it did without a table (960 keys over 256 slots: 90 us per layer call against
 * 84 of plain launches and 81 of replays; a wait and a destruction were part of a miss).  So a captured loop leaves only when REPLAY_IDLE calls have not asked for it, and
 * a key that has only been seen takes the place of another such, chosen at random: with more keys in use than slots, as many as there are slots settle
 * in the table and the others run with plain launches. */
#include <string.h>
#include "replay.h"

#define HEADS 4096
static ReplaySlot T[REPLAY_SLOTS];
static int head[HEADS], n[2];            /* slots in use: of stacks (from 0), of layer calls (behind them); chains of slot index + 1, 0 = end */
static uint64_t calls, rnd = 1;

static unsigned chain_of(const ReplayKey *k) {
    uint64_t h = 0;
    const int v[7] = {k->nb, k->l0, k->nl, k->bias, k->path, k->prof, k->ep};
    for (int i = 0; i < 7; i++) h = (h ^ (unsigned)v[i]) * 0x9E3779B97F4A7C15u, h ^= h >> 29;
    return (unsigned)(h >> 32) % HEADS;
}
static int same(const ReplayKey *a, const ReplayKey *b) {
    return a->nb == b->nb && a->l0 == b->l0 && a->nl == b->nl && a->bias == b->bias && a->path == b->path && a->prof == b->prof && a->ep == b->ep;
}
ReplaySlot *replay_find(const ReplayKey *k) {
    calls++;
    for (int i = head[chain_of(k)]; i; i = T[i - 1].next)
        if (same(&T[i - 1].key, k)) { T[i - 1].used = calls; return &T[i - 1]; }
    return NULL;
}
ReplaySlot *replay_admit(const ReplayKey *k, void **gone) {
    int s = -1;
    *gone = NULL;
    const int kind = k->nl == 0, base = kind ? REPLAY_STACKS : 0, size = kind ? REPLAY_LAYERS : REPLAY_STACKS;
    if (n[kind] < size) s = base + n[kind]++;
    for (int i = 0; i < 16 && s < 0; i++) {
        rnd = rnd * 6364136223846793005u + 1442695040888963407u;
        const int c = base + (int)((rnd >> 33) % (unsigned)size);
        if (T[c].exec && calls - T[c].used < REPLAY_IDLE) continue;
        int *p = &head[chain_of(&T[c].key)];
        while (*p != c + 1) p = &T[*p - 1].next;
        *p = T[c].next;
        *gone = T[c].exec; s = c;
    }
    if (s < 0) return NULL;
    int *h = &head[chain_of(k)];
    memset(&T[s], 0, sizeof T[s]);
    T[s].key = *k; T[s].used = calls; T[s].next = *h; *h = s + 1;
    return &T[s];
}
void replay_clear(void (*destroy)(void *exec)) {
    for (int i = 0; i < REPLAY_SLOTS; i++) if (T[i].exec) destroy(T[i].exec);
    memset(T, 0, sizeof T); memset(head, 0, sizeof head); n[0] = n[1] = 0;
}
