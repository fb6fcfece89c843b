/* replay.h -- which captured layer loops are kept. */
#ifndef MAPLE_REPLAY_H
#define MAPLE_REPLAY_H
#include <stdint.h>
/* Layer calls (nl = 0): 24 layers x 96 batch sizes whose rows are used in place; measured for all of them: 300 MB of device memory and 125 MB of the host's.
 * Stacks: 0.4 MB of device memory and 1.3 MB of the host's each (24 layers). */
#define REPLAY_LAYERS 2304
#define REPLAY_STACKS 256
#define REPLAY_SLOTS (REPLAY_LAYERS + REPLAY_STACKS)
#define REPLAY_IDLE (4 * REPLAY_SLOTS)      /* a captured loop that so many calls have not asked for may go */
typedef struct { int nb, l0, nl, bias, path, prof, ep; } ReplayKey;
typedef struct { ReplayKey key; int next, tried; long launches; uint64_t used; void *exec; } ReplaySlot;
/* the slot of a key that has been asked for before (counts as a use), NULL: it is new, or was not kept */
ReplaySlot *replay_find(const ReplayKey *k);
/* a slot for a new key; *gone = the captured loop that has to make room and is for the caller to destroy, else NULL.  Returns NULL when no slot can be
 * spared: the call then runs without a replay, as a call that comes once does. */
ReplaySlot *replay_admit(const ReplayKey *k, void **gone);
/* empties the table; destroy is called for every captured loop */
void replay_clear(void (*destroy)(void *exec));
#endif
