// asv_tally.cuh -- counts of a block, gathered in shared memory.
//
// Labels of neighbouring voxels are few, so all blocks in flight count into the
// same few words of a global table, and such updates wait for each other: one
// atomic per run of equal labels took 84 us for the label counts of a
// 320x240x85 volume (6.5 M voxels), a tenth of which is the bytes' time.  A block
// adds to a small hash table first and hands each of its labels out once.  A key
// that finds no place after four probes is handed out at once.
#ifndef ASV_TALLY_CUH
#define ASV_TALLY_CUH

#define TALLY_LOG 8
#define TALLY_SLOTS (1 << TALLY_LOG)

struct Tally {
    int key[TALLY_SLOTS];
    unsigned cnt[TALLY_SLOTS];
};

// by a block of at least TALLY_SLOTS threads; a barrier must follow
__device__ __forceinline__ void tally_clear(Tally &t)
{
    if (threadIdx.x < TALLY_SLOTS) {
        t.key[threadIdx.x] = -1;
        t.cnt[threadIdx.x] = 0u;
    }
}

// adds c to key (>= 0); false: no place, the caller hands it out itself
__device__ __forceinline__ bool tally_add(Tally &t, int key, unsigned c)
{
    const unsigned h = ((unsigned)key * 2654435761u) >> (32 - TALLY_LOG);
    for (unsigned p = 0; p < 4; p++) {
        const unsigned i = (h + p) & (TALLY_SLOTS - 1);
        int k = *(volatile int *)&t.key[i];
        if (k == -1) k = atomicCAS(&t.key[i], -1, key);
        if (k == -1 || k == key) {
            atomicAdd(&t.cnt[i], c);
            return true;
        }
    }
    return false;
}

#endif
