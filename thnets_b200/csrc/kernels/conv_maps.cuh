// What the tensor-core convolution launchers share: TMA descriptors (cached by what they encode) and the launch knobs.
// Defined in conv_tc.cu.
#pragma once
#include <cuda.h>
#include <pthread.h>
#include <string.h>
#include "thb200_kernels.h"

// TMA descriptors (one, or the few of a launch) by what they encode, an address and a shape: they cannot go stale when memory is
// reused.  The oldest makes way for the SIZE-th and later ones.  Found and kept as copies under a lock: launches of several host
// threads share the cache, and one launch's later descriptors may take the place of its earlier ones.
template <typename Key, typename Maps, int SIZE> class ThbMapCache {
    struct Entry {
        Key key;
        Maps maps;
    } entries[SIZE];
    unsigned used = 0, next = 0;
    pthread_mutex_t mutex = PTHREAD_MUTEX_INITIALIZER;

public:
    // (keys are compared as bytes: their padding is zero)
    bool find(const Key &key, Maps *out)
    {
        pthread_mutex_lock(&mutex);
        unsigned i = 0;
        while (i < used && memcmp(&entries[i].key, &key, sizeof(Key))) i++;
        if (i < used) *out = entries[i].maps;
        const bool found = i < used;
        pthread_mutex_unlock(&mutex);
        return found;
    }
    void keep(const Key &key, const Maps &maps)
    {
        pthread_mutex_lock(&mutex);
        Entry &e = entries[used < SIZE ? used++ : next++ % SIZE];
        e.key = key;
        e.maps = maps;
        pthread_mutex_unlock(&mutex);
    }
};

// Each into *out; false: the driver refuses it.
// a plain row-major matrix [rows][cols] with a row pitch, in boxes of 128 rows x box_cols
bool thb_matrix_tmap(const void *x, long rows, int cols, int ld, int dtype, int box_cols, CUtensorMap *out);
// the activation operand: mode 1 plain matrix, 2 im2col, 3 im2col over rows stored with their padding
bool thb_activation_tmap(const thb_conv_desc *d, const void *x, int mode, CUtensorMap *out);
// the packed weights in boxes of box_rows output channels x 128 or 64 bytes
bool thb_weights_tmap(const thb_conv_desc *d, int box_rows, int box_bytes, CUtensorMap *out);
// a rank-4 im2col descriptor can describe this convolution's input
bool thb_im2col_ok(const thb_conv_desc *d);

struct ThbConvLaunch {
    int pdl, test_withhold, sms, a_tma;
    int few_tiles, few_stages; // conv_few_tc.cu: THB200_FEW_TILES (most tiles of an unsplit launch, 0: off), THB200_FEW_STAGES; -1: not set
    long long wait_limit;
};
ThbConvLaunch thb_conv_launch_knobs();
