// What the forms of the decayed linear attention share: how q, k and v enter the recurrence.
#pragma once

#include <math.h>

// Rotary positions on q and k on their way in (positions null: none), and a factor on k after them.  The first
// `rotary` elements of a head are rotated by the token's position: the pair (u, v), elements (i, i + rotary / 2)
// or, `interleaved`, (2i, 2i + 1), becomes (u c - v s, v c + u s) with c = mag cos(pos * freq[i]), s = mag sin(same);
// position x frequency is one fp32 product, sine and cosine are in full precision.
struct RotaryArgs {
    const int* positions;
    const float* freq;
    int rotary, interleaved;
    float mag, k_scale;
};

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
