// Plain C++ (the host's checks compile it too): which keys a tile of 128 copies.
#pragma once
#ifdef __CUDACC__
#define KTB_HOST_DEVICE __host__ __device__
#else
#define KTB_HOST_DEVICE
#endif

namespace ktb {

// A tile of 128 keys from k0 (a multiple of 128) is copied as two runs of 64, each inside one page.  The first key of what is copied for run i when
// the keys lo .. hi are looked at: a run without any of them has no page to be looked up (its column of the page table may never have
// been written), and the tile's other run, which then has some, stands in for it.  lo <= hi, and the tile holds one of them.
KTB_HOST_DEVICE inline int key_run(int k0, int i, int lo, int hi) {
    const int k = k0 + 64 * i;
    return k + 63 < lo || k > hi ? k0 + 64 * (1 - i) : k;
}

}  // namespace ktb
