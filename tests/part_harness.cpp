// Host check that a failed allocation of the partial sums' buffer leaves no
// capacity behind (zeno_gb300/csrc/zc_reduce.cu): the allocation asked for here,
// for a state of 2^58 amplitudes, fails on every machine, before any launch.
// Links the built libzeno_cuda.so; no GPU.
#include <cstdio>

#include "zc_internal.h"

int main() {
    for (bool exact : {false, true}) {
        zc_state st;
        st.n = 58;
        st.len = 1ull << 58;
        st.num_sms = 148;
        st.part_cap = 16;  // as if a buffer of 16 sums had been there
        size_t nch = 0;
        if (zc::launch_chunk_sums(&st, 0, 0, &nch, exact) == ZC_OK) return std::printf("FAIL: allocated\n"), 1;
        if (st.d_part || st.part_cap) return std::printf("FAIL: capacity %zu without a buffer\n", st.part_cap), 1;
    }
    std::printf("ok\n");
    return 0;
}
