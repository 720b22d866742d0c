// phase_bits.h -- which phase of an mbarrier a thread waits for next.  Plain C++, so that
// the host can test it.  Not part of the C ABI.
#pragma once

#ifdef __CUDACC__
#define CHAN_HD __host__ __device__ __forceinline__
#else
#define CHAN_HD inline
#endif

// The parity of the next wait on each of up to 32 barriers whose phases are waited for in
// order.  The bit moves on with every wait, also with one that runs out: moved on success
// only, it cost the persistent ensemble kernel 1 to 1.7% in spills.
struct PhaseBits {
    unsigned bits = 0u;
    CHAN_HD unsigned next(int s) const { return (bits >> s) & 1u; }
    CHAN_HD void waited(int s) { bits ^= 1u << s; }
    // the parity of the phase of barrier s that is not complete: the one last waited for, if
    // that wait ran out, else the next.  (A test of the other parity succeeds at once.)
    CHAN_HD unsigned open(int s, bool ran_out) const { return ((bits >> s) & 1u) ^ (ran_out ? 1u : 0u); }
};

// The phases of up to 32 barriers that one thread's commits complete: whether a barrier has
// had one, and the parity of its last, the one to wait for before leaving.
struct CommitBits {
    unsigned bits, any;   // start from {} (no initialisers: it is also a shared variable)
    CHAN_HD void committed(int s)
    {
        bits ^= 1u << s;
        any |= 1u << s;
    }
    CHAN_HD bool some(int s) const { return (any >> s) & 1u; }
    CHAN_HD unsigned last(int s) const { return ((bits >> s) & 1u) ^ 1u; }
};
