// How a kernel's failure reaches the host: a status word in device memory, which later CTAs and launches look at, and a
// mirror of it in host memory, which the host looks at after a synchronise.  Both halves are written over their memory
// operations, so that a plain C++ test can interleave them.
#pragma once

#if defined(__CUDACC__)
#define TXB_HD __host__ __device__ __forceinline__
#else
#define TXB_HD inline
#endif

namespace txb {

// Kernel side.  `claim(code)`: stores the code in the word if that is 0, returns what was there.  `tell(code)`: writes the
// mirror.  The first code stays; every report reaches the mirror, also one that comes while the host is clearing up
// after an earlier one and has the mirror cleared but not yet the word.
template <class Claim, class Tell>
TXB_HD void make_report(Claim claim, Tell tell, int code)
{
    const int before = claim(code);
    tell(before != 0 ? before : code);
}

// Host side, one caller at a time.  `exchange(v)`: puts v in the mirror, returns what was there.  `clear()`: zeroes the word
// and waits for it; false if that failed.  Returns the code, 0 if there is none.  The mirror goes first: a report that comes
// between the two steps leaves the mirror set and the word zero, where the other order would leave a word that stops every
// later launch and that nobody asks for.  A word that could not be cleared keeps its mirror.
template <class Exchange, class Clear>
inline int take_report(Exchange exchange, Clear clear)
{
    const int code = exchange(0);
    if (code != 0 && !clear()) exchange(code);
    return code;
}

}  // namespace txb
