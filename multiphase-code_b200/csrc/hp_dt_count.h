// hp_dt_count.h -- finished blocks of a launch, counted in a word that
// launches share one after another.
//
// Each call has a number, larger than that of every call before it, and
// counts in the range of values that starts at number << DT_COUNT_BITS.
// Opening raises the word to the start of that range, so whatever an earlier
// call left there (calls that overlapped and mixed their counts too) is
// overwritten, no call has to leave the word at zero, and no operation of
// another launch has to clear it.  Every block opens before it arrives, so
// the first to arrive finds the range open.  Not for launches that are
// repeated with the same number.
#ifndef HP_DT_COUNT_H
#define HP_DT_COUNT_H

namespace hp {

enum { DT_COUNT_BITS = 20 };

#if defined(__CUDACC__)
__device__ __forceinline__ void dt_raise(unsigned long long* w, unsigned long long v) { atomicMax(w, v); }
__device__ __forceinline__ unsigned long long dt_next(unsigned long long* w) { return atomicAdd(w, 1ull); }
#define HP_DT_FN __device__ __forceinline__
#else
// one thread
inline void dt_raise(unsigned long long* w, unsigned long long v) { if (*w < v) *w = v; }
inline unsigned long long dt_next(unsigned long long* w) { return (*w)++; }
#define HP_DT_FN inline
#endif

HP_DT_FN void dt_count_open(unsigned long long* word, unsigned long long call) {
    dt_raise(word, call << DT_COUNT_BITS);
}
// true for the block of the call that arrives last
HP_DT_FN bool dt_count_arrive(unsigned long long* word, unsigned long long call, unsigned blocks) {
    return dt_next(word) - (call << DT_COUNT_BITS) == blocks - 1;
}
#undef HP_DT_FN

}  // namespace hp
#endif
