// Joins a second stream at the end of a scope.
#pragma once
#include <cuda_runtime.h>

namespace bsrg {

// Work queued on `aux` writes a workspace that belongs to `st`.  However the scope is left, `st` waits for it, so
// that the next call on `st` cannot meet a kernel that still writes there; done() where `st` has been joined already.
class AuxJoin {
    cudaStream_t aux, st;
    cudaEvent_t ev;

public:
    AuxJoin(cudaStream_t aux_, cudaStream_t st_, cudaEvent_t ev_) : aux(aux_), st(st_), ev(ev_) {}
    AuxJoin(const AuxJoin &) = delete;
    AuxJoin &operator=(const AuxJoin &) = delete;
    ~AuxJoin()
    {
        if (aux && cudaEventRecord(ev, aux) == cudaSuccess) cudaStreamWaitEvent(st, ev, 0);
    }
    void done() { aux = nullptr; }
};

}  // namespace bsrg
