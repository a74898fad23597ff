// StreamFork against a runtime that only keeps account: which stream waits for
// which work.  One argument: the call to fail (1-based; 0: none).  The script is
// a plan run with two side streams, one with a look-ahead stream, whose third
// launch fails.  Prints the calls made and ends with 0 if the caller's stream is
// behind everything that was launched.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>

#include "stream_fork.h"

static std::map<cudaStream_t, std::set<int>> behind;   // work a stream is ordered behind
static std::map<cudaEvent_t, std::set<int>> recorded;  // work an event stands for
static int launched = 0, calls = 0, fail_at = 0;
static cudaError_t last = cudaSuccess;

static cudaError_t step(const char *what)
{
    std::printf("%s ", what);
    if (++calls != fail_at) return cudaSuccess;
    return last = cudaErrorUnknown;
}
extern "C" {
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st)
{
    const cudaError_t e = step("record");
    if (e == cudaSuccess) recorded[ev] = behind[st];
    return e;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned)
{
    const cudaError_t e = step("wait");
    if (e == cudaSuccess) behind[st].insert(recorded[ev].begin(), recorded[ev].end());
    return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    std::printf("sync ");
    for (auto &b : behind) b.second.insert(behind[st].begin(), behind[st].end());
    return cudaSuccess;
}
}
static void launch(cudaStream_t st) { behind[st].insert(++launched); }

static cudaStream_t S(long i) { return reinterpret_cast<cudaStream_t>(i); }
static cudaEvent_t E(long i) { return reinterpret_cast<cudaEvent_t>(i); }

static int run(bool launch_fails)
{
    mgpu::StreamFork fork(S(1), E(1));
    launch(S(1));
    if (fork.begin()) return 1;
    if (fork.to(S(2), E(2), S(3), E(3))) return 1;
    if (behind[S(2)].empty()) return 2;  // not after the caller's work
    launch(S(2));
    launch(S(3));
    if (!launch_fails) {  // the look-ahead stream joins its main stream on the way through
        if (cudaEventRecord(E(4), S(3)) || cudaStreamWaitEvent(S(2), E(4), 0)) return 1;
    }
    if (fork.to(S(5), E(5))) return 1;
    launch(S(5));
    if (launch_fails) return 1;
    launch(S(1));
    return fork.join() ? 1 : 0;
}

int main(int argc, char **argv)
{
    fail_at = argc > 1 ? std::atoi(argv[1]) : 0;
    const int rc = run(argc > 2);
    // an error of the join on the way out reaches nobody: it must not be left for the next launch check either
    if (argc > 2 && fail_at > 3 && last != cudaSuccess) return 3;
    std::printf("\n%d of %d\n", (int)behind[S(1)].size(), launched);
    if (rc == 2 || (int)behind[S(1)].size() != launched) return 1;
    return (rc != 0) == (argc > 2 || (fail_at > 0 && fail_at <= calls)) ? 0 : 2;
}
