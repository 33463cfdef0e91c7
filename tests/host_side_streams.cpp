// Side streams on the fake runtime: each caller's stream has its own on each
// device, a bounded number of them, given back with the working sets.
#include <set>

#include "fake_cuda.hpp"
#include "common.cuh"

using imops::SideStream;

static cudaStream_t caller(size_t k) { return reinterpret_cast<cudaStream_t>(k << 4); }

int main() {
    std::set<cudaStream_t> sides;
    for (int dev = 0; dev < 2; dev++) {
        cudaSetDevice(dev);
        for (size_t k = 0; k < imops::SIDE_STREAMS; k++) {  // the default stream among them
            SideStream ss, again;
            EXPECT(imops::side_stream(caller(k), &ss) == IMOPS_OK && ss.side != caller(k));
            EXPECT(imops::side_stream(caller(k), &again) == IMOPS_OK && again.side == ss.side);
            EXPECT(sides.insert(ss.side).second);
            EXPECT(ss.fork(caller(k)) == IMOPS_OK && ss.record(caller(k)) == IMOPS_OK && ss.wait(caller(k)) == IMOPS_OK);
        }
        SideStream more;  // one caller too many: its work stays on its stream
        EXPECT(imops::side_stream(caller(1000), &more) == IMOPS_OK && more.side == caller(1000) && !more.forked);
        EXPECT(more.fork(caller(1000)) == IMOPS_OK && more.record(caller(1000)) == IMOPS_OK &&
               more.wait(caller(1000)) == IMOPS_OK);
    }
    EXPECT(fake::streams == 2 * imops::SIDE_STREAMS && fake::events == 4 * imops::SIDE_STREAMS);
    EXPECT(imops::release_working_sets(1) == IMOPS_OK);
    EXPECT(fake::streams == imops::SIDE_STREAMS && fake::events == 2 * imops::SIDE_STREAMS);
    cudaSetDevice(0);
    EXPECT(imops::release_working_sets(0) == IMOPS_OK && fake::streams == 0 && fake::events == 0);
    return 0;
}
