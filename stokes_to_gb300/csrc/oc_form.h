// The launch form of an optimality-criteria update (topo.cu oc_update_device), host arithmetic only.
#pragma once

namespace stg {

constexpr int OC_CB = 16;             // blocks of the cluster form
constexpr int OC_CR = 8, OC_GR = 16;  // cells a thread holds, cluster and grid form
constexpr int OC_MAX_BLOCKS = 304;    // blocks of the grid form at most
// Doubles of block sums that an update needs at most: two buffers, so that a probe never
// overwrites the sums that the previous one's reduction still reads.
constexpr int OC_PARTS = 2 * OC_MAX_BLOCKS;
template <int R>
constexpr int OC_T = R ? 128 : 512;  // threads of a block that holds R cells each (0: reads them)
constexpr int OC_CLUSTER_MAX = OC_CB * OC_T<OC_CR> * OC_CR;

struct OcForm {
    bool cluster = false;  // one cluster of OC_CB blocks, sums in shared memory
    bool held = true;      // the cells stay in registers
    int blocks = OC_CB, threads = OC_T<OC_CR>;
    int parts() const { return cluster ? 0 : 2 * blocks; }
};

// One cluster while its threads hold at most eight cells each: a cluster barrier is 0.3 us and
// one over the device 1.3, but the cells of a probe take 1.3 us of sixteen SMs' FP64 units at
// the line (16384 cells: 178 us an update) and next to none of all of them. Else as many blocks
// as have cells, one on each SM.
inline OcForm oc_form(long long ncell, int sms, bool cluster_ok) {
    OcForm f;
    f.cluster = cluster_ok && ncell <= OC_CLUSTER_MAX;
    if (f.cluster) return f;
    if (sms > OC_MAX_BLOCKS) sms = OC_MAX_BLOCKS;
    if (sms < 1) sms = 1;
    f.held = ncell <= (long long)sms * OC_T<OC_GR> * OC_GR;
    f.threads = f.held ? OC_T<OC_GR> : OC_T<0>;
    const long long all = (ncell + f.threads - 1) / f.threads;
    f.blocks = (int)(all < sms ? all : sms);
    return f;
}

}  // namespace stg
