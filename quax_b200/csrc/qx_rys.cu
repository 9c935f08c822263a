// qx_rys.cu -- the Rys quadrature table on the device, and the sum over the work items
// that share a quartet of a first-derivative tensor.
//
// The node/weight table (qx_rys_table.inc, ~345 KB) is a statically initialised
// __device__ array: it is loaded with the module, so no allocation or copy is
// needed.  Host code reaches it through qx_rys_table(), which looks up the
// array's device address once per device (cudaGetSymbolAddress) -- the symbol
// itself is only a host-side stand-in.
#include <cuda_runtime.h>

#include <mutex>

#include "qx_rys.cuh"

__device__ const double g_qx_rys_table[qx::RYS_TABLE_DOUBLES] = {QX_RYS_TAB_DATA QX_RYS_ASYM_Y_DATA,
                                                                 QX_RYS_ASYM_W_DATA};

namespace qx {

// The parts' sums of a quartet (block: its position in the processing order), added in
// order and written by one thread per component, so that the images of a derivative
// integral are equal to the bit and repeated calls give the same tensor; atomics of every
// part gave neither.  Ten molecules of two and three atoms with f shells: 2.0 to 67 ms by
// atomics, 14 to 118 by one team per quartet, 1.9 to 43 in order (the join reads each sum
// once, where the atomics went to up to eight images of it).
__global__ void __launch_bounds__(128) k_rys_join(RysArgs ra, int ncomp, int nb, int nc, int nd) {
    __shared__ long long slot[12];
    __shared__ double mult[12];
    const EriArgs& a = ra.e;
    const long long w = blockIdx.x, n = a.n, n4 = n * n * n * n;
    const int2 pq = a.quartets[list_index(a, w)];
    const PairInfo P = a.pairs[pq.x], Q = a.pairs[pq.y];
    const int atoms[4] = {P.atom1, P.atom2, Q.atom1, Q.atom2};
    // what the parts skipped
    if (atoms[0] == atoms[1] && atoms[0] == atoms[2] && atoms[0] == atoms[3]) return;
    if (ra.slice_k) {
        const int at = ra.slice_nu[0] / 3;
        if (at != atoms[0] && at != atoms[1] && at != atoms[2] && at != atoms[3]) return;
    }
    if (threadIdx.x < 12) {
        int ops;
        double m;
        const bool keep = rys_derk_index(1, threadIdx.x, atoms, ra.M, ra.slice_nu, ra.slice_k, ops, slot[threadIdx.x], m);
        mult[threadIdx.x] = keep ? m : 0.0;
    }
    __syncthreads();
    const bool s12 = P.s1 != P.s2, s34 = Q.s1 != Q.s2, sPQ = pq.x != pq.y;
    const int parts = min(ra.parts, P.nprim * Q.nprim);
    for (int kc = blockIdx.y * blockDim.x + threadIdx.x; kc < ncomp; kc += gridDim.y * blockDim.x) {
        const int id = kc % nd, ic = (kc / nd) % nc, ib = (kc / (nd * nc)) % nb, ia = kc / (nd * nc * nb);
        for (int m = 0; m < 12; ++m) {
            if (mult[m] == 0.0) continue;
            const double* q = ra.partial + (w * ra.parts * 12 + m) * ncomp + kc;
            double v = 0.0;
            for (int p = 0; p < parts; ++p) v += q[(long long)p * 12 * ncomp];
            atomic_images_w(a.out + slot[m] * n4, n, P.bf1 + ia, P.bf2 + ib, Q.bf1 + ic, Q.bf2 + id, s12, s34, sPQ,
                            mult[m] * v);
        }
    }
}

}  // namespace qx

void qx_launch_rys_join(const qx::RysArgs& ra, int ncomp, int nb, int nc, int nd, cudaStream_t s) {
    const dim3 grid((unsigned)ra.e.nq, (unsigned)((ncomp + 127) / 128));
    qx::k_rys_join<<<grid, 128, 0, s>>>(ra, ncomp, nb, nc, nd);
}

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mu;
const double* g_addr[kMaxDevices] = {};
}  // namespace

// Device address of the table on the current device (nullptr on failure).
const double* qx_rys_table() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_addr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_qx_rys_table) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        g_addr[dev] = static_cast<const double*>(p);
    }
    return g_addr[dev];
}
