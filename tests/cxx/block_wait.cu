// Two groups of 128 threads apply a pass's blocks to tiles of their own, as
// the complex64 pass kernels do, while the completion of one group's products
// never reaches the threads that wait for it: its mbarrier expects one arrival
// more than it gets, so every wait runs into its (short) limit. Prints, per
// group, whether it gave up and how many tiles it finished, and fails when
// threads of one group disagree.
#include <cstdio>

#include "k_block.cuh"

using namespace kate;
using namespace kate::blk;

constexpr int G = 128, NG = NT / G, TILES = 5;
constexpr uint32_t OFF_S = KATE_C64_MAX_BLOCKS * KATE_BLOCK_IMG_BYTES, OFF_MISC = OFF_S + NG * S_BYTES;
constexpr uint32_t SMEM = OFF_MISC + 64 + 1024;

// out[2 t]: tiles that thread t saw its group finish with the right values
// (zero operand images: every amplitude becomes 0); out[2 t + 1]: gave up.
__global__ void __launch_bounds__(NT) k_blocks(const __grid_constant__ BlockProg P, int lost, int* out) {
    extern __shared__ uint8_t raw_smem[];
    const uint32_t raw = smem_u32(raw_smem), base = (raw + 1023u) & ~1023u;
    uint8_t* g = raw_smem + (base - raw);
    const uint32_t t = threadIdx.x, grp = t / G;
    GroupSync* groups = reinterpret_cast<GroupSync*>(g + OFF_MISC);
    uint32_t* slot = reinterpret_cast<uint32_t*>(groups + NG);
    for (uint32_t i = t; i < OFF_S / 4; i += NT) reinterpret_cast<uint32_t*>(g)[i] = 0;
    if (t == 0) {
        for (int i = 0; i < NG; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&groups[i].mbar)),
                         "r"(1u + (uint32_t)((lost >> i) & 1))
                         : "memory");
            groups[i].gave_up = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tmem_alloc(slot, NG * TMEM_COLS);
    Pass<G> X;
    setup(P, X);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *slot + grp * TMEM_COLS;
    float2* S = reinterpret_cast<float2*>(g + OFF_S + grp * S_BYTES);
    uint32_t phase = 0;
    int tiles = 0;
    bool ok = true;
    for (int i = 0; i < TILES && ok; i++) {
        for (uint32_t x = t % G; x < (uint32_t)TS; x += G) S[x] = make_float2(1.f, (float)i);
        group_bar<G>();
        ok = apply_blocks(P, X, S, base, tmem, smem_u32(&groups[grp]), phase);
        if (!ok) break;
        bool zero = true;
        for (uint32_t x = t % G; x < (uint32_t)TS; x += G) zero = zero && S[x].x == 0.f && S[x].y == 0.f;
        tiles += zero;
        group_bar<G>();
    }
    out[2 * t] = tiles;
    out[2 * t + 1] = !ok;
    tmem_free(*slot, NG * TMEM_COLS);
}

int main() {
    BlockProg P{};
    P.m = TB;
    P.nblocks = 2;
    for (int i = 0; i < TB; i++) P.tphys[i] = P.outsrc[i] = (uint8_t)i;
    for (int i = 0; i < 5; i++) P.btb[0][i] = (uint8_t)i, P.btb[1][i] = (uint8_t)(i + 6);
    int* d = nullptr;
    int h[2 * NT];
    auto check = [](cudaError_t e) {
        if (e != cudaSuccess) std::printf("%s\n", cudaGetErrorString(e));
        return e == cudaSuccess;
    };
    if (!check(cudaMalloc(&d, sizeof h)) ||
        !check(cudaFuncSetAttribute(k_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM)))
        return 2;
    int bad = 0;
    for (int lost = 0; lost < 1 << NG; lost++) {
        k_blocks<<<1, NT, SMEM>>>(P, lost, d);
        if (!check(cudaGetLastError()) || !check(cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost))) return 2;
        for (int grp = 0; grp < NG; grp++) {
            const int* a = h + 2 * G * grp;
            for (int t = 1; t < G; t++) bad += a[2 * t] != a[0] || a[2 * t + 1] != a[1];
            std::printf("lost %d group %d: gave up %d tiles %d\n", lost, grp, a[1], a[0]);
        }
    }
    std::printf("disagreements %d\n", bad);
    return bad != 0;
}
