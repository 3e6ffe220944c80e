// qgru_rec_reg.cu - the recurrence with R in registers and warp-level int8 tensor instructions.
//
// A step of the recurrence is latency: a product with few batch rows, the cell, an exchange.  Here a CTA's slice
// of R (up to 196 KB) is held in registers in the order mma.sync takes its A operand (m16n8k32, eight batch
// rows per instruction), so a step reads only the state from shared memory and its sums appear in the
// registers of the threads that go on with them: no descriptors, no commit, no tensor-memory load
// between the product and the cell.  Measured on a B200: mma.sync.m16n8k32.s8 issues every 8 cycles per
// scheduler with 21 cycles latency, so the slice of 128 units of H = 512 takes 768 cycles for up to eight
// rows; the same rows on tcgen05 (whose throughput these small tiles cannot use: 16 columns at least,
// 128 x 16 x 32 per instruction, 53 cycles per issuing thread) are complete 1970 cycles after the state.
// For one row it equals dp4a (64 lanes per clock and SM).
//
// Split: clusters of P CTAs own Bt batch rows; a CTA owns U units as groups of 16 (three tiles of 16 rows of R, one
// per gate, so that one thread ends up with all three gates of a cell); K is split over KS warps per group
// where one warp's 96 registers do not hold it (H > 256), and their partial sums meet in shared memory,
// redistributed so that every warp gets an equal share of the cells.  H <= 256 is one CTA per row group:
// nothing leaves the SM and a step ends with one block barrier.  Larger layers send the new state to the
// peers with st.async, counted on their mbarrier: no fence on the sending side.  A peer can be at most
// one step ahead, so two state buffers are enough.
// W*x + bw arrives D steps ahead: one bulk copy a step where one CTA owns the rows, 16-byte copies by every warp of what its
// own cells read in clusters.
#include "qgru_rec_reg_kernel.cuh"

namespace qgru {
namespace {

RegKernel kernel_of(RecCell cell, int ih_bytes, int kst, int ks, bool hu, bool few) {
    switch (cell) {
        case CELL_INT_FAST: return ih_bytes == 2 ? pick<int16_t, CELL_INT_FAST>(kst, ks, hu, few) : pick<int32_t, CELL_INT_FAST>(kst, ks, hu, few);
        case CELL_INT_FAST_NOTIE: return ih_bytes == 2 ? pick<int16_t, CELL_INT_FAST_NOTIE>(kst, ks, hu, few) : pick<int32_t, CELL_INT_FAST_NOTIE>(kst, ks, hu, few);
        case CELL_INT_GENERIC: return ih_bytes == 1 ? pick<int8_t, CELL_INT_GENERIC>(kst, ks, hu, few) : pick<int16_t, CELL_INT_GENERIC>(kst, ks, hu, few);
        default: return rec_reg_float_kernel(cell, ih_bytes, kst, ks, hu, few);
    }
}

}  // namespace

bool rec_reg_plan(qgru_handle *h, int B, int sms, int ih_bytes, RecCell cell, int n_table, RecRegPlan *pl) {
    const int H = h->H;
    if (pl->H == H && pl->B == B && pl->sms == sms && pl->ih_bytes == ih_bytes && pl->cell == (int)cell && pl->n_table == n_table) return pl->ok;
    *pl = RecRegPlan{};
    pl->H = H;
    pl->B = B;
    pl->sms = sms;
    pl->ih_bytes = ih_bytes;
    pl->cell = (int)cell;
    pl->n_table = n_table;
    const int chunks = (H + 63) / 64;                    // of 64 inputs; at most four to a warp (96 registers)
    if (chunks > 16) return false;
    const int KS = chunks <= 4 ? 1 : chunks <= 8 ? 2 : 4;
    const int KST = std::max(KS > 1 ? 6 : 2, 2 * ((chunks + KS - 1) / KS));
    const int groups = (H + 15) / 16, most = 16 / KS;
    const int P = (groups + most - 1) / most;
    if (P > 16) return false;
    const int U = 16 * ((groups + P - 1) / P), threads = U / 16 * KS * 32;
    const RegKernel kern = kernel_of(cell, ih_bytes, KST, KS, h->h_uns, false);
    const int K = KS * KST * 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P);
    cfg.blockDim = dim3((unsigned)threads);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (P > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    // Rows per cluster: as few as the clusters that fit the chip at once allow.
    int D = 3, Bt = 0;
    for (int pass = 0; pass < 3; ++pass) {
        const int NT = (std::max(Bt, 1) + 7) / 8;
        for (D = 3; D > 1 && reg_smem(K, U, KS, NT, D, ih_bytes, cell, n_table).total > (size_t)h->smem_optin; --D) {}
        const size_t smem = reg_smem(K, U, KS, NT, D, ih_bytes, cell, n_table).total;
        if (smem > (size_t)h->smem_optin) {
            if (Bt <= 8) return false;
            Bt = (NT - 1) * 8;                           // more waves of clusters instead
            --pass;
            continue;
        }
        cfg.dynamicSmemBytes = smem;
        int active = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, kern, &cfg) != cudaSuccess || active < 1) {
            cudaGetLastError();
            return false;
        }
        active = std::max(1, std::min(active, (int)((long long)active * sms / h->sm_count)));
        pl->smem = smem;
        pl->D = D;
        const int want = (B + active - 1) / active;
        if (Bt >= want || (pass > 0 && Bt > 0)) break;
        Bt = want;
    }
    // Up to 128 inputs the few rows' form takes ten registers more (above, R alone fills the register file's share of a CTA):
    // only for a last tile that gains by it, and where as many CTAs still fit.  us a step: H = 128, 592 rows 1.53 -> 1.08, float storage
    // 2.70 -> 1.65; H = 64, 2000 rows 1.62 -> 1.06; with one row a CTA (H = 64, 592 rows) 1.04, and 1.06 in this form.
    const int tail = (Bt - 1) % 8 + 1;
    if (KS == 1 && KST <= 4 && tail > 1 && tail <= 4) {
        const RegKernel other = kernel_of(cell, ih_bytes, KST, KS, h->h_uns, true);
        int active = 0;
        if (cudaFuncSetAttribute(other, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl->smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, other, &cfg) != cudaSuccess)
            cudaGetLastError();
        pl->few = (long long)active * sms / h->sm_count * Bt >= B;
    }
    pl->KST = KST;
    pl->KS = KS;
    pl->U = U;
    pl->P = P;
    pl->Bt = Bt;
    pl->G = (B + Bt - 1) / Bt;
    pl->ok = true;
    return true;
}

int rec_reg_launch(qgru_handle *h, const RecRegPlan &pl, RecRegArgs a, RecCell cell, int ih_bytes, cudaStream_t st) {
    const RegKernel kern = kernel_of(cell, ih_bytes, pl.KST, pl.KS, h->h_uns, pl.few);
    a.U = pl.U;
    a.P = pl.P;
    a.Bt = pl.Bt;
    a.NT = (pl.Bt + 7) / 8;
    a.D = pl.D;
    // fp32 output only, through running pointers with 32-bit row offsets; where one CTA owns all units, in pairs of
    // neighbouring units (8-byte stores: every row's first unit has to be aligned)
    const bool plain = a.out.hf && !a.out.hq && !a.out.h8 && a.out.bs <= (1u << 24);
    a.vec2 = pl.KS > 1 ? plain : plain && a.H % 2 == 0 && a.out.ts % 2 == 0 && a.out.bs % 2 == 0 &&
             (reinterpret_cast<uintptr_t>(a.out.hf) & 7u) == 0 && (reinterpret_cast<uintptr_t>(a.out.hn_f) & 7u) == 0;
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
    if (pl.P > 8) CK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(pl.G * pl.P));
    cfg.blockDim = dim3((unsigned)(pl.U / 16 * pl.KS * 32));
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)pl.P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.pdl ? 2 : 1;
    CK(cudaLaunchKernelEx(&cfg, kern, (const GateConsts)h->gc_host, (const RecRegArgs)a));
    h->launches++;
    return QGRU_OK;
}

}  // namespace qgru
