// Batched form: one launch of a pass covers the tiles of every problem of a
// group (same order p, same tile shape). Each problem contributes a table
// item -- its grid description, its pass arguments and the index of its
// first block in the launch -- and a block finds its item by binary search,
// copies it to shared memory and runs the same kernel body as the
// single-problem launch, on its problem-local tile index.
#pragma once
#include "spdk_kernelset.cuh"

namespace spdk {

struct DtArgs {
    double* dt;
    unsigned long long* dtmin;
};

template <typename Args>
struct BatchItem {
    DevGrid G;
    Args A;
    long long first;  // first block of this problem in the launch
};

// the item of block `block`, copied to shared memory (all threads return it)
template <typename Item>
__device__ __forceinline__ const Item& batch_item(const Item* __restrict__ items, int n, long long* local, long long block) {
    __shared__ __align__(16) unsigned char raw[sizeof(Item)];
    __shared__ int q;
    if (threadIdx.x == 0) {
        int lo = 0, hi = n - 1;
        const long long b = block;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (items[mid].first <= b) lo = mid;
            else hi = mid - 1;
        }
        q = lo;
    }
    __syncthreads();
    const int* src = reinterpret_cast<const int*>(items + q);
    int* dst = reinterpret_cast<int*>(raw);
    static_assert(sizeof(Item) % 4 == 0, "item size");
    for (int w = threadIdx.x; w < (int)(sizeof(Item) / 4); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    const Item& it = *reinterpret_cast<const Item*>(raw);
    *local = block - it.first;
    return it;
}

template <typename R, int P, int TX, int TY, int MODE>
__global__ void __launch_bounds__(picard_threads<R, 2, P, TX, TY>(), picard_blocks<R, 2, P, MODE>())
    picard_batched(const BatchItem<PicardArgsT<R>>* __restrict__ items, int n, DevMatsT<R> M) {
    long long b;
    const BatchItem<PicardArgsT<R>>& it = batch_item(items, n, &b, blockIdx.x);
    picard2d_body<R, P, TX, TY, MODE, false>(it.G, M, it.A, b);
}

// the batched detect takes one block per SM more than the single-problem
// kernel in 2D: the groups' many small members leave its sizing's occupancy
// unused (measured on the first 16 problems of the ensemble, FP32)
template <int D>
constexpr int kDetectBlocksPerSMBatched = D == 2 ? 5 : kDetectBlocksPerSM<D>;

template <typename R, int D, int P, int TX, int TY, int TZ>
__global__ void __launch_bounds__(kThreads, kDetectBlocksPerSMBatched<D>) detect_batched(const BatchItem<DetectArgs>* __restrict__ items, int n) {
    long long b;
    const BatchItem<DetectArgs>& it = batch_item(items, n, &b, blockIdx.x);
    fv_detect_kernel_body<R, D, P, TX, TY, TZ>(it.G, it.A, b);
}

// the tiles of all members that the detection listed, shared out among the blocks
template <typename R, int D, int P, int TX, int TY, int TZ>
__global__ void __launch_bounds__(kThreads, kBlendBlocksPerSM<R, D>)
    blend_batched(const BatchItem<BlendArgsT<R>>* __restrict__ items, int n, DevMatsT<R> M) {
    const BlendList list = items[0].A.list;
    const int count = *list.count;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int tile = list.tiles[i];
        long long b;
        const BatchItem<BlendArgsT<R>>& it = batch_item(items, n, &b, tile);
        fv_blend_kernel_body<R, D, P, TX, TY, TZ>(it.G, M, it.A, b);
        __syncthreads();  // the next tile reuses the shared memory
        if (threadIdx.x == 0) list.mark[tile] = 0;
    }
}

template <typename R, int D, int P>
__global__ void __launch_bounds__(kThreads, kUpdateBlocksPerSM<R, D, P>)
    update_batched(const BatchItem<FallbackArgsT<R>>* __restrict__ items, int n, DevMatsT<R> M) {
    long long b;
    const BatchItem<FallbackArgsT<R>>& it = batch_item(items, n, &b, blockIdx.x);
    fv_update_kernel_body<R, D, P>(it.G, M, it.A, b);
}

// dt hand-over of every problem of the batch: one thread per problem
__global__ void dt_batched(const DtArgs* __restrict__ a, int n);

template <typename R>
struct BatchSetT {
    void (*predict)(const BatchItem<PicardArgsT<R>>*, int, DevMatsT<R>) = nullptr;
    void (*correct)(const BatchItem<PicardArgsT<R>>*, int, DevMatsT<R>) = nullptr;
    void (*flux)(const BatchItem<PicardArgsT<R>>*, int, DevMatsT<R>) = nullptr;
    void (*detect)(const BatchItem<DetectArgs>*, int) = nullptr;
    void (*blend)(const BatchItem<BlendArgsT<R>>*, int, DevMatsT<R>) = nullptr;
    void (*update)(const BatchItem<FallbackArgsT<R>>*, int, DevMatsT<R>) = nullptr;
    size_t picard_smem[3] = {0, 0, 0}, blend_smem = 0, update_smem = 0;  // predict, correct, flux
    int picard_threads = kThreads;
    int picard_tile[3] = {1, 1, 1};  // a Picard block's elements (may hang over a domain's edge)
    int tile[3] = {1, 1, 1};         // a detect block's elements
    int blend_tile[3] = {1, 1, 1};
    int update_elems = 1;            // consecutive elements of an update block
};

template <typename R, int P, int TX, int TY>
BatchSetT<R> make_batch_set() {
    BatchSetT<R> k;
    constexpr int PX = kLineTX<P>, PY = kLineTY<P>;
    k.predict = picard_batched<R, P, PX, PY, kPredict>;
    k.correct = picard_batched<R, P, PX, PY, kCorrect>;
    k.flux = picard_batched<R, P, PX, PY, kFlux>;
    k.picard_threads = picard_threads<R, 2, P, PX, PY>();
    k.picard_tile[0] = PX;
    k.picard_tile[1] = PY;
    k.detect = detect_batched<R, 2, P, TX, TY, 1>;
    using BT = BlendTile<2, P>;
    k.blend = blend_batched<R, 2, P, BT::X, BT::Y, 1>;
    k.blend_smem = BlendSmem<R, 2, P, BT::X, BT::Y, 1>::bytes;
    k.blend_tile[0] = BT::X;
    k.blend_tile[1] = BT::Y;
    k.update = update_batched<R, 2, P>;
    k.update_elems = UpdateBlock<2, P>::NE;
    k.picard_smem[kPredict] = picard_smem_bytes<R, 2, P, PX, PY, kPredict>();
    k.picard_smem[kCorrect] = picard_smem_bytes<R, 2, P, PX, PY, kCorrect>();
    k.picard_smem[kFlux] = picard_smem_bytes<R, 2, P, PX, PY, kFlux>();
    k.update_smem = UpdateSmem<R, 2, P>::bytes;
    k.tile[0] = TX;
    k.tile[1] = TY;
    return k;
}

// the batched kernels of one (form, order, tile) -- false when not instantiated
// (2D; orders 2, 3, 5; tiles 1x1, 2x2 and, for p <= 3, 4x4)
bool batch_set(int p, int tile, BatchSetT<double>* k);
bool batch_set(int p, int tile, BatchSetT<float>* k);

}  // namespace spdk
