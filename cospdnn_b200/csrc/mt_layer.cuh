// Multi-layer tile kernel interface (implementation in mt_layer.cu).
#pragma once

#include <vector>

#include "engine.cuh"

namespace cospdnn {

// True when a CUDA-core net of width N in precision `prec` whose layers each
// have one weight value runs on the multi-layer tile kernel: two tiles of
// 16-byte feature columns (8 rows, FP32 4) in shared memory.
bool mt_supported(int N, int prec);
// Builds and uploads the entry list of one layer (S, dW and K already in ld).
int mt_build_entries(const std::vector<int32_t> &colptr, const std::vector<int32_t> &rowidx,
                     const std::vector<float> &vals, int N, int prec, const LayerDev &ld, MtLayer &ml,
                     std::vector<void *> &owned);
// Launch description of the kernel for the nets of precision `prec`, the
// widest of max_n neurons.
int mt_layer_spec(KSpec &k, NetDev *nets, int nnets, int prec, unsigned long long *launches, int sms, int max_n);
// Tiles up to which a layer is faster on k_layer_cc (0: never, -1: all `rows` of the
// network are); entries: of the fullest output.
int mt_few_tiles(int N, int prec, double entries, int sms, int64_t rows);
// CTAs of that launch.
int mt_layer_ctas(int sms, int max_n);

}  // namespace cospdnn
