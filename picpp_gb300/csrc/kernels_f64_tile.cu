// FP64 instantiation of the per-tile particle kernels, with fused
// multiply-adds: their time is the number of FP64 instructions.
#include "kernels_tile_impl.cuh"
namespace pic {
template size_t PK<double>::tile_smem_bytes(const TileShape&, bool);
template void PK<double>::push_deposit_tiled(cudaStream_t, const GridP&, const TileGeom&, const TileGeom&, const TileShape&,
                                             const SpeciesSet<double>&, const void*, const void*, double*, int);
template float PK<double>::fixed_scale(const GridP&, const SpeciesSet<double>&);
template void PK<double>::assemble_j(cudaStream_t, const GridP&, const TileGeom&, const TileShape&, const double*,
                                     const double*, double*, double, int);
template ImpBlock PK<double>::implicit_block(const GridP&, const TileGeom&, int, bool);
template size_t PK<double>::implicit_tile_smem(const ImpBlock&, int, int);
template void PK<double>::implicit_deposit_tiled(cudaStream_t, const GridP&, const TileGeom&, const TileGeom&,
                                                 const ImpBlock&, const ImpSpecies<double>&, const double*, const double*,
                                                 double*, double*, double*, double*);
template bool PK<double>::implicit_push_tiled(cudaStream_t, const GridP&, const TileGeom&, const TileGeom&, const ImpSpecies<double>&,
                                              const double*, const double*, const double*);
}  // namespace pic
