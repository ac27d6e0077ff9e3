// Lattice and all-cohort instantiations of the tensor-memory tile kernel.
#include "tile_tc_launch.cuh"
#include "tile_tc_nvq.cuh"

namespace mfqb {

cudaError_t launch_tile_nvq(const TileArgs& a, const TilePlan& p, int terms, cudaStream_t stream) {
    const NintDevB& w = a.pools[0];
    if (!w.jsc) return w.index_bits == 8 ? launch_tile<TileOne<TileNvq<8, false, 1>>>(a, p, stream) : cudaErrorNotSupported;
    switch (w.index_bits * 2 + terms - 1) {
        case 16: return launch_tile<TileOne<TileNvq<8, true, 1>>>(a, p, stream);
        case 17: return launch_tile<TileOne<TileNvq<8, true, 2>>>(a, p, stream);
        case 18: return launch_tile<TileOne<TileNvq<9, true, 1>>>(a, p, stream);
        case 19: return launch_tile<TileOne<TileNvq<9, true, 2>>>(a, p, stream);
        case 20: return launch_tile<TileOne<TileNvq<10, true, 1>>>(a, p, stream);
        case 21: return launch_tile<TileOne<TileNvq<10, true, 2>>>(a, p, stream);
        default: return cudaErrorNotSupported;
    }
}

// Every cohort of an expert record in one launch: the codecs of the per-expert precision profiles.
template <int TERMS_, int XTERMS_>
struct TileExperts {
    static constexpr bool ONE = false;
    static constexpr int TERMS = TERMS_, XTERMS = XTERMS_;
    template <class Fn>
    __device__ static __forceinline__ void dispatch(const NintDevB& w, Fn&& f) {
        switch (w.bits * 16 + w.t8) {
            case 2 * 16 + 2: f(TileNint<2, 2, TERMS>{}); break;
            case 3 * 16 + 3: f(TileNint<3, 3, TERMS>{}); break;
            case 4 * 16 + 3: f(TileNint<4, 3, TERMS>{}); break;
            case 5 * 16 + 4: f(TileNint<5, 4, TERMS>{}); break;
            case 6 * 16 + 3: f(TileNint<6, 3, TERMS>{}); break;
            case 8 * 16 + 3: f(TileNint<8, 3, TERMS>{}); break;
            case 8 * 16 + 6: f(TileNint<8, 6, TERMS>{}); break;
            default: break;
        }
    }
    __device__ static void ctx_init(unsigned char*, const TileArgs&, int, int) {}
};
cudaError_t launch_tile_experts(const TileArgs& a, const TilePlan& p, int terms, int x_terms, cudaStream_t stream) {
    if (terms == 1) return launch_tile_form<TileExperts<1, 1>, false>(a, p, stream);
    return x_terms == 1 ? launch_tile_form<TileExperts<2, 1>, false>(a, p, stream) : launch_tile_form<TileExperts<2, 2>, false>(a, p, stream);
}

}  // namespace mfqb
