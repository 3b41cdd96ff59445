// The batched lattice step kernel, instantiated per storage form in batch_step_f32.cu,
// batch_step_f16.cu and batch_step_bf16.cu (FSI_BATCH_STEP_STORAGE, FSI_BATCH_STEP_NAME),
// so that the forms' many template instances compile in parallel.
#include "batch_types.cuh"

namespace fsi {
namespace {

struct BatchStepArgs {
  const BatchLattice* lat;
  const Tile* tiles;
  int reps;  // passes of kStepBlock * lanes cells over the tile
  void* pops;
  float* macro;
  const float* force;
  const float* force_prev;
  const uint32_t* flags;
  bool pairs;  // every lattice has an even number of cells, the arrays are aligned (even_pairs)
};

// Minimum resident blocks per SM of register-cap variant kVar (0..2), 1 being the default.
// Measured on 64 scenes with tiles of 1,024 cells, us per step, by blocks. FP16, even: 606 at 4,
// 570 at 6, 572 at 8 (rho and u read); odd: 650 at 4, 851 at 5, 967 at 6 (spills), and with rho and
// u recomputed 669, 649, 740. FP32 exact, even: 906 at 4, 928 at 6, 808 at 8; odd: 927 at 6, 903 at 8.
template <bool kFast, bool kOdd, bool kRecompute, int kVar>
constexpr int batch_min_blocks() {
  if (kFast && kOdd) return kVar == 0 ? 4 : kVar == 1 ? (kRecompute ? 5 : 4) : 6;
  if (kFast) return kVar == 0 ? 4 : kVar == 1 ? 6 : 8;
  return !kOdd ? (kVar == 0 ? 4 : kVar == 1 ? 8 : 6) : (kVar == 0 ? 6 : 8);
}

// kStepBlock threads cover a tile of reps * kStepBlock * lanes cells: the exact form takes
// one cell per thread and pass, the fast forms two (the packed lanes; kPairs: neighbours in memory,
// on even steps of lattices that allow it, see step_even_pair).
template <int kStore, bool kFast, bool kOdd, bool kRecompute, int kVar, bool kPairs>
__global__ void __launch_bounds__(kStepBlock, (batch_min_blocks<kFast, kOdd, kRecompute, kVar>()))
    batch_step_kernel(BatchStepArgs b) {
  constexpr int NL = StepLanes<kFast>::n;
  const int kReps = b.reps;
  const Tile t = b.tiles[blockIdx.x];
  const BatchLattice& L = b.lat[t.lattice];
  __shared__ Rates rates;
  load_rates(L, rates);
  __syncthreads();
  const LatticeView v = view_of<kStore>(L, rates, b.pops, b.macro, b.force, b.force_prev, b.flags);
  for (int r = 0; r < kReps; ++r) {
    if constexpr (kPairs) {
      const uint32_t c = 2 * (uint32_t)(t.first + r * kStepBlock + threadIdx.x);
      if (c < (uint32_t)L.g.n) step_even_pair<kStore, kRecompute, LatticeView>(v, c);
      continue;
    }
    int ci[NL], cj[NL], ck[NL];
    bool has[NL];
    if (step_unit<NL>(L.g, (long long)t.first + r * kStepBlock + threadIdx.x, ci, cj, ck, has))
      step_cells<kStore, kFast, kOdd, kRecompute, LatticeView>(v, ci, cj, ck, has);
  }
}

template <int S, bool F, int V>
void launch_variant(const BatchStepArgs& a, int ntiles, bool odd, bool recompute, cudaStream_t s) {
  if constexpr (F) {
    if (!odd && a.pairs) {
      if (recompute) batch_step_kernel<S, F, false, true, V, true><<<ntiles, kStepBlock, 0, s>>>(a);
      else batch_step_kernel<S, F, false, false, V, true><<<ntiles, kStepBlock, 0, s>>>(a);
      return;
    }
  }
  if (recompute) {
    if (odd) batch_step_kernel<S, F, true, true, V, false><<<ntiles, kStepBlock, 0, s>>>(a);
    else batch_step_kernel<S, F, false, true, V, false><<<ntiles, kStepBlock, 0, s>>>(a);
  } else {
    if (odd) batch_step_kernel<S, F, true, false, V, false><<<ntiles, kStepBlock, 0, s>>>(a);
    else batch_step_kernel<S, F, false, false, V, false><<<ntiles, kStepBlock, 0, s>>>(a);
  }
}

template <int S, bool F>
void launch_form(const BatchStepArgs& a, int ntiles, int variant, bool odd, bool recompute,
                 cudaStream_t s) {
  if (variant == 0) launch_variant<S, F, 0>(a, ntiles, odd, recompute, s);
  else if (variant == 2) launch_variant<S, F, 2>(a, ntiles, odd, recompute, s);
  else launch_variant<S, F, 1>(a, ntiles, odd, recompute, s);
}

}  // namespace

int FSI_BATCH_STEP_NAME(const void* lat, const void* tiles, int ntiles, int tile_cells,
                        int variant, bool fast, bool odd, bool recompute, bool even_cells, void* pops,
                        float* macro, const float* force, const float* force_prev,
                        const uint32_t* flags, cudaStream_t stream) {
  BatchStepArgs a{static_cast<const BatchLattice*>(lat), static_cast<const Tile*>(tiles), 0,
                  pops, macro, force, force_prev, flags,
                  even_cells && even_pairs(0, pops, flags, force, force_prev)};
  a.reps = tile_cells / (kStepBlock * (fast ? 2 : 1));
#if FSI_BATCH_STEP_STORAGE == FSI_STORAGE_F32
  if (fast) launch_form<FSI_STORAGE_F32, true>(a, ntiles, variant, odd, recompute, stream);
  else launch_form<FSI_STORAGE_F32, false>(a, ntiles, variant, odd, recompute, stream);
#else
  launch_form<FSI_BATCH_STEP_STORAGE, true>(a, ntiles, variant, odd, recompute, stream);
#endif
  return check_launch("batch_step_kernel");
}

}  // namespace fsi
