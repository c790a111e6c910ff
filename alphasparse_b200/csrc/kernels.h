// Launch entry of the kernel families (kernels.cu); used by the C ABI only.
#ifndef ASP_KERNELS_H
#define ASP_KERNELS_H
#include <cuda_runtime.h>
#include "kernel_args.h"
namespace asp
{
// templ: asp_template_type; vec: TLBs handled per thread by the ELL-like / SELL-like families
cudaError_t launch_template(int templ, int val_is_f64, int col_width, const KArgs &a, unsigned grid, unsigned block, size_t smem, cudaStream_t st, int vec);
cudaError_t allow_dynamic_smem(int templ, int val_is_f64, int col_width, size_t smem);
// CSR5-like family specialised on the TLB size (kernels_csr5.cu). mode: bit 0 = the second template's whole-warp
// fast path, bit 1 = staged contiguous write-out, bit 2 = write-out through KArgs::y_mc (needs bit 1).
bool csr5_specialised(int tlb_size, int col_width, int bits_word);
cudaError_t launch_csr5(int val_is_f64, int col_width, int mode, const KArgs &a, unsigned grid, unsigned block, cudaStream_t st);
// block-value template (kernels_block.cu): blocked ELL over dense r x c blocks; KArgs::n_tlb = padded block rows,
// tlb_size = block slots per block row, effective = rows of the sub-matrix
bool block_ell_supported(int r, int c);
cudaError_t launch_block_ell(int val_is_f64, int r, int c, const KArgs &a, unsigned block, cudaStream_t st);
// diagonal-value template (kernels_diag.cu): KArgs::col = u64 offsets biased by the column count, n_tlb = padded rows,
// tlb_size = diagonals, effective = rows, n_units = columns of the sub-matrix
cudaError_t launch_diag(int val_is_f64, const KArgs &a, unsigned grid, unsigned block, cudaStream_t st);
// y[0, n) = 0 (kernels_tiled.cu)
cudaError_t launch_clear(int val_is_f64, void *y, unsigned long long n, unsigned n_sm, cudaStream_t st);
// end rows of the warps (the rows the CSR5-like kernel accumulates with `red`): cleared before, published after
cudaError_t launch_zero_rows(int val_is_f64, void *y, const unsigned *rows, unsigned long long n, cudaStream_t st);
cudaError_t launch_publish_rows(int val_is_f64, const void *y, void *y_mc, const unsigned *rows, unsigned long long n, cudaStream_t st);
// whole rows whose elements lie one after the other (kernels_rows.cu): rows[i] = {first element, row of y}, rows[n].x = where the last row
// ends; cta: threads of a CTA per row, 0: a warp per row
struct RowArgs
{
    const void *val, *col, *x;
    void *y;
    const uint2 *rows;
    const uint4 *tlbs; // row-grouped, instead: {first element, row of y, TLBs | elements of one << 16, distance of a TLB's elements}
    const uint4 *strips; // ELL- and SELL-like, instead: groups of up to 32 TLBs side by side, a TLB a row: {first element, first TLB, elements of a TLB |
                         // TLBs << 16, distance of a TLB's elements}; `place` rows of y by TLB (NULL: as numbered, from first_row on)
    const unsigned *place;
    unsigned first_row;
    const uint4 *runs; // CSR5-like, instead: {first element, row of y, elements, 0}, the first `hubs` of them for a CTA each; TLBs of `size`
    unsigned hubs, size;
    unsigned n, cta, lanes; // lanes: of a row with TLBs; warps of a group of them
};
cudaError_t launch_own_rows(int val_is_f64, int col_width, const RowArgs &a, cudaStream_t st);
} // namespace asp
#endif
