"""CPU suite: offsets into val_arr are checked one by one, not only the last of an array: the kernels, and the host when it lays a
group out by column tiles, walk from every entry to the next."""
import numpy as np
import pytest

import specs
from alphasparse_b200 import capi, matrices as M
from alphasparse_b200.graph import Matrix
from test_plan_validate_cpu import _array_of, _expect_bounds


def descs_of(spec):
    m, _ = M.from_row_lengths(np.random.default_rng(3).integers(1, 400, size=300), 2_000, seed=3)
    fmt = Matrix.from_csr(m).execute(specs.full_spec(spec))
    descs = fmt.plan_descs()
    capi.validate_descs(descs)
    return fmt, descs


@pytest.mark.parametrize("spec,role", [("S4_K4", "global_warp_nz_begin_offset"), ("S8_K7", "block_nz_begin_offset"), ("S6_K8", "global_warp_block_first_nz")])
@pytest.mark.parametrize("entry", [1, 37, -2])
def test_an_inner_offset_beyond_the_values_is_rejected(spec, role, entry):
    fmt, descs = descs_of(spec)
    _, off = _array_of(descs[0], role)
    if off is None:  # equal chunks, a closed form: the same offsets as an array
        a = next(descs[0].arrays[k] for k in range(descs[0].n_arrays) if descs[0].arrays[k].role == capi.ROLE[role])
        off = (np.arange(a.len) * a.coef + a.icpt).astype(np.uint32)
        a.host_ptr, a.dtype, a.compress = off.ctypes.data, capi.U32, capi.COMPRESS["none"]
    off[entry] = int(off[-1])
    capi.validate_descs(descs)  # out of order, but inside val_arr: its unit takes more elements, the next one none
    off[entry] = np.iinfo(off.dtype).max
    _expect_bounds(descs, "an nz offset outside val_arr")
    fmt.close()


@pytest.mark.parametrize("spec", ["X_K1", "X_K5"])
@pytest.mark.parametrize("role,needle", [("warp_nz_begin_offset", "a WLB reaches outside"), ("warp_begin_thread_index_offset", "a WLB reaches outside"),
                                         ("thread_block_size_in_warp", "a WLB reaches outside"), ("block_nz_begin_offset", "a WLB reaches outside")])
def test_a_wlb_beyond_the_values_is_rejected(spec, role, needle):
    fmt, descs = descs_of(spec)
    a = next(descs[0].arrays[k] for k in range(descs[0].n_arrays) if descs[0].arrays[k].role == capi.ROLE[role])
    _, arr = _array_of(descs[0], role)
    if arr is None:
        a.icpt += 1 << 40
    else:
        arr[len(arr) // 2] = np.iinfo(arr.dtype).max
        if int(arr.max()) * 64 < 1_000_000:
            pytest.skip("the narrowed type cannot express a value that reaches outside")
    _expect_bounds(descs, needle)
    fmt.close()


@pytest.mark.parametrize("spec,role", [("S1_K2", "thread_block_size_in_block"), ("S2_K6", "thread_block_size_in_block"), ("X_K1", "thread_block_size_in_warp"), ("X_K5", "thread_block_size_in_warp")])
def test_too_few_tlb_sizes_are_rejected(spec, role):
    fmt, descs = descs_of(spec)
    a = next(descs[0].arrays[k] for k in range(descs[0].n_arrays) if descs[0].arrays[k].role == capi.ROLE[role])
    sizes = np.full(a.len, a.icpt if a.compress else 1, dtype=np.uint32)
    _, arr = _array_of(descs[0], role)
    if arr is not None:
        sizes[:] = arr
    a.host_ptr, a.dtype, a.compress = sizes.ctypes.data, capi.U32, capi.COMPRESS["none"]
    capi.validate_descs(descs)
    a.len -= 1
    _expect_bounds(descs, "fewer TLB sizes")
    fmt.close()
