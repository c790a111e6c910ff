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
