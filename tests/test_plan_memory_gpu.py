"""GPU test of the device memory that plans keep: tables in proportion to the axes'
lengths."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(4000, 2, 2), (2, 3969, 2), (2, 2, 4096)])
def test_plans_keep_their_tables_only(torch_cuda, ff, n):
    torch = torch_cuda
    ff.Plan(n)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    plans = [ff.Plan(n) for _ in range(32)]
    torch.cuda.synchronize()
    used = free0 - torch.cuda.mem_get_info()[0]
    # per plan: at most 2 twiddle tables of about 16 bytes a point with some padding
    # of odd radices, three integer tables and 16 KB steps: 2 * 1.5 * 16 + 3 * 4 = 60
    # bytes a point, and the allocator's 2 MB pages shared by several
    per_point = 60
    assert used <= 32 * (per_point * max(n) + 64 * 1024) + (2 << 20), used
    assert len(plans) == 32
