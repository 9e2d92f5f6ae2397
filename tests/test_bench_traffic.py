"""The bench's measured DRAM bytes of the spikes' back substitution, against
the FP32 tiles that kernel must move per 64-row block (checked without a GPU)."""
import bench


def test_back_substitution_reads_its_tiles_once_for_both_spikes():
    # G and E in once for V and W together, the one forward-swept spike in, both out
    need = 5 * 64 * 64 * 4
    assert 0.9 * need <= bench.TRAFFIC_PER_BLOCK["factor_bwd"] <= 1.1 * need
