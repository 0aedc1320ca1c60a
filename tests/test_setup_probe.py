"""Properties of the set-up kernels' data that need no GPU."""
import probe


def test_inverse_candidates_are_aligned_for_their_vector_access():
    # a candidate moves through memory as one 16-byte access
    assert probe.load("setup_probe").probe_inv_cand_align() == 16
