"""Workspace sizes of the split form, from the shapes alone (no GPU needed)."""


def test_full_workspace_size(fmm):
    f = fmm.strassen_fmm()
    for fmt, s in (("bf16", 6), ("fp8", 10)):
        for m, n, k in ((300, 700, 450), (64, 64, 64), (1, 1, 1), (1100, 260, 300)):
            plain = fmm.split_workspace_size(m, n, k, None, 0, s, fmt)
            assert plain < fmm.split_workspace_size(m, n, k, None, 0, s, fmt, full=True) <= plain + (128 << 20)
            assert (fmm.split_workspace_size(m, n, k, f, 1, s, fmt, full=True)
                    == fmm.split_workspace_size(m, n, k, f, 1, s, fmt))
        for m, n, k in ((0, 5, 5), (5, 0, 5), (5, 5, 0), (8192, 8192, 100)):
            assert (fmm.split_workspace_size(m, n, k, None, 0, s, fmt, full=True)
                    == fmm.split_workspace_size(m, n, k, None, 0, s, fmt))
    assert fmm.split_workspace_size(64, 64, 64, None, 0, 9, full=True) == 0
