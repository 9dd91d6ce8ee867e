"""CPU: the captured runs that a stretch of plain iterations is replayed in. Each
costs a graph launch, so runs of 2, 4, 16 and 64 alone are not enough: eight
iterations between two Monitor outputs, or in a call, are one launch, as with runs of
2 and 8, and no stretch needs more launches than those took."""


def test_no_more_launches_than_runs_of_2_and_8(built):
    import imexlb as im
    run = im.lib().imexlb_testing_graph_run

    def launches(n):
        k = 0
        while run(n):
            n -= run(n)
            k += 1
        return k + n

    assert run(0) == run(1) == 0 and run(8) == 8
    for n in range(1, 200):
        assert run(n) <= n and run(n) % 2 == 0
        assert launches(n) <= n // 8 + n % 8 // 2 + n % 2
