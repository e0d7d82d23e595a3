"""Shapes that take the prefill kernel on pairs of SMs through each form of its work, on 74 pairs (a B200): tokens, weight rows, k,
then tokens per tile T, row tiles per item R and how the items left over after whole waves run: "whole"; "parts": all tiles split
by k, no pair on two of them; "straddle": the same with parts that straddle tiles; "tail": split behind whole waves.
test_pair_cpu.py checks that each takes the form it names, test_prefill_pair_gpu.py runs them.  Rows and tokens are ragged; with
R = 2 the number of row tiles is odd but in the last one, so half an item lies beyond the weight (split: a part of zeros)."""

FP4 = [
    (130, 19056, 256, 160, 2, "whole"),       # one stage an item: rings and accumulators run across items
    (161, 19104, 256, 192, 2, "whole"),
    (65, 19488, 256, 96, 2, "whole"),
    (17, 1600, 16128, 32, 1, "parts"),
    (38, 1632, 13056, 64, 1, "parts"),
    (72, 264, 16640, 32, 1, "parts"),
    (200, 1056, 5888, 128, 1, "parts"),
    (303, 1608, 4096, 160, 1, "parts"),
    (174, 2208, 8704, 192, 1, "parts"),
    (1314, 8, 4096, 96, 1, "parts"),
    (199, 4992, 8448, 128, 1, "straddle"),
    (17, 10368, 8960, 32, 1, "straddle"),
    (214, 9536, 4096, 96, 1, "tail"),
    (869, 3608, 3584, 128, 1, "tail"),
    (2474, 1344, 4096, 160, 1, "tail"),
    (1645, 2064, 4608, 192, 1, "tail"),
    (235, 19520, 2560, 128, 2, "tail"),
    (783, 7744, 3072, 160, 2, "tail"),
    (1740, 3600, 3840, 192, 2, "tail"),
]

BF16 = [
    (163, 19000, 256, 192, 2, "whole"),
    (194, 19048, 256, 224, 2, "whole"),
    (129, 19584, 1024, 160, 2, "whole"),      # units of 64 k, several stages, an odd number of row tiles
    (391, 9232, 1024, 160, 2, "whole"),       # units of 128 k from here on
    (484, 19488, 1024, 192, 2, "whole"),
    (649, 19144, 1024, 224, 2, "whole"),
    (327, 19152, 5376, 192, 2, "tail"),       # 4 of 152 tiles in parts
    (387, 19136, 6656, 224, 2, "tail"),
    (327, 21080, 6400, 192, 2, "tail"),       # 20 of 168: units of 64 k
    (643, 15208, 5120, 224, 2, "tail"),
    (86, 552, 7424, 32, 1, "parts"),
    (194, 616, 4096, 64, 1, "parts"),
    (150, 1784, 4096, 96, 1, "parts"),
    (105, 2208, 8448, 128, 1, "parts"),
    (142, 2104, 8448, 160, 1, "parts"),
    (98, 9696, 11776, 128, 1, "straddle"),
    (17, 19976, 5120, 32, 1, "tail"),
    (512, 14336, 8192, 128, 2, "tail"),
]
