"""Tag reading where coordinates fall on the borders between pixels: quads along
the axes with corners on whole, half and quarter pixels put sample points
there, and which pixel a point takes is decided by the last bit of its FP64
coordinate.  The expected values are those of the FP64 form of every
coordinate, on an image where any other pixel shows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _image():
    y, x = np.mgrid[0:480, 0:640].astype(np.uint32)
    h = (x * np.uint32(73856093)) ^ (y * np.uint32(19349663))
    return ((h >> np.uint32(9)) & np.uint32(255)).astype(np.uint8)


def _decode(quads, width_at_border, refine):
    from atag import decode
    k = width_at_border - 2
    layout = type("Layout", (), {"width_at_border": width_at_border, "total_width": k,
                                 "bit_x": [1 + i % k for i in range(k * k)], "bit_y": [1 + i // k for i in range(k * k)]})
    prm = decode.default_params(refine_edges=refine, min_contrast=-300.0)
    q = torch.tensor(quads, dtype=torch.float32, device="cuda")
    return decode.to_numpy(decode.decode_quads(torch.from_numpy(_image()).cuda(), q,
                                               decode.Family(layout, [0x123456789]), prm))


# (quad, refined corners)
REFINED = [
    ([[30, 268], [206, 268], [206, 299], [30, 299]],
     [[29.5945, 267.1528], [206.6676, 267.4542], [206.3956, 299.0972], [28.4088, 299.0718]]),
    ([[31, 240], [148, 240], [148, 286], [31, 286]],
     [[32.0146, 239.9839], [148.7122, 239.5666], [146.7792, 286.0], [30.4956, 286.0174]]),
    ([[307, 15], [344, 15], [344, 58], [307, 58]],
     [[307.7519, 14.7825], [342.0498, 15.4942], [343.7642, 58.0261], [308.1022, 57.4748]]),
    ([[94, 375], [125.5, 375], [125.5, 397.5], [94, 397.5]],
     [[94.304, 374.4409], [124.8842, 374.0246], [124.8193, 397.8622], [94.3586, 397.1411]]),
    ([[132, 229], [165.5, 229], [165.5, 254.5], [132, 254.5]],
     [[131.585, 228.5708], [165.7962, 229.1867], [166.3259, 253.7196], [132.4828, 255.2613]]),
    ([[63, 10], [137.5, 10], [137.5, 30], [63, 30]],
     [[63.779, 9.5316], [138.5458, 9.7067], [138.0433, 29.9754], [63.7589, 29.1929]]),
    ([[281, 15], [316.25, 15], [316.25, 23.25], [281, 23.25]],
     [[281.0542, 15.8107], [314.75, 15.6326], [314.75, 23.8479], [280.9715, 23.5965]]),
    ([[11, 92], [30, 92], [30, 116.25], [11, 116.25]],
     [[11.7199, 92.5247], [30.8214, 91.7866], [29.1557, 115.3245], [10.4092, 116.9735]]),
    ([[56, 27], [68.75, 27], [68.75, 62], [56, 62]],
     [[55.8215, 28.1456], [67.275, 27.4271], [68.6398, 61.1818], [56.167, 62.5261]]),
    ([[14, 139], [99, 138], [96, 215], [14, 217]],
     [[13.962, 139.5899], [98.5714, 138.1117], [96.7597, 213.9476], [11.9196, 217.8245]]),
    ([[15, 149], [77, 154], [81, 213], [15, 212]],
     [[15.6158, 149.1256], [75.9121, 153.9801], [82.1537, 215.0484], [15.6102, 210.5847]]),
]


def test_edges_walked_along_pixel_borders():
    g = _decode([q for q, _ in REFINED], 8, 1)
    # the values above are rounded to 1e-4
    assert np.abs(g["corners"] - np.array([c for _, c in REFINED])).max() <= 1e-3


# (cells of a side, quad, white, black)
MODELS = [
    (8, [[233, 351], [311, 350], [307, 370], [230, 366]], 139.84375, 148.0),
    (7, [[74, 339], [270, 339], [270, 400], [74, 400]], 133.25, 124.67857),
    (7, [[52, 164], [248, 164], [248, 267], [52, 267]], 102.5, 131.07143),
    (7, [[39, 70], [218, 70], [218, 252], [39, 252]], 127.57143, 130.10715),
    (7, [[190, 13], [262, 13], [262, 97], [190, 97]], 119.57143, 141.0),
    (6, [[9, 398], [81, 398], [81, 443], [9, 443]], 116.58334, 115.91666),
    (6, [[33, 321], [153, 321], [153, 344], [33, 344]], 145.91667, 97.5),
    (6, [[43, 35], [143, 35], [143, 167], [43, 167]], 108.66666, 149.16667),
    (6, [[39, 29], [231, 29], [231, 102], [39, 102]], 104.66666, 152.25),
]


@pytest.mark.parametrize("width", [6, 7, 8])
def test_grey_model_samples_on_pixel_borders(width):
    rows = [m for m in MODELS if m[0] == width]
    g = _decode([m[1] for m in rows], width, 0)
    # a sample's grey value changes a model by at least 1 / 32 of a grey level
    assert np.abs(g["white"] - [m[2] for m in rows]).max() <= 1e-3
    assert np.abs(g["black"] - [m[3] for m in rows]).max() <= 1e-3
