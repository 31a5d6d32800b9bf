// gx_dop853_nystrom.cuh -- generated by gen_dop853_nystrom.py; do not edit.
// DOP853 for x' = v, v' = a(x): nIJ = (A^2)_IJ, nbJ = (b A)_J, nerJ = (er A)_J,
// nbhJ = ((b - bhh) A)_J, ncI = sum_J a_IJ.
#pragma once

namespace gx {
namespace dop {
constexpr double nc2 = 0x1.aee6838dae63ap-5;
constexpr double nc3 = 0x1.432ce2aa42cacp-4;
constexpr double n3_1 = 0x1.97fa4bd857c3ap-9;
constexpr double nc4 = 0x1.e4c353ff64302p-4;
constexpr double n4_1 = 0x1.caf9955362bc1p-10;
constexpr double n4_2 = 0x1.583b2ffe8a0d1p-8;
constexpr double nc5 = 0x1.2068c499c08d9p-2;
constexpr double n5_1 = 0x1.44ebe53a4526dp-7;
constexpr double n5_2 = -0x1.accbfefe6d3edp-5;
constexpr double n5_3 = 0x1.503e7575108dfp-4;
constexpr double nc6 = 0x1.5555555555555p-2;
constexpr double n6_1 = 0x1.217d036868b4cp-5;
constexpr double n6_3 = -0x1.8879abc79e49bp-4;
constexpr double n6_4 = 0x1.db4962f6f8284p-4;
constexpr double nc7 = 0x1.0000000000000p-2;
constexpr double n7_1 = 0x1.35fe4221648cap-6;
constexpr double n7_3 = -0x1.388b7e0e7b3ffp-5;
constexpr double n7_4 = 0x1.af9d9aa51cc97p-5;
constexpr double n7_5 = -0x1.2113da753cfcep-9;
constexpr double nc8 = 0x1.3b13b13b13b14p-2;
constexpr double n8_1 = 0x1.f68031439116bp-6;
constexpr double n8_3 = -0x1.46acff29807b4p-4;
constexpr double n8_4 = 0x1.915f39fadea93p-4;
constexpr double n8_5 = -0x1.7542aa816a524p-10;
constexpr double n8_6 = -0x1.3101454da6cdfp-13;
constexpr double nc9 = 0x1.4d74d74d74d75p-1;
constexpr double n9_1 = -0x1.37e44a3a3d286p-3;
constexpr double n9_3 = 0x1.e0eec7f1761d7p-2;
constexpr double n9_4 = -0x1.171b710b3b662p-4;
constexpr double n9_5 = 0x1.5f0192e399b99p-7;
constexpr double n9_6 = 0x1.3f75068de373cp-2;
constexpr double n9_7 = -0x1.707642fcde52bp-2;
constexpr double nc10 = 0x1.3333333333333p-1;
constexpr double n10_1 = -0x1.c36897302cb72p-4;
constexpr double n10_3 = 0x1.34853e327dabcp-2;
constexpr double n10_4 = 0x1.422e368da0510p-4;
constexpr double n10_5 = 0x1.f9439ccc790f3p-6;
constexpr double n10_6 = -0x1.47464f4598605p-2;
constexpr double n10_7 = -0x1.5ecf653d1571ep-1;
constexpr double n10_8 = 0x1.c4b612b71fecap-1;
constexpr double nc11 = 0x1.b6db6db6db6dbp-1;
constexpr double n11_1 = 0x1.7d1f3e8130efap-2;
constexpr double n11_3 = -0x1.029902a47a1c0p-1;
constexpr double n11_4 = -0x1.d893209d33c96p-2;
constexpr double n11_5 = -0x1.0aff864b4e24bp-4;
constexpr double n11_6 = 0x1.064642de96f87p+2;
constexpr double n11_7 = 0x1.f233f254578bcp+1;
constexpr double n11_8 = -0x1.c19e285005301p+2;
constexpr double n11_9 = 0x1.fb72c96a00a96p-5;
constexpr double nc12 = 0x1.0000000000000p+0;
constexpr double n12_1 = -0x1.87b7e9647bf30p-1;
constexpr double n12_3 = 0x1.ab6ad6747361bp-1;
constexpr double n12_4 = 0x1.c1858e30e981dp+0;
constexpr double n12_5 = 0x1.dc3c5a4906312p-3;
constexpr double n12_6 = 0x1.7ceb44dbdbac1p+3;
constexpr double n12_7 = -0x1.e74b71c5bf258p+0;
constexpr double n12_8 = -0x1.5e707259e25a6p+3;
constexpr double n12_9 = 0x1.5a624e7cc0091p+0;
constexpr double n12_10 = -0x1.f5d400c8d1709p+0;
constexpr double nb1 = 0x1.bcc6368d1177cp-5;
constexpr double nb6 = 0x1.7bc2918e723d8p+1;
constexpr double nb7 = 0x1.6b2be346040b7p+0;
constexpr double nb8 = -0x1.0109b7c05dbccp+2;
constexpr double nb9 = 0x1.bc738374d6d62p-4;
constexpr double nb10 = -0x1.f299db205e669p-5;
constexpr double nb11 = 0x1.d74f62f6d9a7dp-6;
constexpr double ner1 = -0x1.825beab80ca51p-3;
constexpr double ner4 = 0x1.fe0fe8f118cc8p-1;
constexpr double ner5 = 0x1.e352b7cd95f78p-3;
constexpr double ner6 = -0x1.6d6489c76d7b6p+1;
constexpr double ner7 = -0x1.054cbd65f2e73p+2;
constexpr double ner8 = 0x1.8274300ebeaafp+2;
constexpr double ner9 = 0x1.95587b9df5488p-2;
constexpr double ner10 = -0x1.0d460aa2428f6p-1;
constexpr double ner11 = -0x1.d74f62f6d9a7dp-7;
constexpr double nbh1 = -0x1.d0bf40d812c55p-2;
constexpr double nbh4 = 0x1.5970eb2982213p+1;
constexpr double nbh5 = 0x1.5cd04f410d935p-1;
constexpr double nbh6 = -0x1.0e2a5d3ab05f5p+4;
constexpr double nbh7 = -0x1.bf9cafd65a23fp+3;
constexpr double nbh8 = 0x1.bf6359ba252c3p+4;
constexpr double nbh9 = 0x1.3788f4dcb4394p-2;
constexpr double nbh10 = -0x1.55874d65582b7p-2;
constexpr double nbh11 = 0x1.dd8f901379b8ep-7;
}  // namespace dop
}  // namespace gx

