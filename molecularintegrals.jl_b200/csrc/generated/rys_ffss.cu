// Generated by gen_rys.py -- Rys class (ff|ss).  Do not edit.
// roots 4, block 74 x 1, outputs 100 x 1, group 32 threads, 4 ket pairs a round,
// 2 primitive quartets per ket pair and batch, 25600 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_ffss {
    static constexpr int LA = 3, LB = 3, LC = 0, LD = 0;
    static constexpr int E = 6, F = 0, NR = 4;
    static constexpr int NA = 74, NC = 1, NBLK = 74;
    static constexpr int NB = 10, ND = 1;
    static constexpr int NAB = 100, NCD = 1;
    static constexpr int G = 32, W = 4, H = 8, PB = 2;
    static constexpr int S = 7, SI = 21, NCP = 1, NCDP = 1;
    static constexpr int SMEM_GROUP = 800;
    // stage 2: acc[row] += x[ax] y[ay] z[az] for the column's table columns
    template <typename T, typename A>
    __device__ __forceinline__ static void col_update(const T *x, const T *y, const T *z, A *acc) {
        acc[0] = fma(x[3] * y[0], z[0], acc[0]);
        acc[1] = fma(x[2] * y[1], z[0], acc[1]);
        acc[2] = fma(x[2] * y[0], z[1], acc[2]);
        acc[3] = fma(x[1] * y[2], z[0], acc[3]);
        acc[4] = fma(x[1] * y[0], z[2], acc[4]);
        acc[5] = fma(x[1] * y[1], z[1], acc[5]);
        acc[6] = fma(x[0] * y[3], z[0], acc[6]);
        acc[7] = fma(x[0] * y[2], z[1], acc[7]);
        acc[8] = fma(x[0] * y[1], z[2], acc[8]);
        acc[9] = fma(x[0] * y[0], z[3], acc[9]);
        acc[10] = fma(x[4] * y[0], z[0], acc[10]);
        acc[11] = fma(x[3] * y[1], z[0], acc[11]);
        acc[12] = fma(x[3] * y[0], z[1], acc[12]);
        acc[13] = fma(x[2] * y[2], z[0], acc[13]);
        acc[14] = fma(x[2] * y[1], z[1], acc[14]);
        acc[15] = fma(x[2] * y[0], z[2], acc[15]);
        acc[16] = fma(x[1] * y[3], z[0], acc[16]);
        acc[17] = fma(x[1] * y[2], z[1], acc[17]);
        acc[18] = fma(x[1] * y[1], z[2], acc[18]);
        acc[19] = fma(x[1] * y[0], z[3], acc[19]);
        acc[20] = fma(x[0] * y[4], z[0], acc[20]);
        acc[21] = fma(x[0] * y[3], z[1], acc[21]);
        acc[22] = fma(x[0] * y[2], z[2], acc[22]);
        acc[23] = fma(x[0] * y[1], z[3], acc[23]);
        acc[24] = fma(x[0] * y[0], z[4], acc[24]);
        acc[25] = fma(x[5] * y[0], z[0], acc[25]);
        acc[26] = fma(x[4] * y[1], z[0], acc[26]);
        acc[27] = fma(x[4] * y[0], z[1], acc[27]);
        acc[28] = fma(x[3] * y[2], z[0], acc[28]);
        acc[29] = fma(x[3] * y[1], z[1], acc[29]);
        acc[30] = fma(x[3] * y[0], z[2], acc[30]);
        acc[31] = fma(x[2] * y[3], z[0], acc[31]);
        acc[32] = fma(x[2] * y[2], z[1], acc[32]);
        acc[33] = fma(x[2] * y[1], z[2], acc[33]);
        acc[34] = fma(x[2] * y[0], z[3], acc[34]);
        acc[35] = fma(x[1] * y[4], z[0], acc[35]);
        acc[36] = fma(x[1] * y[3], z[1], acc[36]);
        acc[37] = fma(x[1] * y[2], z[2], acc[37]);
        acc[38] = fma(x[1] * y[1], z[3], acc[38]);
        acc[39] = fma(x[1] * y[0], z[4], acc[39]);
        acc[40] = fma(x[0] * y[5], z[0], acc[40]);
        acc[41] = fma(x[0] * y[4], z[1], acc[41]);
        acc[42] = fma(x[0] * y[3], z[2], acc[42]);
        acc[43] = fma(x[0] * y[2], z[3], acc[43]);
        acc[44] = fma(x[0] * y[1], z[4], acc[44]);
        acc[45] = fma(x[0] * y[0], z[5], acc[45]);
        acc[46] = fma(x[6] * y[0], z[0], acc[46]);
        acc[47] = fma(x[5] * y[1], z[0], acc[47]);
        acc[48] = fma(x[5] * y[0], z[1], acc[48]);
        acc[49] = fma(x[4] * y[2], z[0], acc[49]);
        acc[50] = fma(x[4] * y[1], z[1], acc[50]);
        acc[51] = fma(x[4] * y[0], z[2], acc[51]);
        acc[52] = fma(x[3] * y[3], z[0], acc[52]);
        acc[53] = fma(x[3] * y[2], z[1], acc[53]);
        acc[54] = fma(x[3] * y[1], z[2], acc[54]);
        acc[55] = fma(x[3] * y[0], z[3], acc[55]);
        acc[56] = fma(x[2] * y[4], z[0], acc[56]);
        acc[57] = fma(x[2] * y[3], z[1], acc[57]);
        acc[58] = fma(x[2] * y[2], z[2], acc[58]);
        acc[59] = fma(x[2] * y[1], z[3], acc[59]);
        acc[60] = fma(x[2] * y[0], z[4], acc[60]);
        acc[61] = fma(x[1] * y[5], z[0], acc[61]);
        acc[62] = fma(x[1] * y[4], z[1], acc[62]);
        acc[63] = fma(x[1] * y[3], z[2], acc[63]);
        acc[64] = fma(x[1] * y[2], z[3], acc[64]);
        acc[65] = fma(x[1] * y[1], z[4], acc[65]);
        acc[66] = fma(x[1] * y[0], z[5], acc[66]);
        acc[67] = fma(x[0] * y[6], z[0], acc[67]);
        acc[68] = fma(x[0] * y[5], z[1], acc[68]);
        acc[69] = fma(x[0] * y[4], z[2], acc[69]);
        acc[70] = fma(x[0] * y[3], z[3], acc[70]);
        acc[71] = fma(x[0] * y[2], z[4], acc[71]);
        acc[72] = fma(x[0] * y[1], z[5], acc[72]);
        acc[73] = fma(x[0] * y[0], z[6], acc[73]);
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[25], in[46]);
        const double h1 = fma(x, in[10], in[25]);
        const double h2 = fma(x, h1, h0);
        const double h3 = fma(x, in[0], in[10]);
        const double h4 = fma(x, h3, h1);
        const double h5 = fma(x, h4, h2);
        const double h6 = fma(y, in[25], in[47]);
        const double h7 = fma(y, in[10], in[26]);
        const double h8 = fma(x, h7, h6);
        const double h9 = fma(y, in[0], in[11]);
        const double h10 = fma(x, h9, h7);
        const double h11 = fma(x, h10, h8);
        const double h12 = fma(z, in[25], in[48]);
        const double h13 = fma(z, in[10], in[27]);
        const double h14 = fma(x, h13, h12);
        const double h15 = fma(z, in[0], in[12]);
        const double h16 = fma(x, h15, h13);
        const double h17 = fma(x, h16, h14);
        const double h18 = fma(y, in[26], in[49]);
        const double h19 = fma(y, in[11], in[28]);
        const double h20 = fma(x, h19, h18);
        const double h21 = fma(y, h10, h20);
        const double h22 = fma(z, in[27], in[51]);
        const double h23 = fma(z, in[12], in[30]);
        const double h24 = fma(x, h23, h22);
        const double h25 = fma(z, h16, h24);
        const double h26 = fma(z, in[26], in[50]);
        const double h27 = fma(y, h13, h26);
        const double h28 = fma(z, in[11], in[29]);
        const double h29 = fma(y, h15, h28);
        const double h30 = fma(x, h29, h27);
        const double h31 = fma(y, in[28], in[52]);
        const double h32 = fma(y, h19, h31);
        const double h33 = fma(y, h9, h19);
        const double h34 = fma(y, h33, h32);
        const double h35 = fma(z, in[28], in[53]);
        const double h36 = fma(y, h28, h35);
        const double h37 = fma(y, h29, h36);
        const double h38 = fma(z, in[29], in[54]);
        const double h39 = fma(y, h23, h38);
        const double h40 = fma(z, h29, h39);
        const double h41 = fma(z, in[30], in[55]);
        const double h42 = fma(z, h23, h41);
        const double h43 = fma(z, h15, h23);
        const double h44 = fma(z, h43, h42);
        const double h45 = fma(x, in[26], in[47]);
        const double h46 = fma(x, in[11], in[26]);
        const double h47 = fma(x, h46, h45);
        const double h48 = fma(x, in[1], in[11]);
        const double h49 = fma(x, h48, h46);
        const double h50 = fma(x, h49, h47);
        const double h51 = fma(y, in[1], in[13]);
        const double h52 = fma(x, h51, h19);
        const double h53 = fma(x, h52, h20);
        const double h54 = fma(x, h28, h26);
        const double h55 = fma(z, in[1], in[14]);
        const double h56 = fma(x, h55, h28);
        const double h57 = fma(x, h56, h54);
        const double h58 = fma(y, in[13], in[31]);
        const double h59 = fma(x, h58, h31);
        const double h60 = fma(y, h52, h59);
        const double h61 = fma(z, in[14], in[33]);
        const double h62 = fma(x, h61, h38);
        const double h63 = fma(z, h56, h62);
        const double h64 = fma(z, in[13], in[32]);
        const double h65 = fma(y, h55, h64);
        const double h66 = fma(x, h65, h36);
        const double h67 = fma(y, in[31], in[56]);
        const double h68 = fma(y, h58, h67);
        const double h69 = fma(y, h51, h58);
        const double h70 = fma(y, h69, h68);
        const double h71 = fma(z, in[31], in[57]);
        const double h72 = fma(y, h64, h71);
        const double h73 = fma(y, h65, h72);
        const double h74 = fma(z, in[32], in[58]);
        const double h75 = fma(y, h61, h74);
        const double h76 = fma(z, h65, h75);
        const double h77 = fma(z, in[33], in[59]);
        const double h78 = fma(z, h61, h77);
        const double h79 = fma(z, h55, h61);
        const double h80 = fma(z, h79, h78);
        const double h81 = fma(x, in[27], in[48]);
        const double h82 = fma(x, in[12], in[27]);
        const double h83 = fma(x, h82, h81);
        const double h84 = fma(x, in[2], in[12]);
        const double h85 = fma(x, h84, h82);
        const double h86 = fma(x, h85, h83);
        const double h87 = fma(y, in[27], in[50]);
        const double h88 = fma(y, in[12], in[29]);
        const double h89 = fma(x, h88, h87);
        const double h90 = fma(y, in[2], in[14]);
        const double h91 = fma(x, h90, h88);
        const double h92 = fma(x, h91, h89);
        const double h93 = fma(z, in[2], in[15]);
        const double h94 = fma(x, h93, h23);
        const double h95 = fma(x, h94, h24);
        const double h96 = fma(y, in[29], in[53]);
        const double h97 = fma(y, in[14], in[32]);
        const double h98 = fma(x, h97, h96);
        const double h99 = fma(y, h91, h98);
        const double h100 = fma(z, in[15], in[34]);
        const double h101 = fma(x, h100, h41);
        const double h102 = fma(z, h94, h101);
        const double h103 = fma(y, h93, h61);
        const double h104 = fma(x, h103, h39);
        const double h105 = fma(y, in[32], in[57]);
        const double h106 = fma(y, h97, h105);
        const double h107 = fma(y, h90, h97);
        const double h108 = fma(y, h107, h106);
        const double h109 = fma(y, h103, h75);
        const double h110 = fma(y, h100, h77);
        const double h111 = fma(z, h103, h110);
        const double h112 = fma(z, in[34], in[60]);
        const double h113 = fma(z, h100, h112);
        const double h114 = fma(z, h93, h100);
        const double h115 = fma(z, h114, h113);
        const double h116 = fma(x, in[28], in[49]);
        const double h117 = fma(x, in[13], in[28]);
        const double h118 = fma(x, h117, h116);
        const double h119 = fma(x, in[3], in[13]);
        const double h120 = fma(x, h119, h117);
        const double h121 = fma(x, h120, h118);
        const double h122 = fma(y, in[3], in[16]);
        const double h123 = fma(x, h122, h58);
        const double h124 = fma(x, h123, h59);
        const double h125 = fma(x, h64, h35);
        const double h126 = fma(z, in[3], in[17]);
        const double h127 = fma(x, h126, h64);
        const double h128 = fma(x, h127, h125);
        const double h129 = fma(y, in[16], in[35]);
        const double h130 = fma(x, h129, h67);
        const double h131 = fma(y, h123, h130);
        const double h132 = fma(z, in[17], in[37]);
        const double h133 = fma(x, h132, h74);
        const double h134 = fma(z, h127, h133);
        const double h135 = fma(z, in[16], in[36]);
        const double h136 = fma(y, h126, h135);
        const double h137 = fma(x, h136, h72);
        const double h138 = fma(y, in[35], in[61]);
        const double h139 = fma(y, h129, h138);
        const double h140 = fma(y, h122, h129);
        const double h141 = fma(y, h140, h139);
        const double h142 = fma(z, in[35], in[62]);
        const double h143 = fma(y, h135, h142);
        const double h144 = fma(y, h136, h143);
        const double h145 = fma(z, in[36], in[63]);
        const double h146 = fma(y, h132, h145);
        const double h147 = fma(z, h136, h146);
        const double h148 = fma(z, in[37], in[64]);
        const double h149 = fma(z, h132, h148);
        const double h150 = fma(z, h126, h132);
        const double h151 = fma(z, h150, h149);
        const double h152 = fma(x, in[30], in[51]);
        const double h153 = fma(x, in[15], in[30]);
        const double h154 = fma(x, h153, h152);
        const double h155 = fma(x, in[4], in[15]);
        const double h156 = fma(x, h155, h153);
        const double h157 = fma(x, h156, h154);
        const double h158 = fma(y, in[30], in[54]);
        const double h159 = fma(y, in[15], in[33]);
        const double h160 = fma(x, h159, h158);
        const double h161 = fma(y, in[4], in[18]);
        const double h162 = fma(x, h161, h159);
        const double h163 = fma(x, h162, h160);
        const double h164 = fma(z, in[4], in[19]);
        const double h165 = fma(x, h164, h100);
        const double h166 = fma(x, h165, h101);
        const double h167 = fma(y, in[33], in[58]);
        const double h168 = fma(y, in[18], in[37]);
        const double h169 = fma(x, h168, h167);
        const double h170 = fma(y, h162, h169);
        const double h171 = fma(z, in[19], in[39]);
        const double h172 = fma(x, h171, h112);
        const double h173 = fma(z, h165, h172);
        const double h174 = fma(z, in[18], in[38]);
        const double h175 = fma(y, h164, h174);
        const double h176 = fma(x, h175, h110);
        const double h177 = fma(y, in[37], in[63]);
        const double h178 = fma(y, h168, h177);
        const double h179 = fma(y, h161, h168);
        const double h180 = fma(y, h179, h178);
        const double h181 = fma(y, h174, h148);
        const double h182 = fma(y, h175, h181);
        const double h183 = fma(z, in[38], in[65]);
        const double h184 = fma(y, h171, h183);
        const double h185 = fma(z, h175, h184);
        const double h186 = fma(z, in[39], in[66]);
        const double h187 = fma(z, h171, h186);
        const double h188 = fma(z, h164, h171);
        const double h189 = fma(z, h188, h187);
        const double h190 = fma(x, in[29], in[50]);
        const double h191 = fma(x, in[14], in[29]);
        const double h192 = fma(x, h191, h190);
        const double h193 = fma(x, in[5], in[14]);
        const double h194 = fma(x, h193, h191);
        const double h195 = fma(x, h194, h192);
        const double h196 = fma(y, in[5], in[17]);
        const double h197 = fma(x, h196, h97);
        const double h198 = fma(x, h197, h98);
        const double h199 = fma(z, in[5], in[18]);
        const double h200 = fma(x, h199, h61);
        const double h201 = fma(x, h200, h62);
        const double h202 = fma(y, in[17], in[36]);
        const double h203 = fma(x, h202, h105);
        const double h204 = fma(y, h197, h203);
        const double h205 = fma(x, h174, h77);
        const double h206 = fma(z, h200, h205);
        const double h207 = fma(y, h199, h132);
        const double h208 = fma(x, h207, h75);
        const double h209 = fma(y, in[36], in[62]);
        const double h210 = fma(y, h202, h209);
        const double h211 = fma(y, h196, h202);
        const double h212 = fma(y, h211, h210);
        const double h213 = fma(y, h207, h146);
        const double h214 = fma(z, h207, h181);
        const double h215 = fma(z, h174, h183);
        const double h216 = fma(z, h199, h174);
        const double h217 = fma(z, h216, h215);
        const double h218 = fma(x, in[31], in[52]);
        const double h219 = fma(x, in[16], in[31]);
        const double h220 = fma(x, h219, h218);
        const double h221 = fma(x, in[6], in[16]);
        const double h222 = fma(x, h221, h219);
        const double h223 = fma(x, h222, h220);
        const double h224 = fma(y, in[6], in[20]);
        const double h225 = fma(x, h224, h129);
        const double h226 = fma(x, h225, h130);
        const double h227 = fma(x, h135, h71);
        const double h228 = fma(z, in[6], in[21]);
        const double h229 = fma(x, h228, h135);
        const double h230 = fma(x, h229, h227);
        const double h231 = fma(y, in[20], in[40]);
        const double h232 = fma(x, h231, h138);
        const double h233 = fma(y, h225, h232);
        const double h234 = fma(z, in[21], in[42]);
        const double h235 = fma(x, h234, h145);
        const double h236 = fma(z, h229, h235);
        const double h237 = fma(z, in[20], in[41]);
        const double h238 = fma(y, h228, h237);
        const double h239 = fma(x, h238, h143);
        const double h240 = fma(y, in[40], in[67]);
        const double h241 = fma(y, h231, h240);
        const double h242 = fma(y, h224, h231);
        const double h243 = fma(y, h242, h241);
        const double h244 = fma(z, in[40], in[68]);
        const double h245 = fma(y, h237, h244);
        const double h246 = fma(y, h238, h245);
        const double h247 = fma(z, in[41], in[69]);
        const double h248 = fma(y, h234, h247);
        const double h249 = fma(z, h238, h248);
        const double h250 = fma(z, in[42], in[70]);
        const double h251 = fma(z, h234, h250);
        const double h252 = fma(z, h228, h234);
        const double h253 = fma(z, h252, h251);
        const double h254 = fma(x, in[32], in[53]);
        const double h255 = fma(x, in[17], in[32]);
        const double h256 = fma(x, h255, h254);
        const double h257 = fma(x, in[7], in[17]);
        const double h258 = fma(x, h257, h255);
        const double h259 = fma(x, h258, h256);
        const double h260 = fma(y, in[7], in[21]);
        const double h261 = fma(x, h260, h202);
        const double h262 = fma(x, h261, h203);
        const double h263 = fma(z, in[7], in[22]);
        const double h264 = fma(x, h263, h132);
        const double h265 = fma(x, h264, h133);
        const double h266 = fma(y, in[21], in[41]);
        const double h267 = fma(x, h266, h209);
        const double h268 = fma(y, h261, h267);
        const double h269 = fma(z, in[22], in[43]);
        const double h270 = fma(x, h269, h148);
        const double h271 = fma(z, h264, h270);
        const double h272 = fma(y, h263, h234);
        const double h273 = fma(x, h272, h146);
        const double h274 = fma(y, in[41], in[68]);
        const double h275 = fma(y, h266, h274);
        const double h276 = fma(y, h260, h266);
        const double h277 = fma(y, h276, h275);
        const double h278 = fma(y, h272, h248);
        const double h279 = fma(y, h269, h250);
        const double h280 = fma(z, h272, h279);
        const double h281 = fma(z, in[43], in[71]);
        const double h282 = fma(z, h269, h281);
        const double h283 = fma(z, h263, h269);
        const double h284 = fma(z, h283, h282);
        const double h285 = fma(x, in[33], in[54]);
        const double h286 = fma(x, in[18], in[33]);
        const double h287 = fma(x, h286, h285);
        const double h288 = fma(x, in[8], in[18]);
        const double h289 = fma(x, h288, h286);
        const double h290 = fma(x, h289, h287);
        const double h291 = fma(y, in[8], in[22]);
        const double h292 = fma(x, h291, h168);
        const double h293 = fma(x, h292, h169);
        const double h294 = fma(z, in[8], in[23]);
        const double h295 = fma(x, h294, h174);
        const double h296 = fma(x, h295, h205);
        const double h297 = fma(y, in[22], in[42]);
        const double h298 = fma(x, h297, h177);
        const double h299 = fma(y, h292, h298);
        const double h300 = fma(z, in[23], in[44]);
        const double h301 = fma(x, h300, h183);
        const double h302 = fma(z, h295, h301);
        const double h303 = fma(y, h294, h269);
        const double h304 = fma(x, h303, h181);
        const double h305 = fma(y, in[42], in[69]);
        const double h306 = fma(y, h297, h305);
        const double h307 = fma(y, h291, h297);
        const double h308 = fma(y, h307, h306);
        const double h309 = fma(y, h303, h279);
        const double h310 = fma(y, h300, h281);
        const double h311 = fma(z, h303, h310);
        const double h312 = fma(z, in[44], in[72]);
        const double h313 = fma(z, h300, h312);
        const double h314 = fma(z, h294, h300);
        const double h315 = fma(z, h314, h313);
        const double h316 = fma(x, in[34], in[55]);
        const double h317 = fma(x, in[19], in[34]);
        const double h318 = fma(x, h317, h316);
        const double h319 = fma(x, in[9], in[19]);
        const double h320 = fma(x, h319, h317);
        const double h321 = fma(x, h320, h318);
        const double h322 = fma(y, in[34], in[59]);
        const double h323 = fma(y, in[19], in[38]);
        const double h324 = fma(x, h323, h322);
        const double h325 = fma(y, in[9], in[23]);
        const double h326 = fma(x, h325, h323);
        const double h327 = fma(x, h326, h324);
        const double h328 = fma(z, in[9], in[24]);
        const double h329 = fma(x, h328, h171);
        const double h330 = fma(x, h329, h172);
        const double h331 = fma(y, in[38], in[64]);
        const double h332 = fma(y, in[23], in[43]);
        const double h333 = fma(x, h332, h331);
        const double h334 = fma(y, h326, h333);
        const double h335 = fma(z, in[24], in[45]);
        const double h336 = fma(x, h335, h186);
        const double h337 = fma(z, h329, h336);
        const double h338 = fma(y, h328, h300);
        const double h339 = fma(x, h338, h184);
        const double h340 = fma(y, in[43], in[70]);
        const double h341 = fma(y, h332, h340);
        const double h342 = fma(y, h325, h332);
        const double h343 = fma(y, h342, h341);
        const double h344 = fma(y, h338, h310);
        const double h345 = fma(y, h335, h312);
        const double h346 = fma(z, h338, h345);
        const double h347 = fma(z, in[45], in[73]);
        const double h348 = fma(z, h335, h347);
        const double h349 = fma(z, h328, h335);
        const double h350 = fma(z, h349, h348);
        out[0] = h5;
        out[1] = h11;
        out[2] = h17;
        out[3] = h21;
        out[4] = h25;
        out[5] = h30;
        out[6] = h34;
        out[7] = h37;
        out[8] = h40;
        out[9] = h44;
        out[10] = h50;
        out[11] = h53;
        out[12] = h57;
        out[13] = h60;
        out[14] = h63;
        out[15] = h66;
        out[16] = h70;
        out[17] = h73;
        out[18] = h76;
        out[19] = h80;
        out[20] = h86;
        out[21] = h92;
        out[22] = h95;
        out[23] = h99;
        out[24] = h102;
        out[25] = h104;
        out[26] = h108;
        out[27] = h109;
        out[28] = h111;
        out[29] = h115;
        out[30] = h121;
        out[31] = h124;
        out[32] = h128;
        out[33] = h131;
        out[34] = h134;
        out[35] = h137;
        out[36] = h141;
        out[37] = h144;
        out[38] = h147;
        out[39] = h151;
        out[40] = h157;
        out[41] = h163;
        out[42] = h166;
        out[43] = h170;
        out[44] = h173;
        out[45] = h176;
        out[46] = h180;
        out[47] = h182;
        out[48] = h185;
        out[49] = h189;
        out[50] = h195;
        out[51] = h198;
        out[52] = h201;
        out[53] = h204;
        out[54] = h206;
        out[55] = h208;
        out[56] = h212;
        out[57] = h213;
        out[58] = h214;
        out[59] = h217;
        out[60] = h223;
        out[61] = h226;
        out[62] = h230;
        out[63] = h233;
        out[64] = h236;
        out[65] = h239;
        out[66] = h243;
        out[67] = h246;
        out[68] = h249;
        out[69] = h253;
        out[70] = h259;
        out[71] = h262;
        out[72] = h265;
        out[73] = h268;
        out[74] = h271;
        out[75] = h273;
        out[76] = h277;
        out[77] = h278;
        out[78] = h280;
        out[79] = h284;
        out[80] = h290;
        out[81] = h293;
        out[82] = h296;
        out[83] = h299;
        out[84] = h302;
        out[85] = h304;
        out[86] = h308;
        out[87] = h309;
        out[88] = h311;
        out[89] = h315;
        out[90] = h321;
        out[91] = h327;
        out[92] = h330;
        out[93] = h334;
        out[94] = h337;
        out[95] = h339;
        out[96] = h343;
        out[97] = h344;
        out[98] = h346;
        out[99] = h350;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0] * (nrm * 1.0);
    }
};

__device__ const double kNormAB_ffss[100] = {
    0.06666666666666665, 0.14907119849998599, 0.14907119849998599, 0.14907119849998599,
    0.14907119849998599, 0.2581988897471611, 0.06666666666666665, 0.14907119849998599,
    0.14907119849998599, 0.06666666666666665, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.3333333333333334, 0.3333333333333334, 0.5773502691896258,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.14907119849998599,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.14907119849998599, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.3333333333333334, 0.3333333333333334, 0.5773502691896258,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.14907119849998599,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.14907119849998599, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 1.0,
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.2581988897471611,
    0.06666666666666665, 0.14907119849998599, 0.14907119849998599, 0.14907119849998599,
    0.14907119849998599, 0.2581988897471611, 0.06666666666666665, 0.14907119849998599,
    0.14907119849998599, 0.06666666666666665, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.3333333333333334, 0.3333333333333334, 0.5773502691896258,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.14907119849998599,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.14907119849998599, 0.06666666666666665, 0.14907119849998599,
    0.14907119849998599, 0.14907119849998599, 0.14907119849998599, 0.2581988897471611,
    0.06666666666666665, 0.14907119849998599, 0.14907119849998599, 0.06666666666666665,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_ffss[1] = { 0 };

__device__ __forceinline__ RysClassTabs tabs_ffss() {
    return RysClassTabs{kNormAB_ffss, kCol_ffss};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_ffss(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_ffss, MIXED>(Q, R, tabs_ffss());
}

static void rys_prepare_ffss() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_ffss<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 25600);
        cudaFuncSetAttribute(rys_queue_ffss<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 25600);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_ffss(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_ffss();
    constexpr int ng = 128 / C_ffss::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_ffss<1><<<grid, 128, 25600, s>>>(Q, R);
    else rys_queue_ffss<0><<<grid, 128, 25600, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_ffss(int mixed) {
    rys_prepare_ffss();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_ffss<1>, 128, 25600);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_ffss<0>, 128, 25600);
    return n;
}

}  // namespace molints
